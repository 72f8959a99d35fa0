"""Polynomials that have a kernel written out at build time ("static" kernels).

For a polynomial whose path list is known when the library is built, the whole evaluation
of one (row, channel) pair can be emitted as straight-line FP32 code: every operand segment
is loaded into a register once, every path is a couple of multiplies, and permutation-
equivalent paths of repeated operands (x*x*x) are merged.  The reference obtains the same
effect by JIT-compiling one kernel per polynomial with NVRTC (CHANGELOG.md:38,49); here the
source is generated ahead of time by ``csrc/gen_u1d_static.py`` for the polynomials listed in
`registered_polynomials` and matched at run time by a digest of the serialised tables.
"""
from __future__ import annotations

import hashlib
import struct
from typing import Dict, List, Tuple

import numpy as np

from .polynomial import Operation, Polynomial
from .stp import Path, SegmentedTensorProduct


def merge_symmetric_paths(poly: Polynomial) -> Polynomial:
    """Within each operation, paths that differ only by a permutation of the segment indices
    of operands bound to the same buffer describe the same monomial; they are merged (their
    coefficients added).  The polynomial function is unchanged."""
    new_ops = []
    for ope, stp in poly.operations:
        groups: Dict[int, List[int]] = {}
        for k, b in enumerate(ope.buffers):
            groups.setdefault(b, []).append(k)
        acc: Dict[Tuple[int, ...], float] = {}
        order: List[Tuple[int, ...]] = []
        for p in stp.paths:
            idx = list(p.indices)
            for ks in groups.values():
                if len(ks) > 1:
                    vals = sorted(idx[k] for k in ks)
                    for k, v in zip(ks, vals):
                        idx[k] = v
            key = tuple(idx)
            if key not in acc:
                acc[key] = 0.0
                order.append(key)
            acc[key] += float(p.coefficients)
        d = stp.copy()
        d.paths = [Path(k, np.float64(acc[k])) for k in order if acc[k] != 0.0]
        new_ops.append((ope, d))
    return Polynomial(poly.inputs, poly.outputs, new_ops)


def digest(poly: Polynomial) -> str:
    """Digest of the structure a static kernel depends on: segment counts, scalar/vector kind,
    operations, path indices and coefficients (float64 bit patterns) - not the extent."""
    h = hashlib.sha1()
    h.update(struct.pack("<ii", poly.num_inputs, poly.num_outputs))
    for o in poly.operands:
        h.update(struct.pack("<ii", o.ndim, o.num_segments))
    for ope, stp in poly.operations:
        h.update(struct.pack(f"<{len(ope.buffers) + 1}i", len(ope.buffers), *ope.buffers))
        for p in stp.paths:
            h.update(struct.pack(f"<{len(p.indices)}i", *p.indices))
            h.update(struct.pack("<d", float(p.coefficients)))
    return h.hexdigest()[:16]


def registered_polynomials() -> List[Tuple[str, Polynomial]]:
    """(name, flattened polynomial) of everything that gets a static kernel: the MACE symmetric contractions
    0e+1o[+2e[+3o]] -> 0e[+1o] of degree 2 and 3 and their first derivatives, each alone and both together.  The path
    tables of these shapes ship with the package, so that the digest cannot depend on the host that evaluates it (tables
    ship for 0e -> 0e, for outputs 0e+1o+2e and for degree 1 too; those run on the table-driven kernel)."""
    from . import descriptors

    out = []
    for l_in in (1, 2, 3):
        for l_out in (0, 1):
            for degree in (2, 3):
                irreps = ["+".join(f"4x{l}{'eo'[l % 2]}" for l in range(n + 1)) for n in (l_in, l_out)]  # noqa: E741
                e, _ = descriptors.symmetric_contraction(*irreps, tuple(range(1, degree + 1)))
                fwd = e.polynomial.flatten_coefficient_modes().squeeze_modes()
                name = f"sc_l{l_in}_l{l_out}_d{degree}"
                out.append((f"{name}_fwd", fwd))
                out.append((f"{name}_bwd_wx", fwd.backward([True, True], [True])))
                out.append((f"{name}_bwd_x", fwd.backward([False, True], [True])))
                out.append((f"{name}_bwd_w", fwd.backward([True, False], [True])))
    return out
