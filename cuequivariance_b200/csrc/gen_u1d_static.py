"""Generates ``generated/u1d_static.cuh``: one straight-line FP32 kernel body per registered
polynomial (see ``cuequivariance_b200/static_poly.py``).

Each body evaluates one (row, channel) pair: operand segments are loaded into registers at
first use, products of two segments of the same buffer are shared between paths, and each output
segment is handed to a caller-supplied sink exactly once.

The sum of an output segment is factored as in Horner's rule for several variables: the factor
that most of its terms share is taken out, its cofactor and the remainder are treated the same
way, down to sums of ``coefficient * segment`` or ``coefficient * shared product``, one multiply-add
per term.  Factors are taken from the buffers that occur once in a term first (cotangent and weight,
the one with fewer segments first) and from the repeated buffer last, which leaves its products as
the innermost terms.  A body runs straight through once, so its time goes with its instructions and with the loads that
nothing but other warps overlaps (47-64 % of the issue slots are used); for 0e+1o+2e+3o -> 0e+1o of degree 3, against one
product and one multiply-add per term and a factored first operand only: forward 1089 -> 747, weight gradient 1155 -> 747,
feature gradient 2664 -> 1786 instructions.

    python cuequivariance_b200/csrc/gen_u1d_static.py
"""
from __future__ import annotations

import os
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.dirname(os.path.dirname(HERE)))

from cuequivariance_b200.static_poly import digest, merge_symmetric_paths, registered_polynomials  # noqa: E402


def fl(c: float) -> str:
    t = f"{float(c):.9g}"
    if "." not in t and "e" not in t and "n" not in t:
        t += ".0"
    return t + "f"


def emit(name: str, poly) -> str:
    merged = merge_symmetric_paths(poly)
    n_in = merged.num_inputs
    L = []
    A = L.append
    A(f"// {name}: " + "; ".join(f"{ope.buffers}:{stp.num_paths}" for ope, stp in merged.operations))
    A(f"struct U1dStatic_{name} {{")
    A(f"  static constexpr int NUM_INPUTS = {n_in};")
    A(f"  static constexpr int NUM_OUTPUTS = {merged.num_outputs};")
    A("  static constexpr const char* digest() { return \"%s\"; }" % digest(poly))
    A("  static constexpr const char* name() { return \"%s\"; }" % name)
    A("  // in(b, s): value of segment s of input buffer b for this (row, channel); out(j, s, v): add v to output j")
    A("  template <class In, class Out>")
    A("  __device__ __forceinline__ static void run(const In& in, Out& out) {")
    loaded = set()
    prods = {}
    B = []  # lines of the block being built; definitions above go to function scope (L)

    def seg(b, s):
        v = f"x{b}_{s}"
        if (b, s) not in loaded:
            loaded.add((b, s))
            L.append(f"    const float {v} = in({b}, {s});")
        return v

    def prod(b, s1, s2):
        key = (b, min(s1, s2), max(s1, s2))
        v = f"p{b}_{key[1]}_{key[2]}"
        if key not in prods:
            a, c = seg(b, key[1]), seg(b, key[2])
            prods[key] = v
            L.append(f"    const float {v} = {a} * {c};")
        return v

    # accumulate per output segment over ALL operations bound to it
    by_out = {}
    repeated = set()
    for ope, stp in merged.operations:
        k_out = [k for k, b in enumerate(ope.buffers) if b >= n_in][0]
        j = ope.buffers[k_out] - n_in
        ins = [k for k in range(len(ope.buffers)) if k != k_out]
        repeated |= {b for b in ope.buffers if ope.buffers.count(b) > 1}
        for p in stp.paths:
            by_out.setdefault((j, p.indices[k_out]), []).append(
                (sorted((ope.buffers[k], p.indices[k]) for k in ins), float(p.coefficients)))
    order = sorted(range(n_in), key=lambda b: (b in repeated, merged.inputs[b].num_segments))
    tmp = 0

    def is_leaf(factors):
        return len(factors) <= 1 or (len(factors) == 2 and factors[0][0] == factors[1][0])

    def accumulate(terms, acc):
        """Adds the sum of ``terms`` to the variable ``acc`` (None: a new one); returns its name."""
        nonlocal tmp
        deep = [f for f, _ in terms if not is_leaf(f)]
        if not deep:
            for factors, c in terms:
                expr = "1.f" if not factors else seg(*factors[0]) if len(factors) == 1 else prod(factors[0][0], factors[0][1], factors[1][1])
                if acc is None:
                    acc, tmp = f"t{tmp}", tmp + 1
                    B.append(f"      float {acc} = {fl(c)} * {expr};")
                else:
                    B.append(f"      {acc} = fmaf({fl(c)}, {expr}, {acc});")
            return acc
        count = {}
        for f in deep:
            for q in dict.fromkeys(map(tuple, f)):
                count[q] = count.get(q, 0) + 1
        first = min(order.index(b) for b, _ in count)
        v = max((q for q in count if q[0] == order[first]), key=lambda q: (count[q], -q[1]))
        cofactor, rest = [], []
        for f, c in terms:
            if v in f:
                f = list(f)
                f.remove(v)
                cofactor.append((f, c))
            else:
                rest.append((f, c))
        inner = accumulate(cofactor, None)
        if acc is None:
            acc, tmp = f"t{tmp}", tmp + 1
            B.append(f"      float {acc} = {seg(*v)} * {inner};")
        else:
            B.append(f"      {acc} = fmaf({seg(*v)}, {inner}, {acc});")
        return accumulate(rest, acc) if rest else acc

    # every segment is handed out, zero where no term feeds it: batched outputs are not cleared beforehand
    for j, so in [(j, so) for j, o in enumerate(merged.outputs) for so in range(o.num_segments)]:
        B.append("    {")
        acc = accumulate(by_out[j, so], None) if (j, so) in by_out else "0.f"
        B.append(f"      out({j}, {so}, {acc});")
        B.append("    }")
        L.extend(B)
        B.clear()
    A("  }")
    A("};")
    return "\n".join(L)


def main():
    parts = ["// GENERATED by gen_u1d_static.py - do not edit.", "#pragma once", ""]
    names = []
    for name, poly in registered_polynomials():
        parts.append(emit(name, poly))
        parts.append("")
        names.append(name)
    parts.append("#define U1D_STATIC_FOR_EACH(X) \\")
    parts.append(" \\\n".join(f"  X(U1dStatic_{n})" for n in names))
    parts.append("")
    os.makedirs(os.path.join(HERE, "generated"), exist_ok=True)
    path = os.path.join(HERE, "generated", "u1d_static.cuh")
    text = "\n".join(parts)
    if not os.path.exists(path) or open(path).read() != text:
        open(path, "w").write(text)
    return names


if __name__ == "__main__":
    print(main())
