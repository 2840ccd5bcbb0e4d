"""Generates sgh_hex_geometry.cuh: straight-line device code for one hex's
outward corner area normals B (geometry.cpp:40-234), exact volume
(geometry.cpp:271-310) and the velocity-divergence sums (momentum.cpp:221-292).

Every expression keeps the reference's operands and association order, so the
generated code is bit-for-bit equivalent to it when compiled without
contraction.  The work is shared where that is exact:
  * each cofactor combo is evaluated once for all the node pairs it belongs to;
    the other orientation, and the pairs whose terms are the negated ones, are
    its exact negation (term-by-term negated sums round to the negated value);
  * the volume reuses the B-matrix products y_j * comb_ij of component 0.
The volume's products and sums (and with them component 0 of B) go through
FX_MUL / FX_ADD, which stay separately rounded in the fused-multiply-add build
too: the cofactor sum cancels terms of size ~|x| h^2 down to a volume ~h^3, so
contracting it would move the volume (and the density) by ~|x|/h ulps, 1e-11
relative on a 256^3 mesh, while every other field moves by ~1e-16.

The tables are parsed from sgh_hex.h so there is one source of truth.
Run:  python gen_hex_geometry.py   (writes sgh_hex_geometry.cuh beside it)
"""
import os
import re

HERE = os.path.dirname(os.path.abspath(__file__))


def parse_tables():
    src = open(os.path.join(HERE, "sgh_hex.h")).read()

    def arr(name):
        m = re.search(r"constexpr[^=]*\b%s\b[^=]*=\s*\{(.*?)\};" % name, src, re.S)
        return [int(v) for v in re.findall(r"-?\d+", m.group(1))]

    J = arr("J")
    T = arr("TERMS")
    VI = arr("VI")
    VJ = arr("VJ")
    J = [J[p * 6:(p + 1) * 6] for p in range(8)]
    T = [[T[(p * 6 + t) * 4:(p * 6 + t + 1) * 4] for t in range(6)] for p in range(8)]
    VJ = [VJ[a * 6:(a + 1) * 6] for a in range(8)]
    return J, T, VI, VJ


def combo_expr(I, terms):
    """The combo's signed terms summed left to right, as the reference writes them."""
    expr = ("-" if terms[0] < 0 else "") + "%s[%d]" % (I, abs(terms[0]) - 1)
    for v_ in terms[1:]:
        expr = "(%s %s %s[%d])" % (expr, "+" if v_ > 0 else "-", I, abs(v_) - 1)
    return expr


def emit_combos(w, I, pairs, T, indent="    "):
    """Declares the combos the pairs need and returns pair index -> signed name.
    A combo equal to an earlier one or to its term-by-term negation is that one
    (the compiler does not see that (-a - b) + c + d is -((a + b) - c - d)), and
    a four-term combo whose first two terms are a two-term combo starts from it:
    12 + 16 additions per component instead of the 40 left of 48 when each pair
    forms its own."""
    seen, name_of = {}, {}
    order = sorted(range(len(pairs)), key=lambda k: len([v for v in T[pairs[k][0]][pairs[k][1]] if v]))
    for k in order:
        p, t, j = pairs[k]
        terms = tuple(v for v in T[p][t] if v)
        neg = tuple(-v for v in terms)
        if terms in seen:
            name_of[k] = seen[terms]
            continue
        if neg in seen:
            name_of[k] = "(-%s)" % seen[neg]
            continue
        head, neg_head = terms[:2], neg[:2]
        expr = combo_expr(I, terms)
        if len(terms) == 4 and (head in seen or neg_head in seen):
            expr = seen[head] if head in seen else "(-%s)" % seen[neg_head]
            for v_ in terms[2:]:
                expr = "(%s %s %s[%d])" % (expr, "+" if v_ > 0 else "-", I, abs(v_) - 1)
        w("%sconst double cm%d = %s;  // pair (%d,%d)" % (indent, k, expr, p, j))
        seen[terms] = "cm%d" % k
        name_of[k] = "cm%d" % k
    return name_of


def negated(name):
    return name[2:-1] if name.startswith("(-") else "(-%s)" % name


def main():
    J, T, VI, VJ = parse_tables()
    # unordered pairs, stored in the p < j orientation
    pairs = []  # (p, t, j)
    pair_of = {}
    for p in range(8):
        for t in range(6):
            j = J[p][t]
            if p < j:
                pair_of[(p, j)] = len(pairs)
                pairs.append((p, t, j))
    for p in range(8):
        for t in range(6):
            j = J[p][t]
            if p > j:
                k = pair_of[(j, p)]
                a = T[j][pairs[k][1]]
                b = T[p][t]
                assert [-v for v in a if v] == [v for v in b if v], (p, j)
    comps = [("y", "z"), ("z", "x"), ("x", "y")]  # (O, I) for c = 0, 1, 2
    L = []
    w = L.append
    w("// GENERATED by gen_hex_geometry.py from sgh_hex.h -- do not edit.")
    w("// Straight-line hex geometry; see the generator's docstring for the exactness argument.")
    w("#pragma once")
    w("")
    w("// Separately rounded product and sum, also where the unit contracts (FIERRO_FMA=1).")
    w("#if FIERRO_FMA")
    w("#define FX_MUL(a, b) __dmul_rn((a), (b))")
    w("#define FX_ADD(a, b) __dadd_rn((a), (b))")
    w("#else")
    w("#define FX_MUL(a, b) ((a) * (b))")
    w("#define FX_ADD(a, b) ((a) + (b))")
    w("#endif")
    w("")
    w("// a + b c and a b + c d: fused in the FMA build (which product is the fused one is")
    w("// part of the result), the reference's products and sum in the exact build.")
    w("__device__ __forceinline__ double mul_add(double a, double b, double c) {")
    w("#if FIERRO_FMA")
    w("  return fma(b, c, a);")
    w("#else")
    w("  return a + b * c;")
    w("#endif")
    w("}")
    w("__device__ __forceinline__ double mul_mul(double a, double b, double c, double d) {")
    w("#if FIERRO_FMA")
    w("  return fma(a, b, __dmul_rn(c, d));")
    w("#else")
    w("  return a * b + c * d;")
    w("#endif")
    w("}")
    w("")
    w("// In: x,y,z,u,v,w[8] (node lids 0..7).  Out: vol; bmat rows lid*3+dim at")
    w("// bmat[row*ne + e]; Sx,Sy,Sz = sum_p u_p B(p,0), v_p B(p,1), w_p B(p,2) (p order).")
    w("__device__ __forceinline__ void hex_geometry(const double* __restrict__ x, const double* __restrict__ y,")
    w("    const double* __restrict__ z, const double* __restrict__ u, const double* __restrict__ v,")
    w("    const double* __restrict__ w, double* __restrict__ bmat, int ne, int e, double& vol,")
    w("    double& Sx, double& Sy, double& Sz) {")
    w("  const double twelth = 1. / 12.;")
    vel = {0: "u", 1: "v", 2: "w"}
    for c, (O, I) in enumerate(comps):
        w("  {  // component %d: O = %s, I = %s" % (c, O, I))
        combo = emit_combos(w, I, pairs, T)
        # products
        prod = {}
        for p in range(8):
            for t in range(6):
                j = J[p][t]
                cm = combo[pair_of[(p, j)]] if p < j else negated(combo[pair_of[(j, p)]])
                if c == 0:
                    w("    const double pr%d_%d = FX_MUL(%s[%d], %s);" % (p, t, O, j, cm))
                else:
                    prod[(p, t)] = "%s[%d], %s" % (O, j, cm)
        if c == 0:
            # volume: sum_a x[VI[a]] * (sum_b products in VJ order)
            for a in range(8):
                i = VI[a]
                slots = [J[i].index(jj) for jj in VJ[a]]
                expr = "pr%d_%d" % (i, slots[0])
                for s_ in slots[1:]:
                    expr = "FX_ADD(%s, pr%d_%d)" % (expr, i, s_)
                w("    const double vi%d = FX_MUL(x[%d], %s);" % (a, i, expr))
            expr = "vi0"
            for a in range(1, 8):
                expr = "FX_ADD(%s, vi%d)" % (expr, a)
            w("    vol = FX_MUL(%s, twelth);" % expr)
        S = "S" + "xyz"[c]
        for p in range(8):
            if c == 0:
                expr = "pr%d_0" % p
                for t in range(1, 6):
                    expr = "(%s + pr%d_%d)" % (expr, p, t)
            else:
                expr = "mul_mul(%s, %s)" % (prod[(p, 0)], prod[(p, 1)])
                for t in range(2, 6):
                    expr = "mul_add(%s, %s)" % (expr, prod[(p, t)])
            w("    const double b%d = %s * twelth;" % (p, expr))
            w("    bmat[(size_t)%d * ne + e] = b%d;" % (p * 3 + c, p))
            if p == 1:
                w("    %s = mul_mul(%s[0], b0, %s[1], b1);" % (S, vel[c], vel[c]))
            elif p > 1:
                w("    %s = mul_add(%s, %s[%d], b%d);" % (S, S, vel[c], p, p))
        w("  }")
    w("}")
    w("")
    w("// The exact hex volume alone (geometry.cpp:271-310), the same operations in the")
    w("// same order as hex_geometry's volume.")
    w("__device__ __forceinline__ double hex_volume(const double* __restrict__ x, const double* __restrict__ y,")
    w("    const double* __restrict__ z) {")
    w("  const double twelth = 1. / 12.;")
    O, I = comps[0]
    combo = emit_combos(w, I, pairs, T, "  ")
    used = set()
    for a in range(8):
        i = VI[a]
        for jj in VJ[a]:
            used.add((i, J[i].index(jj)))
    for (p_, t) in sorted(used):
        j = J[p_][t]
        cm = combo[pair_of[(p_, j)]] if p_ < j else negated(combo[pair_of[(j, p_)]])
        w("  const double pr%d_%d = %s[%d] * %s;" % (p_, t, O, j, cm))
    for a in range(8):
        i = VI[a]
        slots = [J[i].index(jj) for jj in VJ[a]]
        expr = "pr%d_%d" % (i, slots[0])
        for s_ in slots[1:]:
            expr = "(%s + pr%d_%d)" % (expr, i, s_)
        w("  const double vi%d = x[%d] * %s;" % (a, i, expr))
    expr = "vi0"
    for a in range(1, 8):
        expr = "(%s + vi%d)" % (expr, a)
    w("  return %s * twelth;" % expr)
    w("}")
    w("")
    # four-term combos as sums of two two-term ones: -a - b + c + d = (c - a) + (d - b)
    def two_term(i, j):
        """(name, sign) of the two-term combo worth I[i] - I[j], 1-based."""
        for k, (p_, t, _) in enumerate(pairs):
            terms = sorted(v for v in T[p_][t] if v)
            if len(terms) == 2:
                if terms == [-j, i]:
                    return k, 1
                if terms == [-i, j]:
                    return k, -1
        return None

    fours, four_of = [], {}  # distinct four-term combos (terms, [(k, sign) of its halves]); pair -> (four, sign)
    for k, (p_, t, j) in enumerate(pairs):
        terms = tuple(sorted(v for v in T[p_][t] if v))
        if len(terms) != 4:
            continue
        neg = tuple(sorted(-v for v in terms))
        known = [i for i, f in enumerate(fours) if f[0] in (terms, neg)]
        if not known:
            plus, minus = [v for v in terms if v > 0], [-v for v in terms if v < 0]
            for m in (minus, minus[::-1]):
                halves = [two_term(plus[0], m[0]), two_term(plus[1], m[1])]
                if None not in halves:
                    break
            assert None not in halves, terms
            fours.append((terms, halves))
            known = [len(fours) - 1]
        four_of[k] = (known[0], 1 if fours[known[0]][0] == terms else -1)

    w("// Reverse mode of the corner normals: given Bbar[lid*3+dim] (the adjoint of")
    w("// B(lid, dim)), accumulate the coordinate adjoints xbar, ybar, zbar[8].  B is")
    w("// bilinear, B(p,c) = sum_t O[j_t] comb_t(I) / 12, and each unordered pair (p, j)")
    w("// enters B(p) as O[j] cm and B(j) as -O[p] cm with one shared combo cm, so")
    w("//   Obar[j] += g_p cm,  Obar[p] -= g_j cm,  wbar(cm) += g_p O[j] - g_j O[p]")
    w("// with g = Bbar / 12 (multiply-adds fused: the adjoint has no parity target).  The 24")
    w("// pairs share 12 two-term and 6 four-term combos, a four-term one is the sum of two")
    w("// two-term ones, and the combos' adjoints take the same tree back: 164 FP64")
    w("// operations per component where a scatter of every pair's terms took 216.")
    w("__device__ __forceinline__ void hex_bmatrix_adjoint(const double* __restrict__ x, const double* __restrict__ y,")
    w("    const double* __restrict__ z, const double* __restrict__ Bbar, double* __restrict__ xbar,")
    w("    double* __restrict__ ybar, double* __restrict__ zbar) {")
    w("  const double twelth = 1. / 12.;")
    bar = {"x": "xbar", "y": "ybar", "z": "zbar"}
    sgn = {1: "", -1: "-"}
    for c, (O, I) in enumerate(comps):
        w("  {  // component %d: O = %s, I = %s" % (c, O, I))
        for p_ in range(8):
            w("    const double g%d = Bbar[%d] * twelth;" % (p_, p_ * 3 + c))
        two = [k for k, (p_, t, _) in enumerate(pairs) if len([v for v in T[p_][t] if v]) == 2]
        for k in two:
            p_, t, j = pairs[k]
            i_, j_ = max(T[p_][t][:2]), -min(T[p_][t][:2])
            w("    const double cm%d = %s[%d] - %s[%d];" % (k, I, i_ - 1, I, j_ - 1))
        for f, (_, h) in enumerate(fours):
            w("    const double c4_%d = %scm%d %s cm%d;" % (f, sgn[h[0][1]], h[0][0], "+" if h[1][1] > 0 else "-", h[1][0]))
        w("    double %s;" % ", ".join("w4_%d = 0.0" % f for f in range(len(fours))))
        first = {}
        for k, (p_, t, j) in enumerate(pairs):
            if k in four_of:
                f, sg = four_of[k]
                cm = "%sc4_%d" % (sgn[sg], f)
            else:
                cm = "cm%d" % k
            w("    %s[%d] = fma(g%d, %s, %s[%d]);  // pair (%d,%d)" % (bar[O], j, p_, cm, bar[O], j, p_, j))
            w("    %s[%d] = fma(-g%d, %s, %s[%d]);" % (bar[O], p_, j, cm, bar[O], p_))
            if k in four_of:
                ps, ns = ("", "-") if sg > 0 else ("-", "")
                if f in first:
                    w("    w4_%d = fma(%sg%d, %s[%d], fma(%sg%d, %s[%d], w4_%d));" % (f, ps, p_, O, j, ns, j, O, p_, f))
                else:
                    w("    w4_%d = fma(%sg%d, %s[%d], %sg%d * %s[%d]);" % (f, ps, p_, O, j, ns, j, O, p_))
                    first[f] = True
            else:
                w("    double w%d = fma(g%d, %s[%d], -(g%d * %s[%d]));" % (k, p_, O, j, j, O, p_))
        for f, (_, h) in enumerate(fours):
            for k, sg in h:
                w("    w%d %s= w4_%d;" % (k, "+" if sg > 0 else "-", f))
        for k in two:
            p_, t, j = pairs[k]
            i_, j_ = max(T[p_][t][:2]), -min(T[p_][t][:2])
            w("    %s[%d] += w%d;" % (bar[I], i_ - 1, k))
            w("    %s[%d] -= w%d;" % (bar[I], j_ - 1, k))
        w("  }")
    w("}")
    out = os.path.join(HERE, "sgh_hex_geometry.cuh")
    with open(out, "w") as f:
        f.write("\n".join(L) + "\n")
    print("wrote", out, "pairs", len(pairs))


if __name__ == "__main__":
    main()
