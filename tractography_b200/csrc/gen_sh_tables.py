#!/usr/bin/env python3
"""Generate the real symmetric spherical-harmonic tables used by the tracker.

Basis (the MRtrix3 convention the reference uses, ``tractography/core.py:
169-202`` and ``resources/kernels/utils/spharm.cl:216-413``): for even
``l <= 8`` and ``-l <= m <= l`` the coefficient index is
``i = l (l + 1) / 2 + m`` and

    Y_{l,0}  = N_l^0 P_l^0(cos t)
    Y_{l,m}  = sqrt(2) N_l^m P_l^m(cos t) cos(m p)        (m > 0)
    Y_{l,-m} = sqrt(2) N_l^m P_l^m(cos t) sin(m p)        (m > 0)

with ``N_l^m = sqrt((2l+1)/(4 pi) (l-m)!/(l+m)!)`` and ``P_l^m`` carrying
the Condon-Shortley phase.  Writing ``P_l^m(x) = (-1)^m (1-x^2)^{m/2}
d^m P_l / dx^m`` gives ``Y = sin(t)^m R_l^m(cos t) trig(m p)`` where
``R_l^m`` is a polynomial of degree ``l - m`` with parity ``l - m``.  The
tables store ``R_l^m`` and its derivative ``dR/dx`` as polynomials in
``u = x^2`` (times ``x`` for odd parity), rounded once from exact rational
Legendre coefficients and double-precision normalisations.

Outputs (committed next to this script):
  tg_sh_table.h   -- plain C data: coefficient array and per-(l,m) index.
  tg_sh_eval.cuh  -- CUDA device code: straight-line evaluation for
                     LMAX in {0, 2, 4, 6, 8} performing, in the same order,
                     the operations the table-driven CPU evaluation performs.
  tg_sh_fold.h    -- plain C: the fold of a coefficient vector into per-order
                     polynomials in u (tgsh_fold, double sums).
  tg_sh_folded.cuh -- CUDA device code: the same fold in straight line, and
                     the straight-line evaluation of the folded form (what
                     the tracking kernels run per step).
"""

from fractions import Fraction
from math import comb, factorial, pi, sqrt
from pathlib import Path

import numpy as np

LMAX = 8
HERE = Path(__file__).resolve().parent


def legendre(l):
    """Exact coefficients of P_l(x), ascending powers."""
    coeffs = [Fraction(0)] * (l + 1)
    for k in range(l // 2 + 1):
        coeffs[l - 2 * k] += Fraction((-1) ** k * comb(l, k) * comb(2 * l - 2 * k, l), 2 ** l)
    return coeffs


def derivative(coeffs):
    return [coeffs[i] * i for i in range(1, len(coeffs))] or [Fraction(0)]


def r_poly(l, m):
    """Exact R_l^m without the normalisation, ascending powers of x."""
    p = legendre(l)
    for _ in range(m):
        p = derivative(p)
    sign = (-1) ** m
    return [sign * c for c in p]


def norm(l, m):
    n = sqrt((2 * l + 1) / (4 * pi) * factorial(l - m) / factorial(l + m))
    return n * (sqrt(2.0) if m > 0 else 1.0)


def in_u(coeffs, parity):
    """Split a parity polynomial into coefficients of u = x^2."""
    return [coeffs[parity + 2 * j] for j in range((len(coeffs) - parity + 1) // 2)]


def f32(x):
    return float(np.float32(x))


def pairs():
    """Canonical (l, m) order: m ascending, then l ascending (even l >= m)."""
    out = []
    for m in range(LMAX + 1):
        l0 = m if m % 2 == 0 else m + 1
        for l in range(l0, LMAX + 1, 2):
            out.append((l, m))
    return out


def table():
    entries = []
    for l, m in pairs():
        exact = r_poly(l, m)
        k = norm(l, m)
        deg = l - m
        parity = deg & 1
        r = [f32(float(c) * k) for c in in_u(exact[: deg + 1], parity)]
        if deg >= 1:
            d = derivative(exact[: deg + 1])
            rp = [f32(float(c) * k) for c in in_u(d[:deg], 1 - parity)]
        else:
            rp = []
        entries.append((l, m, parity, r, rp))
    return entries


def hexf(x):
    if x == 0.0:
        return "0.0f"
    return float(x).hex().replace("0000000p", "p").replace("000000p", "p") + "f"


def write_c_table(entries):
    flat = []
    rows = []
    for l, m, parity, r, rp in entries:
        r_off = len(flat)
        flat += r
        rp_off = len(flat)
        flat += rp
        rows.append((l, m, parity, r_off, len(r), rp_off, len(rp)))
    lines = [
        "/* Generated by gen_sh_tables.py -- do not edit. */",
        "/* Real symmetric SH (l <= 8): R_l^m and dR_l^m/dx as polynomials in u = x^2,",
        " * times x when the parity flag is set (the derivative has the opposite parity). */",
        "#ifndef TG_SH_TABLE_H",
        "#define TG_SH_TABLE_H",
        "",
        f"#define TG_SH_LMAX {LMAX}",
        f"#define TG_SH_NPAIRS {len(rows)}",
        "",
        "/* Per (l, m) pair in canonical order (m ascending, then l ascending):",
        " * l, m, parity of R, offset/length of R in TG_SH_COEF, offset/length of dR/dx. */",
        "static const int TG_SH_PAIRS[TG_SH_NPAIRS][7] = {",
    ]
    for row in rows:
        lines.append("    {" + ", ".join(str(v) for v in row) + "},")
    lines += ["};", "", f"static const float TG_SH_COEF[{len(flat)}] = {{"]
    for i in range(0, len(flat), 4):
        lines.append("    " + ", ".join(hexf(v) for v in flat[i:i + 4]) + ",")
    lines += ["};", "", "#endif", ""]
    (HERE / "tg_sh_table.h").write_text("\n".join(lines))


def write_cuda(entries):
    by_m = {}
    for e in entries:
        by_m.setdefault(e[1], []).append(e)

    out = [
        "/* Generated by gen_sh_tables.py -- do not edit. */",
        "/* Straight-line evaluation of the real symmetric SH model value, d/dtheta and",
        " * (d/dphi)/sin(theta) at one orientation.  Operation order equals the",
        " * table-driven evaluation described in gen_sh_tables.py. */",
        "#ifndef TG_SH_EVAL_CUH",
        "#define TG_SH_EVAL_CUH",
        "",
        "namespace tg {",
        "",
    ]

    def horner(lines, name, coeffs, parity, u, x):
        lines.append(f"        float {name} = {hexf(coeffs[-1])};")
        for c in reversed(coeffs[:-1]):
            lines.append(f"        {name} = fmaf({name}, {u}, {hexf(c)});")
        if parity:
            lines.append(f"        {name} = {name} * {x};")

    for lmax in range(0, LMAX + 1, 2):
        out += [
            f"template <> __device__ __forceinline__ void sh_eval<{lmax}>(",
            "    const float* c, float ct, float st, float cp, float sp,",
            "    float* val_out, float* dth_out, float* dph_out)",
            "{",
            "    const float u = ct * ct;",
            "    const float tc = cp + cp;",
            "    (void)u; (void)tc;",
        ]
        # trig recurrences
        out.append("    const float cm0 = 1.0f, sm0 = 0.0f;")
        if lmax >= 1:
            out.append("    float cm1 = cp, sm1 = sp;")
        for m in range(2, lmax + 1):
            out.append(f"    const float cm{m} = fmaf(tc, cm{m-1}, -cm{m-2});")
            out.append(f"    const float sm{m} = fmaf(tc, sm{m-1}, -sm{m-2});")
        out.append("    (void)cm0; (void)sm0;")
        out.append("    float stp0 = 1.0f;")
        for k in range(1, lmax + 2):
            out.append(f"    const float stp{k} = stp{k-1} * st;")
        out.append("    (void)stp0;")
        out.append("    float val = 0.0f, dth = 0.0f, dph = 0.0f;")
        for m in range(0, lmax + 1):
            ents = [e for e in by_m.get(m, []) if e[0] <= lmax]
            if not ents:
                continue
            out.append("    {")
            out.append("        float A = 0.0f, Ap = 0.0f;")
            if m > 0:
                out.append("        float B = 0.0f, Bp = 0.0f;")
            for (l, mm, parity, r, rp) in ents:
                ip = l * (l + 1) // 2 + m
                im = l * (l + 1) // 2 - m
                out.append("        {")
                horner(out, "R", r, parity, "u", "ct")
                out.append(f"        A = fmaf(c[{ip}], R, A);")
                if m > 0:
                    out.append(f"        B = fmaf(c[{im}], R, B);")
                if l > m:
                    horner(out, "Rp", rp, 1 - parity, "u", "ct")
                    out.append(f"        Ap = fmaf(c[{ip}], Rp, Ap);")
                    if m > 0:
                        out.append(f"        Bp = fmaf(c[{im}], Rp, Bp);")
                out.append("        }")
            if m == 0:
                out.append("        val = val + A;")
                out.append("        dth = fmaf(-stp1, Ap, dth);")
            else:
                out += [
                    f"        const float F = fmaf(B, sm{m}, A * cm{m});",
                    f"        const float Fp = fmaf(Bp, sm{m}, Ap * cm{m});",
                    f"        const float G = fmaf(-A, sm{m}, B * cm{m});",
                    f"        val = fmaf(stp{m}, F, val);",
                    f"        const float mw = {float(m)}f * stp{m-1};",
                    "        const float wct = mw * ct;",
                    "        dth = fmaf(wct, F, dth);",
                    f"        dth = fmaf(-stp{m+1}, Fp, dth);",
                    "        dph = fmaf(mw, G, dph);",
                ]
            out.append("    }")
        out += [
            "    *val_out = val;",
            "    *dth_out = dth;",
            "    *dph_out = dph;",
            "}",
            "",
        ]

    # value-only basis (used by seeds_from_fod): Y_i for i < (lmax+1)(lmax+2)/2
    for lmax in range(0, LMAX + 1, 2):
        out += [
            f"template <> __device__ __forceinline__ void sh_basis<{lmax}>(",
            "    float ct, float st, float cp, float sp, float* Y)",
            "{",
            "    const float u = ct * ct;",
            "    const float tc = cp + cp;",
            "    (void)u;",
        ]
        if lmax >= 1:
            out.append("    const float cm0 = 1.0f, sm0 = 0.0f; (void)cm0; (void)sm0;")
            out.append("    float cm1 = cp, sm1 = sp;")
        else:
            out.append("    (void)tc; (void)st; (void)sp;")
        if lmax >= 1:
            out.append("    float stp0 = 1.0f; (void)stp0;")
        order = 0
        for (l, m, parity, r, rp) in [e for e in entries if e[0] <= lmax]:
            while order < m:     # an order's cosine, sine and power of sin(theta) right before its terms
                order += 1
                if order >= 2:
                    out.append(f"    const float cm{order} = fmaf(tc, cm{order-1}, -cm{order-2});")
                    out.append(f"    const float sm{order} = fmaf(tc, sm{order-1}, -sm{order-2});")
                out.append(f"    const float stp{order} = stp{order-1} * st;")
            ip = l * (l + 1) // 2 + m
            im = l * (l + 1) // 2 - m
            out.append("    {")
            horner(out, "R", r, parity, "u", "ct")
            if m == 0:
                out.append(f"        Y[{ip}] = R;")
            else:
                out.append(f"        const float P = R * stp{m};")
                out.append(f"        Y[{ip}] = P * cm{m};")
                out.append(f"        Y[{im}] = P * sm{m};")
            out.append("    }")
        out += ["}", ""]

    out += ["}  // namespace tg", "", "#endif", ""]
    (HERE / "tg_sh_eval.cuh").write_text("\n".join(out))


# ----------------------------------------------------------------------------
# Folded form.  For one order m and one trigonometric part (cos: index +m,
# sin: index -m) every R_l^m has the parity p = m & 1, so
#     sum_l c_{l,+-m} R_l^m(x) = x^p S(u),  S(u) = sum_j a_j u^j,
#     a_j = sum_l c_{l,+-m} r_{l,m,j}
# with K = number of l values coefficients.  A field voxel is folded once
# (tgsh_fold, in double, then rounded to binary32); a step then evaluates S
# and S' by one Horner pass (two fused multiply-adds per coefficient)
# instead of one Horner pass per (l, m) pair.

def fold_blocks(lmax):
    """Blocks of the folded vector for band limit lmax: (m, part, parity, K, offset, ls);
    a[offset + t] is the coefficient of u^(K-1-t) (Horner order)."""
    blocks = []
    off = 0
    for m in range(0, lmax + 1):
        ls = [l for l in range(0, lmax + 1, 2) if l >= m]
        if not ls:
            continue
        for part in ([0] if m == 0 else [0, 1]):
            blocks.append((m, part, m & 1, len(ls), off, ls))
            off += len(ls)
    return blocks, off


def fold_coefficients():
    """r_{l,m,j} in double: the normalised coefficient of u^j in R_l^m / x^p."""
    r = {}
    for l, m in pairs():
        exact = r_poly(l, m)
        k = norm(l, m)
        deg = l - m
        parity = deg & 1
        for j, c in enumerate(in_u(exact[: deg + 1], parity)):
            r[(l, m, j)] = float(c) * k
    return r


def fold_terms(lmax):
    """(dst, src, r) in accumulation order: per destination, ascending l."""
    r = fold_coefficients()
    blocks, n = fold_blocks(lmax)
    terms = []
    for m, part, parity, K, off, ls in blocks:
        for j in range(K):
            dst = off + (K - 1 - j)
            for l in ls:
                if (l, m, j) in r:
                    src = l * (l + 1) // 2 + (m if part == 0 else -m)
                    terms.append((dst, src, r[(l, m, j)]))
    return terms, n


def hexd(x):
    return float(x).hex()


def write_fold_header():
    lines = [
        "/* Generated by gen_sh_tables.py -- do not edit. */",
        "/* Folded real symmetric SH coefficients (see gen_sh_tables.py): per band",
        " * limit, the terms dst += c[src] * r of the fold, in accumulation order, and",
        " * the block layout (m, part, parity, K, offset) of the folded vector. */",
        "#ifndef TG_SH_FOLD_H",
        "#define TG_SH_FOLD_H",
        "",
        "#define TGSH_FN static inline",
        "#define TGSH_TABLE static const",
        "",
    ]
    offsets = []
    total = 0
    all_terms = []
    for lmax in range(0, LMAX + 1, 2):
        terms, n = fold_terms(lmax)
        offsets.append((lmax, total, len(terms), n))
        total += len(terms)
        all_terms += terms
    lines.append(f"#define TGSH_NTERMS {total}")
    lines.append("/* per band limit 0, 2, .., 8: first term, term count, folded length */")
    lines.append("TGSH_TABLE int TGSH_FOLD_RANGE[5][3] = {")
    for lmax, first, count, n in offsets:
        lines.append(f"    {{{first}, {count}, {n}}},   /* lmax {lmax} */")
    lines.append("};")
    lines.append("TGSH_TABLE unsigned char TGSH_FOLD_DST[TGSH_NTERMS] = {")
    for i in range(0, total, 16):
        lines.append("    " + ", ".join(str(t[0]) for t in all_terms[i:i + 16]) + ",")
    lines.append("};")
    lines.append("TGSH_TABLE unsigned char TGSH_FOLD_SRC[TGSH_NTERMS] = {")
    for i in range(0, total, 16):
        lines.append("    " + ", ".join(str(t[1]) for t in all_terms[i:i + 16]) + ",")
    lines.append("};")
    lines.append("TGSH_TABLE double TGSH_FOLD_R[TGSH_NTERMS] = {")
    for i in range(0, total, 4):
        lines.append("    " + ", ".join(hexd(t[2]) for t in all_terms[i:i + 4]) + ",")
    lines.append("};")
    blocks8, _ = fold_blocks(LMAX)
    lines.append("")
    lines.append("/* Block layout for band limit 8; a smaller band limit L keeps the blocks")
    lines.append(" * with m <= L, each with K = (L - m - parity) / 2 + 1, packed in order. */")
    lines.append(f"#define TGSH_NBLOCKS {len(blocks8)}")
    lines.append("TGSH_TABLE int TGSH_BLOCKS[TGSH_NBLOCKS][2] = {   /* m, part (0 cos, 1 sin) */")
    for m, part, parity, K, off, ls in blocks8:
        lines.append(f"    {{{m}, {part}}},")
    lines.append("};")
    lines += [
        "",
        "/* Fold the coefficients c (zero-padded to the full band of lmax) into a:",
        " * each a[d] is the double sum of its terms in table order, rounded once. */",
        "TGSH_FN void tgsh_fold(int lmax, const float* c, float* a)",
        "{",
        "    const int* range = TGSH_FOLD_RANGE[lmax / 2];",
        "    double acc[48];",
        "    for (int i = 0; i < range[2]; ++i) acc[i] = 0.0;",
        "    for (int t = range[0]; t < range[0] + range[1]; ++t) {",
        "        const double prod = (double)c[TGSH_FOLD_SRC[t]] * TGSH_FOLD_R[t];",
        "        acc[TGSH_FOLD_DST[t]] = acc[TGSH_FOLD_DST[t]] + prod;",
        "    }",
        "    for (int i = 0; i < range[2]; ++i) a[i] = (float)acc[i];",
        "}",
        "",
        "#endif",
        "",
    ]
    (HERE / "tg_sh_fold.h").write_text("\n".join(lines))


def write_fold_eval():
    """Straight-line CUDA fold (tgsh_fold's sums) and evaluation of the folded form,
    in the operation order of the oracle's block loop."""
    out = [
        "/* Generated by gen_sh_tables.py -- do not edit. */",
        "/* The fold of a voxel's SH coefficients (tgsh_fold's sums), and the value,",
        " * d/dtheta and (d/dphi)/sin(theta) of the real symmetric SH model from it: per",
        " * order m and part, S(u) and S'(u) by one Horner pass, then A = x^p S and dA/dx.",
        " * Written for scalar instructions: with cosine and sine part of an order in",
        " * register pairs (tg_f32x2.cuh) it took 147 instructions instead of 182 but, at",
        " * 96 registers, 40 to 150 bytes of spills, and the paired multiply-adds hold the",
        " * arithmetic pipe for two cycles each: 593 ms against 558 ms for 100k SDE seeds.",
        " * Each order's trigonometric factors and powers stand right before their block:",
        " * all of them up front took 570 ms where this order takes 540 ms. */",
        "#ifndef TG_SH_FOLDED_CUH",
        "#define TG_SH_FOLDED_CUH",
        "",
        "namespace tg {",
        "",
    ]
    for lmax in range(0, LMAX + 1, 2):
        sums = {}
        for dst, src, r in fold_terms(lmax)[0]:
            sums[dst] = f"({sums.get(dst, '0.0')} + (double)c[{src}] * {hexd(r)})"
        out += [f"template <> __device__ __forceinline__ void sh_fold<{lmax}>(const float* c, float* a)", "{"]
        out += [f"    a[{dst}] = (float){sums[dst]};" for dst in sorted(sums)]
        out += ["}", ""]
        blocks, n = fold_blocks(lmax)
        out += [
            f"template <> __device__ __forceinline__ void sh_eval_folded<{lmax}>(",
            "    const float* a, float ct, float st, float cp, float sp,",
            "    float* val_out, float* dth_out, float* dph_out)",
            "{",
            "    const float u = ct * ct;",
            "    const float x2 = ct + ct;",
            "    const float u2 = u + u;",
            "    const float tc = cp + cp;",
            "    (void)x2; (void)u2; (void)tc; (void)sp;",
            "    const float cm0 = 1.0f, sm0 = 0.0f;",
            "    (void)cm0; (void)sm0;",
        ]
        if lmax >= 1:
            out.append("    const float cm1 = cp, sm1 = sp;")
        out.append("    const float stp0 = 1.0f;")
        out.append("    (void)stp0;")
        out.append("    float val = 0.0f, dth = 0.0f, dph = 0.0f;")
        by_m = {}
        for blk in blocks:
            by_m.setdefault(blk[0], []).append(blk)
        powers = 0
        for m in sorted(by_m):
            # each order's cosine, sine and powers of sin(theta) right before its block
            if m >= 2:
                out.append(f"    const float cm{m} = fmaf(tc, cm{m-1}, -cm{m-2});")
                out.append(f"    const float sm{m} = fmaf(tc, sm{m-1}, -sm{m-2});")
            while powers < min(m + 1, lmax + 1):
                powers += 1
                out.append(f"    const float stp{powers} = stp{powers-1} * st;")
            out.append("    {")
            names = ["A", "B"]
            has_deriv = False
            for (mm, part, parity, K, off, ls), nm in zip(by_m[m], names):
                # S and S' by Horner (a[off] is the highest power)
                if K == 1:
                    out.append(f"        const float S{nm} = a[{off}];")
                else:
                    out.append(f"        float D{nm} = a[{off}];")
                    out.append(f"        float S{nm} = fmaf(a[{off}], u, a[{off + 1}]);")
                    for t in range(2, K):
                        out.append(f"        D{nm} = fmaf(D{nm}, u, S{nm});")
                        out.append(f"        S{nm} = fmaf(S{nm}, u, a[{off + t}]);")
                if parity:
                    out.append(f"        const float {nm} = S{nm} * ct;")
                    if K == 1:
                        out.append(f"        const float {nm}p = S{nm};")
                    else:
                        out.append(f"        const float {nm}p = fmaf(u2, D{nm}, S{nm});")
                    has_deriv = True
                else:
                    out.append(f"        const float {nm} = S{nm};")
                    if K > 1:
                        out.append(f"        const float {nm}p = x2 * D{nm};")
                        has_deriv = True
            if m == 0:
                out.append("        val = val + A;")
                if has_deriv:
                    out.append("        dth = fmaf(-stp1, Ap, dth);")
            else:
                out.append(f"        const float F = fmaf(B, sm{m}, A * cm{m});")
                if has_deriv:
                    out.append(f"        const float Fp = fmaf(Bp, sm{m}, Ap * cm{m});")
                out.append(f"        const float G = fmaf(-A, sm{m}, B * cm{m});")
                out.append(f"        val = fmaf(stp{m}, F, val);")
                out.append(f"        const float mw = {float(m)}f * stp{m-1};")
                out.append("        const float wct = mw * ct;")
                out.append("        dth = fmaf(wct, F, dth);")
                if has_deriv:
                    out.append(f"        dth = fmaf(-stp{m+1}, Fp, dth);")
                out.append("        dph = fmaf(mw, G, dph);")
            out.append("    }")
        out += ["    *val_out = val;", "    *dth_out = dth;", "    *dph_out = dph;", "}", ""]
    out += ["}  // namespace tg", "", "#endif", ""]
    (HERE / "tg_sh_folded.cuh").write_text("\n".join(out))


def main():
    entries = table()
    write_c_table(entries)
    write_cuda(entries)
    write_fold_header()
    write_fold_eval()


if __name__ == "__main__":
    main()
