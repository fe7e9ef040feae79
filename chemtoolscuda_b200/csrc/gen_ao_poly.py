"""Generate ctc_ao_poly.inc: per-type AO polynomial evaluators with literal exponents.

For every segment type (s, p, Cartesian/pure d, f, g) one device function
evaluates all components and, depending on DERIV, their first and second
derivatives (written to o[q * ld_q + component * ldc]), given the powers
X[i] = x^i (Y, Z alike) and the contracted radial sums R0, R1, R2 (see
ctc_ao.cu).  With P the component's angular polynomial, P_k and P_kl its
derivatives, S_k = -2 R1 P_k, T = -2 R1 P and U = 4 R2 P:
    phi        = P R0
    d_k phi    = P_k R0 + x_k T
    d_k d_l phi = P_kl R0 + x_l (S_k + x_k U) + x_k S_l          (k != l)
    d_k d_k phi = P_kk R0 + T + x_k (2 S_k + x_k U)
Only the non-zero terms of the polynomials are written, so a component costs
about 40 operations for all ten quantities whatever its number of terms.

With TRACK = 1 the running maximum of the high word of |value| (sign cleared;
its exponent is the exponent of the largest |value|) over the components is
kept in mx[0], with TRACK = 4 also those of the three first derivatives in
mx[1..3] (the row scales of the tensor-core split operands).  With TRACK = -1
the weighted row w = wv[0] value + wv[1..3] . gradient (the adjoint's second
operand) is written as quantity 10, with TRACK = -2 the value and w (as
quantity 1) are all that is written.  The terms come from gen_terms.py;
writing their exponents as literals lets the compiler keep the power arrays in
registers and share the monomials between components.

    python chemtoolscuda_b200/csrc/gen_ao_poly.py > chemtoolscuda_b200/csrc/ctc_ao_poly.inc
"""
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from gen_terms import TYPES, comps  # noqa: E402


AX = "XYZ"
SECOND = [(0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)]  # quantities 4 .. 9


def deriv(poly, k):
    out = []
    for c, *e in poly:
        if e[k]:
            f = list(e)
            f[k] -= 1
            out.append((c * e[k], *f))
    return out


def expr(poly):
    """C expression of a polynomial, None when it is zero, a number when constant."""
    terms = []
    for c, *e in poly:
        m = [f"{AX[k]}[{n}]" for k, n in enumerate(e) if n]
        C = repr(float(c))
        if not m:
            terms.append(C)
        elif c == 1:
            terms.append("(" + " * ".join(m) + ")")
        else:
            terms.append(f"{C} * (" + " * ".join(m) + ")")
    return " + ".join(terms) if terms else None


def emit_type(ti, l, pure):
    cs = comps(l, pure)
    out = [f"// type {ti}: l = {l}{' (pure)' if pure else ''}, {len(cs)} components",
           "template <int DERIV, int TRACK>",
           f"__device__ __forceinline__ void ao_poly_{ti}(const double* X, const double* Y, const double* Z,",
           "    double R0, double R1, double R2, double* __restrict__ o, int64_t ld_q, int64_t ldc, int nq_out,",
           "    unsigned* mx, const double* wv) {",
           "  const double M1 = -2.0 * R1, M2 = 4.0 * R2;"]
    for j, comp in enumerate(cs):
        poly = [tuple(t) for t in comp]
        d1 = [expr(deriv(poly, k)) for k in range(3)]
        out.append("  {")
        out.append("    double q0, q1 = 0.0, q2 = 0.0, q3 = 0.0, q4 = 0.0, q5 = 0.0, q6 = 0.0, q7 = 0.0, q8 = 0.0, q9 = 0.0;")
        out.append(f"    const double P = {expr(poly)};")
        out.append("    q0 = P * R0;")
        out.append("    if (DERIV >= 1) {")
        out.append("      const double T = P * M1;")
        for k in range(3):
            x = f"{AX[k]}[1]"
            if d1[k]:
                out.append(f"      const double P{k} = {d1[k]};")
                out.append(f"      q{1 + k} = fma({x}, T, P{k} * R0);")
            else:
                out.append(f"      q{1 + k} = {x} * T;")
        out.append("      if (DERIV >= 2) {")
        out.append("        const double U = P * M2;")
        for k in range(3):
            x = f"{AX[k]}[1]"
            if d1[k]:
                out.append(f"        const double S{k} = P{k} * M1, W{k} = fma({x}, U, S{k});")
            else:
                out.append(f"        const double W{k} = {x} * U;")
        for q, (k, m) in enumerate(SECOND):
            pkl = expr(deriv(deriv(poly, k), m))
            xk, xm = f"{AX[k]}[1]", f"{AX[m]}[1]"
            if k == m:
                base = f"fma({pkl}, R0, T)" if pkl else "T"
                inner = f"(W{k} + S{k})" if d1[k] else f"W{k}"
                out.append(f"        q{4 + q} = fma({xk}, {inner}, {base});")
            else:
                base = None
                if pkl:
                    base = f"({pkl}) * R0"
                if d1[m]:
                    base = f"fma({xk}, S{m}, {base})" if base else f"{xk} * S{m}"
                out.append(f"        q{4 + q} = " + (f"fma({xm}, W{k}, {base});" if base else f"{xm} * W{k};"))
        out.append("      }")
        out.append("    }")
        c = f"{j} * ldc"
        out.append(f"    o[{c}] = q0;")
        out.append("    if (TRACK < 0) {")
        out.append("      const double w = wv[0] * q0 + wv[1] * q1 + wv[2] * q2 + wv[3] * q3;")
        out.append(f"      o[(TRACK == -1 ? 10 : 1) * ld_q + {c}] = w;")
        out.append("    }")
        out.append(f"    if (TRACK != -2 && DERIV >= 1) {{ if (nq_out > 1) {{ o[ld_q + {c}] = q1; o[2 * ld_q + {c}] = q2; o[3 * ld_q + {c}] = q3; }} }}")
        out.append(f"    if (DERIV >= 2) {{ if (nq_out > 4) {{ o[4 * ld_q + {c}] = q4; o[5 * ld_q + {c}] = q5; o[6 * ld_q + {c}] = q6;")
        out.append(f"      o[7 * ld_q + {c}] = q7; o[8 * ld_q + {c}] = q8; o[9 * ld_q + {c}] = q9; }} }}")
        out.append("    if (TRACK >= 1) mx[0] = max(mx[0], abs_hi(q0));")
        out.append("    if (TRACK >= 4 && DERIV >= 1) { mx[1] = max(mx[1], abs_hi(q1)); mx[2] = max(mx[2], abs_hi(q2)); mx[3] = max(mx[3], abs_hi(q3)); }")
        out.append("  }")
    out.append("}")
    return out


def main():
    print("// Generated by gen_ao_poly.py -- do not edit.")
    for ti, (l, pure) in enumerate(TYPES):
        print("\n".join(emit_type(ti, l, pure)))
        print()


if __name__ == "__main__":
    main()
