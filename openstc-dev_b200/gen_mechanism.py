"""Generates csrc/mech_h2air9.cuh: the finite-rate chemistry source of the
9-species, 19-reaction H2-air mechanism as straight-line device code.

The generic kernel (csrc/chem.cuh: chemistry_omega) walks the reactions in
a runtime loop and, for each, all nine species through stoichiometric
tables in __constant__ memory. For a mechanism known at build time the
structure (reaction types, stoichiometric coefficients, reaction orders)
becomes code: only the participating species are touched, with literal
coefficients. The rate parameters (A, b, Ea, the second Arrhenius set,
third-body efficiencies, Troe constants) stay runtime values read from the
same __constant__ tables, so a context uses the generated code whenever its
mechanism has this structure (checked on the host against the tables
below) and the generic code otherwise. The arithmetic is the generic
code's, operation by operation, with the exact no-ops left out (terms with
a zero coefficient, multiplications by one, a zero reaction order); the
compiler may still contract products into FMAs differently.

    python openstc-dev_b200/gen_mechanism.py      # rewrites csrc/mech_h2air9.cuh
"""
from pathlib import Path

import numpy as np

import chemdata

OUT = Path(__file__).resolve().parent / "csrc" / "mech_h2air9.cuh"


def _lit(v):
    return repr(float(v))


def generate(mech) -> str:
    t = mech.tables
    ns, nr = mech.n_spec, mech.n_reac
    rt = np.asarray(t["reac_type"]).astype(int)
    nuf = np.asarray(t["stoi_f"]).reshape(nr, ns).astype(int)
    nub = np.asarray(t["stoi_b"]).reshape(nr, ns).astype(int)
    order = np.asarray(t["reac_order"]).astype(int)
    L = []
    w = L.append
    w("// mech_h2air9.cuh — GENERATED by openstc-dev_b200/gen_mechanism.py from")
    w("// data/h2_air_9sp.json (%s); regenerate instead of editing." % ", ".join(mech.names))
    w("//")
    w("// The chemistry source of this mechanism's structure as straight-line code")
    w("// (the generic form is chem.cuh: chemistry_omega, FiniteRateChem.cu:7-194);")
    w("// rate parameters are read from c_p at run time.")
    w("#pragma once")
    w('#include "chem.cuh"')
    w("")
    w("namespace ostc {")
    w("namespace mech_h2air9 {")
    w("")
    w("constexpr int NS = %d, NR = %d;" % (ns, nr))
    w("// the structure a context's mechanism must have to use the generated code")
    w("constexpr int reac_type[NR] = {%s};" % ", ".join(map(str, rt)))
    w("constexpr int reac_order[NR] = {%s};" % ", ".join(map(str, order)))
    w("constexpr int stoi_f[NR][NS] = {%s};" % ", ".join("{%s}" % ", ".join(map(str, r)) for r in nuf))
    w("constexpr int stoi_b[NR][NS] = {%s};" % ", ".join("{%s}" % ", ".join(map(str, r)) for r in nub))
    w("")
    w("__device__ __forceinline__ void omega(double rho, double t, const double *Y, double *om) {")
    w("  double c[NS], g[NS];")
    w("  double lnT, invT, ln_temp_t;")
    w("  chemistry_setup<NS>(rho, t, Y, c, g, lnT, invT, ln_temp_t);")
    w("  double cre[NS], des[NS];")
    w("#pragma unroll")
    w("  for (int l = 0; l < NS; ++l) {")
    w("    cre[l] = 0;")
    w("    des[l] = 0;")
    w("  }")
    def rates(r):
        """q1, q2 of reaction r (the body of a scope)"""
        ty = int(rt[r])
        eq = " + ".join(("%d %s" % (nuf[r, l], mech.names[l])).replace("1 ", "") for l in range(ns) if nuf[r, l])
        eqb = " + ".join(("%d %s" % (nub[r, l], mech.names[l])).replace("1 ", "") for l in range(ns) if nub[r, l])
        w("  {  // %d: %s = %s (type %d)" % (r, eq, eqb, ty))
        w("    double kf = arrhenius(lnT, invT, c_p.A[%d], c_p.b[%d], c_p.Ea[%d]);" % (r, r, r))
        if ty == 3:
            w("    kf += arrhenius(lnT, invT, c_p.A2[%d], c_p.b2[%d], c_p.Ea2[%d]);" % (r, r, r))
        if ty > 3:
            w("    double cc = 0;")
            for l in range(ns):
                w("    cc += c[%d] * c_p.tb[%d][%d];" % (l, r, l))
            if ty == 4:
                w("    kf *= cc;")
            else:
                w("    {")
                w("      const double kf_low = arrhenius(lnT, invT, c_p.A2[%d], c_p.b2[%d], c_p.Ea2[%d]);" % (r, r, r))
                w("      const double kf_high = kf;")
                w("      const double pr = kf_low * cc / kf_high;")
                w("      double F = 1.0;")
                if ty > 5:
                    w("      double f_cent = (1 - c_p.troe_alpha[%d]) * exp(-t / c_p.troe_t3[%d]) + "
                      "c_p.troe_alpha[%d] * exp(-t / c_p.troe_t1[%d]);" % (r, r, r, r))
                    if ty == 7:
                        w("      f_cent += exp(-c_p.troe_t2[%d] / t);" % r)
                    w("      const double logFc = log10(f_cent);")
                    w("      const double cc2 = -0.4 - 0.67 * logFc;")
                    w("      const double nn = 0.75 - 1.27 * logFc;")
                    w("      const double logPr = log10(pr);")
                    w("      const double tempo = (logPr + cc2) / (nn - 0.14 * (logPr + cc2));")
                    w("      const double pp = logFc / (1.0 + tempo * tempo);")
                    w("      F = pow(10.0, pp);")
                w("      kf = kf_high * pr / (1.0 + pr) * F;")
                w("    }")
        if ty == 2:
            w("    const double kb = arrhenius(lnT, invT, c_p.A2[%d], c_p.b2[%d], c_p.Ea2[%d]);" % (r, r, r))
        elif ty != 0:
            w("    double dg = 0;")
            for l in range(ns):
                d = int(nub[r, l] - nuf[r, l])
                if d == 1:
                    w("    dg += g[%d];" % l)
                elif d == -1:
                    w("    dg -= g[%d];" % l)
                elif d:
                    w("    dg += g[%d] * %s;" % (l, _lit(d)))
            if order[r] == 0:
                w("    const double kb = kf * exp(dg);")
            else:
                w("    const double kb = kf * exp(dg - %s * ln_temp_t);" % _lit(order[r]))
        prod_f = ["ipow(c[%d], %d)" % (l, nuf[r, l]) if nuf[r, l] > 1 else "c[%d]" % l
                  for l in range(ns) if nuf[r, l]]
        prod_b = ["ipow(c[%d], %d)" % (l, nub[r, l]) if nub[r, l] > 1 else "c[%d]" % l
                  for l in range(ns) if nub[r, l]]
        w("    double q1 = 1.0, q2 = 1.0;")
        for f in prod_f:
            w("    q1 *= %s;" % f)
        if ty != 0:
            for f in prod_b:
                w("    q2 *= %s;" % f)
        w("    q1 *= kf;")
        w("    q2 %s;" % ("*= kb" if ty != 0 else "= 0.0"))

    for r in range(nr):
        rates(r)
        def term(q, k):
            return q if k == 1 else "%s * %s" % (q, _lit(k))

        for l in range(ns):
            a, b = int(nuf[r, l]), int(nub[r, l])
            if a and b:
                w("    cre[%d] += q2 * %s + q1 * %s;" % (l, _lit(a), _lit(b)))
                w("    des[%d] += q1 * %s + q2 * %s;" % (l, _lit(a), _lit(b)))
            elif a:
                w("    cre[%d] += %s;" % (l, term("q2", a)))
                w("    des[%d] += %s;" % (l, term("q1", a)))
            elif b:
                w("    cre[%d] += %s;" % (l, term("q1", b)))
                w("    des[%d] += %s;" % (l, term("q2", b)))
        w("  }")
    w("#pragma unroll")
    w("  for (int l = 0; l < NS; ++l) om[l] = cre[l] * (c_p.mw[l] * 1e+3) - des[l] * (c_p.mw[l] * 1e+3);")
    w("}")
    w("")
    # the chemical Jacobian over the species that take part in a reaction
    act = [l for l in range(ns) if nuf[:, l].any() or nub[:, l].any()]
    w("// species that take part in a reaction")
    w("constexpr int NA = %d;" % len(act))
    w("__host__ __device__ constexpr int active(int m) {")
    w("  constexpr int a[NA] = {%s};" % ", ".join(map(str, act)))
    w("  return a[m];")
    w("}")
    w("")
    w("// net molar production wd[NA] (mol/(cm^3 s)) and its sensitivities")
    w("// Z[m][n] = sum_r (nu''_m - nu'_m) (nu'_n q1 - nu''_n q2) over the active species:")
    w("// d omega_m / d(rho Y_n) = 1e3 W_m Z[m][n] / (rho Y_n) (chem.cuh: chemistry_jacobian).")
    w("// Each reaction adds to the entries of its own species only, and every index is a")
    w("// literal, so Z stays in registers.")
    w("__device__ __forceinline__ void production_jacobian(double rho, double t, const double *Y, double *wd,")
    w("                                                    double (&Z)[NA][NA]) {")
    w("  double c[NS], g[NS];")
    w("  double lnT, invT, ln_temp_t;")
    w("  chemistry_setup<NS>(rho, t, Y, c, g, lnT, invT, ln_temp_t);")
    w("#pragma unroll")
    w("  for (int m = 0; m < NA; ++m) {")
    w("    wd[m] = 0;")
    w("#pragma unroll")
    w("    for (int n = 0; n < NA; ++n) Z[m][n] = 0;")
    w("  }")

    def add(to, k, q):
        if k:
            w("    %s %s= %s;" % (to, "+" if k > 0 else "-", q if abs(k) == 1 else "%s * %s" % (_lit(abs(k)), q)))

    for r in range(nr):
        rates(r)
        w("    const double net = q1 - q2;")
        for l in act:
            add("wd[%d]" % act.index(l), int(nub[r, l] - nuf[r, l]), "net")
        for n in act:
            for m in act:
                k = int(nub[r, m] - nuf[r, m])
                add("Z[%d][%d]" % (act.index(m), act.index(n)), k * int(nuf[r, n]), "q1")
                if rt[r] != 0:
                    add("Z[%d][%d]" % (act.index(m), act.index(n)), -k * int(nub[r, n]), "q2")
        w("  }")
    w("}")
    w("")
    w("}  // namespace mech_h2air9")
    w("}  // namespace ostc")
    return "\n".join(L) + "\n"


if __name__ == "__main__":
    OUT.write_text(generate(chemdata.h2_air_9sp()))
    print("wrote", OUT)
