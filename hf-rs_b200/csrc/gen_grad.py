"""Generate the straight-line ERI-derivative code of the light classes (grad_gen.cuh).

For every class (la lb|lc ld) of s, p and d shells with la + lb + lc + ld <= 4
but (21|10), whose body no longer fits the compiler's register allocation, this
emits GradClass<LA,LB,LC,LD>::prim: the derivatives of one primitive
quartet's contribution sum_{abcd} G_abcd (ab|cd), G the two-particle density
block, in the McMurchie-Davidson form

  sum_{h,k} (-1)^|k| E^{ab}_h E^{cd}_k G_abcd R_{h+k},   h, k Hermite triples.

With P the bra's product centre and R_AB = A - B,
  d/dA = (alpha/p) d/dP + d/dR_AB,   d/dB = (beta/p) d/dP - d/dR_AB,
where d/dP raises R and d/dR_AB acts on E^{ab} only (and the same for the
ket, with d/dQ = -d/dP).  prim() returns
  e     = the quartet's value,
  gp[3] = d/dP,
  gb[3], gk[3] = d/dR_AB, d/dR_CD of the Hermite coefficients, the Gaussian
          product factors apart (the caller adds -2 mu R_AB e).
Two passes keep few values live: over k with t_ab = sum_cd G E^{cd}_k, then
over h with x_cd = sum_ab G E^{ab}_h.

Run:  python gen_grad.py   (writes grad_gen.cuh next to this file)
"""
import os

from gen_eri import cart

AX = "xyz"
LTOT = 4
VMAX = 40  # accumulators of one pass that still stay in registers


def herm(l):
    return [(t, u, v) for t in range(l + 1) for u in range(l + 1 - t) for v in range(l + 1 - t - u)]


class Side:
    """Hermite coefficients of a side as C expressions over named scalars."""

    def __init__(self, n, l1, l2):
        self.n, self.l1, self.l2 = n, l1, l2
        self.c1, self.c2 = cart(l1), cart(l2)
        self.pairs = [(a, b) for a in self.c1 for b in self.c2]
        self.lines = []
        self.E, self.D = {}, {}  # (axis, i, j, t) -> expression ("0" and "1" folded)
        for ax in range(3):
            for i in range(l1 + 1):
                for j in range(l2 + 1):
                    for t in range(i + j + 1):
                        self.coef(ax, i, j, t)

    def get(self, tab, ax, i, j, t):
        return tab.get((ax, i, j, t), "0") if 0 <= t <= i + j else "0"

    def put(self, tab, pre, key, terms):
        """terms: list of factor lists; names the sum."""
        out = []
        for fs in terms:
            if "0" in fs:
                continue
            fs = [f for f in fs if f != "1"]
            out.append(" * ".join(fs) if fs else "1.0")
        if not out:
            tab[key] = "0"
        elif len(out) == 1 and " " not in out[0] and out[0] != "1.0":
            tab[key] = out[0]
        else:
            name = "%s%s%s%d%d%d" % (self.n, pre, AX[key[0]], key[1], key[2], key[3])
            self.lines.append("const double %s = %s;" % (name, " + ".join(out)))
            tab[key] = name

    def coef(self, ax, i, j, t):
        key = (ax, i, j, t)
        if i + j == 0:
            self.E[key], self.D[key] = "1", "0"
            return
        q = (i - 1, j) if i else (i, j - 1)
        x = "%s%s%s" % (self.n, "a" if i else "b", AX[ax])       # P - A or P - B
        dx = "%s%s" % (self.n, "da" if i else "db")              # its derivative: -beta/p or alpha/p
        e = lambda s: self.get(self.E, ax, q[0], q[1], s)
        d = lambda s: self.get(self.D, ax, q[0], q[1], s)
        k = "1" if t == 0 else "%d.0" % (t + 1)
        self.put(self.E, "e", key, [["%si2p" % self.n, e(t - 1)], [x, e(t)], [k, e(t + 1)]])
        self.put(self.D, "d", key, [["%si2p" % self.n, d(t - 1)], [x, d(t)], [dx, e(t)], [k, d(t + 1)]])

    def product(self, pair, h, d=None):
        """Factors of E^{pair}_h (axis d differentiated), or None if zero."""
        a, b = self.pairs[pair]
        fs = []
        for ax in range(3):
            f = self.get(self.D if ax == d else self.E, ax, a[ax], b[ax], h[ax])
            if f == "0":
                return None
            if f != "1":
                fs.append(f)
        return fs

    def support(self, pair):
        a, b = self.pairs[pair]
        return [(t, u, v) for t in range(a[0] + b[0] + 1) for u in range(a[1] + b[1] + 1) for v in range(a[2] + b[2] + 1)]


def add(h, k):
    return tuple(x + y for x, y in zip(h, k))


def rname(h):
    return "r%d%d%d" % h


def emit(la, lb, lc, ld):
    out = []
    w = out.append
    B, K = Side("b", la, lb), Side("k", lc, ld)
    lab, lcd = la + lb, lc + ld
    L = lab + lcd + 1
    ncd = len(K.pairs)
    w("template <> struct GradClass<%d, %d, %d, %d> {" % (la, lb, lc, ld))
    w("  static constexpr int L = %d;" % (L - 1))
    w("  // F: (-2 alpha)^m pref F_m, m <= L + 1; G: the density block, element x at G[x * gs]")
    w("  static __device__ __forceinline__ void prim(const double* __restrict__ G, int gs, const double* F, double PQx,")
    w("      double PQy, double PQz, double bax, double bay, double baz, double bbx, double bby, double bbz, double bi2p,")
    w("      double bda, double bdb, double kax, double kay, double kaz, double kbx, double kby, double kbz, double ki2p,")
    w("      double kda, double kdb, double& e_out, double* gp, double* gb, double* gk) {")
    # R_tuv of degree <= L
    names = {(m, (0, 0, 0)): "F[%d]" % m for m in range(L + 1)}

    def need(m, h):
        if (m, h) in names:
            return names[(m, h)]
        ax = 0 if h[0] else (1 if h[1] else 2)
        h1 = tuple(x - (k == ax) for k, x in enumerate(h))
        s = "PQ%s * %s" % (AX[ax], need(m + 1, h1))
        c = h1[ax]
        if c:
            h2 = tuple(x - (k == ax) for k, x in enumerate(h1))
            s += " + %s%s" % ("" if c == 1 else "%d.0 * " % c, need(m + 1, h2))
        n = rname(h) if m == 0 else "r%d_%d%d%d" % ((m,) + h)
        w("    const double %s = %s;" % (n, s))
        names[(m, h)] = n
        return n

    R = {h: need(0, h) for h in sorted(herm(L), key=lambda h: (sum(h), h))}
    for l in B.lines + K.lines:
        w("    " + l)

    def named(side, pair, h, d=None):
        """A name for E^{pair}_h (or its derivative), declared once."""
        fs = side.product(pair, h, d)
        if fs is None:
            return None
        if not fs:
            return "1"
        if len(fs) == 1:
            return fs[0]
        n = "%sp%s%d_%d%d%d" % ((side.n, "" if d is None else AX[d], pair) + h)
        if n not in declared:
            declared.add(n)
            w("    const double %s = %s;" % (n, " * ".join(fs)))
        return n

    declared = set()
    mul = lambda a, b: b if a == "1" else (a if b == "1" else "%s * %s" % (a, b))
    G = lambda ab, cd: "G[%d * gs]" % (ab * ncd + cd)
    w("    double e = 0.0, gpx = 0.0, gpy = 0.0, gpz = 0.0, gbx = 0.0, gby = 0.0, gbz = 0.0, gkx = 0.0, gky = 0.0, gkz = 0.0;")
    hb, hk = herm(lab), herm(lcd)
    nnzb = sum(len(B.support(p)) for p in range(len(B.pairs)))
    vacc = lab > 0 and len(hk) > 1 and nnzb <= VMAX
    if vacc:
        for p in range(len(B.pairs)):
            for h in B.support(p):
                w("    double v%d_%d%d%d = 0.0;" % ((p,) + h))
    # pass 1: over the ket's Hermite triples
    for k in hk:
        sg = "-" if sum(k) & 1 else "+"
        w("    {")
        ts = []
        for ab in range(len(B.pairs)):
            terms = []
            for cd in range(ncd):
                n = named(K, cd, k)
                if n is not None:
                    terms.append(mul(n, G(ab, cd)))
            w("    const double t%d = %s;" % (ab, " + ".join(terms)))
            ts.append("t%d" % ab)
        # y_h = sum_ab t_ab E^{ab}_h, against the raised R
        for h in hb:
            terms = []
            for ab in range(len(B.pairs)):
                n = named(B, ab, h)
                if n is not None:
                    terms.append(mul(n, ts[ab]))
            w("    const double y%d%d%d = %s;" % (h + (" + ".join(terms),)))
        for ax in range(3):
            s = " + ".join("y%d%d%d * %s" % (h + (R[add(add(h, k), tuple(int(x == ax) for x in range(3)))],)) for h in hb)
            w("    gp%s %s= %s;" % (AX[ax], sg, s))
        w("    e %s= %s;" % (sg, " + ".join("y%d%d%d * %s" % (h + (R[add(h, k)],)) for h in hb)))
        if lab > 0:
            if vacc:
                for ab in range(len(B.pairs)):
                    for h in B.support(ab):
                        w("    v%d_%d%d%d %s= t%d * %s;" % ((ab,) + h + (sg, ab, R[add(h, k)])))
            else:
                for ax in range(3):
                    tot = []
                    for h in hb:
                        terms = []
                        for ab in range(len(B.pairs)):
                            fs = B.product(ab, h, ax)
                            if fs is not None:
                                terms.append(" * ".join(fs + [ts[ab]]))
                        if terms:
                            tot.append("(%s) * %s" % (" + ".join(terms), R[add(h, k)]))
                    if tot:
                        w("    gb%s %s= %s;" % (AX[ax], sg, " + ".join(tot)))
        w("    }")
        declared = {n for n in declared if not n.startswith(("bp", "kp"))}
    if vacc:
        for ax in range(3):
            terms = []
            for ab in range(len(B.pairs)):
                for h in B.support(ab):
                    fs = B.product(ab, h, ax)
                    if fs is not None:
                        terms.append(" * ".join(fs + ["v%d_%d%d%d" % ((ab,) + h)]))
            w("    gb%s = %s;" % (AX[ax], " + ".join(terms)))
    # pass 2: over the bra's Hermite triples, the ket's coefficients differentiated
    if lcd > 0:
        for cd in range(ncd):
            for k in K.support(cd):
                w("    double u%d_%d%d%d = 0.0;" % ((cd,) + k))
        for h in hb:
            w("    {")
            for cd in range(ncd):
                terms = []
                for ab in range(len(B.pairs)):
                    n = named(B, ab, h)
                    if n is not None:
                        terms.append(mul(n, G(ab, cd)))
                w("    const double x%d = %s;" % (cd, " + ".join(terms)))
            for cd in range(ncd):
                for k in K.support(cd):
                    w("    u%d_%d%d%d += x%d * %s;" % ((cd,) + k + (cd, R[add(h, k)])))
            w("    }")
            declared = {n for n in declared if not n.startswith(("bp", "kp"))}
        for ax in range(3):
            terms = []
            for cd in range(ncd):
                for k in K.support(cd):
                    fs = K.product(cd, k, ax)
                    if fs is not None:
                        terms.append(("-" if sum(k) & 1 else "+") + " " + " * ".join(fs + ["u%d_%d%d%d" % ((cd,) + k)]))
            w("    gk%s = 0.0 %s;" % (AX[ax], " ".join(terms)))
    w("    e_out = e;")
    for v in ("p", "b", "k"):
        w("    " + " ".join("g%s[%d] = g%s%s;" % (v, i, v, AX[i]) for i in range(3)))
    w("  }")
    w("};")
    return out


def render():
    """The text of grad_gen.cuh."""
    lines = ["// Generated by gen_grad.py; do not edit.", "#pragma once", "", "namespace hfg {", "",
             "template <int LA, int LB, int LC, int LD> struct GradClass;", ""]
    pairs = [(a, b) for a in range(3) for b in range(a + 1)]
    for i, (la, lb) in enumerate(pairs):
        for lc, ld in pairs[:i + 1]:
            if la + lb + lc + ld <= LTOT and (la, lb, lc, ld) != (2, 1, 1, 0):
                lines += emit(la, lb, lc, ld) + [""]
    lines.append("}  // namespace hfg")
    return "\n".join(lines) + "\n"


def main():
    with open(os.path.join(os.path.dirname(os.path.abspath(__file__)), "grad_gen.cuh"), "w") as f:
        f.write(render())


if __name__ == "__main__":
    main()
