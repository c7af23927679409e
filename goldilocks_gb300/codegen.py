"""Generator of the straight-line DFT codelets used inside the GPU kernels.

The reference generates its small NTTs (ntt/src/ntt/small.rs) with
ntt/src/bin/codegen.rs: naive 2- and 3-point transforms, Rader for the primes
5 and 17, and a `split()`-driven recursion into Good-Thomas (coprime factors)
or Cooley-Tukey (otherwise), with every twiddle whose order divides 384 turned
into shifts.  This generator applies the same selection rules but emits CUDA
device code in single-assignment form for register-resident data:

* `gl_dft_lazy<R, INV>(uint64_t *x)` transforms R values held in registers,
  natural order in and out, with omega_R = 2717^((p-1)/R) (INV: omega_R^-1);
  inputs are any words, outputs words congruent to the transform (`gl_dft`
  reduces them below p).
* additions, subtractions and twiddles of order dividing 192 (powers of two,
  omega_192 = 2: `gl_lshl<k>`) work on three unreduced limbs; other twiddles
  and the Rader constants are `gl_mont_mul` by the literal's Montgomery form
  c*2^64 mod p (the product is exactly x*c).

Usage: python -m goldilocks_gb300.codegen   (rewrites csrc/gl_codelets.cuh)
"""
import bisect
import math
import os

P = 0xFFFF_FFFF_0000_0001
ORDER = P - 1
GENERATOR = 2717
FACTORS = [3, 5, 17, 257, 65537]


def _divisors():
    d = [1 << i for i in range(33)]
    for f in FACTORS:
        d = d + [i * f for i in d]
    return sorted(d)


DIVISORS = _divisors()


def split(n):
    """Divisor of n nearest below sqrt(n), as ntt/src/divisors.rs:67-89 picks it."""
    isqrt = int(math.sqrt(float(n)))
    isqrt = (isqrt + n // isqrt) // 2
    i = bisect.bisect_left(DIVISORS, isqrt)
    for d in reversed(DIVISORS[: i + 1]):
        if n % d == 0 and n // d >= d:
            return d
    raise AssertionError


def root(n, inv=False):
    w = pow(GENERATOR, ORDER // n, P)
    return pow(w, P - 2, P) if inv else w


# Rader generators (primitive roots) for the primes dividing p - 1.
RADER_G = {5: 2, 17: 3}


class Val:
    """A generated variable and what is known of it: the exact interval
    [lo, hi] of the stored integer, and whether the value meant is its
    negation.  `wide`: three limbs (gl_l3), else one 64-bit word (any u64)."""

    def __init__(self, name, lo, hi, wide, neg=False):
        self.name, self.lo, self.hi, self.wide, self.neg = name, lo, hi, wide, neg

    def negated(self):
        return Val(self.name, self.lo, self.hi, self.wide, not self.neg)


class Gen:
    """Emits lazy arithmetic: additions, subtractions and products by powers of
    two keep three limbs without reducing; a value is folded to 64 bits where a
    general product or the end of the codelet needs it, and the values folded
    together are kept non-negative by a multiple of p on one input of their
    transform (which adds the same multiple to each of its outputs)."""

    def __init__(self, inv):
        self.inv = inv
        self.lines = []
        self.n = 0

    def word(self, expr, hi=2**64 - 1):
        return Val(self.var("uint64_t", expr), 0, hi, False)

    def limbs(self, expr, lo, hi, neg=False):
        assert -2**95 <= lo and hi < 2**95
        return Val(self.var("gl_l3", expr), lo, hi, True, neg)

    def var(self, kind, expr):
        self.n += 1
        name = "v%d" % self.n
        self.lines.append("  const %s %s = %s;" % (kind, name, expr))
        return name

    def add(self, a, b):
        if a.neg == b.neg:
            return self.limbs("gl_ladd(%s, %s)" % (a.name, b.name), a.lo + b.lo, a.hi + b.hi, a.neg)
        if a.neg:
            a, b = b, a
        return self.limbs("gl_lsub(%s, %s)" % (a.name, b.name), a.lo - b.hi, a.hi - b.lo)

    def sub(self, a, b):
        return self.add(a, b.negated())

    def shift(self, x, k):
        """x * 2^k, 2^96 = -1 by the sign."""
        neg = x.neg ^ (k % 192 >= 96)
        k %= 96
        if k == 0:
            return Val(x.name, x.lo, x.hi, x.wide, neg)
        q, s = divmod(k, 32)
        fits = lambda v: -2**31 <= (v.lo << s) >> 64 and (v.hi << s) >> 64 < 2**31  # noqa: E731
        if not fits(x):
            x = self.norm(x)
        if not fits(x):  # only by 31 bits: in two steps
            r = self.shift(self.shift(x, s - 16), k - s + 16)
            return Val(r.name, r.lo, r.hi, r.wide, r.neg ^ neg ^ x.neg)
        y0, y1, eps = 2**32 - 2**s, 2**32 - 1, 2**32 - 1
        y2lo, y2hi = (x.lo << s) >> 64, (x.hi << s) >> 64
        if q == 0:
            lo, hi = x.lo << s, x.hi << s
        elif q == 1:
            lo, hi = -y2hi, y0 * 2**32 + y1 * eps - y2lo
        else:
            lo, hi = -y1 - y2hi * 2**32, y0 * eps - y2lo * 2**32
        r = self.limbs("gl_lshl<%d>(%s)" % (k, x.name), lo, hi, neg)
        # Room for the additions that follow.
        return r if -2**91 <= lo and hi < 2**91 else self.norm(r)

    def norm(self, x):
        lo, hi = (x.lo >> 64) * (2**32 - 1), 2**64 - 1 + (x.hi >> 64) * (2**32 - 1)
        return self.limbs("gl_lnorm(%s)" % x.name, lo, hi, x.neg)

    def bias(self, x, least):
        """x plus the smallest multiple of p that is at least `least`."""
        m = -(-least // P)
        return self.limbs("gl_lbias<%d>(%s)" % (m, x.name), x.lo + m * P, x.hi + m * P, x.neg)

    def fold(self, x):
        """x as a 64-bit word congruent to it (not necessarily below p)."""
        if x.neg:
            m = max(0, -(-x.hi // P))
            x = self.limbs("gl_lnegb<%d>(%s)" % (m, x.name), m * P - x.hi, m * P - x.lo)
        if not x.wide:
            return x
        if x.lo < 0:
            x = self.bias(x, -x.lo)
        assert x.hi >> 64 < 2**31
        return self.word("gl_lfold(%s)" % x.name)

    def twiddle(self, x, order, exp):
        """x * omega_order^exp (inverse direction if self.inv)."""
        exp %= order
        if exp == 0:
            return x
        if self.inv:
            exp = (order - exp) % order
        if 192 % order == 0:
            return self.shift(x, (192 // order) * exp % 192)
        return self.mulc(x, pow(root(order), exp, P))

    def mulc(self, x, c):
        """x * c for a constant c: Montgomery product by c*2^64 mod p."""
        if x.neg:
            x, c = x.negated(), (P - c) % P
        x = self.fold(x)
        return self.word("gl_mont_mul(%s, 0x%016xull)" % (x.name, c * 2**64 % P), P - 1)

    def dft_above_zero(self, xs):
        """dft(xs) with every output that is not a word non-negative and of
        positive sign where a multiple of p on xs[0] can do it: the coefficient
        of xs[0] is 1 in each output."""
        least = 0
        for _ in range(4):
            mark, n = len(self.lines), self.n
            ys = self.dft([self.bias(xs[0], least)] + xs[1:] if least else xs)
            short = -min(y.lo for y in ys)
            if short <= 0 or any(y.neg for y in ys):
                return ys
            least += short
            del self.lines[mark:]
            self.n = n
        return self.dft(xs)

    # -- transforms on lists of variable names, natural order in/out --------
    def dft(self, xs):
        n = len(xs)
        if n == 1:
            return list(xs)
        if n == 2:
            return [self.add(xs[0], xs[1]), self.sub(xs[0], xs[1])]
        if n == 3:
            return self.dft3(xs)
        if n in RADER_G:
            return self.rader(xs)
        a = split(n)
        b = n // a
        if math.gcd(a, b) == 1:
            return self.good_thomas(xs, a, b)
        return self.cooley_tukey(xs, a, b)

    def dft3(self, xs):
        # One product instead of four: with w = omega_3 (2^64; the inverse
        # uses w^2 = -2^32) and w^2 = -1 - w,
        #   X1 = a + w b + w^2 c = (a - c) + w (b - c)
        #   X2 = a + w^2 b + w c = (a - b) - w (b - c).
        # The same field values as the reference's naive form
        # (ntt/src/bin/codegen.rs), in 7 additions and 1 product.
        a, b, c = xs
        x0 = self.add(self.add(a, b), c)
        m = self.twiddle(self.sub(b, c), 3, 1)
        x1 = self.add(self.sub(a, c), m)
        x2 = self.sub(self.sub(a, b), m)
        return [x0, x1, x2]

    def cooley_tukey(self, xs, a, b):
        # n = a*b, j = b*ja + jb, k = ka + a*kb:
        # X[ka + a*kb] = sum_jb w_b^(jb*kb) * w_n^(jb*ka) * sum_ja x[b*ja+jb] w_a^(ja*ka)
        n = a * b
        y = [[None] * b for _ in range(a)]
        for jb in range(b):
            col = self.dft([xs[b * ja + jb] for ja in range(a)])
            for ka in range(a):
                y[ka][jb] = self.twiddle(col[ka], n, jb * ka)
        out = [None] * n
        for ka in range(a):
            row = self.dft(y[ka])
            for kb in range(b):
                out[ka + a * kb] = row[kb]
        return out

    def good_thomas(self, xs, a, b):
        # gcd(a, b) = 1: input j = (b*ja + a*jb) mod n, output k = CRT(ka, kb).
        n = a * b
        y = [[None] * b for _ in range(a)]
        for jb in range(b):
            col = self.dft([xs[(b * ja + a * jb) % n] for ja in range(a)])
            for ka in range(a):
                y[ka][jb] = col[ka]
        ea = b * pow(b, -1, a)
        eb = a * pow(a, -1, b)
        out = [None] * n
        for ka in range(a):
            row = self.dft(y[ka])
            for kb in range(b):
                out[(ka * ea + kb * eb) % n] = row[kb]
        return out

    def rader(self, xs):
        # Prime q, generator g: X[g^u] = x0 + sum_v x[g^-v] w^(g^(u-v)), a cyclic
        # convolution of length q-1 done with two (q-1)-point transforms.
        q = len(xs)
        g = RADER_G[q]
        m = q - 1
        ginv = pow(g, -1, q)
        a = [xs[pow(ginv, v, q)] for v in range(m)]
        ah = self.dft_above_zero(a)
        x0 = self.add(xs[0], ah[0])
        w = root(q, self.inv)
        bvec = [pow(w, pow(g, t, q), P) for t in range(m)]
        bh = dft_int(bvec, self.inv)  # same direction as the inner transforms
        scale = pow(m, P - 2, P)
        y = [self.mulc(ah[f], bh[f] * scale % P) for f in range(m)]
        y[0] = self.add(y[0], xs[0])
        wh = self.dft_above_zero(y)
        out = [None] * q
        out[0] = x0
        for u in range(m):
            out[pow(g, u, q)] = wh[(-u) % m]
        return out


def dft_int(x, inv=False):
    n = len(x)
    w = root(n, inv)
    return [sum(x[j] * pow(w, j * k % n, P) for j in range(n)) % P for k in range(n)]


SIZES = [2, 3, 4, 5, 6, 8, 10, 12, 15, 16, 17, 32, 60, 64, 68]


def emit(sizes=SIZES):
    out = [
        "// Generated by goldilocks_gb300/codegen.py -- do not edit.",
        "// Straight-line DFT codelets on register-resident values, natural order",
        "// in and out: gl_dft_lazy<R, INV>(x) replaces x[0..R) (any words) by its",
        "// R-point DFT with omega_R = 2717^((p-1)/R) (INV: omega_R^-1, no 1/R",
        "// scaling) as words congruent to it; gl_dft<R, INV> reduces them below p.",
        "#pragma once",
        '#include "gl_field.cuh"',
        "",
        "template <int R, bool INV> struct gl_dft_impl;",
        "template <int R, bool INV> GL_HD void gl_dft_lazy(uint64_t *x) { gl_dft_impl<R, INV>::run(x); }",
        "template <int R, bool INV> GL_HD void gl_dft(uint64_t *x) {",
        "  gl_dft_lazy<R, INV>(x);",
        "  for (int i = 0; i < R; i++) x[i] = gl_canon(x[i]);",
        "}",
        "template <bool INV> struct gl_dft_impl<1, INV> { static GL_HD void run(uint64_t *) {} };",
        "",
    ]
    for r in sizes:
        for inv in (False, True):
            g = Gen(inv)
            ins = [g.word("x[%d]" % i) for i in range(r)]
            res = [g.fold(v) for v in g.dft_above_zero(ins)]
            out.append("template <> struct gl_dft_impl<%d, %s> {" % (r, "true" if inv else "false"))
            out.append(" static GL_HD void run(uint64_t *x) {")
            out.extend(g.lines)
            for i, v in enumerate(res):
                out.append("  x[%d] = %s;" % (i, v.name))
            out.append(" }")
            out.append("};")
            out.append("")
    return "\n".join(out) + "\n"


def main():
    here = os.path.dirname(os.path.abspath(__file__))
    path = os.path.join(here, "csrc", "gl_codelets.cuh")
    text = emit()
    with open(path, "w") as f:
        f.write(text)


if __name__ == "__main__":
    main()
