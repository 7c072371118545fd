"""Writes mt_jump.inc: jump polynomials of the Mersenne twister MT19937.

The twister's state (19,937 bits: the top bit of word 0 and words 1..623) moves
by a linear map over GF(2) with characteristic polynomial p, so the state N
words on is sum_i g_i state_i with g(x) = x^N mod p(x) (Haramoto, Matsumoto,
Nishimura, Panneton, L'Ecuyer, "Efficient jump ahead for F2-linear random number
generators", INFORMS J. Comput. 20, 2008).  p comes from the generator's own
output by the Berlekamp-Massey algorithm.  The file holds g for N = s * JUMP,
s = 1 .. SEGMENTS - 1, 624 32-bit words each (bit i of the polynomial is bit
i % 32 of word i // 32).  The polynomials are checked on another seed before they
are written.

    python -m ccpp_physics_b200.data.make_mt_jump
"""
import os

STATE, JUMP, SEGMENTS = 624, 33 * 624, 16


def words(seed, n):
    """x_0 .. x_{n-1}: the seeding mt(i) = 69069^i seed, then the recurrence."""
    x = [seed & 0xffffffff]
    for _ in range(1, STATE):
        x.append(x[-1] * 69069 & 0xffffffff)
    for i in range(n - STATE):
        y = (x[i] & 0x80000000) | (x[i + 1] & 0x7fffffff)
        x.append(x[i + 397] ^ (y >> 1) ^ (0x9908B0DF if y & 1 else 0))
    return x


def characteristic(bits):
    """Berlekamp-Massey: p(x) with bit k = the coefficient of x^k."""
    c, b, length, gap, past = 1, 1, 0, 1, 0
    for n, s in enumerate(bits):
        past = (past << 1) | s
        if (c & past).bit_count() & 1 == 0:
            gap += 1
        elif 2 * length <= n:
            c, b, length, gap = c ^ (b << gap), c, n + 1 - length, 1
        else:
            c ^= b << gap
            gap += 1
    return int(bin(c)[2:].zfill(length + 1)[::-1], 2)


def mulmod(a, b, p):
    d = p.bit_length() - 1
    r = 0
    for i in range(b.bit_length()):
        if b >> i & 1:
            r ^= a << i
    while r.bit_length() > d:
        r ^= p << (r.bit_length() - 1 - d)
    return r


def main():
    p = characteristic([w & 1 for w in words(4357, 2 * 19937 + 64)[1:]])
    assert p.bit_length() == 19938
    step = 1
    for bit in bin(JUMP)[2:]:   # x^JUMP mod p
        step = mulmod(step, step, p)
        if bit == "1":
            step = mulmod(step, 2, p)
    polys, g = [], 1
    for _ in range(1, SEGMENTS):
        g = mulmod(g, step, p)
        polys.append(g)
    x = words(12345, SEGMENTS * JUMP + STATE)
    for s, g in enumerate(polys, 1):
        for j in (0, 1, 300, 623):
            v = 0
            for i in range(19937):
                if g >> i & 1:
                    v ^= x[i + j]
            keep = 0x80000000 if j == 0 else 0xffffffff
            assert (v ^ x[s * JUMP + j]) & keep == 0, (s, j)
    path = os.path.join(os.path.dirname(os.path.abspath(__file__)), "mt_jump.inc")
    with open(path, "w") as f:
        f.write("// x^(s * %d) mod p, s = 1 .. %d (make_mt_jump.py)\n" % (JUMP, SEGMENTS - 1))
        for g in polys:
            for k in range(0, STATE, 8):
                f.write(" ".join("0x%08xu," % (g >> 32 * (k + q) & 0xffffffff) for q in range(8)) + "\n")


if __name__ == "__main__":
    main()
