"""Constants of csrc/kpmath.cuh, computed in 60 digits: prints the table and coefficient blocks of that header, which
tests/test_sampler_math.py compares with what it holds."""
import struct

import mpmath as mp

mp.mp.dps = 60
GRID = mp.mpf(2) ** -47   # the high parts of the logarithms are multiples of this


def high_word(x):
    """x rounded to what a double's high word holds (20 bits behind the leading one)."""
    if x == 0:
        return 0
    bits = struct.unpack("<Q", struct.pack("<d", float(x)))[0]
    return (bits + (1 << 31)) >> 32


def split(x):
    """x as a multiple of GRID and the high word of the rest."""
    hi = mp.nint(x / GRID) * GRID
    return float(hi), high_word(x - hi)


def log_table():
    rows = []
    for j in range(128):
        # the number of 18 fractional bits (19 from j = 48 on, where it is below 3/4) next to one over the interval's middle
        f = 2 ** (18 if j < 48 else 19)
        c = mp.mpf("0.5") if j == 127 else mp.nint(f / (1 + (2 * mp.mpf(j) + 1) / 256)) / f
        assert max(abs(c * (1 + mp.mpf(j + i) / 128) - 1) for i in (0, 1)) <= mp.mpf(2) ** -8
        hi, lo = split(-mp.log(c))
        word = struct.unpack("<Q", struct.pack("<d", float(c)))[0]
        assert word & 0xffffffff == 0
        rows.append((hi, struct.unpack("<d", struct.pack("<Q", word | lo))[0]))
    return rows


def rest(f, f0):
    """(f(sqrt z) - f0) / z, from its series at 0."""
    return lambda z: (f(mp.sqrt(z)) - f0) / z if z > mp.mpf(10) ** -12 else (f(mp.mpf(10) ** -6) - f0) / mp.mpf(10) ** -12


def fit(f, b, n):
    return [float(x) for x in mp.chebyfit(f, [mp.mpf(0), b], n)]


def block(name, values):
    text = ",\n    ".join(", ".join(v.hex() for v in values[i:i + 4]) for i in range(0, len(values), 4))
    return "static __constant__ const double %s[%d] = {\n    %s};" % (name, len(values), text)


def low(x):
    return [float(x), float(x - mp.mpf(float(x)))]


def blocks():
    rows = log_table()
    table = "\n".join("    " + " ".join("{%s, %s}," % (a.hex(), b.hex()) for a, b in rows[i:i + 2]) for i in range(0, 128, 2))
    hi, lo = split(mp.log(2))
    lo = struct.unpack("<d", struct.pack("<Q", lo << 32))[0]
    return ["static __device__ const double2 kKpLog[128] = {\n%s\n};" % table,
            block("kKpSin2Pi", fit(rest(lambda y: mp.sin(2 * mp.pi * y) / y, 2 * mp.pi), mp.mpf(1) / 64, 6)),
            block("kKpCos2Pi", fit(rest(lambda y: mp.cos(2 * mp.pi * y), mp.mpf(1)), mp.mpf(1) / 64, 7)),
            block("kKp2Pi", low(2 * mp.pi)),
            block("kKpLn2", [hi, lo])]


if __name__ == "__main__":
    print("\n".join(blocks()))
