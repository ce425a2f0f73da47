"""FP64 products on the integer pipes (mulq): a bit-exact model of it agrees with the IEEE product wherever
it takes the product itself; and grids from the size on where the kernels use it (64x32x19 cells, and one
row of cells less, which multiplies) match the oracle bit for bit, with a cross flow of ordinary size, of
zero (whole products of zeros) and of a size whose products underflow."""
import random
import struct

import numpy as np
import pytest

CELLS = ["roCon", "u1Con", "u2Con", "u3Con", "ronCon", "u1nCon", "u2nCon", "u3nCon"]
FACES = [f"{v}{d}" for d in "123" for v in ("p", "u1", "u2", "u3")]
U32 = 0xFFFFFFFF


def bits(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0]


def from_bits(b):
    return struct.unpack("<d", struct.pack("<Q", b))[0]


def mulq_model(a, b):
    """The product's bits by mulq's words, or None where another path takes it."""
    ha, a0, hb, lb = bits(a) >> 32, bits(a) & U32, bits(b) >> 32, bits(b) & U32
    exp, one = 0x7FF00000, 1 << 20
    A = (((ha & 0xFFFFF) | one) << 32) | a0
    B = (((((hb << 11) | (lb >> 21)) & U32) | 0x80000000) << 32) | ((lb << 11) & U32)
    P = A * B
    w = [(P >> (32 * q)) & U32 for q in range(4)]
    s = 1 - (w[3] >> 20)
    P <<= s
    hi, lo, r = (P >> 96) & U32, (P >> 64) & U32, P & ((1 << 64) - 1)
    e = ((ha & exp) + (hb & exp) - 1023 * one - s * one) & U32
    carry = (r + (1 << 63) - 1 + (lo & 1)) >> 64
    low = lo + carry
    top = (hi + e + (low >> 32)) & U32
    if not ((ha ^ (ha << 1)) & (hb ^ (hb << 1)) & 0x40000000 and e < 2044 * one):
        return None
    return ((top | ((ha ^ hb) & 0x80000000)) << 32) | (low & U32)


def test_integer_product_model_matches_ieee_product():
    rng = random.Random(7)
    taken = 0
    for t in range(200000):
        x, y = rng.getrandbits(64), rng.getrandbits(64)
        if t % 4 == 1:  # short significands: ties
            x &= ~((1 << rng.randint(0, 52)) - 1)
            y &= ~((1 << rng.randint(0, 52)) - 1)
        elif t % 4 == 2:  # ordinary sizes, long runs of ones
            x = (x & 0x800FFFFFFFFFFFFF) | (rng.randint(983, 1063) << 52) | (0xFFFFFFFFFFF00 if t % 8 == 2 else 0)
            y = (y & 0x800FFFFFFFFFFFFF) | (rng.randint(983, 1063) << 52)
        elif t % 4 == 3:  # the range's edges
            x = (x & 0x800FFFFFFFFFFFFF) | (rng.choice([0, 1, 511, 512, 513, 1534, 1535, 1536, 2046, 2047]) << 52)
            y = (y & 0x800FFFFFFFFFFFFF) | (rng.choice([0, 1, 511, 512, 513, 1534, 1535, 1536, 2046, 2047]) << 52)
        a, b = from_bits(x), from_bits(y)
        got = mulq_model(a, b)
        if got is not None:
            taken += 1
            with np.errstate(all="ignore"):
                assert got == bits(a * b), (a.hex(), b.hex())
    assert taken >= 50000  # every pair of ordinary sizes


@pytest.mark.gpu
@pytest.mark.parametrize("px,pz", [(1, 1), (0, 0)])
@pytest.mark.parametrize("u3", [1.0, 0.0, 1e-170])
@pytest.mark.parametrize("C", [(64, 32, 19), (64, 31, 19), (33, 35, 37)])
def test_fp64_grids_with_integer_products_match_oracle(ark, port, C, u3, px, pz):
    p = port.channel_params(*C, seed=29)
    st = port.channel_state(p)
    for n in st:
        if n.startswith("u3"):
            st[n] = st[n] * u3
    st["condition"][4, 3, 5] = 1.0
    for n in CELLS:
        if n[0] == "u":
            st[n][4, 3, 5] = 0.0
    gp = ark.make_params(*C, vis=p["nu"], sound=p["sound"], rho0=p["rho0"], cfl=p["cfl"], lx=p["lx"], ly=p["ly"], lz=p["lz"],
                         ub=p["ub"], precision=ark.FP64)
    gp.periodic_x, gp.periodic_z = px, pz
    o = port.Port(p, periodic_x=bool(px), periodic_z=bool(pz))
    o.load(st)
    o.run(3)
    with ark.Context(gp) as c:
        c.upload(st)
        c.step(3)
        c.sync()
        out = c.download(CELLS + FACES)
    for n in CELLS + FACES:
        a, b = port.interior(n, out[n]), port.interior(n, o.get(n))
        assert np.array_equal(np.ascontiguousarray(a).view(np.uint64), np.ascontiguousarray(b).view(np.uint64)), n
