"""The short square root and reciprocals of the element kernels where they are
hardest to round: bit for bit the IEEE values (the host's)."""
import ctypes as C

import numpy as np
import pytest

from snac_b200.context import load_library

pytestmark = pytest.mark.gpu

_DP = C.POINTER(C.c_double)

# Significands b (53 bits) for which b m = 2^k + j with a 54-bit odd m and |j| <= 8
# (times the powers of two in b): 1/b lies that near to the midpoint m between two
# doubles.  They are the divisors of these sizes of 2^k + j.
RECIPROCALS = [
    0x1014ca35e947b6, 0x1024a3bd98da02, 0x10699d36aec84e, 0x109107683ee29e, 0x10aadc6f562fdc, 0x10af911aa26396,
    0x10d03f8a57cc76, 0x10ed85c351e224, 0x110af85de838ce, 0x110d10000221a2, 0x1125e52b034982, 0x115efb8b10aa42,
    0x11d3799c32581e, 0x11f98ea5d9b262, 0x120a8f5bbf2106, 0x12af4d6bc06922, 0x12bf5907e316d2, 0x12d2d2d2d2d2d4,
    0x12e3c6a0509ca4, 0x12e93952a2ed6e, 0x130a0dd90e13a2, 0x132160ccc0848c, 0x134d8fe343ef42, 0x13541c0067f83c,
    0x1379cb88f092f2, 0x13a324a526d5ee, 0x13a7a1d01d1ec2, 0x13d75d54b37492, 0x1403e897077b16, 0x14873ecade304c,
    0x14a6fb45f5d782, 0x14cad5a5fa03ee, 0x15555555555554, 0x155f2490c86132, 0x156a8cb0234262, 0x159aa11aaecb86,
    0x16026c81a85766, 0x163baaac17d1e2, 0x163dd0554d0122, 0x16d6422e5cf246, 0x16f0f27bf434d6, 0x16fae7ba173812,
    0x172f10bf899124, 0x17641c46f799ee, 0x178cb7d5d6e322, 0x178d42e524dcdc, 0x17f52093014f0e, 0x1806c89fcb9452,
    0x181efe51ead722, 0x18401cbcdb5596, 0x184a12efef626e, 0x194ab05a4ecedc, 0x194c4511fa3124, 0x1960a45d1a71e6,
    0x199d2b42ffe9f4, 0x199e1b447e99c2, 0x19f142d24e1352, 0x1a0b8ffffcbe8e, 0x1a149bad85de72, 0x1a2ce4d7478a06,
    0x1a6f41dab98cb2, 0x1aa7c88ee59082, 0x1ae6849e786ad2, 0x1b227794e85702, 0x1bea3278b789d2, 0x1c2693dcf34742,
    0x1c36899addce3c, 0x1c384d119331c4, 0x1c4d3aabd478f6, 0x1c69bf28eba166, 0x1c928b5b9dc714, 0x1d5b9032f086be,
    0x1da210daeb138e, 0x1de441d5331432, 0x1de4a0d00fa9b2, 0x1e20adbc4078a2, 0x1e756f08df1792, 0x1e8d517d09c5c2,
    0x1e9a9473949bf6, 0x1ef7930608393e, 0x1f65fad23b0d86, 0x1f739bd459bea2, 0x1fe24bffeb8794, 0x1ffb8a8b628dbc,
    0x1ffffff8000001, 0x1fffffffffffff,
]


def near_midpoint_squares():
    """(Q, e): Q 2^e + j = m^2 for an odd 54-bit m, |j| < 512: the root of Q 2^e is
    that near to the midpoint m between two doubles."""
    for e in (54, 55):
        for j in range(-511, 512):
            if j % 8 != 1:
                continue  # no odd square is anything else modulo 8
            roots = [x for x in (1, 3, 5, 7) if (x * x - j) % 8 == 0]
            for k in range(3, e):
                roots = {y % (1 << (k + 1)) for x in roots for y in (x, x + (1 << (k - 1)), x + (1 << k))
                         if (y * y - j) % (1 << (k + 1)) == 0}
            for m in roots:
                if (1 << 53) <= m < (1 << 54) and (1 << 52) <= (m * m - j) >> e < (1 << 53):
                    yield (m * m - j) >> e, e


def device(q):
    f = load_library().snac_gpu_selftest_roots
    f.argtypes = [_DP, C.c_longlong, _DP, _DP, _DP]
    f.restype = C.c_int
    q = np.ascontiguousarray(q)
    out = [np.zeros_like(q) for _ in range(3)]
    assert f(q.ctypes.data_as(_DP), q.size, *(o.ctypes.data_as(_DP) for o in out)) == 0
    return out


def low_word_all_ones(x):
    return (x.view(np.uint64) & 0xFFFFFFFF) == 0xFFFFFFFF


def test_roots_nearest_to_a_midpoint():
    hard = sorted(set(near_midpoint_squares()))
    assert len(hard) > 150
    q = np.array([np.ldexp(float(Q), (e & 1) + 2 * k) for Q, e in hard for k in range(-380, 177, 13)])
    assert q.min() >= 2.0 ** -714 and q.max() < 2.0 ** 408
    root, recip_root, _ = device(q)
    assert np.array_equal(root, np.sqrt(q))
    keep = ~low_word_all_ones(root)
    assert np.array_equal(recip_root[keep], 1.0 / root[keep])


def test_reciprocals_nearest_to_a_midpoint():
    s = np.array([np.ldexp(float(b), k) for b in RECIPROCALS for k in range(-404, 150, 11)])
    # every q whose root rounds to s
    q = s * s
    q = np.concatenate([(q.view(np.int64) + d).view(np.float64) for d in range(-3, 4)])
    q = q[np.isin(np.sqrt(q), s)]
    assert q.size > 2 * s.size
    root, recip_root, _ = device(q)
    assert np.array_equal(root, np.sqrt(q))
    keep = ~low_word_all_ones(root)
    assert np.count_nonzero(~keep) > 0  # the all-ones significand, which the callers turn away
    assert np.array_equal(recip_root[keep], 1.0 / root[keep])
    y = np.array([np.ldexp(float(b), k) for b in RECIPROCALS for k in range(-52, 12)])
    y = y[~low_word_all_ones(y)]
    assert np.array_equal(device(y)[2], 1.0 / y)


def test_random_operands():
    rng = np.random.default_rng(17)
    q = np.ldexp(1.0 + rng.random(1 << 22), rng.integers(-714, 408, 1 << 22))
    root, recip_root, _ = device(q)
    assert np.array_equal(root, np.sqrt(q))
    keep = ~low_word_all_ones(root)
    assert np.array_equal(recip_root[keep], 1.0 / root[keep])
