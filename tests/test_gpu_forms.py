"""Sizes and special cases at which the kernels change form, against the oracle (bit-exact):
transform passes, the point operations over groups of lanes, the bit-wise bucket reduction and
the sums of crowded buckets."""
import numpy as np
import pytest

from oracle.oracle import ints_to_limbs, random_field, R
from tests.gpu_common import random_points

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from cusnarks_b200 import Context
    c = Context(0)
    yield c
    c.close()


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()


def _host(t):
    return t.cpu().numpy().view(np.uint32)


# 1..8 one pass, 9.. two; even and odd passes; 15/16 and 17/18: one thread per butterfly or per
# four elements
@pytest.mark.parametrize("L", [1, 2, 3, 4, 7, 8, 9, 10, 11, 13, 14, 15, 17, 18])
def test_ntt_pass_forms(ctx, oracle, L):
    rng = np.random.Generator(np.random.PCG64(300 + L))
    A = oracle.to_mont(random_field(rng, 1 << L, 1), 1)
    roots = oracle.find_roots(L)
    fwd, inv = oracle.ntt(A, roots, L, 1, 1, 1, 1), oracle.intt(A, roots, L, 1, 0, 1)
    for direction, want in ((1, fwd), (-1, inv)):
        d, out = _dev(A), _dev(np.zeros_like(A))
        ctx.ntt_device(d.data_ptr(), out.data_ptr(), L, direction, fmat=0)
        ctx.ntt_device(d.data_ptr(), d.data_ptr(), L, direction, fmat=0)  # in place
        ctx.sync()
        assert np.array_equal(_host(out), want) and np.array_equal(_host(d), want), direction


@pytest.mark.parametrize("L", [8, 9, 11, 12])
@pytest.mark.parametrize("shift", [-1, 1, 100])
def test_ntt_output_partly_over_its_input(ctx, oracle, L, shift):
    rng = np.random.Generator(np.random.PCG64(350 + L))
    n = 1 << L
    A = oracle.to_mont(random_field(rng, n, 1), 1)
    buf = _dev(np.concatenate([np.zeros((100, 8), np.uint32), A, np.zeros((100, 8), np.uint32)]))
    ctx.ntt_device(buf.data_ptr() + 32 * 100, buf.data_ptr() + 32 * (100 + shift), L, 1)
    ctx.sync()
    assert np.array_equal(_host(buf)[100 + shift:100 + shift + n], oracle.ntt(A, oracle.find_roots(L), L, 1, 1, 1, 1))


# 18, 19: two and three blocks a SM
@pytest.mark.parametrize("L", [1, 2, 3, 8, 9, 10, 15, 16, 17, 18, 19])
def test_hstep_forms(ctx, oracle, L):
    rng = np.random.Generator(np.random.PCG64(400 + L))
    m = 1 << L
    A, B, C = (oracle.to_mont(random_field(rng, m, 1), 1) for _ in range(3))
    dA, dB, dC = _dev(A), _dev(B), _dev(C)
    both = _dev(np.concatenate([A, B]))  # the output over its own inputs
    row = _dev(np.concatenate([B, A, np.zeros((2 * m, 8), np.uint32), C, B]))  # next to them
    M, H = _dev(np.zeros((2 * m, 8), np.uint32)), _dev(np.zeros((m, 8), np.uint32))
    ctx.hstep_device(0, dA.data_ptr(), dB.data_ptr(), 0, L, M.data_ptr())
    ctx.hstep_device(1, dA.data_ptr(), dB.data_ptr(), dC.data_ptr(), L, H.data_ptr())
    ctx.hstep_device(0, both.data_ptr(), both.data_ptr() + 32 * m, 0, L, both.data_ptr())
    at = lambda k: row.data_ptr() + 32 * m * k  # noqa: E731
    ctx.hstep_device(0, at(1), at(0), 0, L, at(2))
    ctx.sync()
    side = _host(row)[2 * m:4 * m].copy()
    ctx.hstep_device(1, at(1), at(0), at(4), L, at(3))
    ctx.sync()
    want = oracle.interpolandmul(A, B, oracle.find_roots(L + 1), L, 2)
    assert np.array_equal(_host(M), want) and np.array_equal(_host(both), want)
    assert np.array_equal(side, want) and np.array_equal(_host(row)[3 * m:4 * m], oracle.hstep_coset(A, B, C, L))
    assert np.array_equal(_host(H), oracle.hstep_coset(A, B, C, L))
    assert np.array_equal(_host(dA), A) and np.array_equal(_host(dB), B)


def _fixed(ctx, s, pts, c, ec2):
    dp, ds, out = _dev(pts), _dev(s), _dev(np.zeros(32 if ec2 else 16, np.uint32))
    table = _dev(np.zeros(ctx.msm_fixed_table_points(len(s), c) * (32 if ec2 else 16), np.uint32))
    ctx.msm_fixed_table_device(dp.data_ptr(), len(s), c, table.data_ptr(), ec2=ec2)
    ctx.msm_fixed_device(ds.data_ptr(), table.data_ptr(), len(s), c, out.data_ptr(), ec2=ec2)
    ctx.sync()
    return _host(out)


# bucket counts of one to three stages of the bit tree, with and without levels of eight before it
@pytest.mark.parametrize("ec2,c", [(False, 4), (False, 5), (False, 7), (False, 8), (False, 13), (False, 14), (False, 19),
                                   (False, 20), (True, 4), (True, 7), (True, 8), (True, 13), (True, 17), (True, 18)])
def test_reduction_by_bits(ctx, oracle, ec2, c):
    rng = np.random.Generator(np.random.PCG64(500 + c))
    pts = random_points(oracle, rng, 150, ec2=ec2)
    s = random_field(rng, 150, 1)
    want = oracle.msm(s, pts, ec2=int(ec2))
    assert np.array_equal(_fixed(ctx, s, pts, c, ec2), want)
    if c <= 17:
        assert np.array_equal(ctx.msm(s, pts, ec2=ec2, window=c), want)


@pytest.mark.parametrize("ec2", [False, True])
@pytest.mark.parametrize("window", [0, 4, 8])
def test_equal_and_opposite_sums(ctx, oracle, ec2, window):
    """One point throughout: every addition of two buckets, partial sums or windows meets equal
    or opposite points or infinity."""
    rng = np.random.Generator(np.random.PCG64(600))
    n = 128
    one = random_points(oracle, rng, 1, ec2=ec2)
    pts = np.repeat(one, n, axis=0)
    runs = [list(range(1, n + 1)), [1] * n, [R - 1, 1] * (n // 2), [2, R - 2, 4, R - 4] * (n // 4),
            [1 << (k % 253) for k in range(n)], [0] * n, [R - 1] * n]
    for ks in runs:
        s = ints_to_limbs(ks)
        want = oracle.msm(s, pts, ec2=int(ec2))
        assert np.array_equal(ctx.msm(s, pts, ec2=ec2, window=window), want), ks[:4]
        assert np.array_equal(_fixed(ctx, s, pts, window or 6, ec2), want), ks[:4]


# partial sums of one bucket: within one pass (8), one more, a warp's worth, thousands
@pytest.mark.parametrize("ec2,n", [(False, 127), (False, 130), (False, 260), (False, 2000), (False, 40000), (True, 130),
                                   (True, 300), (True, 6000)])
def test_crowded_bucket(ctx, oracle, ec2, n):
    rng = np.random.Generator(np.random.PCG64(700 + n))
    pts = random_points(oracle, rng, n, ec2=ec2)
    s = np.zeros((n, 8), np.uint32)
    s[:, 0] = 1
    s[::7, 0] = 3
    s[-3:] = random_field(rng, 3, 1)
    want = oracle.msm(s, pts, ec2=int(ec2))
    assert np.array_equal(ctx.msm(s, pts, ec2=ec2), want)
    assert np.array_equal(_fixed(ctx, s, pts, ctx.msm_fixed_window(n, ec2), ec2), want)


@pytest.mark.parametrize("pidx", [0, 1])
def test_inverse_edges(ctx, oracle, pidx):
    from oracle.oracle import limbs_to_int, Q
    p = R if pidx else Q
    vals = [0, 1, 2, 3, p - 1, p - 2, (p + 1) // 2] + [1 << k for k in (29, 30, 31, 32, 61, 62, 63, 64, 200, 252)]
    vals += [p - (1 << k) for k in (30, 62, 128, 250)]
    rng = np.random.Generator(np.random.PCG64(800 + pidx))
    vals += [limbs_to_int(x) % p for x in random_field(rng, 500, 1)]
    a = ints_to_limbs(vals)  # Montgomery form of vals / 2^256
    d, out = _dev(a), _dev(np.zeros_like(a))
    ctx.field_op_device("inv", pidx, d.data_ptr(), 0, out.data_ptr(), len(vals))
    ctx.sync()
    mont = 1 << 256
    want = [pow(v, -1, p) * mont * mont % p if v else 0 for v in vals]
    assert np.array_equal(_host(out), ints_to_limbs(want))
