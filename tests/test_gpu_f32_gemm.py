"""fp32 GEMM on the bf16 tensor cores (nnb200_gemm_f32) at the edges of its tiles and splits, against float64."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g():
    from tests import gpu_util
    return gpu_util


# one element; one tile and one past it (128 rows, 64 or 128 columns, 64 of K); K that splits over 2, 4 and 8 CTAs of a
# cluster, with a last rank that has nothing; rows no 16-byte load can take; several tiles per persistent CTA
SHAPES = [(1, 1, 1), (128, 64, 64), (129, 65, 65), (128, 128, 192), (100, 60, 1000), (384, 128, 1024), (70, 40, 577), (805, 377, 697),
          (3000, 2600, 200)]


@pytest.mark.parametrize("a_mn,b_mn", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gemm_f32_against_float64(g, M, N, K, a_mn, b_mn):
    r = np.random.default_rng(M + N + K)
    A, B = r.standard_normal((M, K)).astype(np.float32), r.standard_normal((N, K)).astype(np.float32)
    c0, bias = r.standard_normal((M, N)).astype(np.float32), r.standard_normal(N).astype(np.float32)
    a, b, bv = g.dev(A.T if a_mn else A), g.dev(B.T if b_mn else B), g.dev(bias)
    scale = np.abs(A.astype(np.float64)) @ np.abs(B.astype(np.float64)).T
    for accumulate in (0, 1):
        c = g.dev(c0)
        g.call("nnb200_gemm_f32", g.ptr(a), g.ptr(b), g.ptr(c), M, N, K, M if a_mn else K, N if b_mn else K, N, a_mn, b_mn, C.c_float(0.5),
               g.ptr(bv), None, accumulate, g.stream())
        want = 0.5 * A.astype(np.float64) @ B.astype(np.float64).T + bias + (c0 if accumulate else 0)
        # dropped products below 2^-24 of |a||b|; at most six steps of the tensor core's sum at full size per 64 of K, each
        # off by 2^-23; one rounding per 64 of K and per split, and three in the epilogue
        bound = 0.5 * scale * (2.0 ** -24 + 6 * 2.0 ** -23 + (K / 64 + 8) * 2.0 ** -24) + 3 * 2.0 ** -23 * (np.abs(want) + np.abs(c0) + 1)
        assert (np.abs(g.host(c) - want) <= bound).all()
    assert g.gemm_status() == 0


def test_gemm_f32_non_finite_and_huge_operands(g):
    """What an infinity, a NaN or a value that bf16 rounds to infinity makes of a result is what fp32 arithmetic makes of it."""
    r = np.random.default_rng(3)
    A, B = r.standard_normal((300, 200)).astype(np.float32), r.standard_normal((150, 200)).astype(np.float32)
    A[5, 3], A[9, 2], B[4, 9], A[7, 1], B[3, 1] = np.inf, np.nan, -np.inf, 3.3e38, 0.0
    a, b, c = g.dev(A), g.dev(B), g.dev(np.zeros((300, 150), np.float32))
    g.call("nnb200_gemm_f32", g.ptr(a), g.ptr(b), g.ptr(c), 300, 150, 200, 200, 200, 150, 0, 0, C.c_float(1.0), None, None, 0, g.stream())
    with np.errstate(all="ignore"):
        want = A.astype(np.float64) @ B.astype(np.float64).T
        want = np.where(np.abs(want) > np.finfo(np.float32).max, np.sign(want) * np.inf, want)
    got = g.host(c)
    rows, cols = np.delete(np.arange(300), 7), np.arange(150)          # row 7 overflows in part: order-dependent, except at B = 0
    assert np.array_equal(np.isnan(got[rows]), np.isnan(want[rows])) and np.array_equal(np.isposinf(got[rows]), np.isposinf(want[rows]))
    fine = np.isfinite(want[rows])
    assert np.abs(got[rows][fine] - want[rows][fine]).max() < 1e-3
    assert abs(got[7, 3] - want[7, 3]) < 1e-3


@pytest.mark.parametrize("dk", [8, 32, 64, 128])
@pytest.mark.parametrize("S", [1, 63, 64, 65, 200])
@pytest.mark.parametrize("docs", [False, True])
def test_attention_f32_tile_edges(g, dk, S, docs):
    """Sequence lengths around the 64-row tiles of the fp32 attention kernels, with documents that close whole tiles: against
    float64 autograd."""
    import torch
    B, H = 2, 3
    d = H * dk
    gen = torch.Generator(device="cuda").manual_seed(S + dk)
    qkv = torch.randn(B * S, 3 * d, device="cuda", generator=gen)
    dout = torch.randn(B * S, d, device="cuda", generator=gen)
    doc = (torch.arange(B * S, device="cuda", dtype=torch.int32) // 50).contiguous() if docs else None
    out, lse, dqkv, dvec = torch.empty_like(dout), torch.empty(B * H * S, device="cuda"), torch.empty_like(qkv), torch.empty(B * H * S, device="cuda")
    g.call("nnb200_attention_forward", g.ptr(qkv), g.ptr(out), g.ptr(lse), g.ptr(doc), None, B, S, H, dk, 1, 0, g.stream())
    g.call("nnb200_attention_backward", g.ptr(qkv), g.ptr(out), g.ptr(dout), g.ptr(lse), g.ptr(dvec), g.ptr(dqkv), g.ptr(doc), None, B, S, H, dk, 1, 0,
           g.stream())
    x = qkv.double().requires_grad_()
    q, k, v = x.view(B, S, 3, H, dk).permute(2, 0, 3, 1, 4)
    i = torch.arange(S, device="cuda")
    slope = torch.exp2(-8.0 * torch.arange(H, device="cuda", dtype=torch.float64) / H)
    s = q @ k.transpose(-1, -2) / dk ** 0.5 - slope[None, :, None, None] * (i[:, None] - i[None, :])
    mask = (i[None, :] <= i[:, None])[None, None]
    if docs:
        mask = mask & (doc.view(B, 1, S, 1) == doc.view(B, 1, 1, S))
    ref = (s.masked_fill(~mask, float("-inf")).softmax(-1) @ v).transpose(1, 2).reshape(B * S, d)
    ref.backward(dout.double())
    # fp32 sums of up to 200 terms and an exponential of arguments up to about 50 (error 50 x 2^-24): 1e-5 of the norm
    assert (out - ref).norm() <= 1e-5 * ref.norm()
    assert (dqkv - x.grad).norm() <= 1e-5 * x.grad.norm()


def _attention(g, qkv, dout, doc, B, S, H, dk, precision):
    import torch
    out, lse, dqkv, dvec = torch.empty_like(dout), torch.empty(B * H * S, device="cuda"), torch.empty_like(qkv), torch.empty(B * H * S, device="cuda")
    g.call("nnb200_attention_forward", g.ptr(qkv), g.ptr(out), g.ptr(lse), g.ptr(doc), None, B, S, H, dk, 0, precision, g.stream())
    g.call("nnb200_attention_backward", g.ptr(qkv), g.ptr(out), g.ptr(dout), g.ptr(lse), g.ptr(dvec), g.ptr(dqkv), g.ptr(doc), None, B, S, H, dk, 0, precision,
           g.stream())
    torch.cuda.synchronize()
    return [t.float().view(B, S, -1, H * dk) for t in (out, dqkv)]


# fp32 at every head size, and the bf16 forms that run the same kernels (small heads, heads of 128 at a ragged length)
@pytest.mark.parametrize("dk,precision", [(8, 0), (32, 0), (64, 0), (128, 0), (8, 1), (16, 1), (128, 1)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_attention_keeps_non_finite_rows_from_queries_that_do_not_see_them(g, dk, precision, value):
    """An infinite or NaN row reaches the positions that attend to it (or that it attends to, in the gradients of keys and
    values) and leaves every other result bit for bit what it is without that row."""
    import torch
    B, H, S, at = 1, 2, 200, 100                                 # `at` in the middle of a 64-row tile
    d = H * dk
    dt = torch.bfloat16 if precision else torch.float32
    gen = torch.Generator(device="cuda").manual_seed(dk)
    qkv = torch.randn(B * S, 3 * d, device="cuda", generator=gen).to(dt)
    dout = torch.randn(B * S, d, device="cuda", generator=gen).to(dt)
    out, dqkv = _attention(g, qkv, dout, None, B, S, H, dk, precision)
    for part in range(4):                                        # a row of q, k, v or dout
        x, y = qkv.clone(), dout.clone()
        if part < 3:
            x[at, part * d:(part + 1) * d] = value
        else:
            y[at] = value
        o, dx = _attention(g, x, y, None, B, S, H, dk, precision)
        before, after = slice(0, at), slice(at + 1, S)
        if part == 3:                                            # no output depends on it
            assert torch.equal(o, out)
        elif part == 0:                                          # its own output
            assert not torch.isfinite(o[:, at]).any()
            assert torch.equal(o[:, before], out[:, before]) and torch.equal(o[:, after], out[:, after])
        else:                                                    # a key or value: the queries from there on
            assert torch.equal(o[:, before], out[:, before])
            if part == 2 or value != value:                      # (an infinite key may score minus infinity)
                assert not torch.isfinite(o[:, after]).any()
        assert torch.equal(dx[:, before, 0], dqkv[:, before, 0])               # dQ of earlier queries
        if part in (0, 3):                                       # a query's row: no later query, no later key or value
            assert torch.equal(dx[:, after], dqkv[:, after])
            assert not torch.isfinite(dx[:, at, 0]).any() and not torch.isfinite(dx[:, before, 1]).any()
    # one document in which every row of everything is broken, between documents that are whole
    doc = (torch.arange(S, device="cuda") // 50).to(torch.int32).contiguous()
    out, dqkv = _attention(g, qkv, dout, doc, B, S, H, dk, precision)
    x, y = qkv.clone(), dout.clone()
    x[50:100], y[50:100] = value, value
    o, dx = _attention(g, x, y, doc, B, S, H, dk, precision)
    whole = torch.cat([torch.arange(50), torch.arange(100, S)]).cuda()
    assert torch.equal(o[:, whole], out[:, whole]) and torch.equal(dx[:, whole], dqkv[:, whole])


@pytest.mark.parametrize("dk", [16, 64])
def test_attention_loses_no_precision_with_the_length_of_the_sequence(g, dk):
    """Every output adds a term per key or query.  In one chain over 2048 of them the error is sqrt(2048 / 64) = 5.7 times that
    over 64 (2.8 to 5 measured, with what the terms bring along); in runs of 8, tiles of 8 runs and a chain over tiles it goes
    with 8 + 8 + n / 64: sqrt(48 / 17) = 1.7 times."""
    import torch
    err = []
    for S in (64, 2048):
        B, H = 2048 // S, 2
        d = H * dk
        gen = torch.Generator(device="cuda").manual_seed(dk)
        qkv, dout = torch.randn(B * S, 3 * d, device="cuda", generator=gen), torch.randn(B * S, d, device="cuda", generator=gen)
        out, dqkv = (t.double().reshape(B * S, -1) for t in _attention(g, qkv, dout, None, B, S, H, dk, 0))
        x = qkv.double().requires_grad_()
        q, k, v = x.view(B, S, 3, H, dk).permute(2, 0, 3, 1, 4)
        s = (q @ k.transpose(-1, -2) / dk ** 0.5).masked_fill(torch.ones(S, S, device="cuda", dtype=torch.bool).triu(1), float("-inf"))
        ref = (s.softmax(-1) @ v).transpose(1, 2).reshape(B * S, d)
        ref.backward(dout.double())
        pairs = [(out, ref.detach())] + [(dqkv[:, c * d:(c + 1) * d], x.grad[:, c * d:(c + 1) * d]) for c in range(3)]
        err.append([float((a - b).norm() / b.norm()) for a, b in pairs])
    assert all(long < 1.8 * short for short, long in zip(*err)), err


# persistent and split forms (K over 2, 4, 8 CTAs), tiles of 64 and 128 columns, edges in M, N and K
@pytest.mark.parametrize("a_mn,b_mn", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K", [(130, 70, 65), (300, 150, 200), (100, 60, 1000), (384, 128, 1024), (805, 377, 697), (3000, 2600, 70)])
def test_gemm_f32_tiles_with_non_finite_results(g, M, N, K, a_mn, b_mn):
    """Rows and columns with infinities and NaNs, or that overflow in bf16 or in the sum, next to finite ones in the same tiles."""
    r = np.random.default_rng(M + N)
    A, B = r.standard_normal((M, K)).astype(np.float32), r.standard_normal((N, K)).astype(np.float32)
    rows, cols = r.choice(M, 6, replace=False), r.choice(N, 3, replace=False)
    A[rows[0], K // 2], A[rows[1], 0], A[rows[2], K - 1] = np.inf, -np.inf, np.nan
    B[cols[0], K // 3], B[cols[1], 1] = np.nan, np.inf
    A[rows[3], 0], B[:, 0] = 3.4e38, np.abs(B[:, 0]) * 1e-30         # beyond bf16, results of 1e8
    A[rows[4]] = np.abs(A[rows[4]]) * 3e37                           # infinite where a column adds up to more than about ten
    c0 = r.standard_normal((M, N)).astype(np.float32)
    a, b, c = g.dev(A.T if a_mn else A), g.dev(B.T if b_mn else B), g.dev(c0)
    g.call("nnb200_gemm_f32", g.ptr(a), g.ptr(b), g.ptr(c), M, N, K, M if a_mn else K, N if b_mn else K, N, a_mn, b_mn, C.c_float(2.0), None, None, 1,
           g.stream())
    got = g.host(c)
    with np.errstate(all="ignore"):
        A64, B64 = A.astype(np.float64), B.astype(np.float64)
        dot = A64 @ B64.T
        scale = np.abs(A64) @ np.abs(B64).T
    fine = np.isfinite(scale) & (scale < 1e38)                       # no fp32 sum overflows whatever its order
    want = 2.0 * dot + c0
    # one FMA chain over K where a result was computed again, else far less
    assert (np.abs(got[fine] - want[fine]) <= (2.0 * scale * K * 2.0 ** -24 + 2.0 ** -22 * (np.abs(want) + np.abs(c0) + 1))[fine]).all()
    special = ~np.isfinite(dot)
    assert np.array_equal(np.isnan(got[special]), np.isnan(dot[special])) and np.array_equal(np.isposinf(got[special]), np.isposinf(dot[special]))
    assert g.gemm_status() == 0


def test_gemm_f32_full_of_nans_is_not_slow(g):
    """A diverged run multiplies matrices full of NaNs, whose results are all computed again: each chain ends at its first NaN (5 times the
    time of a finite product; 150 times with chains that run to their end)."""
    import torch
    M, N, K = 1024, 8192, 384
    a, b, c = (torch.randn(*s, device="cuda") for s in ((M, K), (N, K), (M, N)))
    times = []
    for value in (None, float("nan")):
        if value is not None:
            a.fill_(value)
        for _ in range(3):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            g.call("nnb200_gemm_f32", g.ptr(a), g.ptr(b), g.ptr(c), M, N, K, K, K, N, 0, 0, C.c_float(1.0), None, None, 0, g.stream())
            e1.record()
            torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1))
    assert times[1] < 15 * times[0], times


@pytest.mark.parametrize("M,N,K", [(130, 70, 65), (384, 128, 1024), (3000, 2600, 70)])
@pytest.mark.parametrize("ea,eb", [(-112, 100), (-118, 118), (-126, 120), (-140, 124), (100, -126), (-60, -60), (-120, 0), (40, 40)])
def test_gemm_f32_keeps_the_bits_of_small_operands(g, M, N, K, ea, eb):
    """Operands whose lower bits lie below the smallest bf16 number count in full, as they do in fp32 arithmetic."""
    r = np.random.default_rng(K)
    A = (r.standard_normal((M, K)) * 2.0 ** ea).astype(np.float32)         # subnormal ones hold the bits that fp32 has for them
    B = (r.standard_normal((N, K)) * 2.0 ** eb).astype(np.float32)
    a, b, c = g.dev(A), g.dev(B), g.dev(np.zeros((M, N), np.float32))
    g.call("nnb200_gemm_f32", g.ptr(a), g.ptr(b), g.ptr(c), M, N, K, K, K, N, 0, 0, C.c_float(1.0), None, None, 0, g.stream())
    want = A.astype(np.float64) @ B.astype(np.float64).T
    scale = np.abs(A.astype(np.float64)) @ np.abs(B.astype(np.float64)).T
    # the bound of test_gemm_f32_against_float64, and half the smallest fp32 number for results down there
    bound = scale * (2.0 ** -24 + 6 * 2.0 ** -23 + (K / 64 + 8) * 2.0 ** -24) + 2.0 ** -23 * np.abs(want) + 2.0 ** -149
    assert (np.abs(g.host(c) - want) <= bound).all()
    assert g.gemm_status() == 0
