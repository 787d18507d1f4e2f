"""Vector and one-launch forms of the surrogate kernels at the sizes where they
can go wrong: GEMM epilogues with whole, cut and unaligned 32-column groups,
split-K sums around the sixteen slabs in flight, the two lowerings against
the oracle at strides and taps on both sides of their rules, the activation's
reverse pass with cut and unaligned rows, Adam over many
tensors of ragged sizes and alignments."""
import numpy as np
import pytest

from photonfdtd_b200 import _native as N
from oracle.surrogate_ref import bf16, col2im, im2col

pytestmark = pytest.mark.gpu


def _t():
    import torch
    return torch


def _p(x):
    return x.data_ptr()


def _chk(rc):
    assert rc == N.PF_OK, N.lib().pfs_last_error().decode()


def _s():
    return _t().cuda.current_stream().cuda_stream


def _ints(rng, shape):
    """Small integers: exact in BF16, and their products and sums in FP32."""
    return rng.integers(-4, 5, shape).astype(np.float32)


@pytest.mark.parametrize("M,n,ldc,off", [(1, 1, 1, 0), (129, 32, 32, 0), (130, 33, 36, 0),
                                         (257, 288, 288, 0), (128, 64, 65, 0), (200, 96, 96, 1),
                                         (127, 31, 32, 0)])
@pytest.mark.parametrize("beta", [0.0, 2.0])
def test_gemm_epilogue_columns(M, n, ldc, off, beta):
    t = _t()
    rng = np.random.default_rng(M + n)
    K = 64
    A, B, C0 = _ints(rng, (M, K)), _ints(rng, (n, K)), _ints(rng, (M, ldc))
    a, b = (t.from_numpy(x).cuda().bfloat16() for x in (A, B))
    buf = t.full((M * ldc + 8,), 7.0, device="cuda")
    c = buf[off:off + M * ldc].view(M, ldc)
    c.copy_(t.from_numpy(C0))
    _chk(N.lib().pfs_gemm_bf16(M, n, K, _p(a), K, _p(b), K, _p(c), ldc, 1.0, beta, _s()))
    want = C0.copy()
    want[:, :n] = A @ B.T + beta * C0[:, :n]
    assert np.array_equal(c.cpu().numpy(), want)
    rest = buf.cpu().numpy()
    assert (rest[:off] == 7).all() and (rest[off + M * ldc:] == 7).all()


@pytest.mark.parametrize("n,ldy", [(32, 32), (40, 40), (64, 66)])
def test_gemm_bias_act_columns(n, ldy):
    t = _t()
    rng = np.random.default_rng(n)
    M, K = 131, 32
    A, B, bias = _ints(rng, (M, K)), _ints(rng, (n, K)), _ints(rng, n)
    a, b = (t.from_numpy(x).cuda().bfloat16() for x in (A, B))
    db = t.from_numpy(bias).cuda()
    y = t.full((M, ldy), -1.0, device="cuda")
    h = t.full((M, ldy), -1.0, device="cuda", dtype=t.bfloat16)
    _chk(N.lib().pfs_gemm_bf16_bias_act(M, n, K, _p(a), K, _p(b), K, _p(db), 1, _p(y), _p(h), ldy,
                                        _s()))
    want = np.full((M, ldy), -1.0, np.float32)
    want[:, :n] = np.maximum(A @ B.T + bias, 0)
    assert np.array_equal(y.cpu().numpy(), want)
    assert np.array_equal(h.float().cpu().numpy(), bf16(want).astype(np.float32))


@pytest.mark.parametrize("splits", [2, 8, 15, 16, 17, 127, 128, 129, 293])
@pytest.mark.parametrize("M,n", [(32, 32), (33, 45)])
def test_split_k_sum(M, n, splits):
    t = _t()
    rng = np.random.default_rng(splits)
    K = 64 * splits
    A, B = _ints(rng, (M, K)), _ints(rng, (n, K))
    a, b = (t.from_numpy(x).cuda().bfloat16() for x in (A, B))
    c = t.full((M, n), 3.0, device="cuda")
    work = t.zeros(splits * M * n, device="cuda")
    _chk(N.lib().pfs_gemm_bf16_splitk(M, n, K, _p(a), K, _p(b), K, _p(c), n, 1.0, 1.0, splits,
                                      _p(work), work.numel(), _s()))
    assert np.array_equal(c.cpu().numpy(), A @ B.T + 3.0)


@pytest.mark.parametrize("C,kh,kw,stride,ph,pw", [(1, 3, 3, 1, 1, 1), (3, 3, 3, 2, 1, 1),
                                                  (5, 1, 3, 1, 0, 1), (8, 3, 3, 1, 1, 1),
                                                  (8, 3, 3, 2, 1, 1), (16, 4, 4, 2, 1, 1),
                                                  (8, 5, 5, 2, 2, 2), (8, 2, 2, 3, 0, 0),
                                                  (8, 3, 1, 2, 2, 0)])
@pytest.mark.parametrize("H,W", [(9, 7), (6, 8)])
def test_lowerings_match_oracle(H, W, C, kh, kw, stride, ph, pw):
    t = _t()
    rng = np.random.default_rng(C * 100 + kh * 10 + stride)
    nb, K = 2, kh * kw * C
    Kp = (K + 31) // 32 * 32
    Ho, Wo = (H + 2 * ph - kh) // stride + 1, (W + 2 * pw - kw) // stride + 1
    x = _ints(rng, (nb, H, W, C))
    dx16 = t.from_numpy(x).cuda().bfloat16()
    col = t.full((nb * Ho * Wo, Kp), 9.0, device="cuda", dtype=t.bfloat16)
    args = (nb, H, W, C, kh, kw, stride, ph, pw)
    _chk(N.lib().pfs_im2col(*args, _p(dx16), _p(col), Kp, _s()))
    got = col.float().cpu().numpy()
    want = im2col(x, kh, kw, stride, ph, pw)[0]
    assert np.array_equal(got[:, :K], want) and not got[:, K:].any()
    d = np.zeros((nb * Ho * Wo, Kp), np.float32)
    d[:, :K] = _ints(rng, (nb * Ho * Wo, K))
    dcol = t.from_numpy(d).cuda()
    out = t.full((nb, H, W, C), 9.0, device="cuda")
    _chk(N.lib().pfs_col2im(*args, _p(dcol), Kp, _p(out), _s()))
    want = col2im(d[:, :K], x.shape, kh, kw, stride, ph, pw)
    assert np.array_equal(out.cpu().numpy(), want.reshape(x.shape))


@pytest.mark.parametrize("M,n,rb,off", [(1, 4, 1, 0), (63, 32, 1, 0), (65, 36, 3, 0),
                                        (200, 64, 7, 0), (130, 33, 2, 0), (130, 32, 2, 1),
                                        (10, 32, 16, 0)])
@pytest.mark.parametrize("relu", [0, 1])
def test_act_bwd_vectors(M, n, rb, off, relu):
    t = _t()
    rng = np.random.default_rng(M + n)
    dy, y = _ints(rng, (M, n)), _ints(rng, (M, n))
    y[0, 0] = np.nan
    buf = t.zeros(M * n + 4, device="cuda")
    d = buf[off:off + M * n].view(M, n)
    d.copy_(t.from_numpy(dy))
    dyv = t.from_numpy(y).cuda()
    d32 = t.full((M, n), 9.0, device="cuda")
    d16 = t.full((M, n), 9.0, device="cuda", dtype=t.bfloat16)
    gb, part = t.zeros(n, device="cuda"), t.zeros(rb * n, device="cuda")
    _chk(N.lib().pfs_act_bwd(M, n, _p(d), _p(dyv), relu, _p(d32), _p(d16), _p(gb), _p(part), rb,
                             _s()))
    want = np.where(y > 0, dy, 0) if relu else dy
    assert np.array_equal(d32.cpu().numpy(), want)
    assert np.array_equal(d16.float().cpu().numpy(), want)
    assert np.array_equal(gb.cpu().numpy(), want.sum(0))


def test_adam_many_ragged():
    """The tensors of one launch (33: two launches) give the bits of one call
    each, aligned or not, with and without a BF16 copy."""
    t = _t()
    rng = np.random.default_rng(5)
    sizes = [1, 2, 3, 4, 5, 31, 32, 1023, 1024, 1025, 4096] * 3
    base = [[t.from_numpy(np.abs(rng.standard_normal(n + 1)).astype(np.float32)).cuda()
             for _ in range(4)] for n in sizes]

    def views(i, off):
        return [x.clone()[off:off + sizes[i]] for x in base[i]]
    many, one, h1, h2, tab = [], [], [], [], []
    for i, n in enumerate(sizes):
        off = i % 2
        many.append(views(i, off))
        one.append(views(i, off))
        h1.append(t.zeros(n, device="cuda", dtype=t.bfloat16))
        h2.append(t.zeros(n, device="cuda", dtype=t.bfloat16))
        w, g, m, v = many[i]
        tab.append((n, _p(w), _p(g), _p(m), _p(v), _p(h1[i]) if i % 3 else 0, 0.1 * (i % 2)))
    hyper = (1e-2, 0.9, 0.999, 1e-8)
    _chk(N.lib().pfs_adam_many(len(tab), (N.AdamTensor * len(tab))(*tab), *hyper, 3, _s()))
    for i, n in enumerate(sizes):
        w, g, m, v = one[i]
        _chk(N.lib().pfs_adam(n, _p(w), _p(g), _p(m), _p(v), *hyper, 3, 0.1 * (i % 2),
                              _p(h2[i]) if i % 3 else 0, _s()))
        g64, m0, v0 = (x[i % 2:i % 2 + n].double() for x in base[i][1:])
        w0 = base[i][0][i % 2:i % 2 + n].double()
        m1, v1 = 0.9 * m0 + 0.1 * g64, 0.999 * v0 + 0.001 * g64 * g64
        want = w0 - 1e-2 * (m1 / (1 - 0.9 ** 3) / ((v1 / (1 - 0.999 ** 3)).sqrt() + 1e-8)
                            + 0.1 * (i % 2) * w0)
        assert t.allclose(many[i][0].double(), want, rtol=1e-5, atol=1e-6)
        assert all(t.equal(a, b) for a, b in zip(many[i], one[i])) and t.equal(h1[i], h2[i])
