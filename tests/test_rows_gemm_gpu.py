"""Projections of 1-64 rows with norm, residual add and SwiGLU inside (q_gemm_rows_*), against the
same rounding points in plain torch: fp64 products, everything else as the oracle rounds it."""
import ctypes as C

import pytest
import torch

from starter_b200 import _lib, ops
from starter_b200._lib import check, lib

pytestmark = pytest.mark.gpu
EPS = 1e-6
# fp32 sums of up to 9728 products against fp64: 2^-24 per addition; a bf16 rounding that falls the
# other way is one ulp, up to 2^-7 of the value (8 significant bits).
ERR_ARG = -1          # q_status Q_ERR_ARG
F32_RTOL, BF16_ULP = 2e-5, 2.0 ** -7


def _p(t):
    return C.c_void_p(t.data_ptr())


def _bf16(shape, seed, scale=1.0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, scale, generator=gen)


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _rms(x, ss, gain):
    inv = torch.rsqrt(ss / x.shape[1] + EPS)
    return ((x.float() * inv[:, None]).bfloat16().float() * gain.float()).bfloat16()


def _parts(x, parts):
    """Sums of squares of the rows of x, cut into `parts` unequal parts [parts][rows]."""
    out = torch.zeros((parts, x.shape[0]), device="cuda")
    out[0] = x.float().pow(2).sum(1)
    for p in range(1, parts):
        out[p] = out[0] / (4 * parts)
        out[0] -= out[p]
    return out


def _close_add(got, want, branch):
    """Where fp32 and fp64 sums round to different bf16 values the branch moves by one ulp of ITS size (the
    total may be much smaller), and the total then rounds once more; that happens to few elements. (1e-4: what
    fp32 sums of K products of order 0.05 are off by where the branch is near zero.)"""
    got, want = got.float(), want.float()
    diff = (got - want).abs()
    assert bool((diff <= BF16_ULP * (branch.abs() + want.abs()) + 1e-4).all())
    assert float((diff > 0).float().mean()) < 0.02


# rows at the edges of the 8-row slices, the 16-row warps and the clusters' row runs; widths of one atom,
# of runs that cross a 128-row block, and the benchmark's
ROWS = [1, 3, 8, 9, 16, 17, 33, 64]


@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("N,K", [(8, 64), (1032, 128), (6144, 2560)])
@pytest.mark.parametrize("norm", [False, True])
def test_f32(rows, N, K, norm):
    x, w, gain = _bf16((rows, K), 1), _bf16((N, K), 2, 0.05), _bf16((K,), 3)
    ss = _parts(x, 37)
    out = torch.full((rows, N), float("nan"), device="cuda")
    tc = ops.pack_weight_tc(w)
    check(lib.q_gemm_rows_f32(_p(x), _p(gain) if norm else None, _p(ss), 37, _p(tc), _p(out), rows, N, K, EPS, _stream()))
    a = _rms(x, ss.sum(0), gain) if norm else x
    want = a.double() @ w.double().T
    err = (out.double() - want).norm() / want.norm()
    # (a normalised value that rounds the other way, because rsqrt or the sum differs by an ulp: 2^-9 of a product)
    assert float(err) < (5e-4 if norm else F32_RTOL)
    assert ops.device_status() == [0, 0, 0, 0]


@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("N,K", [(8, 64), (136, 192), (2560, 4096), (2560, 9728)])
def test_add(rows, N, K):
    x, w, resid = _bf16((rows, K), 1), _bf16((N, K), 2, 0.05), _bf16((rows, N), 3)
    parts = lib.q_gemm_rows_parts(rows, N, K)
    assert parts >= 1
    ss = torch.full((parts, rows), float("nan"), device="cuda")
    got = resid.clone()
    check(lib.q_gemm_rows_add(_p(x), _p(ops.pack_weight_tc(w)), _p(got), _p(ss), rows, N, K, _stream()))
    branch = (x.double() @ w.double().T).bfloat16().float()
    _close_add(got, (resid.float() + branch).bfloat16(), branch)
    assert torch.allclose(ss.sum(0), got.float().pow(2).sum(1), rtol=1e-5)
    assert ops.device_status() == [0, 0, 0, 0]


@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("inter,K", [(8, 64), (264, 128), (9728, 2560)])
def test_swiglu(rows, inter, K):
    x, w, gain = _bf16((rows, K), 1), _bf16((2 * inter, K), 2, 0.05), _bf16((K,), 3)
    ss = _parts(x, 36)
    act = torch.full((rows, inter), float("nan"), dtype=torch.bfloat16, device="cuda")
    check(lib.q_gemm_rows_swiglu(_p(x), _p(gain), _p(ss), 36, _p(ops.pack_weight_tc(w)), _p(act), rows, inter, K, EPS,
                                 _stream()))
    y = (_rms(x, ss.sum(0), gain).double() @ w.double().T).bfloat16().float()
    g, u = y[:, :inter], y[:, inter:]
    want = (torch.nn.functional.silu(g).bfloat16().float() * u).bfloat16()
    # the norm's flipped roundings move the sums as in test_f32: 2-norm, and no element far off
    err = (act.float() - want.float()).norm() / want.float().norm()
    assert float(err) < 4e-3
    assert float((act.float() - want.float()).abs().max()) < 0.05 * float(want.float().abs().max())
    assert ops.device_status() == [0, 0, 0, 0]


# K of 14, 41, 172 and 173 tiles of 64: clusters whose CTAs have different, odd and even, numbers of k tiles, with rows
# that leave the last CTAs of a cluster none to finish.
@pytest.mark.parametrize("rows", [1, 9, 17, 33, 64])
@pytest.mark.parametrize("N,K", [(896, 896), (2048, 2624), (4096, 2624), (896, 11008), (2560, 11072)])
def test_uneven_splits(rows, N, K):
    splits = [lib.q_gemm_rows_splits(rows, N, K, add) for add in (0, 1)]
    assert all(s > 1 and (K // 64) % s for s in splits), splits
    test_f32(rows, N, K, False)
    test_f32(rows, N, K, True)
    test_add(rows, N, K)


@pytest.mark.parametrize("K", [896, 2560])
def test_norm_is_rounded_as_the_row_norm(K):
    """Through an identity weight every normalised value comes out exactly, and it is the one that
    bf16(x * rsqrt(sum / K + eps)) * gain gives: same division, same roundings."""
    tc = ops.pack_weight_tc(torch.eye(K, dtype=torch.bfloat16, device="cuda"))
    for seed in range(8):
        x, gain = _bf16((64, K), seed), _bf16((K,), 100 + seed)
        ss = _parts(x, 1)
        out = torch.full((64, K), float("nan"), device="cuda")
        check(lib.q_gemm_rows_f32(_p(x), _p(gain), _p(ss), 1, _p(tc), _p(out), 64, K, K, EPS, _stream()))
        assert torch.equal(out, _rms(x, ss[0], gain).float())


@pytest.mark.parametrize("rows", [9, 33, 64])
@pytest.mark.parametrize("inter,K", [(264, 128), (9728, 2560)])
def test_swiglu_of_each_element(rows, inter, K):
    """With the row's sum in one part the normalised values are those of the oracle bit for bit; then g and u can
    only round the other way (one ulp of each, rarely), and so can silu(g) (whose slope is at most 1.1) and the product."""
    x, w, gain = _bf16((rows, K), 1), _bf16((2 * inter, K), 2, 0.05), _bf16((K,), 3)
    ss = _parts(x, 1)
    act = torch.full((rows, inter), float("nan"), dtype=torch.bfloat16, device="cuda")
    check(lib.q_gemm_rows_swiglu(_p(x), _p(gain), _p(ss), 1, _p(ops.pack_weight_tc(w)), _p(act), rows, inter, K, EPS,
                                 _stream()))
    y = (_rms(x, ss[0], gain).double() @ w.double().T).bfloat16().float()
    g, u = y[:, :inter], y[:, inter:]
    want = (torch.nn.functional.silu(g).bfloat16().float() * u).bfloat16().float()
    diff = (act.float() - want).abs()
    assert bool((diff <= BF16_ULP * (1.1 * g.abs() * u.abs() + 3 * want.abs()) + 1e-4).all())
    assert float((diff > 0).float().mean()) < 0.02
    assert ops.device_status() == [0, 0, 0, 0]


def test_refused():
    z = torch.zeros(4096, dtype=torch.bfloat16, device="cuda")
    for rows, N, K in ((0, 64, 64), (65, 64, 64), (4, 12, 64), (4, 64, 96)):
        assert lib.q_gemm_rows_parts(rows, N, K) == 0
        assert lib.q_gemm_rows_add(_p(z), _p(z), _p(z), _p(z), rows, N, K, _stream()) == ERR_ARG
