"""The prompt pass's projections (q_gemm_prompt_*, CTA pairs) through the C ABI against the CPU
oracle, at the edges of their 256-row x 128..256-column tiles."""
import ctypes as C

import pytest
import torch

from oracle import qwen3_oracle as O
from tests.parity import bit_equal_fraction

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("needs CUDA")
    from starter_b200 import ops as ops_mod
    return ops_mod


def rand(shape, seed, scale):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(shape, generator=g) * scale).to(torch.bfloat16)


def gain(n, seed):
    return (1 + 0.1 * rand(n, seed, 1.0).float()).to(torch.bfloat16)


def stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def P(t):
    return None if t is None else C.c_void_p(t.data_ptr())


@pytest.fixture(scope="module", params=["split", "whole"])
def scratch(request, ops):
    """Parts of tiles shared by several SM pairs, or (no scratch) whole tiles only."""
    from starter_b200._lib import lib
    if request.param == "whole":
        return None
    return torch.zeros(lib.q_gemm_prompt_scratch_bytes(), dtype=torch.uint8, device="cuda")


# one row; rows around one CTA, one tile and a raster group of eight row tiles; columns of less than
# a tile; K of less than a 64-k step, odd and long. With scratch: few tiles cut over all pairs,
# shares of more than a tile, a whole wave before the split, and shapes that stay whole.
SHAPES = [(256, 256, 512), (1, 32, 32), (128, 128, 64), (129, 160, 96), (257, 2560, 416), (700, 96, 4096),
          (1000, 2560, 9728), (2048, 2560, 9728), (3800, 2560, 8192), (2103, 2560, 4096), (2305, 4896, 160)]


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_sums_and_residual(ops, scratch, M, N, K):
    """fp32 sums within the bar of the decode projections (rtol = atol = 2e-3), rows past M untouched;
    the residual form equals the two roundings of that sum bit for bit."""
    from starter_b200._lib import check, lib
    x, w, res = rand((M, K), 1, 1.0), rand((N, K), 2, 0.02), rand((M, N), 3, 1.0)
    xd, tiled = x.cuda(), ops.pack_weight_tc(w.cuda())
    out = torch.full((M + 3, N), float("nan"), dtype=torch.float32, device="cuda")
    check(lib.q_gemm_prompt_f32(P(xd), P(tiled.data), P(out), M, N, K, P(scratch), stream()))
    total = torch.full((M + 3, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    total[:M] = res.cuda()
    check(lib.q_gemm_prompt_add(P(xd), P(tiled.data), P(total), M, N, K, P(scratch), stream()))
    got = out.cpu()
    torch.testing.assert_close(got[:M], O.linear_fp32(x, w), rtol=2e-3, atol=2e-3)
    assert torch.isnan(got[M:]).all() and torch.isnan(total[M:].float()).all()
    want = (res.float() + got[:M].to(torch.bfloat16).float()).to(torch.bfloat16)
    assert torch.equal(total[:M].cpu(), want)
    if scratch is not None:
        assert not scratch[:16384].any()                       # every ticket is back to zero
    assert ops.device_status() == [0, 0, 0, 0]


# Tiles of 160 columns: a last tile of 32 and of 96 columns, weight rows that end inside a 128-row block, one
# wave with idle pairs and three waves, a K that is no multiple of 64.
@pytest.mark.parametrize("M,N,K", [(512, 2592, 512), (2100, 2592, 96), (130, 576, 9728), (5000, 672, 160)])
def test_narrow_tiles(ops, scratch, M, N, K):
    test_sums_and_residual(ops, scratch, M, N, K)


# The same edges where the rule takes narrow tiles for either epilogue (q_gemm_prompt_columns): one wave with idle
# pairs, two waves, last tiles of 32 and 96 columns, a K that is no multiple of 64.
@pytest.mark.parametrize("M,N,K", [(512, 2592, 512), (1800, 2592, 96), (8000, 576, 9728), (7000, 672, 160), (1000, 2560, 4096)])
def test_narrow_tiles_where_the_rule_takes_them(ops, scratch, M, N, K):
    from starter_b200._lib import lib
    assert lib.q_gemm_prompt_columns(M, N, K, 0) == lib.q_gemm_prompt_columns(M, N, K, 1) == 160
    test_sums_and_residual(ops, scratch, M, N, K)


@pytest.mark.parametrize("M,inter,K", [(1, 32, 32), (300, 96, 128), (257, 1184, 416), (600, 9728, 256), (600, 1312, 9728)])
def test_swiglu(ops, scratch, M, inter, K):
    """Within one bf16 rounding of the oracle's SwiGLU of the fp32 sums (inter not a multiple of 128
    puts the up rows across the 128-row weight blocks)."""
    from starter_b200._lib import check, lib
    # Gate sums of standard deviation 0.8, so |g| < 4: where the two fp32 sums round to neighbouring bf16
    # values of g, silu moves by at most ulp(g) * |silu'(g) / silu(g)| <= 2^-7 * 1.02 of itself there
    # (at g = -16 one step of g already moves silu by 6 %, whatever the kernel does).
    x, w = rand((M, K), 4, 1.0), rand((2 * inter, K), 5, 0.8 * K ** -0.5)
    xd, tiled = x.cuda(), ops.pack_weight_tc(w.cuda())
    act = torch.full((M + 2, inter), float("nan"), dtype=torch.bfloat16, device="cuda")
    check(lib.q_gemm_prompt_swiglu(P(xd), P(tiled.data), P(act), M, inter, K, P(scratch), stream()))
    ref = O.swiglu(O.linear_fp32(x, w))
    torch.testing.assert_close(act[:M].cpu().float(), ref.float(), rtol=0.02, atol=2e-3)
    assert bit_equal_fraction(act[:M].cpu(), ref) > 0.98
    assert torch.isnan(act[M:].float()).all()
    assert ops.device_status() == [0, 0, 0, 0]


@pytest.mark.parametrize("B,T,nq,nkv,pos", [(1, 1, 1, 1, 0), (2, 130, 4, 2, 70), (3, 301, 8, 1, 0), (1, 1000, 32, 8, 5), (1, 250, 32, 8, 0)])
def test_qkv_norm_rope_pages(ops, scratch, B, T, nq, nkv, pos):
    """q, k within the bar of the separate kernel, v exact; only the slots of this block are written
    in the NaN-poisoned pages."""
    from starter_b200._lib import check, lib
    width, K, rows = (nq + 2 * nkv) * 128, 9728 if T == 250 else 128, B * T
    w, x = rand((width, K), 6, 0.02), rand((rows, K), 7, 4.0)
    qg, kg = gain(128, 8), gain(128, 9)
    capacity = pos + T + 70
    cos, sin = O.rotary_tables(1_000_000.0, capacity)
    cache = ops.PagedKV(B, nkv, capacity, "cuda", poison=float("nan"))
    position = torch.tensor([pos], dtype=torch.int32, device="cuda")
    tiled, xd = ops.pack_weight_tc(w.cuda()), x.cuda()
    q = torch.full((rows + 1, nq, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    dev = [t.cuda() for t in (qg, kg, cos, sin)]
    check(lib.q_gemm_prompt_qkv(P(xd), P(tiled.data), P(dev[0]), P(dev[1]), P(dev[2]), P(dev[3]), P(position), P(q),
                                C.byref(cache.layout), B, T, nq, K, 1e-6, P(scratch), stream()))
    sums = torch.empty((rows, width), dtype=torch.float32, device="cuda")
    check(lib.q_gemm_prompt_f32(P(xd), P(tiled.data), P(sums), rows, width, K, P(scratch), stream()))
    at = (pos + torch.arange(T)).repeat(B)
    eq, ek, ev = O.qkv_norm_rope(sums.cpu(), qg, kg, 1e-6, cos[at], sin[at], nq, nkv)
    got = q.cpu()
    torch.testing.assert_close(got[:rows].float(), eq.float().view(rows, nq, 128), rtol=0.02, atol=0.02)
    assert bit_equal_fraction(got[:rows], eq.view(rows, nq, 128)) > 0.99
    assert torch.isnan(got[rows:].float()).all()
    kc, vc = (t.cpu() for t in cache.gather(capacity))
    knew = kc[:, :, pos:pos + T].transpose(1, 2).reshape(rows, nkv, 128)
    vnew = vc[:, :, pos:pos + T].transpose(1, 2).reshape(rows, nkv, 128)
    torch.testing.assert_close(knew.float(), ek.float().view(rows, nkv, 128), rtol=0.02, atol=0.02)
    assert bit_equal_fraction(knew, ek.view(rows, nkv, 128)) > 0.99
    assert torch.equal(vnew.view(torch.int16), ev.contiguous().view(rows, nkv, 128).view(torch.int16))
    untouched = torch.ones(capacity, dtype=torch.bool)
    untouched[pos:pos + T] = False
    assert torch.isnan(kc[:, :, untouched].float()).all() and torch.isnan(vc[:, :, untouched].float()).all()
    assert ops.device_status() == [0, 0, 0, 0]


@pytest.mark.parametrize("rows,cols", [(296, 2560), (297, 2560), (301, 8), (400, 2568), (333, 4096), (300, 4104), (299, 100)])
def test_rms_norm_many_rows(ops, rows, cols):
    """Both forms of the row norm around the row count and widths where they part."""
    x, g = rand((rows, cols), 10, 2.0), gain(cols, 11)
    out = ops.rms_norm(x.cuda(), g.cuda(), 1e-6).cpu()
    ref = O.rms_norm(x, g, 1e-6)
    torch.testing.assert_close(out.float(), ref.float(), rtol=0.02, atol=0.02)
    assert bit_equal_fraction(out, ref) > 0.99
