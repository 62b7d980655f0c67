"""Split counts of the decode attention (q_attention_decode_splits) and the argument checks of the
prompt entry points."""
import ctypes as C

import pytest
import torch

from oracle import qwen3_oracle as O


@pytest.mark.parametrize("batch", [1, 2, 3, 5, 8, 9, 11, 16, 37, 64])
@pytest.mark.parametrize("kv_heads", [1, 2, 8])
def test_split_count_is_usable(batch, kv_heads):
    """Between 1 and 32, never more than the pages, and within what two CTAs per SM hold."""
    from starter_b200._lib import lib
    for capacity in (1, 64, 65, 150, 700, 2000, 8000, 40000):
        s = lib.q_attention_decode_splits(batch, kv_heads, capacity)
        assert 1 <= s <= 32 and s <= max(1, (capacity + 63) // 64)
        assert s == 1 or s * batch * kv_heads <= 2 * 148
        assert lib.q_attention_block_splits(batch, kv_heads, capacity, 16) == lib.q_attention_splits(batch, kv_heads, capacity)
        b = lib.q_attention_block_splits(batch, kv_heads, capacity, 17)
        assert 1 <= b <= 32 and b <= max(1, (capacity + 63) // 64)


@pytest.mark.parametrize("batch,capacity,splits", [(6, 512, 3), (6, 10240, 3), (3, 14080, 6), (8, 4096, 2), (7, 16384, 5),
                                                   (8, 16000, 2), (4, 16000, 4), (16, 16000, 1), (5, 32000, 7)])
def test_block_splits_fill_waves(batch, capacity, splits):
    """One CTA per SM for more than 16 query rows: one full wave, or two where one would leave a
    quarter of the SMs idle, but no further wave for a page or two (148 SMs, 8 kv heads)."""
    from starter_b200._lib import lib
    assert lib.q_attention_block_splits(batch, 8, capacity, 32) == splits


def test_prompt_entry_points_reject_bad_arguments():
    """Argument errors surface before any launch (no device needed): sizes, alignment, null pointers."""
    from starter_b200 import _lib
    lib, A = _lib.lib, C.c_void_p(1 << 20)
    odd = C.c_void_p((1 << 20) + 16)
    bad = [
        lib.q_gemm_prompt_f32(A, A, A, 0, 64, 64, None, None),            # no rows
        lib.q_gemm_prompt_f32(A, A, A, 4, 48, 64, None, None),            # N not a multiple of 32
        lib.q_gemm_prompt_f32(A, A, A, 4, 64, 80, None, None),            # K not a multiple of 32
        lib.q_gemm_prompt_f32(A, A, odd, 4, 64, 64, None, None),          # output not 32-byte aligned
        lib.q_gemm_prompt_f32(A, odd, A, 4, 64, 64, None, None),          # weight not 1024-byte aligned
        lib.q_gemm_prompt_add(A, A, A, 4, 64, 64, None, None),            # input is the residual
        lib.q_gemm_prompt_swiglu(None, A, A, 4, 64, 64, None, None),
        lib.q_gemm_prompt_qkv(A, A, A, A, A, A, A, A, None, 1, 4, 4, 64, 1e-6, None, None),
        lib.q_prompt_pass(None, None, A, A, 1, 1, 4, A, None),
        lib.q_prompt_pass(C.byref(_lib.Prompt()), (_lib.LayerWeights * 1)(), A, A, 1, 1, 4, A, None),
    ]
    assert bad == [-1] * len(bad)
    assert lib.q_gemm_prompt_scratch_bytes() > 16384


@pytest.mark.gpu
@pytest.mark.parametrize("batch,kv_heads,capacity,splits", [
    (5, 8, 712, 3), (2, 8, 4012, 6),                    # wide CTAs, their clusters resident
    (2, 8, 8012, 18), (3, 4, 16012, 24),                # a long context on few clusters: merged through memory
    (11, 4, 4012, 5), (16, 4, 2012, 4),                 # behind the tcgen05 projections: narrow CTAs
    (9, 4, 412, 3), (9, 8, 1012, 2),                    # ... but wide ones for few tiles, or where they fill the SMs
    (8, 8, 212, 4), (9, 8, 412, 4),                     # splits of one or two tiles: three CTAs per SM
    (12, 8, 2012, 2), (64, 8, 345, 1)])
def test_split_counts_of_the_measured_rule(batch, kv_heads, capacity, splits):
    """One shape per line of q_attention_decode_splits, with the count that measured best there or within
    one per cent of it (148 SMs)."""
    if not torch.cuda.is_available():
        pytest.skip("needs CUDA")
    from starter_b200._lib import lib
    assert lib.q_attention_decode_splits(batch, kv_heads, capacity) == splits


@pytest.mark.gpu
@pytest.mark.parametrize("B,nq,nkv,pos", [(2, 32, 8, 7700), (11, 16, 4, 700), (9, 32, 8, 400), (1, 32, 8, 7000), (2, 8, 2, 90), (3, 32, 8, 2000), (5, 32, 8, 700), (6, 32, 8, 700),
                                          (11, 32, 8, 500), (40, 32, 8, 430), (64, 32, 8, 333)])
def test_decode_attention_at_its_split_count(B, nq, nkv, pos):
    """The fused decode attention with the splits and the ring it is given in a step - one wide CTA
    per SM, two or three narrow ones, more CTAs than fit, splits merged through memory - against the
    separate kernels, with the bars of the other fused-attention tests."""
    if not torch.cuda.is_available():
        pytest.skip("needs CUDA")
    from starter_b200 import ops
    from starter_b200._lib import lib
    from tests.parity import bit_equal_fraction
    capacity = pos + 70
    g = torch.Generator(device="cuda").manual_seed(pos + B)
    width = (nq + 2 * nkv) * 128
    w = (torch.randn((width, 256), generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    x = (torch.randn((B, 256), generator=g, device="cuda") * 4).to(torch.bfloat16)
    gain = [(1 + 0.1 * torch.randn(128, generator=g, device="cuda")).to(torch.bfloat16) for _ in range(2)]
    cos, sin = (t.cuda() for t in O.rotary_tables(1_000_000.0, capacity))
    part = ops.linear_partials(x, w)
    position = torch.tensor([pos], dtype=torch.int32, device="cuda")
    old = [torch.randn((B, nkv, pos, 128), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2)]
    caches = []
    for _ in range(2):
        c = ops.PagedKV(B, nkv, capacity, "cuda", poison=float("nan"))
        c.scatter(old[0], old[1], 0)
        caches.append(c)
    attn = ops.SmallQueryAttention(B, nq, nkv, capacity, "cuda")
    q = ops.qkv_norm_rope_cache(part, gain[0], gain[1], 1e-6, 1e-6, cos, sin, position, caches[0])
    ref = attn.run(q, caches[0], position, 128 ** -0.5)
    attn.splits = lib.q_attention_decode_splits(B, nkv, capacity)
    attn.partials = torch.empty((B * nkv, attn.splits, nq // nkv, 128), dtype=torch.float32, device="cuda")
    attn.stats = torch.empty((B * nkv, attn.splits, nq // nkv, 2), dtype=torch.float32, device="cuda")
    for _ in range(2):
        got = ops.decode_attention(part, gain[0], gain[1], 1e-6, cos, sin, position, caches[1], attn, 128 ** -0.5)
        torch.testing.assert_close(got.float(), ref.float(), rtol=0.02, atol=5e-3)
        assert bit_equal_fraction(got.cpu(), ref.cpu()) > 0.6
    for a, b in zip(caches[0].gather(pos + 1), caches[1].gather(pos + 1)):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))
    assert ops.device_status()[0] == 0
