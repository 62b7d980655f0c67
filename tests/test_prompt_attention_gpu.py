"""The prompt attention kernel where it can go wrong: one and two query tiles per CTA, several items
per CTA, every head grouping, a maximum that keeps growing (a rescale of O in every tile), scales that are not
positive, an output that is only 4-byte aligned."""
import ctypes as C

import pytest
import torch

from oracle import qwen3_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("needs CUDA")
    from starter_b200 import ops as ops_mod
    return ops_mod


def case(ops, B, nq, nkv, T, base, growth, scale, offset=0):
    from starter_b200._lib import check, lib
    g = torch.Generator().manual_seed(900 + T + nq)
    L = base + T
    q = torch.randn((B, T, nq, 128), generator=g).to(torch.bfloat16)
    k = torch.randn((B, nkv, L, 128), generator=g)
    if growth:
        # late keys score far above early ones: rows move their maximum many times
        k = k * torch.linspace(0.05, 4.0, L)[None, None, :, None]
    k = k.to(torch.bfloat16)
    v = torch.randn((B, nkv, L, 128), generator=g).to(torch.bfloat16)
    cache = ops.PagedKV(B, nkv, L + 40, "cuda", poison=float("nan"))
    cache.scatter(k.cuda(), v.cuda(), 0)
    position = torch.tensor([base], dtype=torch.int32, device="cuda")
    qd = q.reshape(B * T, nq, 128).cuda()
    raw = torch.full((B * T * nq * 128 + 64,), float("nan"), dtype=torch.bfloat16, device="cuda")
    out = raw[offset:offset + B * T * nq * 128]
    P = lambda t: C.c_void_p(t.data_ptr())
    check(lib.q_attention_prefill(P(qd), C.byref(cache.layout), P(position), P(out), B, T, nq, scale,
                                  C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    limits = (base + torch.arange(T) + 1)[None].repeat(B, 1)
    ref = O.attention_fp64(q, k, v, limits, scale).reshape(B * T, nq * 128)
    got = out.view(B * T, nq * 128).cpu()
    assert not torch.isnan(got.float()).any()
    assert torch.isnan(raw[:offset].float()).all() and torch.isnan(raw[offset + out.numel():].float()).all()
    torch.testing.assert_close(got.float(), ref.float(), rtol=0.02, atol=5e-3)
    assert ops.device_status()[0] == 0


@pytest.mark.parametrize("B,nq,nkv,T,base", [(1, 4, 1, 31, 0), (1, 32, 8, 576, 0), (1, 32, 8, 600, 0), (4, 16, 8, 700, 0),
                                             (2, 8, 8, 600, 130), (1, 8, 1, 513, 0), (5, 32, 8, 530, 63)])
@pytest.mark.parametrize("growth", [False, True])
def test_against_fp64(ops, B, nq, nkv, T, base, growth):
    case(ops, B, nq, nkv, T, base, growth, 128 ** -0.5)


@pytest.mark.parametrize("scale", [0.0, -0.05])
def test_scale_that_is_not_positive(ops, scale):
    case(ops, 1, 8, 2, 200, 10, False, scale)


def test_output_of_4_byte_alignment(ops):
    case(ops, 1, 8, 2, 200, 0, False, 128 ** -0.5, offset=2)


# Two query tiles per SM of 148: the last count with one tile per item (two items per CTA, every row's maximum
# exchanged among four threads), and the first with two.
@pytest.mark.parametrize("T,base", [(1184, 0), (1185, 0), (1000, 70)])
def test_where_the_forms_part(ops, T, base):
    case(ops, 1, 32, 8, T, base, True, 128 ** -0.5)
