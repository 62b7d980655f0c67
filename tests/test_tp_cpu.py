"""World-size-2 gloo run of the tensor-parallel decomposition on CPU: the weight
shards made by starter_b200.weights, the fp32 all-reduce after the O and down
projections (one bf16 rounding after the cross-rank sum) and the vocabulary-sharded
argmax merge reproduce the single-rank oracle."""
import os
import sys
from pathlib import Path

import pytest
import torch
import torch.distributed as dist
import torch.multiprocessing as mp

ROOT = Path(__file__).resolve().parents[1]


def _tp_forward(rank, world, sd, cfg, ids):
    """Prefill-style forward over ids [B, T] with this rank's shard; returns the
    gathered logits of the last position and the merged greedy token."""
    from oracle import qwen3_oracle as O
    from starter_b200 import weights as W
    D = 128
    pw = W.pack(cfg, sd.__getitem__, sd.__contains__, "cpu", rank, world)
    nq, nkv = pw.local_q_heads, pw.local_kv_heads
    B, T = ids.shape
    cos_t, sin_t = O.rotary_tables(cfg.rope_theta, T)
    cos_r, sin_r = cos_t.repeat(B, 1), sin_t.repeat(B, 1)
    limits = (torch.arange(T) + 1)[None].repeat(B, 1)
    x = pw.embed[ids].reshape(B * T, cfg.hidden)
    normed = O.rms_norm(x, pw.layers[0].ln_in, cfg.rms_eps)
    for i, lt in enumerate(pw.layers):
        q, k, v = O.qkv_norm_rope(O.linear(normed, lt.wqkv), lt.q_gain, lt.k_gain, cfg.rms_eps,
                                  cos_r, sin_r, nq, nkv)
        keys = k.view(B, T, nkv, D).transpose(1, 2)
        vals = v.view(B, T, nkv, D).transpose(1, 2)
        att = O.attention_fp64(q.view(B, T, nq, D), keys, vals, limits, D ** -0.5).reshape(B * T, nq * D)
        part = O.linear_fp32(att, lt.wo)                  # row-parallel: fp32 partial per rank
        dist.all_reduce(part)
        x, normed = O.add_rms_norm(x, part, lt.ln_post, cfg.rms_eps)
        hidden = O.swiglu(O.linear(normed, lt.wgu))
        part = O.linear_fp32(hidden, lt.wdown)
        dist.all_reduce(part)
        gain = pw.layers[i + 1].ln_in if i + 1 < len(pw.layers) else pw.ln_final
        x, normed = O.add_rms_norm(x, part, gain, cfg.rms_eps)
    last = normed.view(B, T, cfg.hidden)[:, -1]
    local = O.linear(last, pw.lm_head)                     # [B, V/world]
    val = local.float().max(-1).values
    idx = O.greedy_pick(local) + pw.vocab_offset
    vals = [torch.empty_like(val) for _ in range(world)]
    idxs = [torch.empty_like(idx) for _ in range(world)]
    dist.all_gather(vals, val)
    dist.all_gather(idxs, idx)
    vals, idxs = torch.stack(vals), torch.stack(idxs)
    best = vals.max(0).values
    token = torch.where(vals == best[None], idxs, torch.full_like(idxs, 2 ** 40)).min(0).values
    logits = [torch.empty_like(local) for _ in range(world)]
    dist.all_gather(logits, local.contiguous())
    return torch.cat(logits, -1), token


def _worker(rank, world, port, result):
    sys.path.insert(0, str(ROOT))
    os.environ["MASTER_ADDR"] = "127.0.0.1"
    os.environ["MASTER_PORT"] = str(port)
    dist.init_process_group("gloo", rank=rank, world_size=world)
    try:
        from safetensors.torch import load_file
        from oracle import qwen3_oracle as O
        from starter_b200 import weights as W
        import json
        gold = ROOT / "tests" / "golden" / "tiny_qwen3"
        sd = load_file(str(gold / "model.safetensors"))
        sd["model.embed_tokens.weight"] = sd["model.embed_tokens.weight"][:126].contiguous()
        hf_cfg = json.loads((gold / "config.json").read_text())
        hf_cfg["vocab_size"] = 126
        cfg = W.ModelConfig.from_hf(hf_cfg)
        torch.manual_seed(3)
        ids = torch.randint(0, 126, (2, 9))
        logits, token = _tp_forward(rank, world, sd, cfg, ids)
        if rank == 0:
            ref = O.RestatedModel(sd, hf_cfg)
            ref_logits = ref.forward(ids)
            diff = float((logits.float() - ref_logits.float()).abs().max())
            same = float((logits.view(torch.int16) == ref_logits.view(torch.int16)).float().mean())
            result.put((diff, same, token.tolist(), O.greedy_pick(ref_logits).tolist()))
    finally:
        dist.destroy_process_group()


def test_two_rank_sharding_matches_single_rank_oracle():
    ctx = mp.get_context("spawn")
    result = ctx.Queue()
    port = 29500 + os.getpid() % 2000
    procs = [ctx.Process(target=_worker, args=(r, 2, port, result)) for r in range(2)]
    for p in procs:
        p.start()
    for p in procs:
        p.join(180)
        assert p.exitcode == 0
    diff, same, token, ref_token = result.get(timeout=5)
    # fp32 partials are added across ranks before the single bf16 rounding, so the
    # only difference to one rank is fp32 summation order: at most a bf16 ulp
    assert diff <= 2e-3, diff
    assert same > 0.97, same
    assert token == ref_token


def test_argmax_merge_prefers_lowest_global_index():
    vals = torch.tensor([[1.0, 5.0], [1.0, 5.0], [0.5, 7.0]])
    idxs = torch.tensor([[10, 3], [4, 70], [9, 200]])
    best = vals.max(0).values
    token = torch.where(vals == best[None], idxs, torch.full_like(idxs, 2 ** 40)).min(0).values
    assert token.tolist() == [4, 200]


# ---- failure detection on the host: a rank that raises, a wrong shard, a rank that never joins ----
def _failure_worker(rank, world, port, result, case):
    sys.path.insert(0, str(ROOT))
    os.environ["MASTER_ADDR"] = "127.0.0.1"
    os.environ["MASTER_PORT"] = str(port)
    from datetime import timedelta
    from starter_b200 import tp, weights as W
    try:
        if case == "absent" and rank == 1:
            # this rank reaches the rendezvous but never the arrival point
            store = dist.TCPStore("127.0.0.1", port, world, is_master=False, timeout=timedelta(seconds=20))
            result.put((rank, "skipped"))
            return
        if case == "absent":
            store = dist.TCPStore("127.0.0.1", port, world, is_master=True, timeout=timedelta(seconds=20))
            try:
                tp.join_or_fail(store, rank, world, "step0", 1.0)
                result.put((rank, "no error"))
            except tp.TensorParallelError as exc:
                result.put((rank, str(exc)))
            return
        dist.init_process_group("gloo", rank=rank, world_size=world, timeout=timedelta(seconds=30))
        group = dist.group.WORLD
        gold = ROOT / "tests" / "golden" / "tiny_qwen3"
        try:
            if case == "raises":
                def load():
                    if rank == 1:
                        raise FileNotFoundError("shard 1 is missing")
                    return 7
                tp.guarded(group, load, "loading the checkpoint shard")
            elif case == "shape":
                from safetensors.torch import load_file
                import json
                sd = load_file(str(gold / "model.safetensors"))
                sd["model.embed_tokens.weight"] = sd["model.embed_tokens.weight"][:126].contiguous()
                hf_cfg = json.loads((gold / "config.json").read_text())
                hf_cfg["vocab_size"] = 126
                cfg = W.ModelConfig.from_hf(hf_cfg)
                # rank 1 cuts its shard as if it were alone
                pw = W.pack(cfg, sd.__getitem__, sd.__contains__, "cpu", *((rank, world) if rank == 0 else (0, 1)))
                tp.check_shards(group, pw)
            elif case == "fine":
                assert tp.guarded(group, lambda: rank + 1, "a step that works") == rank + 1
            result.put((rank, "no error"))
        except tp.TensorParallelError as exc:
            result.put((rank, str(exc)))
        finally:
            dist.destroy_process_group()
    except Exception as exc:             # noqa: BLE001 - the test reads it
        result.put((rank, f"unexpected {type(exc).__name__}: {exc}"))


def _run_failure_case(case):
    ctx = mp.get_context("spawn")
    result = ctx.Queue()
    port = 31500 + (os.getpid() * 7 + hash(case)) % 2000
    procs = [ctx.Process(target=_failure_worker, args=(r, 2, port, result, case)) for r in range(2)]
    for p in procs:
        p.start()
    for p in procs:
        p.join(120)
        assert p.exitcode == 0
    out = dict(result.get(timeout=5) for _ in range(2))
    return out


def test_a_rank_that_raises_fails_every_rank():
    out = _run_failure_case("raises")
    for rank in (0, 1):
        assert "failed on rank(s) [1] of 2" in out[rank], out
    assert "shard 1 is missing" in out[1]
    assert _run_failure_case("fine") == {0: "no error", 1: "no error"}


def test_a_wrong_shard_fails_every_rank():
    out = _run_failure_case("shape")
    for rank in (0, 1):
        assert "shards disagree" in out[rank], out


def test_a_rank_that_never_arrives_is_named():
    out = _run_failure_case("absent")
    assert "rank(s) [1] of 2 did not arrive at 'step0'" in out[0], out


def test_prompt_pass_clears_tickets_of_a_launch_that_gave_up(monkeypatch):
    """The tensor-parallel prompt pass hands q_gemm_prompt_* a scratch whose tickets are zero in every
    run of layers, whatever an earlier launch that gave up left there; the rest of the scratch stays.
    (The library's calls are recorded, nothing runs.)"""
    from types import SimpleNamespace as NS
    from starter_b200 import decode
    cfg = NS(n_layers=2, hidden=64, rms_eps=1e-6)
    weight = NS(tc=lambda: torch.zeros(1))
    layer = NS(wqkv=weight, wo=weight, wgu=weight, wdown=weight, q_gain=torch.zeros(1), k_gain=torch.zeros(1),
               ln_in=torch.zeros(1), ln_post=torch.zeros(1))
    pool = [torch.zeros(1)] * cfg.n_layers
    state = NS(cfg=cfg, w=NS(local_q_heads=2, local_kv_heads=1, local_inter=64, layers=[layer] * 2, ln_final=torch.zeros(1)),
               kpools=pool, vpools=pool, pages_per_seq=1, cos=torch.zeros(1), sin=torch.zeros(1), group=None,
               PROMPT_TICKET_BYTES=16384)
    pf = {n: torch.zeros(4) for n in ("x", "normed", "q", "att", "act", "zero")}
    pf["reduced"] = torch.zeros((300, cfg.hidden))
    pf["split"] = torch.empty(decode.lib.q_gemm_prompt_scratch_bytes(), dtype=torch.uint8)
    seen = []

    class Recorder:
        def __getattr__(self, name):
            def call(*args):
                if name.startswith("q_gemm_prompt"):
                    seen.append((name, bool(pf["split"][:16384].any()), bool(pf["split"][16384:].all())))
                return 0
            return call

    monkeypatch.setattr(decode, "lib", Recorder())
    monkeypatch.setattr(torch.distributed, "all_reduce", lambda t, group=None: None)
    for _ in range(2):
        pf["split"].fill_(3)                                   # what a launch that gave up may leave
        decode.DecodeState._prefill_layers(state, pf, 1, 300, 0, None)
    assert len(seen) == 2 * 4 * cfg.n_layers
    assert all(not drawn and kept for _, drawn, kept in seen)
