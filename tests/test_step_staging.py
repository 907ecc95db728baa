"""Inputs of a step: one launch out of pinned memory, and decode rows staged by the engine core."""

import pytest
import torch

from research_b200 import ops
from research_b200.inference import EngineConfig, InferenceEngine, SamplingParams
from research_b200.models import get_preset, init_random_weights


def _engine(device, **kw):
    cfg = get_preset("tiny-qwen2", num_layers=2, init_std=0.05)
    w = init_random_weights(cfg, seed=1)
    on_gpu = torch.device(device).type == "cuda"
    if on_gpu:
        w = {k: v.bfloat16() for k, v in w.items()}
    return cfg, InferenceEngine(EngineConfig(max_batch_size=6, max_model_len=200, num_kv_blocks=80, ignore_eos=True, cache_type="none", **kw), cfg, w,
                                device=device)


@pytest.mark.parametrize("n", [1, 3, 6])
def test_staged_decode_rows_equal_the_packed_builder(n):
    """The fields of the rows are those that the general builder gives for the same sequences, the rest is padding."""
    cfg, eng = _engine("cpu")
    r, seen = eng.runner, []
    decode = r.decode

    def watch(rows, max_blocks, sample=True):
        mb, o = r.max_batch, r.pf_at
        base, pf = torch.full_like(r.meta_host, 77), torch.full_like(r.pf_host, 77)
        table = torch.full_like(r.bt_host, 77)
        at, pat = base.data_ptr(), pf.data_ptr()
        assert eng._lib.rbe_build_batch(eng._core, 1, at, at + 4 * mb, at + 8 * mb, pat + 4 * o["cu_q"], at + 12 * mb, table.data_ptr(),
                                        r.max_blocks_per_seq, at + 16 * mb, at + 20 * mb, pat + 4 * o["sample_rows"], mb, mb) == rows
        for field in range(5):
            assert torch.equal(base[field * mb:field * mb + rows], r.meta_host[field * mb:field * mb + rows])
        assert torch.equal(base[5 * mb:5 * mb + 2 * rows], r.meta_host[5 * mb:5 * mb + 2 * rows])
        assert max_blocks == -(-int(base[3 * mb:3 * mb + rows].max()) // 16)
        for i in range(rows):
            used = -(-int(base[3 * mb + i]) // 16)
            assert torch.equal(table[i, :used], r.bt_host[i, :used])
        for field, fill in ((0, 0), (1, 0), (2, -1), (3, 0), (7, -1)):
            assert (r.meta_host[field * mb + rows:field * mb + r.step_rows(rows)] == fill).all()
        seen.append(rows)
        decode(rows, max_blocks, sample)

    r.decode = watch
    eng.generate([list(range(5, 20 + 13 * i)) for i in range(n)], SamplingParams(temperature=0.7, max_tokens=20, seed=3))
    assert seen and max(seen) == n


@pytest.mark.gpu
@pytest.mark.parametrize("n,stride,rows,cols", [(1, 1, 1, 1), (3, 5, 2, 5), (4, 9, 7, 3), (1029, 130, 128, 129), (50_003, 1024, 16, 1023), (8, 4, 0, 0)])
def test_stage_step(n, stride, rows, cols):
    g = torch.Generator().manual_seed(n)
    host = torch.randint(-2**31, 2**31 - 1, (n,), generator=g, dtype=torch.int32).pin_memory()
    table = torch.randint(0, 2**31 - 1, (max(rows, 1) + 1, stride), generator=g, dtype=torch.int32).pin_memory()
    dev, dtable = torch.full((n,), 5, dtype=torch.int32, device="cuda"), torch.full(table.shape, 5, dtype=torch.int32, device="cuda")
    ops.stage_step(host, dev, table, dtable, rows, cols)
    want = torch.full(table.shape, 5, dtype=torch.int32)
    want[:rows, :cols] = table[:rows, :cols]
    assert torch.equal(dev.cpu(), host) and torch.equal(dtable.cpu(), want)
    with pytest.raises(ValueError):
        ops.stage_step(torch.zeros(n, dtype=torch.int32), dev, table, dtable, rows, cols)      # not pinned


@pytest.mark.gpu
def test_skipped_rows_keep_their_outputs():
    logits = torch.randn(3, 9000, device="cuda")
    temps, skip = torch.zeros(3, device="cuda"), torch.ones(1, dtype=torch.int32, device="cuda")
    toks, lps = torch.full((3,), 7, dtype=torch.int32, device="cuda"), torch.full((3,), 7.0, device="cuda")
    ops.sample_with_logprobs(logits, temps, None, 0, None, toks, lps, skip=skip)
    assert (toks == 7).all() and (lps == 7).all()
    ops.sample_with_logprobs(logits, temps, None, 0, None, toks, lps, skip=skip.zero_())
    assert torch.equal(toks.long(), logits.argmax(-1))


@pytest.mark.gpu
@pytest.mark.parametrize("graphs", [False, True])
def test_given_and_sampled_tokens_take_turns(graphs):
    """Greedy tokens fed one by one give the logits that generate() drew from, before and behind sampled steps of the same engine."""
    cfg, eng = _engine("cuda", use_cuda_graphs=graphs, graph_batch_sizes=(2, 6))
    prompts = [list(range(3, 20)), list(range(40, 91)), list(range(7, 9))]

    def drawn():
        return [list(s.completion_tokens) for s in eng.generate(prompts, SamplingParams(temperature=0.0, max_tokens=18))]

    want = drawn()
    for _ in range(2):
        ids = [eng.open_stream() for _ in prompts]
        out = [eng.feed([(i, p, [len(p) - 1]) for i, p in zip(ids, prompts)])]
        for t in range(17):
            out.append(eng.feed([(i, [w[t]], [0]) for i, w in zip(ids, want)]))
        for i in ids:
            eng.close_stream(i)
        for r in range(len(prompts)):
            for t in range(18):
                row = out[t][r]
                assert row[want[r][t]] >= row.max() - 0.05, (r, t)
        assert drawn() == want
    eng.shutdown()
