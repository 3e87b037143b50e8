"""Prompt attention with score reductions on several streams and from several threads at once: every call has partial sums of its own."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(S, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(1, h, S, 64, device="cuda", generator=gen).bfloat16() for h in (8, 2, 2)]


def test_calls_on_two_streams_share_no_scratch(monkeypatch):
    from cold_compress_b200 import ops
    from cold_compress_b200.attention_utils import prefill_attention_stats
    held, whole = [], ops.prefill_attention

    def note(*args):
        held.append(args[-1])
        return whole(*args)

    monkeypatch.setattr(ops, "prefill_attention", note)
    q, k, v = _inputs(300, 0)
    torch.cuda.synchronize()
    for stream in (torch.cuda.Stream(), torch.cuda.Stream()):
        with torch.cuda.stream(stream):
            prefill_attention_stats(q, k, v)
    torch.cuda.synchronize()
    a, b = sorted((t.data_ptr(), t.numel()) for t in held)
    assert a[0] + a[1] <= b[0]


def test_results_do_not_depend_on_other_threads():
    from cold_compress_b200.attention_utils import prefill_attention_stats
    jobs = [_inputs(S, S) for S in (200, 333, 700, 901)]
    want = [prefill_attention_stats(*j) for j in jobs]
    torch.cuda.synchronize()
    wrong = []

    def work(j, ref):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(40):
                y, st = prefill_attention_stats(*j)
                if not (torch.equal(y, ref[0]) and torch.equal(st.col_sum, ref[1].col_sum) and torch.equal(st.obs_mean, ref[1].obs_mean)):
                    wrong.append(j[0].shape[2])

    threads = [threading.Thread(target=work, args=x) for x in zip(jobs, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
