"""The package's per-call functions through the C++ front end and through the ctypes bodies: same library calls, so
the same bits (and the same refusals)."""
import threading
import time

import pytest
import torch

from h100_gdn_cuda_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from h100_gdn_cuda_b200 import api, build
    build.build()
    build.build_ext()
    assert api._load_ext(), "the extension is built but does not load"
    return api


def _cuda(p):
    return {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in p.items()}


def _flat(r):
    return [t for t in (r if isinstance(r, tuple) else (r,)) if t is not None]


def _calls(api):
    d = _cuda(synthetic.decode_inputs(3, 2, 2, 4, 64, seed=1))
    p = _cuda(synthetic.prefill_inputs(2, 97, 2, 4, 60, seed=2))
    v = _cuda(synthetic.varlen_inputs([70, 0, 5], 2, 4, 128, seed=3))
    gating = (d["A_log"], d["dt_bias"], d["a"], d["b"])
    slots = torch.tensor([2, 0, 1], dtype=torch.int32, device="cuda")
    conv_in, conv_w = d["v"].reshape(3, 2, 256), torch.randn(256, 4, device="cuda").bfloat16()
    beta = torch.sigmoid(d["b"].float()).bfloat16()
    wide = _cuda(synthetic.prefill_inputs(1, 70, 1, 2, 200, seed=4))
    caps = torch.tensor([2, 0, 1], dtype=torch.int32, device="cuda")
    conv_s, cu = torch.randn(3, 3, 256, device="cuda").bfloat16(), torch.tensor([0, 1, 5, 6], dtype=torch.int32, device="cuda")
    bias, packed_in = torch.randn(256, device="cuda").bfloat16(), conv_in.reshape(6, 256)
    ones = torch.tensor([0, 1, 2, 3], dtype=torch.int32, device="cuda")
    return {
        "recurrent, caps": lambda: api.recurrent_forward(d["q"], d["k"], d["v"], d["state"], beta, d["a"], None, caps, 1, True)[1],
        "recurrent, step states": lambda: api.recurrent_forward(d["q"], d["k"], d["v"], d["state"], beta, d["a"], inference_mode=2),
        "recurrent, in place": lambda: api.recurrent_forward(d["q"], d["k"], d["v"], d["state"].clone(), beta, d["a"], inplace_state=True),
        "recurrent, fp32 state": lambda: api.recurrent_forward(d["q"], d["k"], d["v"], d["state"].float(), beta, d["a"]),
        "recurrent, packed": lambda: api.recurrent_forward(v["q"], v["k"], v["v"], v["state"], v["beta"], v["g"], v["cu_seqlens"]),
        "prefill, d=200": lambda: api.chunked_forward(wide["q"], wide["k"], wide["v"], wide["beta"], wide["g"], None, wide["state"]),
        "conv, bias and state": lambda: api.causal_conv1d(conv_in, conv_w, bias, conv_s, return_final_state=True),
        "conv, packed": lambda: api.causal_conv1d(packed_in, conv_w, bias, conv_s, cu, return_final_state=True),
        "conv, packed in place": lambda: (lambda s: api.causal_conv1d(packed_in[:3], conv_w, None, s, ones, final_state=s))(conv_s.clone()),
        "gating": lambda: api.fused_gdn_gating(*gating),
        "recurrent, gating inside": lambda: api.recurrent_forward(d["q"], d["k"], d["v"], d["state"], None, None, gating=gating,
                                                                  is_qk_norm=True, inference_mode=2),
        "recurrent, no gate, pool": lambda: api.recurrent_forward(d["q"], d["k"], d["v"], d["state"].clone(), beta,
                                                                  scale=0.3, state_indices=slots),
        "recurrent, fp32, no state": lambda: api.recurrent_forward(d["q"], d["k"], d["v"], None, beta, d["a"].float()),
        "prefill, padded dims": lambda: api.chunked_forward(p["q"], p["k"], p["v"], p["beta"], p["g"], None, p["state"]),
        "prefill, no gate": lambda: api.chunked_forward(p["q"], p["k"], p["v"], p["beta"], None, is_qk_norm=True),
        "prefill, packed": lambda: api.chunked_forward(v["q"], v["k"], v["v"], v["beta"], v["g"], 0.2, v["state"], v["cu_seqlens"],
                                                       v["chunk_indices"], v["cu_chunks"]),
        "conv": lambda: api.causal_conv1d(conv_in, conv_w, None, None, return_final_state=True),
        "conv, y only": lambda: api.causal_conv1d(conv_in, conv_w, activation=False),
        "norm": lambda: api.gated_rmsnorm(d["v"], d["v"], conv_w[:64, 0].contiguous()),
    }


def test_both_front_ends_give_the_same_bits(api, monkeypatch):
    for name, call in _calls(api).items():
        fast = _flat(call())
        with monkeypatch.context() as m:
            m.setattr(api, "_ext", False)
            slow = _flat(call())
        assert len(fast) == len(slow), name
        for a, b in zip(fast, slow):
            assert a.shape == b.shape and a.stride() == b.stride() and a.dtype == b.dtype and torch.equal(a, b), name


def test_refusals(api):
    d = _cuda(synthetic.decode_inputs(1, 1, 1, 1, 64, seed=1))
    with pytest.raises(RuntimeError):
        api.recurrent_forward(d["q"], d["k"], d["v"], d["state"])          # beta missing
    with pytest.raises(RuntimeError):
        api.recurrent_forward(d["q"].cpu(), d["k"], d["v"], d["state"], d["b"])
    with pytest.raises(RuntimeError):
        api.chunked_forward(d["q"], d["k"], d["v"], d["b"].cpu(), None)
    with pytest.raises(RuntimeError):
        api.gated_rmsnorm(d["v"], d["q"].float(), d["q"][0, 0, 0])


def test_empty_last_axis_is_refused(api):
    """The row count of these calls is the size divided by the last axis: an empty one raises and does not divide."""
    e = lambda *shape: torch.empty(*shape, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(RuntimeError):
        api.gated_rmsnorm(e(3, 0), e(3, 0), e(0))
    with pytest.raises(RuntimeError):
        api.fused_gdn_gating(e(0), e(0), e(3, 0), e(3, 0))


def test_a_full_queue_does_not_stop_other_threads(api):
    """A launch blocks while the stream's queue is full (some 1000 launches, here behind a kernel of about half a second):
    another Python thread goes on meanwhile."""
    d = _cuda(synthetic.decode_inputs(1, 1, 1, 1, 64, seed=1))
    x = torch.randn(8, 64, device="cuda").bfloat16()
    calls = [lambda: api.fused_gdn_gating(d["A_log"], d["dt_bias"], d["a"], d["b"]), lambda: api.gated_rmsnorm(x, x, x[0]),
             lambda: api.recurrent_forward(d["q"], d["k"], d["v"], d["state"], d["b"]),
             lambda: api.causal_conv1d(x[None], x[:4].T.contiguous()),
             lambda: api.chunked_forward(d["q"], d["k"], d["v"], d["b"], None)]
    for call in calls:
        call()
        torch.cuda.synchronize()
        beats, done = [], threading.Event()

        def beat():
            while not done.is_set():
                beats.append(time.perf_counter())
                time.sleep(0.002)
        t = threading.Thread(target=beat)
        t.start()
        torch.cuda._sleep(900_000_000)
        t0, longest = time.perf_counter(), 0.0
        for _ in range(2500):
            t1 = time.perf_counter()
            call()
            longest = max(longest, time.perf_counter() - t1)
        t1 = time.perf_counter()
        done.set()
        t.join()
        torch.cuda.synchronize()
        during = [t0] + [b for b in beats if t0 <= b <= t1] + [t1]
        assert longest > 0.1, "no launch had to wait"
        assert max(b - a for a, b in zip(during, during[1:])) < longest / 2


def test_counts_and_modes_as_int_takes_them(api):
    v = _cuda(synthetic.varlen_inputs([70, 5], 1, 1, 64, seed=3))
    args = (v["q"], v["k"], v["v"], v["beta"], v["g"], None, None, v["cu_seqlens"], v["chunk_indices"], v["cu_chunks"])
    ref = api.chunked_forward(*args, v["total_chunks"])
    for chunks in (float(v["total_chunks"]), torch.tensor(v["total_chunks"]), torch.tensor(float(v["total_chunks"]), device="cuda")):
        assert torch.equal(api.chunked_forward(*args, chunks)[0], ref[0])
    d = _cuda(synthetic.decode_inputs(1, 2, 1, 1, 64, seed=1))
    for mode in (2.0, torch.tensor(2), api.SpecVerify):
        assert api.recurrent_forward(d["q"], d["k"], d["v"], d["state"], d["b"], inference_mode=mode)[1].dim() == 5


@pytest.mark.parametrize("front", ["extension", "ctypes"])
@pytest.mark.parametrize("B,T,kh,vh", [(1, 2500, 2, 4), (1, 7919, 2, 8)])
def test_given_workspace_with_room_for_fewer_segments(api, monkeypatch, front, B, T, kh, vh):
    """Few chains ask for more scratch than their longer segments did: a buffer laid out for those is used (fewer segments, other roundings of the
    state between them), not passed over for a new one of the full size; below what the call can do with, one is allocated."""
    if front == "ctypes":
        monkeypatch.setattr(api, "_ext", False)
    p = _cuda(synthetic.prefill_inputs(B, T, kh, vh, 128, seed=T, mild_gate=True))
    run = lambda ws: api.chunked_forward(p["q"], p["k"], p["v"], p["beta"], p["g"], None, p["state"], _workspace=ws)
    full = api.chunked_forward_workspace_bytes(B, T, vh, num_k_heads=kh)
    ref = [t.float() for t in run(None)]
    unit = B * vh * 3 * 128 * 128 * 4
    base = B * ((T + 63) // 64) * (vh * 24576 + kh * 512)
    for n, used in ((full, True), (full - unit, True), (base // 2, False)):
        ws = torch.full((n,), 255, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        before = torch.cuda.memory_stats()["allocated_bytes.all.allocated"]
        got = run(ws)
        grown = torch.cuda.memory_stats()["allocated_bytes.all.allocated"] - before
        assert (grown < base // 2 + sum(t.nbytes for t in got)) == used
        assert bool((ws != 255).any()) == used
        for x, y in zip(ref, got):
            assert torch.isfinite(y.float()).all() and ((x - y.float()).norm() / x.norm()).item() <= 1e-2
