"""The workspace-free prefill entry point (gdn_chunked_forward_static_scratch).

Some callers of the library cannot hand it a workspace because they may not allocate device
memory when the call happens (all HBM already given to their own pool, or cudaMalloc ruled
out on their path because it synchronises the device).  For them the library keeps the U/W
scratch of chunked prefill in a fixed array inside its own image.  This test drives that
entry point through the C ABI, twice in a row on different problems (the array is shared
and keeps the previous call's contents), and requires the same bits as the regular entry
point given a caller-provided workspace.  It also checks that a problem beyond the array's
stated limit is refused.  The file name makes pytest collect it last.
"""
import ctypes as C

import pytest
import torch

from h100_gdn_cuda_b200 import synthetic

pytestmark = pytest.mark.gpu


def _args(api, cabi, p, out, final, ws, ws_bytes):
    q, k, v = p["q"], p["k"], p["v"]
    B, T, kh, d = q.shape
    vh = v.shape[2]
    shape = api._shape(B, T, B * T, kh, vh, d, d)
    return cabi.ChunkedArgs(shape, api._token_tensor(q, False), api._token_tensor(k, False),
                            api._token_tensor(v, False), api._token_tensor(out, False),
                            api._token_scalar(p["beta"], False), api._token_scalar(p["g"], False),
                            api._state_desc(p["state"]), api._state_desc(final), float(d) ** -0.5,
                            ws, ws_bytes, None)


def test_static_scratch_matches_workspace_path_twice():
    from h100_gdn_cuda_b200 import _cabi as cabi, api, build
    build.build()
    lib = cabi.load()
    stream = torch.cuda.current_stream().cuda_stream
    # two calls in a row, the second smaller than the first so stale scratch lies beyond it
    for (B, T, kh, vh, seed) in ((2, 300, 2, 4, 5), (1, 130, 2, 4, 6)):
        p = {k: (v.cuda() if torch.is_tensor(v) else v)
             for k, v in synthetic.prefill_inputs(B, T, kh, vh, 128, seed=seed, mild_gate=True).items()}
        outs = []
        for static in (False, True):
            out = torch.full_like(p["v"], float("nan"))
            final = torch.full_like(p["state"], float("nan"))
            if static:
                a = _args(api, cabi, p, out, final, None, 0)
                rc = lib.gdn_chunked_forward_static_scratch(C.byref(a), stream)
            else:
                n = lib.gdn_chunked_forward_workspace_bytes(C.byref(api._shape(B, T, B * T, kh, vh, 128, 128)))
                ws = torch.empty(n, dtype=torch.uint8, device="cuda")
                a = _args(api, cabi, p, out, final, ws.data_ptr(), n)
                rc = lib.gdn_chunked_forward(C.byref(a), stream)
            assert rc == 0, lib.gdn_last_error()
            torch.cuda.synchronize()
            outs.append((out, final))
        (o_ws, s_ws), (o_st, s_st) = outs
        assert torch.isfinite(o_st.float()).all() and torch.isfinite(s_st.float()).all()
        # same kernels, same inputs: the tolerance of the prefill tests (1e-2 relative
        # Frobenius) is met with zero difference
        assert torch.equal(o_st, o_ws) and torch.equal(s_st, s_ws)


def test_static_scratch_refuses_oversize():
    from h100_gdn_cuda_b200 import _cabi as cabi, api, build
    build.build()
    lib = cabi.load()
    # 4097 tokens x 32 heads is one token over the limit; validation precedes any device work
    shape = api._shape(1, 4097, 4097, 16, 32, 128, 128)
    a = cabi.ChunkedArgs()
    a.shape = shape
    rc = lib.gdn_chunked_forward_static_scratch(C.byref(a), None)
    assert rc == -4 and b"built-in" in lib.gdn_last_error()


def test_static_scratch_runs_in_the_segments_that_fit():
    """2 v-heads of 50048 tokens: the states of 31 segments on top of the blocks do not fit the array, those of 29 do.  Other
    segments, other roundings of the state between them: both within the prefill tests' tolerance of each other."""
    from h100_gdn_cuda_b200 import _cabi as cabi, api, build
    build.build()
    lib = cabi.load()
    stream = torch.cuda.current_stream().cuda_stream
    B, T, vh, d = 1, 50048, 2, 128
    n = lib.gdn_chunked_forward_workspace_bytes(C.byref(api._shape(B, T, B * T, vh, vh, d, d)))
    assert n > (49 << 20) + 8704
    p = {k: (v.cuda() if torch.is_tensor(v) else v)
         for k, v in synthetic.prefill_inputs(B, T, vh, vh, d, seed=8, mild_gate=True).items()}
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    outs = []
    for fn, args in ((lib.gdn_chunked_forward, (ws.data_ptr(), n)), (lib.gdn_chunked_forward_static_scratch, (None, 0))):
        out, final = torch.full_like(p["v"], float("nan")), torch.full_like(p["state"], float("nan"))
        assert fn(C.byref(_args(api, cabi, p, out, final, *args)), stream) == 0, lib.gdn_last_error()
        torch.cuda.synchronize()
        outs.append((out.float(), final.float()))
    for a, b in zip(*outs):
        assert torch.isfinite(b).all() and ((a - b).norm() / a.norm()).item() <= 1e-2


def test_static_scratch_wide_heads_need_none():
    """Head dims 192 and 256 run without scratch, so the size of the array is no limit for them (65536 tokens x v-heads
    here; in blocks of 256 columns it would hold some 40000)."""
    from h100_gdn_cuda_b200 import _cabi as cabi, api, build
    build.build()
    lib = cabi.load()
    stream = torch.cuda.current_stream().cuda_stream
    B, T, kh, vh, d = 1, 2048, 16, 32, 256
    assert lib.gdn_chunked_forward_workspace_bytes(C.byref(api._shape(B, T, B * T, kh, vh, d, d))) == 0
    p = {k: (v.cuda() if torch.is_tensor(v) else v)
         for k, v in synthetic.prefill_inputs(B, T, kh, vh, d, seed=7, mild_gate=True).items()}
    outs = []
    for fn in (lib.gdn_chunked_forward, lib.gdn_chunked_forward_static_scratch):
        out, final = torch.full_like(p["v"], float("nan")), torch.full_like(p["state"], float("nan"))
        rc = fn(C.byref(_args(api, cabi, p, out, final, None, 0)), stream)
        assert rc == 0, lib.gdn_last_error()
        torch.cuda.synchronize()
        outs.append((out, final))
    assert torch.isfinite(outs[1][0].float()).all() and torch.isfinite(outs[1][1].float()).all()
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("B,T,kh,vh", [(1, 2500, 2, 4), (1, 5000, 8, 16), (2, 3000, 1, 2)])
def test_scratch_of_a_longer_plan_is_enough(B, T, kh, vh):
    """Scratch that has no room for all the segments a few short sequences would be cut into, down to none of them: fewer segments, the
    same results but for the rounding; below that the call is refused."""
    from h100_gdn_cuda_b200 import _cabi as cabi, api, build
    build.build()
    lib = cabi.load()
    p = {k: (v.cuda() if torch.is_tensor(v) else v)
         for k, v in synthetic.prefill_inputs(B, T, kh, vh, 128, seed=T, mild_gate=True).items()}
    full = lib.gdn_chunked_forward_workspace_bytes(C.byref(api._shape(B, T, B * T, kh, vh, 128, 128)))
    chunks, segment = B * ((T + 63) // 64), B * vh * 3 * 128 * 128 * 4
    base = (chunks * vh * 24576 + 255) // 256 * 256 + (chunks * kh * 512 + 255) // 256 * 256 + 256
    assert full >= base + 3 * segment
    ref = None
    for n in (full, full - segment, base + 2 * segment, base, base - 1):
        ws = torch.full((n,), 255, dtype=torch.uint8, device="cuda")
        out, final = torch.full_like(p["v"], float("nan")), torch.full_like(p["state"], float("nan"))
        rc = lib.gdn_chunked_forward(C.byref(_args(api, cabi, p, out, final, ws.data_ptr(), n)), torch.cuda.current_stream().cuda_stream)
        if n < base:
            assert rc == -4
            continue
        assert rc == 0, lib.gdn_last_error()
        torch.cuda.synchronize()
        got = (out.float(), final.float())
        ref = ref or got
        for x, y in zip(ref, got):
            assert torch.isfinite(y).all() and ((x - y).norm() / x.norm()).item() <= 1e-2
