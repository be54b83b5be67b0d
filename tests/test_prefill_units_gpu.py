"""The chunk-parallel prefill kernel works out the coordinates of its work units 64 per CTA at a time.  Exactly that
many (74 sequences x 8 chunks x 32 k-heads on 296 CTAs), one more for most CTAs (75 sequences), and a table filled five times
(300 sequences, 260 units each): every sequence must come out with the bits it has in a call of its own.  Padded, and packed with
ragged lengths."""
import pytest
import torch

from h100_gdn_cuda_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [74, 75, 300])
@pytest.mark.parametrize("packed", [False, True])
def test_more_units_than_one_table(packed, B):
    import h100_gdn_cuda_b200 as gdn
    T, H, d = 512, 32, 16
    g = torch.Generator(device="cuda").manual_seed(3)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k = (torch.nn.functional.normalize(r(B * T, H, d), dim=-1).bfloat16() for _ in range(2))
    v, beta = r(B * T, H, d).bfloat16(), torch.sigmoid(r(B * T, H)).bfloat16()
    gate, s0 = -torch.nn.functional.softplus(r(B * T, H)), (r(B, H, d, d) * 0.02).bfloat16()
    if packed:
        lens = [T - 1 if i % 2 else T + 1 for i in range(B - B % 2)] + [T] * (B % 2)  # 8 and 9 chunks
        cu = [0]
        for n in lens:
            cu.append(cu[-1] + n)
        meta = [torch.tensor(x, dtype=torch.int32, device="cuda")
                for x in (cu, synthetic.prepare_chunk_indices(cu), synthetic.prepare_cu_chunks(cu))]
        o, s = gdn.chunked_forward(q, k, v, beta, gate, None, s0, *meta)
    else:
        cu = [i * T for i in range(B + 1)]
        x4 = lambda x: x.view(B, T, *x.shape[1:])
        o, s = gdn.chunked_forward(x4(q), x4(k), x4(v), x4(beta), x4(gate), None, s0)
        o = o.view(B * T, H, d)
    for i in (0, 1, B // 2, B - 10, B - 3, B - 1):
        sl = slice(cu[i], cu[i + 1])
        oi, si = gdn.chunked_forward(q[None, sl], k[None, sl], v[None, sl], beta[None, sl], gate[None, sl], None, s0[i:i + 1])
        assert torch.equal(oi[0], o[sl]) and torch.equal(si[0], s[i])


@pytest.mark.parametrize("norm", [False, True])
def test_chunk_entries_without_tokens(norm):
    """chunk_indices may hold entries that name no token (a chunk for an empty sequence, counted in cu_chunks; chunks past a
    sequence's end behind the last one, as a caller with buffers of a fixed size has them): the bits of the exact lists."""
    import h100_gdn_cuda_b200 as gdn
    lens = [70, 0, 130, 0, 1]
    p = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in synthetic.varlen_inputs(lens, 2, 4, 128, seed=4, mild_gate=True).items()}
    args = (p["q"], p["k"], p["v"], p["beta"], p["g"], None, p["state"], p["cu_seqlens"])
    o_ref, s_ref = gdn.chunked_forward(*args, p["chunk_indices"], p["cu_chunks"], is_qk_norm=norm)
    ci = [0, 0, 0, 1, 1, 0, 2, 0, 2, 1, 2, 2, 3, 0, 4, 0] + [4, 1, 3, 0, 0, 2]
    cc = [0, 2, 3, 6, 7, 8]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    o, s = gdn.chunked_forward(*args, i32(ci), i32(cc), is_qk_norm=norm)
    assert torch.equal(o, o_ref) and torch.equal(s, s_ref)


def test_segmented_launches_without_a_second_segment():
    """chunk_indices padded to a fixed number of chunks: the segment plan is made for that number, and no sequence is longer
    than one segment.  The output launch must still find the chunk-parallel kernel's blocks complete: the bits of the exact
    lists (one segment per sequence is the unsegmented run)."""
    import h100_gdn_cuda_b200 as gdn
    lens = [1100, 700]
    p = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in synthetic.varlen_inputs(lens, 2, 4, 128, seed=6, mild_gate=True).items()}
    args = (p["q"], p["k"], p["v"], p["beta"], p["g"], None, p["state"], p["cu_seqlens"])
    o_ref, s_ref = gdn.chunked_forward(*args, p["chunk_indices"], p["cu_chunks"])
    ci = torch.zeros(4096, 2, dtype=torch.int32, device="cuda")  # the surplus entries repeat the first chunk
    ci[:p["total_chunks"]] = p["chunk_indices"].view(-1, 2)
    for _ in range(20):
        o, s = gdn.chunked_forward(*args, ci.flatten(), p["cu_chunks"])
        assert torch.equal(o, o_ref) and torch.equal(s, s_ref)


@pytest.mark.parametrize("lens,kh,vh", [([70, 130, 40], 2, 4), ([1, 64, 1], 1, 3), ([2100, 1500, 900], 1, 2)])  # the last in segments
@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("what", ["q", "k", "v"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_undefined_values_of_a_neighbour(lens, kh, vh, norm, what, bad):
    """a packed sequence whose inputs are not finite: the sequences before and behind it keep their bits"""
    import h100_gdn_cuda_b200 as gdn
    p = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in synthetic.varlen_inputs(lens, kh, vh, 128, seed=4, mild_gate=True).items()}
    run = lambda: gdn.chunked_forward(p["q"], p["k"], p["v"], p["beta"], p["g"], None, p["state"], p["cu_seqlens"], p["chunk_indices"],
                                      p["cu_chunks"], is_qk_norm=norm)
    o0, s0 = run()
    a, b = lens[0], lens[0] + lens[1]
    p[what] = p[what].clone()
    p[what][a:b] = bad
    o1, s1 = run()
    assert torch.equal(o0[:a], o1[:a]) and torch.equal(s0[0], s1[0])
    assert torch.equal(o0[b:], o1[b:]) and torch.equal(s0[2], s1[2])


@pytest.mark.parametrize("what", ["k", "v"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_undefined_values_of_a_neighbour_stage_by_stage(what, bad):
    """the same for the stage kernels of the low-level functions"""
    import h100_gdn_cuda_b200 as gdn
    from h100_gdn_cuda_b200 import api
    lens, vh, d = [70, 130, 40], 4, 128
    p = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in synthetic.varlen_inputs(lens, 2, vh, d, seed=4, mild_gate=True).items()}
    n, nc, cu, ci, cc = sum(lens), p["total_chunks"], p["cu_seqlens"], p["chunk_indices"], p["cu_chunks"]
    gate = api._chunk_local_cumsum_f32(p["g"], 1, n, vh, cu, ci)

    def run():
        new = lambda *s: torch.zeros(*s, device="cuda", dtype=torch.bfloat16)
        u, w, h, fin, o = new(n, vh, d), new(n, vh, d), new(nc, vh, d, d), new(3, vh, d, d), new(n, vh, d)
        gdn.bf16_gdn_compute_u_w(p["k"], p["v"], u, w, p["beta"], gate, cu_seqlens=cu, chunk_indices=ci)
        u_new = u.clone()
        gdn.bf16_chunked_seq_state_update(p["k"], u_new, w, p["state"], h, fin, gate, cu_seqlens=cu, cu_chunks=cc, total_chunks=nc)
        gdn.bf16_gdn_chunked_compute_O(p["q"], h, p["k"], u_new, o, gate, cu_seqlens=cu, chunk_indices=ci, cu_chunks=cc)
        own = lambda x, a, b: torch.cat([x[:a], x[b:]])
        a, b = cc[1].item(), cc[2].item()
        return [own(x, lens[0], lens[0] + lens[1]) for x in (u, w, u_new, o)] + [own(h, a, b), own(fin, 1, 2)]

    ref = run()
    p[what] = p[what].clone()
    p[what][lens[0]:lens[0] + lens[1]] = bad
    assert all(torch.equal(x, y) for x, y in zip(run(), ref))


def test_packed_calls_back_to_back():
    """Small packed batches whose calls follow one another without a pause: their blocks stay in L2, and the state kernel's warps can run
    a whole chunk ahead of those that write the outputs.  No wait may run out (the status word), and every call has the bits of the first."""
    import ctypes as C
    import h100_gdn_cuda_b200 as gdn
    from h100_gdn_cuda_b200 import _cabi
    lens = [700, 70, 300, 64, 1, 900, 130, 33] * 4
    p = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in synthetic.varlen_inputs(lens, 4, 8, 128, seed=8, mild_gate=True).items()}
    run = lambda: gdn.chunked_forward(p["q"], p["k"], p["v"], p["beta"], p["g"], None, p["state"], p["cu_seqlens"], p["chunk_indices"], p["cu_chunks"])
    st = C.c_int(-1)
    assert _cabi.load().gdn_device_status(0, C.byref(st)) == 0
    o0, s0 = run()
    differ = torch.zeros((), dtype=torch.int64, device="cuda")
    for _ in range(30):
        outs = [run() for _ in range(10)]
        for o, s in outs:
            differ += (o != o0).sum() + (s != s0).sum()
    assert differ.item() == 0
    assert _cabi.load().gdn_device_status(0, C.byref(st)) == 0 and st.value == 0


# segments of 5 chunks and more, first ones walked outright: sequences of one segment (empty, at the front), of two, of many, ragged ends;
# and long ones, whose first segments are found like the others
@pytest.mark.parametrize("lens,kh,vh,norm", [([3000], 1, 2, False), ([100, 3840, 2883, 1920], 1, 1, True), ([0, 6400, 5000, 0], 1, 1, False),
                                             ([64 * 36], 2, 4, False), ([64 * 40, 64 * 41 + 1], 1, 3, True), ([700, 9000, 700], 1, 2, False),
                                             ([42000], 1, 1, False)])
@pytest.mark.parametrize("state", [False, True])
def test_short_segments_back_to_back(lens, kh, vh, norm, state):
    """against the oracle, and calls that follow one another without a pause, each from the states of the one before: what a launch
    leaves for the next must be complete, whichever of them run side by side"""
    import h100_gdn_cuda_b200 as gdn
    from oracle import gdn_oracle as O
    p = synthetic.varlen_inputs(lens, kh, vh, 128, seed=sum(lens), mild_gate=True, normalize=not norm)
    s0 = p["state"] if state else None
    o_ref, s_ref = O.recurrent_ref(*(p[k].float() for k in ("q", "k", "v", "beta")), p["g"], s0.float() if state else None,
                                   cu_seqlens=p["cu_seqlens"], is_qk_norm=norm)
    c = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in p.items()}
    run = lambda s: gdn.chunked_forward(c["q"], c["k"], c["v"], c["beta"], c["g"], None, s, c["cu_seqlens"], c["chunk_indices"], c["cu_chunks"],
                                        c["total_chunks"], is_qk_norm=norm)
    o, s = run(c["state"] if state else None)
    for x, ref in ((o, o_ref), (s, s_ref)):
        assert O.rel_fro(x.float().cpu(), ref) <= 1e-2 and O.max_abs_over_max(x.float().cpu(), ref) <= 5e-2

    def chain(sync):
        x, outs = s, []
        for _ in range(12):
            y, x = run(x)
            outs.append(y)
            if sync:
                torch.cuda.synchronize()
        return outs, x

    a, b = chain(True), chain(False)
    assert torch.equal(a[1], b[1]) and all(torch.equal(x, y) for x, y in zip(a[0], b[0]))


# padded short segments: 4 to 8 chains of 34 to 47 chunks, ragged ends, head dims below 128, two sequences
PADDED = [(1, 2500, 2, 4, 128, False), (1, 2177, 4, 8, 64, True), (2, 2200, 1, 2, 96, False), (1, 3008, 2, 4, 40, True), (3, 2176, 1, 1, 128, True)]


@pytest.mark.parametrize("B,T,kh,vh,d,norm", PADDED)
@pytest.mark.parametrize("state", [False, True])
def test_padded_short_segments(B, T, kh, vh, d, norm, state):
    """against the oracle, and cut it is: the scratch has room for the segments' states"""
    import h100_gdn_cuda_b200 as gdn
    from h100_gdn_cuda_b200 import api
    from oracle import gdn_oracle as O
    assert api.chunked_forward_workspace_bytes(B, T, vh, num_k_heads=kh) > B * ((T + 63) // 64) * (vh * 24576 + kh * 512) + 3 * B * vh * 196608
    p = synthetic.prefill_inputs(B, T, kh, vh, d, seed=T + d, mild_gate=True)
    if norm:
        p["q"], p["k"] = (3 * p["q"].float()).bfloat16(), (0.2 * p["k"].float()).bfloat16()
    s0 = p["state"] if state else None
    o_ref, s_ref = O.recurrent_ref(*(p[k].float() for k in ("q", "k", "v", "beta")), p["g"], s0.float() if state else None, is_qk_norm=norm)
    c = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in p.items()}
    o, s = gdn.chunked_forward(c["q"], c["k"], c["v"], c["beta"], c["g"], None, c["state"] if state else None, is_qk_norm=norm)
    for x, ref in ((o, o_ref), (s, s_ref)):
        assert O.rel_fro(x.float().cpu(), ref) <= 1e-2 and O.max_abs_over_max(x.float().cpu(), ref) <= 5e-2


@pytest.mark.parametrize("B,T,kh,vh,d,norm", PADDED[:3])
def test_short_segments_in_a_graph(B, T, kh, vh, d, norm):
    """The five launches of the call, three of which run beside the one before, recorded and replayed without a pause: the bits of a call
    by itself, also after other inputs have been copied into the buffers."""
    import h100_gdn_cuda_b200 as gdn
    ps = [{k: (v.cuda() if torch.is_tensor(v) else v) for k, v in synthetic.prefill_inputs(B, T, kh, vh, d, seed=s, mild_gate=True).items()} for s in (1, 2)]
    run = lambda p: gdn.chunked_forward(p["q"], p["k"], p["v"], p["beta"], p["g"], None, p["state"], is_qk_norm=norm)
    refs = [run(p) for p in ps]
    buf = {k: (v.clone() if torch.is_tensor(v) else v) for k, v in ps[0].items()}
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        o, s = run(buf)
    for i in (0, 1, 0):
        for k, v in ps[i].items():
            if torch.is_tensor(v):
                buf[k].copy_(v)
        o.zero_(), s.zero_()
        for _ in range(5):
            graph.replay()
        assert torch.equal(o, refs[i][0]) and torch.equal(s, refs[i][1])


@pytest.mark.parametrize("B,T,kh,vh,d,norm", PADDED[:3])
def test_short_segments_final_state_over_the_initial_one(B, T, kh, vh, d, norm):
    """the first segments read the state that the last ones write, in another launch"""
    import ctypes as C
    from h100_gdn_cuda_b200 import _cabi as cabi, api
    p = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in synthetic.prefill_inputs(B, T, kh, vh, d, seed=5, mild_gate=True).items()}
    lib, outs = cabi.load(), []
    n = api.chunked_forward_workspace_bytes(B, T, vh, num_k_heads=kh)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    for over in (False, True):
        s0 = p["state"].clone()
        out, final = torch.empty_like(p["v"]), s0 if over else torch.empty_like(s0)
        a = cabi.ChunkedArgs(api._shape(B, T, B * T, kh, vh, d, d), *(api._token_tensor(t, False) for t in (p["q"], p["k"], p["v"], out)),
                             api._token_scalar(p["beta"], False), api._token_scalar(p["g"], False), api._state_desc(s0), api._state_desc(final),
                             d ** -0.5, ws.data_ptr(), n, None, int(norm))
        assert lib.gdn_chunked_forward(C.byref(a), torch.cuda.current_stream().cuda_stream) == 0, lib.gdn_last_error()
        outs.append((out, final))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
