// State propagation + output of chunked Gated DeltaNet prefill for head dims 129 .. 256, on 256 columns.
// The recurrence is that of gdn_fused_seq_kernel (prefill_fused.cuh):
//     R  = V - e^{g} .* (K S^T)
//     O  = scale * e^{g} .* (Q S^T) + PT R
//     S <- e^{g_L} S + R^T Z
// with Z and PT from gdn_zp_kernel<., true> (prefill_zp.cuh).  The rows of S (value columns) are independent of one
// another, so one CTA walks the chunks of one (sequence, v-head, half of the value columns): 128 rows
// x 256 columns of state, 128 fp32 values in each thread of the eight state warps.  Four output warps, a producer, one warp that issues the
// MMAs, and two idle ones that only give their registers to the state warps (setmaxnreg).
//
// Arithmetic.  These head dims used to run on the fp32 token recurrence, so nothing here may be coarser than fp32
// accumulation of near-fp32 operands: S, R, Z and PT are sums of two bf16 terms (hi + lo, 16 significand bits), K, Q
// and V are the caller's bf16 values:
//     S K = S_hi K + S_lo K,   R Z = R_hi Z_hi + R_hi Z_lo + R_lo Z_hi   (S Q and R PT the same way).
// Two to three times the MMAs of plain bf16, which a chain that waits on latency has room for.
//
// Tensor memory (all 512 columns): S_hi 128 | S_lo 128 | D1 = S K^T 64, its halves overwritten by R_hi, R_lo | O1 =
// S Q^T, later O2 = R PT^T 64 | dS 2 x 64.  dS has 256 columns; it comes in four quarters through two buffers (one per
// half of the state warps), so that the MMAs of one quarter run while another is being read.  (Eighths through four
// buffers were slower, 5.1 against 4.5 us a chunk: MMAs of 32 columns last no longer than their issue takes.)
// Shared memory: one buffer per operand (K, V, Q, Z hi/lo, PT hi/lo), each refilled as soon as its MMAs or its readers
// are done, a good part of a chunk before it is needed again (K, V after R, Q after O1, Z and PT after O2).
//
// What bounds it: the chain S -> D1 -> R -> dS -> S of each CTA, 8 500 cycles a chunk (D1 1 300 and dS 3 000 of them with
// the state passes between the quarters, R 1 200); the MMAs alone are 4 000.  B=2, T=1500, 8 v-heads, d=256 (32 CTAs of
// 24 chunks): 104 us after 34 us of gdn_zp_kernel (121 us together, the set-up overlapped), where the token recurrence took
// 1 006 us; same error against fp32.
#pragma once
#include <cuda.h>

#include "prefill_common.cuh"
#include "prefill_fused.cuh"

namespace gdn {

struct WideSmem {
    static constexpr int kTile = kChunk * 256 * 2;  // 32 KB: K, Q, or one term of Z
    static constexpr int kOffK = 0, kOffQ = kTile, kOffZ = 2 * kTile, kOffPT = 4 * kTile;
    static constexpr int kOffV = kOffPT + 2 * 8192;      // 64 x 128 (this CTA's value columns)
    static constexpr int kOffO1 = kOffV + 16384;         // fp32 scale e^g O1 of the chunk, 64 tokens x 128 rows
    static constexpr int kOffO = kOffO1 + 32768;         // output staging tile
    static constexpr int kOffGate = kOffO + 16384;       // 3 x { scale e^g[64], -e^g[64], e^{gL} }
    static constexpr int kGateStride = FusedSmem::kGateStride;
    static constexpr int kOffBar = kOffGate + 3 * kGateStride;
    static constexpr int kBytes = kOffBar + 192 + 1024;
    static_assert(kOffPT - kOffZ == 2 * kTile && kWideBlockBytes == 2 * kTile + 2 * 8192, "one bulk copy fills Z and PT");
    static_assert(kBytes <= 227 * 1024, "shared memory of one CTA");
};

namespace wide {
constexpr int kThreads = 512;
constexpr uint32_t kTmS = 0;      // bf16 S_hi, then S_lo, 128 columns each
constexpr uint32_t kTmX = 256;    // fp32 D1 (columns 32 hf .. + 31 belong to tokens 32 hf ..), then for each 16 tokens R_hi [8], R_lo [8]
constexpr uint32_t kTmO = 320;    // fp32 O1, then O2
constexpr uint32_t kTmDS = 384;   // two buffers of 64 columns: quarters 0, 1 of dS in the first, 2, 3 in the second
}  // namespace wide

__global__ void __launch_bounds__(wide::kThreads, 1)
    gdn_wide_seq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                        const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO,
                        const FusedParams p) {
    using namespace ptx;
    using namespace wide;
    using fused::reg_inc; using fused::reg_dec; using fused::named_bar_sync; using fused::f2; using fused::pk; using fused::unpk;
    using fused::fma2;
    using L = WideSmem;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (ptx::smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
    uint64_t* bar_kv = bars;          // K, V and the gate vectors of a chunk are there
    uint64_t* bar_q = bars + 1;       // Q
    uint64_t* bar_z = bars + 2;       // Z, PT
    uint64_t* bar_s = bars + 3;       // S published (8 warps)
    uint64_t* bar_d1 = bars + 4;
    uint64_t* bar_r = bars + 5;       // R published, V read (8 warps)
    uint64_t* bar_ds = bars + 6;       // [2] a quarter of dS is ready, one barrier per half of the state warps
    uint64_t* bar_dsfree = bars + 8;   // [2] the first quarter has been read (4 warps)
    uint64_t* bar_o1 = bars + 14;      // O1 done (and Q read)
    uint64_t* bar_o1free = bars + 15;  // O1 read (4 warps)
    uint64_t* bar_o2 = bars + 16;      // O2 done (and Z, PT, R read)
    uint64_t* bar_o2free = bars + 17;  // O2 read (4 warps)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
    int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // grid = (sequences, 2 x heads), or (2 x heads, ranks) with seq_order
    const int hh = static_cast<int>(p.seq_order ? blockIdx.x : blockIdx.y);
    const int seq = p.seq_order ? p.seq_order[blockIdx.y] : static_cast<int>(blockIdx.x);
    const int head = hh >> 1, dv0 = (hh & 1) * 128;
    const int khead = head / (p.vh / p.kh);
    int batch, gchunk0;
    long long seq_tok0, seq_tokens;
    if (p.map.cu_seqlens) {
        const int bos = p.map.cu_seqlens[seq], eos = p.map.cu_seqlens[seq + 1];
        seq_tok0 = bos;
        seq_tokens = eos - bos;
        batch = 0;
        gchunk0 = p.map.cu_chunks[seq];
    } else {
        seq_tok0 = 0;
        seq_tokens = p.map.seq_len;
        batch = seq;
        gchunk0 = seq * p.map.chunks_per_seq;
    }
    const int nchunks = static_cast<int>((seq_tokens + kChunk - 1) / kChunk);
    auto chunk_n = [&](int c) {
        const long long rem = seq_tokens - static_cast<long long>(c) * kChunk;
        return rem < kChunk ? static_cast<int>(rem) : kChunk;
    };
    auto gate_buf = [&](int c) { return reinterpret_cast<float*>(smem + L::kOffGate + (c % 3) * L::kGateStride); };

    if (tid == 0) {
        *abort_flag = 0;
        mbar_init(bar_kv, 1);
        mbar_init(bar_q, 1);
        mbar_init(bar_z, 1);
        mbar_init(bar_s, 8);
        mbar_init(bar_d1, 1);
        mbar_init(bar_r, 8);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bar_ds[i], 1);
            mbar_init(&bar_dsfree[i], 4);
        }
        mbar_init(bar_o1, 1);
        mbar_init(bar_o1free, 4);
        mbar_init(bar_o2, 1);
        mbar_init(bar_o2free, 4);
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(tmem_slot, 512);
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;

    if (warp < 8) {
        // =============================================================== state warps
        // setmaxnreg moves registers inside what the CTA was launched with (512 threads x 128): more would wait for ever
        static_assert(8 * 184 + 4 * 88 + 4 * 56 <= 16 * 128, "register pool of the CTA");
        reg_inc<184>();
        const int lq = warp & 3, hf = warp >> 2;
        const int row = 32 * lq + lane;
        const uint32_t tm_lane = static_cast<uint32_t>(32 * lq) << 16;
        const uint32_t tS = tmem + kTmS + tm_lane + 64 * hf;  // this thread's 128 columns: 64 words of S_hi; S_lo 128 columns on
        // element (token i, this row) of the swizzled V tile: i * 128 + ((i & 7) << 4 ^ vx)
        const uint8_t* const sV = smem + L::kOffV + (row >> 6) * 8192 + (row & 7) * 2;
        const uint32_t vx = static_cast<uint32_t>((row & 63) >> 3) << 4;
        const bool row_ok = dv0 + row < p.d;
        float S[128];
        // 16 columns of S -> their two bf16 terms in tensor memory (the operand of the next chunk's MMAs)
        auto publish16 = [&](int q) {
            uint32_t h[8], l[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float a = S[16 * q + 2 * e], b = S[16 * q + 2 * e + 1];
                h[e] = pack_bf16(a, b);
                l[e] = pack_bf16(a - bf16_lo(h[e]), b - bf16_hi(h[e]));
            }
            tmem_st8(tS + 8 * q, h);
            tmem_st8(tS + 128 + 8 * q, l);
        };
        const __nv_bfloat16* src = p.state_in ? p.state_in + seq * p.si_ss + head * p.si_sh +
                                                    static_cast<long long>(dv0 + row) * p.d + 128 * hf
                                              : nullptr;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const uint4 v = (src && row_ok && 128 * hf + 8 * q < p.d) ? __ldg(reinterpret_cast<const uint4*>(src) + q)
                                                                      : make_uint4(0u, 0u, 0u, 0u);
            S[q * 8 + 0] = bf16_lo(v.x); S[q * 8 + 1] = bf16_hi(v.x);
            S[q * 8 + 2] = bf16_lo(v.y); S[q * 8 + 3] = bf16_hi(v.y);
            S[q * 8 + 4] = bf16_lo(v.z); S[q * 8 + 5] = bf16_hi(v.z);
            S[q * 8 + 6] = bf16_lo(v.w); S[q * 8 + 7] = bf16_hi(v.w);
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) publish16(q);
        tmem_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_s);

        for (int c = 0; c < nchunks; ++c) {
            const uint32_t par = static_cast<uint32_t>(c & 1);
            const int nloc = chunk_n(c) - 32 * hf;  // tokens of this half that exist
            const float* gb = gate_buf(c);
            mbar_wait(bar_kv, par, abort_flag);
            // ---- R = V^T - e^g .* (S K^T), its two terms over the columns of D1 this thread has read
            auto load_v = [&](int b, uint32_t* v8) {  // 16 tokens of this row, packed in pairs
                const uint8_t* v = sV + 4096 * hf + 2048 * b;
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const uint32_t lo = *reinterpret_cast<const uint16_t*>(v + 256 * e + (((2 * e & 7) << 4) ^ vx));
                    const uint32_t hi = *reinterpret_cast<const uint16_t*>(v + 256 * e + 128 + (((2 * e + 1 & 7) << 4) ^ vx));
                    v8[e] = lo | (hi << 16);
                }
            };
            uint32_t v8[8];
            load_v(0, v8);
            mbar_wait(bar_d1, par, abort_flag);
            tc_fence_after_sync();
            const uint32_t tX = tmem + kTmX + tm_lane + 32 * hf;
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                uint32_t r[16], h[8], l[8];
                tmem_ld16(tX + 16 * b, r);
                if (b == 1) load_v(1, v8);
                tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int i = 16 * b + 2 * e;
                    const float2 neg = *reinterpret_cast<const float2*>(gb + 64 + 32 * hf + i);  // -e^g (a broadcast)
                    float r0, r1;
                    unpk(fma2(pk(neg.x, neg.y), pk(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1])),
                              pk(bf16_lo(v8[e]), bf16_hi(v8[e]))),
                         r0, r1);
                    h[e] = pack_bf16(r0, r1);
                    l[e] = pack_bf16(r0 - bf16_lo(h[e]), r1 - bf16_hi(h[e]));
                }
                if (nloc < 32) {  // rows past the end may hold a neighbouring sequence's values (one branch for all of them)
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const int i = 16 * b + 2 * e;
                        const uint32_t keep = (i < nloc ? 0xFFFFu : 0u) | (i + 1 < nloc ? 0xFFFF0000u : 0u);
                        h[e] &= keep;
                        l[e] &= keep;
                    }
                }
                tmem_st8(tX + 16 * b, h);
                tmem_st8(tX + 16 * b + 8, l);
            }
            tmem_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_r);
            // ---- S <- e^{g_L} S + dS, a quarter (64 columns) at a time
            const f2 eg2 = pk(gb[128], gb[128]);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                mbar_wait(&bar_ds[hf], static_cast<uint32_t>(q), abort_flag);  // two phases a chunk
                tc_fence_after_sync();
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    uint32_t r[32];
                    tmem_ld32(tmem + wide::kTmDS + 64 * hf + 32 * b + tm_lane, r);
                    tmem_wait_ld();
                    if (q == 0 && b == 1) {
                        tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&bar_dsfree[hf]);
                    }
#pragma unroll
                    for (int e = 0; e < 32; e += 2) {
                        float* s2 = &S[64 * q + 32 * b + e];
                        unpk(fma2(pk(s2[0], s2[1]), eg2, pk(__uint_as_float(r[e]), __uint_as_float(r[e + 1]))), s2[0], s2[1]);
                    }
                    publish16(4 * q + 2 * b);
                    publish16(4 * q + 2 * b + 1);
                }
            }
            tmem_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_s);
        }
        // nothing is written once a wait of this CTA has given up (the results would be garbage)
        if (*abort_flag == 0 && p.state_out && row_ok) {
            uint4* d4 = reinterpret_cast<uint4*>(p.state_out + seq * p.so_ss + head * p.so_sh +
                                                 static_cast<long long>(dv0 + row) * p.d + 128 * hf);
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                if (128 * hf + 8 * q < p.d)
                    d4[q] = make_uint4(pack_bf16(S[q * 8 + 0], S[q * 8 + 1]), pack_bf16(S[q * 8 + 2], S[q * 8 + 3]),
                                       pack_bf16(S[q * 8 + 4], S[q * 8 + 5]), pack_bf16(S[q * 8 + 6], S[q * 8 + 7]));
            }
        }
    } else if (warp < 12) {
        // =============================================================== output warps
        reg_dec<88>();
        const int lq = warp & 3;
        const int row = 32 * lq + lane;
        const int otid = tid - 256;
        const uint32_t tO = tmem + kTmO + (static_cast<uint32_t>(32 * lq) << 16);
        float* const sO1 = reinterpret_cast<float*>(smem + L::kOffO1) + row;
        uint8_t* const sO = smem + L::kOffO;
        uint8_t* const sOrow = sO + (row >> 6) * 8192 + (row & 7) * 2;  // element (token i, row): i * 128 + ((i & 7) << 4 ^ ox)
        const uint32_t ox = static_cast<uint32_t>((row & 63) >> 3) << 4;
        const bool packed = p.map.cu_seqlens != nullptr;
        for (int c = 0; c < nchunks; ++c) {
            const uint32_t par = static_cast<uint32_t>(c & 1);
            const int n = chunk_n(c);
            const float* gb = gate_buf(c);
            // O1 leaves tensor memory at once: O2 uses the same columns.  (O1 was issued after the chunk's gate values
            // were complete, so they are visible here; waiting on bar_kv itself could miss a phase of it.)
            mbar_wait_relaxed<40>(bar_o1, par, abort_flag);
            tc_fence_after_sync();
            {
                uint32_t r[2][32];
                tmem_ld32(tO, r[0]);
                tmem_ld32(tO + 32, r[1]);
                tmem_wait_ld();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_o1free);
#pragma unroll
                for (int b = 0; b < 16; ++b) {
                    const float4 g = *reinterpret_cast<const float4*>(gb + 4 * b);
                    const float gv[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) sO1[(4 * b + e) * 128] = gv[e] * __uint_as_float(r[b >> 3][(4 * b + e) & 31]);
                }
            }
            if (otid == 0) bulk_wait_read<0>();  // the last chunk's store has read the staging tile
            named_bar_sync(1, 128);
            mbar_wait_relaxed<40>(bar_o2, par, abort_flag);
            tc_fence_after_sync();
            {
                uint32_t r[2][32];
                tmem_ld32(tO, r[0]);
                tmem_ld32(tO + 32, r[1]);
                tmem_wait_ld();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_o2free);  // the next O1 is waiting for these columns
#pragma unroll
                for (int b = 0; b < 8; ++b) {
                    float o1[8];  // read before the stores to the staging tile, which they might alias
#pragma unroll
                    for (int e = 0; e < 8; ++e) o1[e] = sO1[(8 * b + e) * 128];
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        *reinterpret_cast<__nv_bfloat16*>(sOrow + (8 * b + e) * 128 + ((e << 4) ^ ox)) =
                            __float2bfloat16(o1[e] + __uint_as_float(r[b >> 2][(8 * b + e) & 31]));
                }
            }
            const long long tok0 = seq_tok0 + static_cast<long long>(c) * kChunk;
            fence_proxy_async_smem();
            named_bar_sync(1, 128);
            if (*abort_flag != 0) {
                // a wait has given up: the tile is garbage and stays on chip
            } else if (!(packed && n < kChunk)) {
                if (otid == 0) {
                    for (int a = 0; a < 2; ++a)
                        if (dv0 + 64 * a < p.d) tma_store_4d(&tmO, sO + a * 8192, dv0 + 64 * a, head, static_cast<int>(tok0), batch);
                    bulk_commit();
                }
            } else {  // a full-box store would spill into the next sequence
                TokenView out = p.out;
                out.ptr += dv0;
                store_tile_rows<128>(sO, out, batch, tok0, head, n, otid, min(16, (p.d - dv0) >> 3));
            }
        }
        if (otid == 0) bulk_wait_read<0>();
    } else {
        reg_dec<56>();
    }
    if (warp == 13) {
        // =============================================================== producer
        uint32_t ra0 = 0u, ra1 = 0u;  // raw gates of the coming chunk, as bits
        auto load_raw = [&](int c) {
            ra0 = 0u;
            ra1 = 0u;
            if (p.gate.ptr && c < nchunks) {
                const long long t0 = static_cast<long long>(c) * kChunk + lane;
                if (t0 < seq_tokens) ra0 = p.gate.load_bits(batch, seq_tok0 + t0, head);
                if (t0 + 32 < seq_tokens) ra1 = p.gate.load_bits(batch, seq_tok0 + t0 + 32, head);
            }
        };
        auto token_of = [&](int c) { return static_cast<int>(seq_tok0 + static_cast<long long>(c) * kChunk); };
        auto load_q = [&](int c) {
            mbar_arrive_expect_tx_w(bar_q, L::kTile);
            for (int a = 0; a < 4; ++a) tma_load_4d_w(smem + L::kOffQ + a * 8192, &tmQ, bar_q, a * 64, khead, token_of(c), batch);
        };
        auto load_z = [&](int c) {
            mbar_arrive_expect_tx_w(bar_z, kWideBlockBytes);
            bulk_load_w(smem + L::kOffZ, p.blocks + (static_cast<size_t>(gchunk0 + c) * p.vh + head) * kWideBlockBytes, kWideBlockBytes, bar_z);
        };
        // K, V and the gate vectors of chunk c, whose raw gates are in ra0, ra1; fetches those of the next chunk
        auto load_kv = [&](int c) {
            const int n = chunk_n(c);
            float g0 = p.gate.value(ra0), g1 = p.gate.value(ra1);
            load_raw(c + 1);
            float rk0 = 1.f, rk1 = 1.f, rq0 = 1.f, rq1 = 1.f;
            if (p.norms) {
                const float* nr = p.norms + (static_cast<size_t>(gchunk0 + c) * p.kh + khead) * 128;
                rk0 = __ldg(nr + lane);
                rk1 = __ldg(nr + 32 + lane);
                rq0 = __ldg(nr + 64 + lane);
                rq1 = __ldg(nr + 96 + lane);
            }
#pragma unroll
            for (int m = 1; m < 32; m <<= 1) {
                const float y0 = __shfl_up_sync(0xffffffffu, g0, m);
                const float y1 = __shfl_up_sync(0xffffffffu, g1, m);
                if (lane >= m) {
                    g0 += y0;
                    g1 += y1;
                }
            }
            g1 += __shfl_sync(0xffffffffu, g0, 31);
            // tokens past the end carry the last valid value (their raw gate was taken as 0)
            const float g_last = __shfl_sync(0xffffffffu, (n - 1 < 32) ? g0 : g1, (n - 1) & 31);
            const float e0 = __expf(g0), e1 = __expf(g1);
            float* gb = gate_buf(c);
            gb[lane] = p.scale * e0 * rq0;
            gb[lane + 32] = p.scale * e1 * rq1;
            gb[64 + lane] = -e0 * rk0;
            gb[64 + lane + 32] = -e1 * rk1;
            if (lane == 0) gb[128] = __expf(g_last);
            __syncwarp();
            mbar_arrive_expect_tx_w(bar_kv, L::kTile + 16384);
            for (int a = 0; a < 4; ++a) tma_load_4d_w(smem + L::kOffK + a * 8192, &tmK, bar_kv, a * 64, khead, token_of(c), batch);
            for (int a = 0; a < 2; ++a) tma_load_4d_w(smem + L::kOffV + a * 8192, &tmV, bar_kv, dv0 + a * 64, head, token_of(c), batch);
        };
        load_raw(0);
        grid_dep_wait();  // from here on the chunk-parallel kernel's blocks and norm factors are read
        for (int c = 0; c < nchunks; ++c) {
            const uint32_t prev = static_cast<uint32_t>((c - 1) & 1);
            // each buffer as soon as the chunk before is done with it: Q after O1, K and V after R, Z and PT after O2
            if (c == 0) {
                load_kv(0);  // what the chain needs first
                load_q(0);
                load_z(0);
                continue;
            }
            mbar_wait_relaxed<40>(bar_o1, prev, abort_flag);
            load_q(c);
            mbar_wait_relaxed<40>(bar_r, prev, abort_flag);
            load_kv(c);
            mbar_wait_relaxed<40>(bar_o2, prev, abort_flag);
            load_z(c);
        }
    } else if (warp == 12) {
        // =============================================================== MMA issuer (the whole warp, one elected lane issues)
        constexpr uint32_t id_sq = make_idesc_bf16(128, 64, false, false);
        constexpr uint32_t id_ds = make_idesc_bf16(128, 64, false, true);
        const uint64_t dK = make_smem_desc_sw128(smem_u32(smem + L::kOffK), 0, 1024);     // K-major B
        const uint64_t dQ = make_smem_desc_sw128(smem_u32(smem + L::kOffQ), 0, 1024);     // K-major B
        const uint64_t dZ = make_smem_desc_sw128(smem_u32(smem + L::kOffZ), 8192, 1024);  // MN-major B
        const uint64_t dP = make_smem_desc_sw128(smem_u32(smem + L::kOffPT), 0, 1024);    // K-major B
        const uint32_t tS = tmem + kTmS, tX = tmem + kTmX, tO = tmem + kTmO;
        // S (both terms) times a 64 x 256 K-major tile
        auto mma_s = [&](uint32_t d, uint64_t b) {
            mma_ts_k128_w<false>(d, tS, b, id_sq);
            mma_ts_k128_w<true>(d, tS + 64, desc_advance(b, 16384), id_sq);
            mma_ts_k128_w<true>(d, tS + 128, b, id_sq);
            mma_ts_k128_w<true>(d, tS + 192, desc_advance(b, 16384), id_sq);
        };
        // R as an A operand: 16 columns per K-step (16 tokens), hi in the first 8, lo in the others
        for (int c = 0; c < nchunks; ++c) {
            const uint32_t par = static_cast<uint32_t>(c & 1), prev = par ^ 1u;
            mbar_wait(bar_kv, par, abort_flag);
            tc_fence_after_sync();
            if (c > 0) {  // D1 overwrites the R that O2 of the chunk before was the last to read
                mbar_wait(bar_o2, prev, abort_flag);
                tc_fence_after_sync();
            }
            mbar_wait(bar_s, par, abort_flag);
            tc_fence_after_sync();
            mma_s(tX, dK);
            mma_commit_w(bar_d1);
            mbar_wait(bar_z, par, abort_flag);  // (a wait costs some 130 cycles even when it is over: not between R and dS)
            mbar_wait(bar_q, par, abort_flag);
            tc_fence_after_sync();
            if (c > 0) {
                mbar_wait(bar_o2free, prev, abort_flag);
                tc_fence_after_sync();
            }
            mma_s(tO, dQ);
            mma_commit_w(bar_o1);
            mbar_wait(bar_r, par, abort_flag);
            tc_fence_after_sync();
            // dS quarters 0, 2 (the first of either half of the state warps), then 1, 3
#pragma unroll 1
            for (int i = 0; i < 4; ++i) {
                const int q = i >> 1, hf = i & 1;
                if (q == 1) {
                    mbar_wait(&bar_dsfree[hf], par, abort_flag);
                    tc_fence_after_sync();
                }
                const uint32_t d = tmem + wide::kTmDS + 64 * hf;
                const uint64_t z = desc_advance(dZ, (2 * hf + q) * 8192);
                mma_ts_k64_w<false, 128, 16>(d, tX, z, id_ds);
                mma_ts_k64_w<true, 128, 16>(d, tX, desc_advance(z, 32768), id_ds);
                mma_ts_k64_w<true, 128, 16>(d, tX + 8, z, id_ds);
                mma_commit_w(&bar_ds[hf]);
            }
            mbar_wait(bar_o1free, par, abort_flag);
            tc_fence_after_sync();
            mma_ts_k64_w<false, 2, 16>(tO, tX, dP, id_sq);
            mma_ts_k64_w<true, 2, 16>(tO, tX, desc_advance(dP, 8192), id_sq);
            mma_ts_k64_w<true, 2, 16>(tO, tX + 8, dP, id_sq);
            mma_commit_w(bar_o2);
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
    if (tid == 0 && *abort_flag && p.status) atomicExch(p.status, 4);
}

}  // namespace gdn
