// Composite transitions of the segments of a segmented prefill run (few long sequences; see FusedParams).
// Per chunk the state obeys S' = S M_c + N_c, so a segment has a composite (M, N) as well: N is what the segment leaves of
// S = 0, M what it leaves of S = I when V is taken as 0.  One CTA of 640 threads walks the chunks of one (sequence, segment,
// v-head) and carries BOTH runs through the recurrence of gdn_fused_seq_kernel (prefill_fused.cuh), without its output:
//     R = V - e^{g} .* (K S^T)  (run 1: R = -e^{g} .* (K S^T)),   S <- e^{g_L} S + R^T Z
// A run is a chain of dependent steps that leaves the tensor pipe idle 80 % of the time and the schedulers 60 %; two runs
// on the same tiles fill each other's gaps and read K, Z and the gates once.  Each run has 8 state warps of its own, the
// first MMA's accumulator shares the columns of the second's (it is dead once R is published), so both fit tensor memory.
// B=2, T=131072, 4 v-heads (136 CTAs of 114 chunks): replaces two waves of one run per CTA, see gdn_chunked_forward.
#pragma once
#include <cuda.h>

#include "prefill_common.cuh"
#include "prefill_fused.cuh"

namespace gdn {

struct TransitionSmem {
    static constexpr int kStages = 3;
    static constexpr int kTile = kChunk * 128 * 2;  // 16 KB
    static constexpr int kOffK = 0, kOffV = kTile, kOffZ = 2 * kTile, kStage = 3 * kTile;
    static constexpr int kGates = kStages + 1;               // a chunk's factors outlive its tiles by a little
    static constexpr int kOffGate = kStages * kStage;        // { -e^g r_k [64], e^{gL} }
    static constexpr int kGateStride = (64 + 4) * 4;
    static constexpr int kOffBar = kOffGate + kGates * kGateStride;
    static constexpr int kBytes = kOffBar + 192 + 1024;
};

namespace transition {
constexpr int kThreads = 640;  // 16 state warps, producer, issuer, two idle warps (their registers go to the state warps)
// tensor-memory columns of run `i`: + 224 i
constexpr uint32_t kTmSbf = 0, kTmR = 64, kTmD = 96, kTmRun = 224;  // bf16 state 64, bf16 R 32, fp32 S K^T (64) and then dS (128)
}  // namespace transition

__global__ void __launch_bounds__(transition::kThreads, 1)
    gdn_seg_transition_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const FusedParams p) {
    using namespace ptx;
    using fused::f2; using fused::fma2; using fused::pk; using fused::reg_dec; using fused::reg_inc; using fused::unpk;
    using transition::kThreads;
    using L = TransitionSmem;
    constexpr int D = 128;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (ptx::smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
    uint64_t* bar_full = bars;        // [3] K, V and the gate factors
    uint64_t* bar_full2 = bars + 3;   // [3] Z
    uint64_t* bar_empty = bars + 6;   // [3]
    uint64_t* bar_sbf = bars + 9;     // [2 runs]
    uint64_t* bar_d1 = bars + 11;
    uint64_t* bar_un = bars + 13;
    uint64_t* bar_ds = bars + 15;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17);
    int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const SegPos sp = locate_segment(p.map, static_cast<int>(blockIdx.x), p.seg_chunks, p.num_segments, p.num_seqs);
    // surplus slot; nothing follows a sequence's last segment; a first one is walked outright
    if (sp.seq < 0 || sp.segment == sp.nseg - 1 || (sp.segment == 0 && p.first_apart)) {
        // The launch behind this one starts when all CTAs here have let it or are gone, or waits for this grid, and takes it that the
        // chunk-parallel kernel is complete then.  So the first CTA, whose segment is a first one, waits for that in any case.
        if (blockIdx.x == 0 && blockIdx.y == 0) {
            grid_dep_wait();
            grid_dep_handover();
        }
        return;
    }
    const int head = static_cast<int>(blockIdx.y), khead = head / (p.vh / p.kh);
    const long long seg_idx = static_cast<long long>(blockIdx.x) * p.vh + head;
    int batch = sp.seq, gchunk0 = sp.seq * p.map.chunks_per_seq;
    long long seq_tok0 = 0;
    if (p.map.cu_seqlens) {
        batch = 0;
        seq_tok0 = p.map.cu_seqlens[sp.seq];
        gchunk0 = p.map.cu_chunks[sp.seq];
    }
    // every chunk of a segment that is not its sequence's last is a full one
    const int nchunks = p.seg_chunks;
    seq_tok0 += static_cast<long long>(sp.segment) * p.seg_chunks * kChunk;
    gchunk0 += sp.segment * p.seg_chunks;

    if (tid == 0) {
        *abort_flag = 0;
        for (int i = 0; i < L::kStages; ++i) {
            mbar_init(&bar_full[i], 1);
            mbar_init(&bar_full2[i], 1);
            mbar_init(&bar_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bar_sbf[i], 8);
            mbar_init(&bar_d1[i], 1);
            mbar_init(&bar_un[i], 8);
            mbar_init(&bar_ds[i], 1);
        }
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(tmem_slot, 512);
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    auto gate_buf = [&](int c) { return reinterpret_cast<float*>(smem + L::kOffGate + (c % L::kGates) * L::kGateStride); };

    if (warp < 16) {
        // =============================================================== state warps
        // setmaxnreg moves registers inside what the CTA was launched with (640 threads x 96): more would wait for ever
        static_assert(16 * 104 + 4 * 64 <= 20 * 96, "register pool of the CTA");
        reg_inc<104>();
        const int run = warp >> 3, lq = warp & 3, hf = (warp >> 2) & 1;
        const int row = 32 * lq + lane;
        const uint32_t tm = tmem + transition::kTmRun * run + (static_cast<uint32_t>(32 * lq) << 16);
        // V^T by transposing matrix loads, as in gdn_fused_seq_kernel
        const uint32_t vlane = static_cast<uint32_t>((lq >> 1) * 8192 + (32 * hf + 8 * (lane >> 4) + (lane & 7)) * 128);
        const uint32_t vchunk = static_cast<uint32_t>(4 * (lq & 1) + ((lane >> 3) & 1));
        const uint32_t vsw0 = vlane + ((vchunk ^ (lane & 7)) << 4), vsw1 = vlane + (((vchunk + 2) ^ (lane & 7)) << 4);
        const int t0 = 32 * hf + 2 * (lane & 3);
        float S[64];
#pragma unroll
        for (int q = 0; q < 64; ++q) S[q] = (run == 1 && row == 64 * hf + q) ? 1.f : 0.f;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            uint32_t w[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) w[e] = pack_bf16(S[q * 32 + 2 * e], S[q * 32 + 2 * e + 1]);
            tmem_st16(tm + transition::kTmSbf + 32 * hf + 16 * q, w);
        }
        tmem_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_sbf[run]);

        int stage = 0;
        uint32_t sphase = 0;
        for (int c = 0; c < nchunks; ++c) {
            const uint32_t par = static_cast<uint32_t>(c & 1);
            const float* gb = gate_buf(c);
            mbar_wait(&bar_full[stage], sphase, abort_flag);
            const uint32_t sV = smem_u32(smem + stage * L::kStage + L::kOffV);
            if (++stage == L::kStages) {
                stage = 0;
                sphase ^= 1u;
            }
            f2 neg[4];  // -e^{g} of this lane's token pairs
#pragma unroll
            for (int i = 0; i < 4; ++i) neg[i] = *reinterpret_cast<const f2*>(gb + t0 + 8 * i);
            const f2 eg2 = pk(gb[64], gb[64]);
            mbar_wait(&bar_d1[run], par, abort_flag);
            tc_fence_after_sync();
            // ---- R, 16 rows at a time
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t r[16], v[2][4] = {{0u, 0u, 0u, 0u}, {0u, 0u, 0u, 0u}}, w[8];
                tmem_ld_frag32(tm + (static_cast<uint32_t>(16 * h) << 16) + transition::kTmD + 32 * hf, r);
                if (run == 0) {
                    ldmatrix_x4_trans(sV + (h ? vsw1 : vsw0), v[0]);
                    ldmatrix_x4_trans(sV + (h ? vsw1 : vsw0) + 2048, v[1]);
                }
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 4; ++i) {
#pragma unroll
                    for (int a = 0; a < 2; ++a) {
                        const uint32_t vv = v[i >> 1][2 * (i & 1) + a];
                        float r0, r1;
                        unpk(fma2(neg[i], pk(__uint_as_float(r[4 * i + 2 * a]), __uint_as_float(r[4 * i + 2 * a + 1])),
                                  pk(bf16_lo(vv), bf16_hi(vv))),
                             r0, r1);
                        w[2 * i + a] = pack_bf16(r0, r1);
                    }
                }
                tmem_st_frag16(tm + (static_cast<uint32_t>(16 * h) << 16) + transition::kTmR + 16 * hf, w);
            }
            tmem_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar_un[run]);
            // ---- S <- e^{g_L} S + dS
            mbar_wait(&bar_ds[run], par, abort_flag);
            tc_fence_after_sync();
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                uint32_t r[16], w[8];
                tmem_ld16(tm + transition::kTmD + 64 * hf + 16 * q, r);
                tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    float& s0 = S[q * 16 + 2 * e];
                    float& s1 = S[q * 16 + 2 * e + 1];
                    unpk(fma2(pk(s0, s1), eg2, pk(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1]))), s0, s1);
                    w[e] = pack_bf16(s0, s1);
                }
                tmem_st8(tm + transition::kTmSbf + 32 * hf + 8 * q, w);
            }
            tmem_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar_sbf[run]);
        }
        if (*abort_flag == 0) {  // nothing is written once a wait has given up
            float4* d4 = reinterpret_cast<float4*>(p.seg_mn + (seg_idx * 2 + run) * (D * D) + static_cast<long long>(row) * D + 64 * hf);
#pragma unroll
            for (int q = 0; q < 16; ++q) d4[q] = make_float4(S[4 * q], S[4 * q + 1], S[4 * q + 2], S[4 * q + 3]);
        }
    } else {
        reg_dec<64>();
    }
    if (warp == 16) {
        // =============================================================== producer
        auto load_raw = [&](int c, uint32_t& a0, uint32_t& a1) {
            a0 = a1 = 0u;
            if (p.gate.ptr && c < nchunks) {
                const long long t = seq_tok0 + static_cast<long long>(c) * kChunk + lane;
                a0 = p.gate.load_bits(batch, t, head);
                a1 = p.gate.load_bits(batch, t + 32, head);
            }
        };
        const uint64_t keep = l2_policy_evict_last();  // the output launch reads the same tiles
        uint32_t ra0, ra1, rb0, rb1;
        load_raw(0, ra0, ra1);
        load_raw(1, rb0, rb1);
        grid_dep_wait();
        int s = 0;
        uint32_t ephase = 1;
        for (int c = 0; c < nchunks; ++c) {
            float g0 = p.gate.value(ra0), g1 = p.gate.value(ra1);
            ra0 = rb0;
            ra1 = rb1;
            load_raw(c + 2, rb0, rb1);
            float rk0 = 1.f, rk1 = 1.f;
            if (p.norms) {
                const float* nr = p.norms + (static_cast<size_t>(gchunk0 + c) * p.kh + khead) * 128;
                rk0 = __ldg(nr + lane);
                rk1 = __ldg(nr + 32 + lane);
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
            const float el = __expf(__shfl_sync(0xffffffffu, g1, 31));
            mbar_wait_relaxed<100>(&bar_empty[s], ephase, abort_flag);
            float* gb = gate_buf(c);
            gb[lane] = -__expf(g0) * rk0;
            gb[lane + 32] = -__expf(g1) * rk1;
            if (lane == 0) gb[64] = el;
            __syncwarp();
            uint8_t* st = smem + s * L::kStage;
            const int tok = static_cast<int>(seq_tok0 + static_cast<long long>(c) * kChunk);
            mbar_arrive_expect_tx_w(&bar_full[s], 2 * L::kTile);
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                tma_load_4d_w(st + L::kOffK + a * 8192, &tmK, &bar_full[s], a * 64, khead, tok, batch);
                tma_load_4d_w(st + L::kOffV + a * 8192, &tmV, &bar_full[s], a * 64, head, tok, batch);
            }
            mbar_arrive_expect_tx_w(&bar_full2[s], L::kTile);
            bulk_load_hint_w(st + L::kOffZ, p.blocks + (static_cast<size_t>(gchunk0 + c) * p.vh + head) * kZPBlockBytes, L::kTile, &bar_full2[s], keep);
            if (++s == L::kStages) {
                s = 0;
                ephase ^= 1u;
            }
        }
    } else if (warp == 17) {
        // =============================================================== MMA issuer (the whole warp, one elected lane issues)
        constexpr uint32_t id_sk = make_idesc_bf16(128, 64, false, false);
        constexpr uint32_t id_ds = make_idesc_bf16(128, 128, false, true);
        const uint64_t dK0 = make_smem_desc_sw128(smem_u32(smem + L::kOffK), 0, 1024);     // K-major B
        const uint64_t dZ0 = make_smem_desc_sw128(smem_u32(smem + L::kOffZ), 8192, 1024);  // MN-major B
        int s = 0;
        uint32_t phase = 0;
        for (int c = 0; c < nchunks; ++c) {
            const uint32_t par = static_cast<uint32_t>(c & 1);
            const uint64_t k = desc_advance(dK0, s * L::kStage), z = desc_advance(dZ0, s * L::kStage);
            mbar_wait(&bar_full[s], phase, abort_flag);
            tc_fence_after_sync();
#pragma unroll
            for (int run = 0; run < 2; ++run) {
                const uint32_t tm = tmem + transition::kTmRun * run;
                mbar_wait(&bar_sbf[run], par, abort_flag);
                tc_fence_after_sync();
                mma_ts_k128_w<false>(tm + transition::kTmD, tm + transition::kTmSbf, k, id_sk);  // S K^T
                mma_commit_w(&bar_d1[run]);
            }
            mbar_wait(&bar_full2[s], phase, abort_flag);
            tc_fence_after_sync();
#pragma unroll
            for (int run = 0; run < 2; ++run) {
                const uint32_t tm = tmem + transition::kTmRun * run;
                mbar_wait(&bar_un[run], par, abort_flag);
                tc_fence_after_sync();
                mma_ts_k64_w<false, 128>(tm + transition::kTmD, tm + transition::kTmR, z, id_ds);  // dS = R Z
                mma_commit_w(&bar_ds[run]);
            }
            mma_commit_w(&bar_empty[s]);
            if (++s == L::kStages) {
                s = 0;
                phase ^= 1u;
            }
        }
    } else if (warp == 18) {
        // What is launched next, the first segments, reads what the chunk-parallel kernel has written, complete now, and runs beside this launch
        // (or it is the start states' kernel, which sets itself up and waits).  By a warp with no loads of its own, which the
        // fence would wait for (4 v-heads of 2500 tokens 43.7 us without fences, 44.0 so, 44.2 by the producer; others are within 0.1 us).
        grid_dep_wait();
        if (lane == 0) {
            grid_dep_handover();
            grid_dep_launch();
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
    if (tid == 0 && *abort_flag && p.status) atomicExch(p.status, 4);
}

}  // namespace gdn
