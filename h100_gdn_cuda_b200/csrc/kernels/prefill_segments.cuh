// Start states of the segments of a segmented prefill run (see FusedParams in prefill_fused.cuh):
//     S_start[0] = initial state (or S_start[1] as the first segment's run has left it),   S_start[p + 1] = S_start[p] M_p + N_p
// with M_p, N_p the composite transition of segment p (fp32, dv x dk and dk x dk with dv = dk = 128)
// produced by gdn_seg_transition_kernel.  Segment p of a sequence sits in launch
// slot first_slot + p (locate_segment in prefill_common.cuh); in packed mode the sequences have
// different numbers of segments.  The work is tiny (one 128 x 128 x 128
// product per chain and segment) and strictly sequential in p; it stays in fp32 on CUDA cores.
// One CTA of 8 warps per (chain, block of 8 state rows); warp w takes the 16 inner indices 16 w .. of the product, a lane
// four columns of all 8 rows on packed pairs (64 two-wide FMAs against 12 shared-memory loads for 4 indices), then the
// warps' partial sums meet in shared memory.  M_p (64 KB) comes by one bulk copy, that of M_{p+1} running while M_p is in use.
// 8 chains x 18 segments: 54 us with a thread per column and scalar FMAs (three quarters of it shared-memory latency).
#pragma once
#include <cuda_bf16.h>

#include "prefill_common.cuh"
#include "prefill_fused.cuh"
#include "sm100_ptx.cuh"

namespace gdn {

struct SegCombineParams {
    const float* seg_mn;   // [slot][head][2][128][128]: N then M
    float* seg_start;      // [slot][head][128][128]; first_apart: those of the second segments are given, and none is made for the first
    const __nv_bfloat16* state_in;  // or NULL; d x d per (sequence, head), zero outside when d < 128
    long long si_ss, si_sh;
    int d, first_apart;
    ChunkMap map;
    int seg_chunks;
    int vh, num_segments;
    int* status;
};

struct SegCombineSmem {
    static constexpr int D = 128, R = 8;
    static constexpr int kOffM = 0;                      // two buffers of D x D fp32
    static constexpr int kOffS = 2 * D * D * 4;          // R x D fp32
    static constexpr int kThreads = 256;
    static constexpr int kOffRed = kOffS + R * D * 4;    // partial sums of the 8 warps
    static constexpr int kOffBar = kOffRed + 8 * R * D * 4;  // 2 mbarriers, abort flag
    static constexpr int kBytes = kOffBar + 32 + 128;
};

__global__ void __launch_bounds__(SegCombineSmem::kThreads) gdn_seg_combine_kernel(const SegCombineParams p) {
    using namespace ptx;
    using fused::f2; using fused::fma2; using fused::pk; using fused::unpk;
    using L = SegCombineSmem;
    constexpr int D = L::D, R = L::R;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((128u - (ptx::smem_u32(smem_raw) & 127u)) & 127u);
    float* sM = reinterpret_cast<float*>(smem + L::kOffM);
    float(*sS)[D] = reinterpret_cast<float(*)[D]>(smem + L::kOffS);
    float(*sRed)[R][D] = reinterpret_cast<float(*)[R][D]>(smem + L::kOffRed);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
    int* abort_flag = reinterpret_cast<int*>(bar + 2);

    // launched as a programmatic dependent of the first segments' launch, or of the transitions'; the output launch may be placed as soon as all CTAs here are
    ptx::grid_dep_launch();
    ptx::grid_dep_wait();
    const long long chain = blockIdx.x;
    const int warp = threadIdx.x >> 5, col = 4 * (threadIdx.x & 31);
    const int row = blockIdx.y * R + warp;  // this thread's piece of the running state: row `row`, columns col .. col + 3
    const int seq = static_cast<int>(chain / p.vh), head = static_cast<int>(chain % p.vh);
    const SegPos sp = sequence_segments(p.map, seq, p.seg_chunks, p.num_segments);
    const int steps = sp.nseg - 1 - p.first_apart;  // products: S_start[first_apart + 1] and on
    if (p.first_apart && steps <= 0) return;
    auto idx = [&](int s) { return static_cast<long long>(sp.first_slot + p.first_apart + s) * p.vh + head; };
    auto request_m = [&](int s) {  // one thread
        mbar_arrive_expect_tx(&bar[s & 1], D * D * 4);
        bulk_load(sM + (s & 1) * D * D, p.seg_mn + (idx(s) * 2 + 1) * (D * D), D * D * 4, &bar[s & 1]);
    };
    if (threadIdx.x == 0) {
        *abort_flag = 0;
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        mbar_fence_init();
        for (int s = 0; s < 2 && s < steps; ++s) request_m(s);
    }
    float4 cur = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p.first_apart) {
        cur = *reinterpret_cast<const float4*>(p.seg_start + idx(0) * (D * D) + row * D + col);
    } else {
        if (p.state_in && row < p.d && col < p.d) {  // (d is a multiple of 8)
            const uint2 w = *reinterpret_cast<const uint2*>(p.state_in + seq * p.si_ss + head * p.si_sh + static_cast<long long>(row) * p.d + col);
            cur = make_float4(bf16_lo(w.x), bf16_hi(w.x), bf16_lo(w.y), bf16_hi(w.y));
        }
        *reinterpret_cast<float4*>(p.seg_start + idx(0) * (D * D) + row * D + col) = cur;
    }
    auto load_n = [&](int s) {
        return s < steps ? *reinterpret_cast<const float4*>(p.seg_mn + idx(s) * 2 * (D * D) + row * D + col) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    float4 nxt = load_n(0);  // N of the coming segment, fetched one iteration ahead
    *reinterpret_cast<float4*>(&sS[warp][col]) = cur;
    __syncthreads();
    for (int s = 0; s < steps; ++s) {
        const float4 n = nxt;
        nxt = load_n(s + 1);
        mbar_wait(&bar[s & 1], static_cast<uint32_t>((s >> 1) & 1), abort_flag);
        const float* M = sM + (s & 1) * D * D;
        f2 acc[R][2];
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r][0] = acc[r][1] = 0ull;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const int k0 = 16 * warp + 4 * kk;
            f2 m[4][2];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(M + (k0 + e) * D + col);
                m[e][0] = w.x;
                m[e][1] = w.y;
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float4 s4 = *reinterpret_cast<const float4*>(&sS[r][k0]);  // one address for all lanes: a broadcast
                const float sv[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const f2 ss = pk(sv[e], sv[e]);
                    acc[r][0] = fma2(ss, m[e][0], acc[r][0]);
                    acc[r][1] = fma2(ss, m[e][1], acc[r][1]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) *reinterpret_cast<ulonglong2*>(&sRed[warp][r][col]) = make_ulonglong2(acc[r][0], acc[r][1]);
        __syncthreads();  // the partial sums are there, sS and this M buffer free
        if (threadIdx.x == 0 && s + 2 < steps) request_m(s + 2);
        cur = n;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            const float4 v = *reinterpret_cast<const float4*>(&sRed[w][warp][col]);
            cur.x += v.x; cur.y += v.y; cur.z += v.z; cur.w += v.w;
        }
        *reinterpret_cast<float4*>(p.seg_start + idx(s + 1) * (D * D) + row * D + col) = cur;
        *reinterpret_cast<float4*>(&sS[warp][col]) = cur;
        __syncthreads();  // sS complete, the partial sums read
    }
    if (threadIdx.x == 0 && *abort_flag && p.status) atomicExch(p.status, 6);
}

}  // namespace gdn
