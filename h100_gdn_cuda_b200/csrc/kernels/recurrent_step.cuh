// Recurrent Gated DeltaNet step on warp matrix instructions: padded inputs of 2 .. 8 tokens per sequence, bf16 states,
// dk = 64 or 128, dv a multiple of 32 (speculative verify, short runs).  Same recurrence as recurrent.cuh:
//     S_t = a_t S_{t-1} + c_t k_t^T,   c_t = beta_t (v_t - a_t S_{t-1} k_t),   o_t = scale S_t q_t,   a_t = e^{g_t}
// rewritten over the state S_0 the call starts from, with G_t = a_1 .. a_t and Gamma_ts = a_{s+1} .. a_t:
//     c_t = beta_t v_t - beta_t G_t (S_0 k_t) - sum_{s<t} beta_t Gamma_ts (k_s.k_t) c_s
//     o_t = scale (G_t (S_0 q_t) + sum_{s<=t} Gamma_ts (k_s.q_t) c_s)
//     S_t = G_t S_0 + sum_{s<=t} Gamma_ts c_s k_s^T
// so all tokens' S_0 k_t and S_0 q_t are one product with the state tile, and the update is one product of rank t.
// Precision is that of fp32 arithmetic: S_0, k and q enter the MMAs as the bf16 values they are (exact products, fp32
// accumulation; the q/k norms are fp32 factors of the results), the coefficients c enter the update as three bf16 terms,
// which is all 24 bits of them.
//
// Why: on FMAs (recurrent.cuh) a warp spends 240 instructions per token and 8 rows of state, and the step is bound by
// their issue.  Here it is 750 per 16 rows for four tokens and the last state, where that would be 1 920 (counted by
// ncu, per-item work included), and 2 390 with five states: B=64, T=4, accepted caps 1..4, 32 v-heads, d=128 52.5 -> 31.7 us
// (140 MB: 21.5 us at the measured copy bandwidth), B=13, T=5 with a state per token 25.4 -> 20.6 us.
// (For ONE token per sequence the FMA kernel is already bound by HBM and stays: 88.7 us at B=256 against 92 - 102 this way.)
//
// Every warp works by itself on items of whole (sequence, v-head) units, dealt round by round; what does not fill a last
// round is cut into ranges of tiles of 16 state rows, of equal length to within a tile (3.5 units a warp at B=256: without
// the cut a seventh of the GPU idles in the fourth round; with ranges for everything the warps' streams are spread over all
// of memory at once).  Each warp has a ring of stages of its own, filled by bulk copies (a tile is 16 x dk
// contiguous; the item's k, q come with its first tile).  A tile is taken into registers at once and its stage requested again, so all stages are in flight
// while the warp computes, and no warp waits for another.  (With tiles of 64 rows shared by
// the four warps of a CTA each of them would repeat the per-item work.)
// Products: [k; q] (tokens 0-7 and 8-15 of M) times S^T (8 state rows of N), so that a 16-byte piece of a state row is two B
// operands as it lies; the contraction index may be permuted freely, and lane (g, t) takes the pieces t, t + 4, .. of rows g
// and g + 8.  Their result has token g, rows 2t, 2t + 1 in lane (g, t), which is how v is read and o written.  Update: rows
// of M, columns of N, the coefficients transposed by movmatrix; the accumulator starts as G S in place of the pieces.
#pragma once
#include "recurrent.cuh"

namespace gdn {

constexpr int kStepTok = 8;      // tokens an item can have
constexpr int kStepRows = 16;    // state rows per tile
constexpr int kStepWarps = kRecThreads / 32;
constexpr int kStepMaxStages = 3;
constexpr int kStepCtasPerSm = 2;  // 249 registers a thread; spilled to fit three, the update's stores to local memory cost more

// The k, q of item i sit in slot i % stages until the item's first tile has been taken in, and at that moment the tile `stages`
// further on is requested.  That one must belong to an item before i + stages: so at least two tiles per unit (only the two
// ends of a warp's range, its first item and its last, can have fewer).
__host__ __device__ constexpr bool step_applies(int dv) { return dv % (2 * kStepRows) == 0; }
static_assert(step_applies(2 * kStepRows) && !step_applies(kStepRows), "one tile per unit would overwrite its k and q");

// shared memory of one warp: the stages, the present item's k, q as MMA operands (16 rows), then for each stage room for the
// k and q of an item's tokens
__host__ __device__ constexpr int step_stages(int tokens) { return tokens <= 6 ? 3 : 2; }  // shared memory of a CTA: at most 100 KB
__host__ __device__ constexpr int step_warp_bytes(int dk, int tokens) {
    return ((step_stages(tokens) + 1) * kStepRows + step_stages(tokens) * 2 * tokens) * dk * 2;
}

struct StepParams {
    RecurrentParams r;
    long long num_tiles;  // 16-row tiles of all (sequence, v-head) units
};
// (As for RecurrentParams.  368 bytes, with the number of stages among them, : 352: B=1, T=3, 4 v-heads 5.5 : 5.2 us a call, on the device alone
// B=1, T=4, 32 v-heads 5.41 : 5.25.)
static_assert(sizeof(StepParams) <= 352, "parameter bytes");

namespace step {
__device__ __forceinline__ void mma16(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma8(float* d, uint32_t a0, uint32_t a1, uint32_t b0) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(b0));
}
// 8x8 bf16 fragment (row l/4, columns 2(l%4), +1) -> the fragment of its transpose
__device__ __forceinline__ uint32_t transpose8(uint32_t a) {
    uint32_t d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
    return d;
}
// A scalar as its bits, to be converted where it is used: a conversion at the load waits for it.
__device__ __forceinline__ uint32_t ld_bits(const void* p, int is_f32, long long i) {
    return is_f32 ? __ldg(reinterpret_cast<const uint32_t*>(p) + i) : __ldg(reinterpret_cast<const unsigned short*>(p) + i);
}
__device__ __forceinline__ float from_bits(uint32_t w, int is_f32) { return __uint_as_float(is_f32 ? w : w << 16); }
}  // namespace step

template <int DK>
__device__ __forceinline__ void gdn_recurrent_step_body(const StepParams& sp) {
    using namespace ptx;
    using namespace step;
    constexpr int NJ = DK / 32;  // 16-byte pieces per lane and row; two K-steps of 16 each
    constexpr int kTileBytes = kStepRows * DK * 2;
    const RecurrentParams& p = sp.r;
    const int stages = step_stages(p.seq_len);
    extern __shared__ __align__(128) uint8_t smem_all[];
    __shared__ uint64_t full_all[kStepWarps][kStepMaxStages];
    __shared__ int abort_flag;
    // per warp and item: [s][t] = beta_t Gamma_ts k_s.k_t, scale Gamma_ts k_s.q_t and [tau][s] = Gamma_{tau,s} r_s
    __shared__ float2 s_ap[kStepWarps][kStepTok][kStepTok];
    __shared__ float s_w[kStepWarps][kStepTok][kStepTok];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    uint8_t* const smem = smem_all + warp * step_warp_bytes(DK, p.seq_len);
    uint4* const smem_kq = reinterpret_cast<uint4*>(smem + stages * kTileBytes) + lane;  // [K-step][lane]
    uint8_t* const smem_tok = smem + (stages + 1) * kTileBytes;
    const int tok_bytes = p.seq_len * DK * 4;
    uint64_t* const full = full_all[warp];
    const int rblocks = p.dv / kStepRows;
    const bool has_in = p.state_in != nullptr;
    const int rep = p.vh / p.kh;
    const int warps = static_cast<int>(gridDim.x) * kStepWarps;
    // (consecutive ranges go to different CTAs, so that few of them spread over all SMs)
    const int me = warp * static_cast<int>(gridDim.x) + static_cast<int>(blockIdx.x);
    const int units = static_cast<int>(sp.num_tiles / rblocks), rounds = units / warps;
    const long long rest = sp.num_tiles - static_cast<long long>(rounds) * warps * rblocks;  // tiles of the last round
    const long long tile0 = rest * me / warps, tile1 = rest * (me + 1) / warps;
    const int unit_rest = static_cast<int>(tile0 / rblocks);  // first unit of this warp's range, counted within the last round
    const int rb_first = static_cast<int>(tile0 - static_cast<long long>(unit_rest) * rblocks), rest_tiles = static_cast<int>(tile1 - tile0);
    const int rest_items = rest_tiles ? (rb_first + rest_tiles + rblocks - 1) / rblocks : 0;
    const int rb_last = rest_items ? rb_first + rest_tiles - (rest_items - 1) * rblocks : rblocks;  // end of the last item
    const int my_items = rounds + rest_items;
    if (tid == 0) abort_flag = 0;
    if (lane == 0) {
        for (int s = 0; s < kStepMaxStages; ++s) mbar_init(&full[s], 1);
        mbar_fence_init();
    }
    __syncthreads();
    // a programmatic dependent of the work before it, and in turn the next launch may be placed while this one runs (every
    // kernel launched that way waits for the whole of its predecessor before its first global access)
    grid_dep_wait();
    grid_dep_launch();

    struct Pos {
        int seq, head, rb0, rb1;  // state rows 16 rb0 .. 16 rb1
    };
    const int vh_shift = (p.vh & (p.vh - 1)) == 0 ? __ffs(p.vh) - 1 : -1;
    const int rep_shift = (rep & (rep - 1)) == 0 ? __ffs(rep) - 1 : -1;
    auto decode = [&](int item) {  // item: index within this warp
        Pos r;
        const int un = item < rounds ? item * warps + me : rounds * warps + unit_rest + item - rounds;
        r.rb0 = item == rounds ? rb_first : 0;
        r.rb1 = item == my_items - 1 ? rb_last : rblocks;
        r.seq = vh_shift >= 0 ? un >> vh_shift : un / p.vh;
        r.head = un - r.seq * p.vh;
        return r;
    };
    // State slot and token count of this warp's items, one lane per item, 32 items at a time and the next 32 fetched ahead:
    // they are needed where a tile is requested, and reading them there would put a global latency in front of every request.
    int slot_a = 0, slot_b = 0, ntok_a = 0, ntok_b = 0, base = 0;
    auto fetch_window = [&](int b0, int& slot, int& ntok) {
        const int i = b0 + lane;
        slot = -1;
        ntok = 0;
        if (i < my_items) {
            const int seq = decode(i).seq;
            slot = p.state_idx ? p.state_idx[seq] : seq;
            ntok = p.num_accepted ? max(0, min(p.seq_len, p.num_accepted[seq])) : p.seq_len;
            if (slot < 0) ntok = 0;
        }
    };
    fetch_window(0, slot_a, ntok_a);
    if (my_items > 32) fetch_window(32, slot_b, ntok_b);
    auto slot_of = [&](int i) { return __shfl_sync(0xffffffffu, i - base < 32 ? slot_a : slot_b, (i - base) & 31); };
    auto ntok_of = [&](int i) { return __shfl_sync(0xffffffffu, i - base < 32 ? ntok_a : ntok_b, (i - base) & 31); };

    // The tile to request when the present one has left its stage, `stages` tiles on.
    int req_item = 0, req_r = rounds ? 0 : rb_first, req_slot = 0;
    bool req_new = true;  // the item's first tile
    const __nv_bfloat16* req_src = nullptr;  // the tile; lane 0 requests
    auto request = [&](int stage) {
        if (req_item >= my_items) return;
        int nt = 0;
        if (req_new) {
            req_slot = slot_of(req_item);
            nt = ntok_of(req_item);
        }
        if (lane == 0) {
            if (req_new) {
                const Pos u = decode(req_item);
                req_src = static_cast<const __nv_bfloat16*>(p.state_in) + static_cast<long long>(max(req_slot, 0)) * p.si_ss +
                          u.head * p.si_sh + u.rb0 * (kStepRows * DK);
                if (nt > 0) {
                    const int kh = rep_shift >= 0 ? u.head >> rep_shift : u.head / rep;
                    const __nv_bfloat16* kp = p.k + u.seq * p.k_sb + kh * p.k_sh;
                    const __nv_bfloat16* qp = p.q + u.seq * p.q_sb + kh * p.q_sh;
                    uint8_t* dst = smem_tok + (req_item % stages) * tok_bytes;
                    mbar_arrive_expect_tx(&full[stage], (has_in ? kTileBytes : 0) + nt * DK * 4);
                    for (int i = 0; i < nt; ++i) {
                        bulk_load(dst + i * DK * 4, kp + i * p.k_st, DK * 2, &full[stage]);
                        bulk_load(dst + i * DK * 4 + DK * 2, qp + i * p.q_st, DK * 2, &full[stage]);
                    }
                }
            }
            if (nt == 0) mbar_arrive_expect_tx(&full[stage], has_in && req_slot >= 0 ? kTileBytes : 0);
            if (has_in && req_slot >= 0) bulk_load(smem + stage * kTileBytes, req_src, kTileBytes, &full[stage]);
            req_src += kStepRows * DK;
        }
        __syncwarp();
        req_new = ++req_r == (req_item == my_items - 1 ? rb_last : rblocks);
        if (req_new) {
            ++req_item;
            req_r = req_item == rounds ? rb_first : 0;
        }
    };
    for (int i = 0; i < stages; ++i) request(i);

    // raw scalars of an item's tokens: lane i < 8 holds those of token i
    struct Scalars {
        uint32_t b, g, al, db;  // beta and the gate, or the raw projections and the head's gating parameters
    };
    auto fetch_scalars = [&](const Pos& u, int ntok) {
        Scalars x{0u, 0u, 0u, 0u};
        if (lane < ntok) {
            x.b = ld_bits(p.beta, p.beta_f32, u.seq * p.beta_sb + lane * p.beta_st + u.head * p.beta_sh);
            if (p.gate) x.g = ld_bits(p.gate, p.gate_f32, u.seq * p.gate_sb + lane * p.gate_st + u.head * p.gate_sh);
            if (p.fused_gating) {
                x.al = ld_bits(p.A_log, p.gating_param_f32, u.head);
                x.db = ld_bits(p.dt_bias, p.gating_param_f32, u.head);
            }
        }
        return x;
    };
    // v of a tile: token g, rows 2t, 2t + 1 and 8 + 2t, 8 + 2t + 1
    auto v_of = [&](const Pos& u) {
        return reinterpret_cast<const uint32_t*>(p.v + u.seq * p.v_sb + g * p.v_st + u.head * p.v_sh + u.rb0 * kStepRows + 2 * t);
    };
    Pos u_next = decode(0);
    int ntok_next = my_items ? ntok_of(0) : 0;
    Scalars sc_next = fetch_scalars(u_next, ntok_next);
    uint32_t v_next0 = 0u, v_next1 = 0u;
    const uint32_t* v_ptr = v_of(u_next);
    if (g < ntok_next) {
        v_next0 = __ldg(v_ptr);
        v_next1 = __ldg(v_ptr + 4);
    }

    int stage = 0;
    uint32_t parity = 0;
#pragma unroll 1
    for (int item = 0; item < my_items; ++item) {
        if (item - base == 32) {
            base += 32;
            slot_a = slot_b;
            ntok_a = ntok_b;
            fetch_window(base + 32, slot_b, ntok_b);
        }
        const int slot = slot_of(item), ntok = ntok_next;
        float beta = from_bits(sc_next.b, p.beta_f32), gate = from_bits(sc_next.g, p.gate_f32);
        if (p.fused_gating && lane < ntok) {
            // softplus and sigmoid on the fast exponential, logarithm and reciprocal, as in recurrent.cuh
            const float x = gate + from_bits(sc_next.db, p.gating_param_f32), e = __expf(x);
            gate = -__expf(from_bits(sc_next.al, p.gating_param_f32)) * (x > 20.f ? x : (x < -15.f ? e : __logf(1.f + e)));
            beta = __fdividef(1.f, 1.f + __expf(-beta));
        }
        const float a_mine = lane < ntok ? __expf(gate) : 1.f;  // a of token `lane`
        uint32_t* out_ptr = reinterpret_cast<uint32_t*>(p.out + u_next.seq * p.o_sb + g * p.o_st + u_next.head * p.o_sh +
                                                        u_next.rb0 * kStepRows + 2 * t);
        const bool steps = p.store_step != 0;
        __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(p.state_out) +
                             (steps ? static_cast<long long>(u_next.seq) * p.seq_len : static_cast<long long>(slot)) * p.so_ss +
                             u_next.head * p.so_sh + u_next.rb0 * (kStepRows * DK) + g * DK + 8 * t;
        const int tpi = u_next.rb1 - u_next.rb0;
        u_next = decode(item + 1);
        ntok_next = item + 1 < my_items ? ntok_of(item + 1) : 0;
        sc_next = fetch_scalars(u_next, ntok_next);
        float G_mine = a_mine;  // lane i < 8: a_0 .. a_i
#pragma unroll
        for (int m = 1; m < kStepTok; m <<= 1) {
            const float y = __shfl_up_sync(0xffffffffu, G_mine, m);
            if (lane >= m) G_mine *= y;
        }
        uint32_t kt[4 * NJ];  // operand fragments of k^T for the update
        float cb = 0.f, ck = 0.f, cq = 0.f;  // coefficients of token g
#pragma unroll 1
        for (int r = 0; r < tpi; ++r) {
            // `ok` turns false when a wait gives up: the data is garbage then and nothing of it is stored
            const bool ok = mbar_wait(&full[stage], parity, &abort_flag);
            uint4 sa[NJ], sb[NJ];  // rows g and g + 8
            {
                const uint8_t* st = smem + stage * kTileBytes + g * DK * 2 + 16 * t;
                if (has_in) {
#pragma unroll
                    for (int j = 0; j < NJ; ++j) {
                        sa[j] = *reinterpret_cast<const uint4*>(st + 64 * j);
                        sb[j] = *reinterpret_cast<const uint4*>(st + 8 * DK * 2 + 64 * j);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < NJ; ++j) sa[j] = sb[j] = make_uint4(0u, 0u, 0u, 0u);
                }
            }
            __syncwarp();  // the stage has been read
            request(stage);
            if (++stage == stages) {
                stage = 0;
                parity ^= 1u;
            }
            const uint32_t v0 = v_next0, v1 = v_next1;
            v_ptr += kStepRows / 2;
            if (r + 1 == tpi) v_ptr = v_of(u_next);
            v_next0 = v_next1 = 0u;
            if (g < (r + 1 == tpi ? ntok_next : ntok)) {
                v_next0 = __ldg(v_ptr);
                v_next1 = __ldg(v_ptr + 4);
            }

            if (r == 0) {
                // ---- products of the tokens and the coefficients made of them
                float d[4] = {0.f, 0.f, 0.f, 0.f}, dq[4] = {0.f, 0.f, 0.f, 0.f};
                const uint8_t* tk = smem_tok + (item % stages) * tok_bytes + g * DK * 4 + 16 * t;
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    uint4 x = make_uint4(0u, 0u, 0u, 0u), y = x;
                    if (g < ntok) {
                        x = *reinterpret_cast<const uint4*>(tk + 64 * j);
                        y = *reinterpret_cast<const uint4*>(tk + DK * 2 + 64 * j);
                    }
                    smem_kq[64 * j] = make_uint4(x.x, y.x, x.y, y.y);  // read back by this lane only
                    smem_kq[64 * j + 32] = make_uint4(x.z, y.z, x.w, y.w);
                    mma16(d, x.x, y.x, x.y, y.y, x.x, x.y);
                    mma16(d, x.z, y.z, x.w, y.w, x.z, x.w);
                    if (p.is_qk_norm) {
                        mma16(dq, x.x, y.x, x.y, y.y, y.x, y.y);
                        mma16(dq, x.z, y.z, x.w, y.w, y.z, y.w);
                    }
                    const uint32_t kw[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) kt[4 * j + e] = transpose8(kw[e]);  // tokens 2t, 2t + 1 of column g
                }
                // d[e]: k_g . k_{2t+e};  d[2+e]: q_g . k_{2t+e};  dq[2+e]: q_g . q_{2t+e}
                float rk_g = 1.f, rq_g = 1.f, rk_u[2] = {1.f, 1.f};
                if (p.is_qk_norm) {
                    const float nk = (g & 1) ? d[1] : d[0], nq = (g & 1) ? dq[3] : dq[2];  // diagonal, valid where t == g / 2
                    rk_g = rsqrtf(__shfl_sync(0xffffffffu, nk, 4 * g + (g >> 1)) + 1e-6f);
                    rq_g = rsqrtf(__shfl_sync(0xffffffffu, nq, 4 * g + (g >> 1)) + 1e-6f);
#pragma unroll
                    for (int e = 0; e < 2; ++e) rk_u[e] = rsqrtf(__shfl_sync(0xffffffffu, nk, 4 * (2 * t + e) + t) + 1e-6f);
                }
                const float bg = __shfl_sync(0xffffffffu, beta, g), Gg = __shfl_sync(0xffffffffu, G_mine, g);
                cb = bg;
                ck = bg * Gg * rk_g;
                cq = p.scale * Gg * rq_g;
                float gam[2] = {1.f, 1.f};  // Gamma between tokens g and 2t + e, whichever is later
#pragma unroll
                for (int i = 1; i < kStepTok; ++i) {
                    const float ai = __shfl_sync(0xffffffffu, a_mine, i);
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int ue = 2 * t + e;
                        gam[e] *= (i > min(g, ue) && i <= max(g, ue)) ? ai : 1.f;
                    }
                }
                __syncwarp();
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int ue = 2 * t + e;
                    s_ap[warp][ue][g] =
                        make_float2(ue < g ? bg * gam[e] * d[e] * rk_g * rk_u[e] : 0.f,
                                    ue <= g ? p.scale * gam[e] * d[2 + e] * rq_g * rk_u[e] : 0.f);
                    s_w[warp][ue][g] = g <= ue && g < ntok ? gam[e] * rk_g : 0.f;
                }
                __syncwarp();
            }
            // ---- S_0 k and S_0 q of token g: rows 2t, 2t + 1 of the first (h = 0) and the second 8 rows
            float R[2][2], O[2][2];
            {
                float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    const uint4 x = smem_kq[64 * j], y = smem_kq[64 * j + 32];
                    mma16(d0, x.x, x.y, x.z, x.w, sa[j].x, sa[j].y);
                    mma16(d1, x.x, x.y, x.z, x.w, sb[j].x, sb[j].y);
                    mma16(d0, y.x, y.y, y.z, y.w, sa[j].z, sa[j].w);
                    mma16(d1, y.x, y.y, y.z, y.w, sb[j].z, sb[j].w);
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    // (rows of tokens that do not exist are zero, whatever the state holds)
                    R[0][e] = g < ntok ? fmaf(cb, e ? bf16_hi(v0) : bf16_lo(v0), -ck * d0[e]) : 0.f;
                    R[1][e] = g < ntok ? fmaf(cb, e ? bf16_hi(v1) : bf16_lo(v1), -ck * d1[e]) : 0.f;
                    O[0][e] = cq * d0[2 + e];
                    O[1][e] = cq * d1[2 + e];
                }
            }
            // ---- c and o (selected, not multiplied by the zeros of s_ap: an infinite or undefined value of a later token
            //      must not reach an earlier one)
#pragma unroll 1
            for (int s = 0; s < ntok; ++s) {
                const float2 ap = s_ap[warp][s][g];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float& Ri = R[i >> 1][i & 1];
                    const float c = __shfl_sync(0xffffffffu, Ri, 4 * s + t);
                    Ri = s < g ? fmaf(-ap.x, c, Ri) : Ri;
                    O[i >> 1][i & 1] = s <= g ? fmaf(ap.y, c, O[i >> 1][i & 1]) : O[i >> 1][i & 1];
                }
            }
            {
                const uint32_t o0 = pack_bf16(O[0][0], O[0][1]), o1 = pack_bf16(O[1][0], O[1][1]);
                if (ok && g < ntok) {  // token g, rows 2t, 2t + 1 (+ 8)
                    out_ptr[0] = o0;
                    out_ptr[4] = o1;
                }
                out_ptr += kStepRows / 2;
            }
            // ---- S_tau = G_tau S_0 + sum_s (Gamma_{tau,s} r_s c_s) k_s^T: the last token's state, or every token's.  Both factors
            //      of a token after tau are zero: either alone would turn the other's infinite or undefined value into a NaN.
            //      (These selects cost 0.4 us of 31.2 at B=64, T=4 and 0.35 of 20.25 at B=13, T=5 with step states; a second copy of
            //      the update for the tiles that need them, behind a vote, costs 0.9 and 0.1.)
            if (slot >= 0) {
                const int last = max(ntok - 1, 0);
#pragma unroll 1
                for (int tau = steps ? 0 : last; tau < (steps ? ntok : last + 1); ++tau) {
                    const float G = ntok > 0 ? __shfl_sync(0xffffffffu, G_mine, tau) : 1.f;
                    uint32_t w[2][3];  // [8 rows][bf16 term]: rows 2t, 2t + 1 of token g, then transposed to row g, tokens 2t, 2t + 1
                    const float f = s_w[warp][tau][g];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float x0 = g <= tau ? f * R[h][0] : 0.f, x1 = g <= tau ? f * R[h][1] : 0.f;
#pragma unroll
                        for (int i = 0; i < 3; ++i) {
                            const uint32_t b = pack_bf16(x0, x1);
                            x0 -= bf16_lo(b);
                            x1 -= bf16_hi(b);
                            if (i == 0) {  // inf - inf: any finite number (fmaxf drops a NaN), the first term outweighs it
                                x0 = fmaxf(x0, -3.0e38f);
                                x1 = fmaxf(x1, -3.0e38f);
                            }
                            w[h][i] = transpose8(b);
                        }
                    }
                    const uint32_t ktok = (2 * t <= tau ? 0xFFFFu : 0u) | (2 * t + 1 <= tau ? 0xFFFF0000u : 0u);
                    __nv_bfloat16* d = steps ? dst + tau * p.so_ss : dst;
#pragma unroll
                    for (int j = 0; j < NJ; ++j) {
                        uint32_t na[4], nb[4];
                        // opaque: unpacked ahead of the loop over tau the state would take twice the registers
                        asm volatile("" : "+r"(sa[j].x), "+r"(sa[j].y), "+r"(sa[j].z), "+r"(sa[j].w));
                        asm volatile("" : "+r"(sb[j].x), "+r"(sb[j].y), "+r"(sb[j].z), "+r"(sb[j].w));
                        const uint32_t wa[4] = {sa[j].x, sa[j].y, sa[j].z, sa[j].w}, wb[4] = {sb[j].x, sb[j].y, sb[j].z, sb[j].w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            float c[4];
                            c[0] = G * bf16_lo(wa[e]); c[1] = G * bf16_hi(wa[e]);
                            c[2] = G * bf16_lo(wb[e]); c[3] = G * bf16_hi(wb[e]);
                            const uint32_t kk = kt[4 * j + e] & ktok;
                            mma16(c, w[0][0], w[1][0], w[0][1], w[1][1], kk, kk);
                            mma8(c, w[0][2], w[1][2], kk);
                            na[e] = pack_bf16(c[0], c[1]);
                            nb[e] = pack_bf16(c[2], c[3]);
                        }
                        if (ok) {
                            *reinterpret_cast<uint4*>(d + 32 * j) = make_uint4(na[0], na[1], na[2], na[3]);
                            *reinterpret_cast<uint4*>(d + 8 * DK + 32 * j) = make_uint4(nb[0], nb[1], nb[2], nb[3]);
                        }
                    }
                }
            }
            dst += kStepRows * DK;
        }
    }
    __syncthreads();
    if (tid == 0 && abort_flag && p.status) atomicExch(p.status, 1);
}

template <int DK>
__global__ void __launch_bounds__(kRecThreads, kStepCtasPerSm) gdn_recurrent_step_kernel(const StepParams p) {
    gdn_recurrent_step_body<DK>(p);
}

}  // namespace gdn
