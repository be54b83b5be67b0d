// Recurrent Gated DeltaNet over long runs of tokens (short prefill through recurrent_forward, head dims above 128 in
// chunked_forward): blocks of 16 tokens on warp matrix instructions.  Same recurrence as recurrent.cuh, rewritten over the
// state S_0 a block starts from as in recurrent_step.cuh, with G_t = a_1 .. a_t and Gamma_ts = a_{s+1} .. a_t:
//     c_t = beta_t v_t - beta_t G_t (S_0 k_t) - sum_{s<t} A_ts c_s,   A_ts = beta_t Gamma_ts (k_s.k_t)
//     o_t = scale G_t (S_0 q_t) + sum_{s<=t} P_ts c_s,                P_ts = scale Gamma_ts (k_s.q_t)
//     S  <- G_n S_0 + sum_s (Gamma_ns c_s) k_s^T
// The state stays in fp32 registers from the first token to the last; it enters S_0 [k; q] as three bf16 terms, which is all 24 bits
// of it, and so do the coefficients of the update; k and q are the bf16 values they are (their norms are fp32 factors of the
// results).  Products of bf16 values are exact; sums inside a matrix instruction are cut off at about 24 bits, sums of their results
// are rounded; the solve and the outputs are fp32 FMAs; the update is added to the decayed state by one fp32 FMA per element and BLOCK, where
// the token recurrence rounds the state at every token.  Share of the bf16 outputs after 1000 tokens that are not the 64-bit value
// rounded to bf16, token recurrence : here, d=256: no decay 4.1e-4 : 1.7e-4, mean gate -0.016 8.0e-4 : 7.8e-4, -0.16 1.8e-4 : 1.6e-4,
// -0.8 9.0e-5 : 8.9e-5, -5 6.5e-5 : 5.4e-5.  (A state kept in fp32 outside would show the sums that are cut off: with a decay it was up to
// 40 % further off than token by token, so those take the token recurrence.)
//
// Why: the token recurrence (recurrent.cuh, ring instance) is a chain of about 1 250 cycles per token, and a sequence of a
// few v-heads gives it only some tiles to work on side by side.  Here a block of 16 tokens is one chain of some 2 800 cycles: products (1 000),
// sums and a triangular solve (500), the update (500), two barriers, the hand-over to the writing warps and the waits between them:
// B=2, T=1500, 8 v-heads, d=256 996 -> 200 us, 4 v-heads B=1 994 -> 138, T=700, d=192 401 -> 84; B=4, T=512, 32 v-heads, d=128 188 us.
// With two CTAs per SM issue, shared memory (each about half of its time) and the matrix instructions (a quarter) share the time without one
// of them filling it; with one CTA the chain does.
//
// A CTA owns 16 state rows (M of the products) of one (sequence, v-head) and walks its blocks:
//   warps 0-3   a quarter of the columns each, kept as accumulator fragments, which are the A operands of the product
//               S_0 [k; q]^T as they lie.  The four partial products meet in shared memory; then each warp solves for c of four rows,
//               eight lanes to a row with two tokens each, and hands them over as an operand of the update, which every warp makes
//               of its own columns.  The substitution is seven exchanges between lanes of about 45 cycles: a lane takes its two
//               tokens in one step.  (Every warp all 16 rows, a row in two lanes, needs no second barrier but four times the
//               loads, and the solve takes 850 cycles: d=256 B=2 T=1500 217 us, B=1 152, T=700 d=192 95; one token per exchange 201, 141, 86.)
//   warps 4-7   prepare blocks in turn (warp 4 + j: blocks j, j + 4, ..), up to four ahead: copies of k, q, v, the Gram matrices
//               k k^T and q k^T on matrix instructions, decay products, norms, and from them the matrices A and P; when a
//               block is through they write its outputs.  (Written by the warps that hold the state they cost 400 cycles a block.)
//               (Four of them, so that their work is spread over the four schedulers.)
// Two CTAs per SM at dk = 256: one's chain fills the gaps of the other (4 300 cycles a block for the pair).  kGroups = 2: one CTA of two such
// groups of four warps, 32 rows, with one preparation for both (4 100 cycles; B=2, T=1500, 8 v-heads, d=256 211 -> 200 us).  Four warps
// with 32 rows each share k and q in registers too, and the substitution, but a warp is a chain of its own: 359 us.  Additions and FMAs of the
// state in pairs (f32x2) spill: 217 us.
#pragma once
#include "recurrent_step.cuh"

namespace gdn {

constexpr int kBlkTok = 16;   // tokens per block
constexpr int kBlkRows = 16;  // state rows of a group of four warps
__host__ __device__ constexpr int blk_threads(int groups) { return 128 * (groups + 1); }

template <int DK, int kGroups>
struct BlockSmem {
    static constexpr int kRows = kGroups * kBlkRows;  // of the CTA
    // rows of k and q are 16 bytes longer than the data: eight rows at one column lie in different banks
    static constexpr int kRow = DK * 2 + 16;
    static constexpr int kOffQ = kBlkTok * kRow, kOffV = 2 * kBlkTok * kRow;
    // What the outputs are made of, per group scale G_t (S_0 q_t) and c, 16 rows of 16 tokens each: over q once the group has its
    // products, behind v where there is another group that may still be at its own.
    static constexpr int kOut = 2 * kBlkRows * kBlkTok * 4, kOffO = kGroups == 1 ? kOffQ : kOffV + kBlkTok * kRows * 2;
    static constexpr int kOffC1 = kOffO + kBlkRows * kBlkTok * 4;
    static constexpr int kStage = kOffV + kBlkTok * kRows * 2 + (kGroups == 1 ? 0 : kGroups * kOut);
    static constexpr int kStages = 4;  // one per preparing warp
    static_assert(kGroups > 1 || kOffO + kOut <= kOffV, "they fit over q");
    // what a block's solve needs, floats: A as [s][t], P as [t][s], beta v as [row][t] (before that: decay products), factors
    static constexpr int kA = 0, kP = 256, kR0 = 512, kLdR = 20, kCk = kR0 + kRows * kLdR, kCq = kCk + 16, kW = kCq + 16, kG = kW + 16;
    static constexpr int kPrepFloats = kG + 4;
    static constexpr int kOffPrep = kStages * kStage;
    static constexpr int kLdD = 36;  // partial products of a warp: 16 rows x (16 k tokens, 16 q tokens)
    static constexpr int kOffD = kOffPrep + kStages * kPrepFloats * 4;
    static constexpr int kDGroup = 2 * 4 * kBlkRows * kLdD * 4;
    static constexpr int kOffC = kOffD + kGroups * kDGroup;  // coefficients as operands: [group][term][row], 48-byte rows
    static constexpr int kRowC = 48;
    static constexpr int kBytes = kOffC + kGroups * 3 * kBlkRows * kRowC;
    static_assert(kStage % 16 == 0 && kOffPrep % 16 == 0 && (kPrepFloats * 4) % 16 == 0 && kOffD % 16 == 0 && kOffC % 16 == 0, "alignment");
};

namespace blk {
using ptx::smem_u32;
template <bool kValue>
struct Flag {  // (the run-time compiler has no standard library)
    static constexpr bool value = kValue;
};
__device__ __forceinline__ void ldmatrix_x4(uint32_t saddr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(saddr)
                 : "memory");
}
// Two fp32 values as three bf16 terms each, cut off at 8 significand bits (so that the terms add up to the value exactly).
// kSafe: an infinity is its own first term; otherwise the rest of it, inf - inf, is undefined.
template <bool kSafe>
__device__ __forceinline__ void split3(float x0, float x1, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    const uint32_t u0 = __float_as_uint(x0), u1 = __float_as_uint(x1);
    hi = __byte_perm(u0, u1, 0x7632);
    float r0 = x0 - __uint_as_float(u0 & 0xFFFF0000u), r1 = x1 - __uint_as_float(u1 & 0xFFFF0000u);
    if (kSafe) {
        r0 = r0 == r0 ? r0 : 0.f;
        r1 = r1 == r1 ? r1 : 0.f;
    }
    const uint32_t w0 = __float_as_uint(r0), w1 = __float_as_uint(r1);
    mid = __byte_perm(w0, w1, 0x7632);
    lo = __byte_perm(__float_as_uint(r0 - __uint_as_float(w0 & 0xFFFF0000u)), __float_as_uint(r1 - __uint_as_float(w1 & 0xFFFF0000u)), 0x7632);
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t bytes) {  // bytes below 16: zeros for the rest
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// this thread's arrival at `bar` once all its copies so far have landed
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// The `rank`-th packed sequence of at least `min_run` tokens, or -1.  The search starts at sequence `from` with `before` such sequences in
// front of it and leaves both where the one found can be found again.  All lanes of a warp.
__device__ __forceinline__ int long_sequence(const int* cu_seqlens, int batch, int min_run, int rank, int& from, int& before) {
    const int lane = threadIdx.x & 31;
    for (; from < batch; from += 32) {
        const int s = from + lane;
        unsigned m = __ballot_sync(0xffffffffu, s < batch && cu_seqlens[s + 1] - cu_seqlens[s] >= min_run);
        const int c = __popc(m);
        if (rank < before + c) {
            for (int i = before; i < rank; ++i) m &= m - 1;
            return from + __ffs(m) - 1;
        }
        before += c;
    }
    return -1;
}
}  // namespace blk

// Packed sequences: this launch takes those of at least p.long_run tokens, the others are gdn_recurrent_kernel's (decided per sequence,
// so that a sequence has the same bits whatever it is packed with).  How many there are is known here alone.
enum class BlkUnits {
    kPadded,  // a CTA per unit
    kPacked,  // a CTA per unit of every sequence; those of shorter ones end at once
    kWalk,    // packed, most sequences are shorter: a wave of CTAs walks the long ones' units with a stride of the grid
};
template <int DK, BlkUnits kUnits = BlkUnits::kPadded, int kGroups = 1>
__device__ __forceinline__ void gdn_recurrent_block_body(const RecurrentParams& p) {
    constexpr bool kPacked = kUnits != BlkUnits::kPadded;
    using namespace ptx;
    using namespace step;
    using namespace blk;
    using L = BlockSmem<DK, kGroups>;
    constexpr int NK = DK / 64;  // K-steps of 16 columns per warp
    static_assert(DK % 64 == 0, "four warps with whole K-steps each");
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t full[4], ready[4], done[4];  // k, q, v have landed / the block is prepared / it is through
    __shared__ int abort_flag;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    auto init_barriers = [&]() {
        for (int i = 0; i < 4; ++i) {
            mbar_init(&full[i], 32);
            mbar_init(&ready[i], 1);
            mbar_init(&done[i], 4 * kGroups);
        }
        mbar_fence_init();
    };
    if (tid == 0) {
        abort_flag = 0;
        init_barriers();
    }
    __syncthreads();
    // a programmatic dependent of the work before it; every kernel launched that way waits for the whole of its predecessor.  (Packed:
    // what precedes this launch is gdn_recurrent_kernel on the batch's other sequences.  It lets this one start when everything
    // before is complete, so only the end has to wait, for whoever waits for this grid; and that one is not let in early, its CTAs
    // would settle unevenly around those that wait here: 64 sequences of 4 tokens 56.8 -> 61.0 us.)
    if (!kPacked) {
        grid_dep_wait();
        grid_dep_launch();
    }

    const int rblocks = p.dv / L::kRows;
    auto run = [&](int seq, int head, int rb) {
        const int khead = head / (p.vh / p.kh);
        long long tok0 = 0, bidx = seq;
        int ntok = p.seq_len;
        if (kPacked) {
            tok0 = p.cu_seqlens[seq];
            ntok = p.cu_seqlens[seq + 1] - static_cast<int>(tok0);
            bidx = 0;
        }
        if (p.num_accepted) ntok = min(ntok, p.num_accepted[seq]);
        const int slot = p.state_idx ? p.state_idx[seq] : seq;
        if (slot < 0) return;  // padding sequence: no tokens, no state
        const int nblk = ntok > 0 ? (ntok + kBlkTok - 1) / kBlkTok : 0;
        // ldmatrix: lane l addresses row l & 7 of 8x8 matrix l >> 3; matrices 1 and 3 are rows 8 .. 15, matrices 2 and 3 columns 8 .. 15
        const int lm_row = lane & 15, lm_col = 8 * (lane >> 4);
        auto prep_of = [&](int b) { return reinterpret_cast<float*>(smem + L::kOffPrep) + (b & 3) * L::kPrepFloats; };

        if (warp >= 4 * kGroups) {
            // =============================================================== preparation and outputs
            const int j = warp - 4 * kGroups;
            uint8_t* const st = smem + j * L::kStage;
            float* const pr = prep_of(j);
            float* const X = pr + L::kR0;  // [t][s] = Gamma_ts, [t][16] = G_t, [t][17], [t][18] = inverse norms of k_t, q_t
            const __nv_bfloat16* const kp = p.k + bidx * p.k_sb + tok0 * p.k_st + khead * p.k_sh;
            const __nv_bfloat16* const qp = p.q + bidx * p.q_sb + tok0 * p.q_st + khead * p.q_sh;
            const __nv_bfloat16* const vp = p.v + bidx * p.v_sb + tok0 * p.v_st + head * p.v_sh + rb * L::kRows;
            const int r = lane & 15, h = lane >> 4;  // for the outputs: row r, tokens 8 h .. 8 h + 7
            __nv_bfloat16* const out = p.out + bidx * p.o_sb + tok0 * p.o_st + head * p.o_sh + rb * L::kRows + r;
            float al = 0.f, db = 0.f;
            if (p.fused_gating) {
                al = __expf(from_bits(ld_bits(p.A_log, p.gating_param_f32, head), p.gating_param_f32));
                db = from_bits(ld_bits(p.dt_bias, p.gating_param_f32, head), p.gating_param_f32);
            }
            uint32_t b_next = 0u, g_next = 0u;  // bits of beta and the gate (or of the raw projections) of token `lane` of the next block
            auto fetch = [&](int b) {
                b_next = g_next = 0u;
                const long long i = static_cast<long long>(b) * kBlkTok + lane;
                if (lane < kBlkTok && i < ntok) {
                    b_next = ld_bits(p.beta, p.beta_f32, bidx * p.beta_sb + (tok0 + i) * p.beta_st + head * p.beta_sh);
                    if (p.gate) g_next = ld_bits(p.gate, p.gate_f32, bidx * p.gate_sb + (tok0 + i) * p.gate_st + head * p.gate_sh);
                }
            };
            fetch(j);
            // false once a wait has given up.  Every lane polls for itself and the answers of two lanes can differ, so the loop is walked to its end: a
            // warp whose lanes parted here would hang in its next shuffle.
            bool ok = true;
            for (int b = j; b < nblk + 4; b += 4) {
                const uint32_t it = static_cast<uint32_t>(b >> 2);
                const bool next = b < nblk;
                const int n = min(kBlkTok, ntok - b * kBlkTok);
                float o[kGroups][8], c0[kGroups][8], c1[kGroups][8];
                if (b >= 4) {  // block b - 4 is through: what its outputs are made of
                    ok = mbar_wait(&done[j], (it - 1) & 1u, &abort_flag) && ok;
                    auto row8 = [&](int off, int c, float* x) {
                        const float4 u = *reinterpret_cast<const float4*>(st + off + row64_off(r, c));
                        const float4 w = *reinterpret_cast<const float4*>(st + off + row64_off(r, c + 1));
                        x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w; x[4] = w.x; x[5] = w.y; x[6] = w.z; x[7] = w.w;
                    };
#pragma unroll
                    for (int q = 0; q < kGroups; ++q) {
                        row8(L::kOffO + q * L::kOut, 2 * h, o[q]);
                        row8(L::kOffC1 + q * L::kOut, 0, c0[q]);
                        row8(L::kOffC1 + q * L::kOut, 2, c1[q]);
                    }
                    __syncwarp();
                }
                if (next) {
                    // rows past the end of the sequence are filled with zeros (their address is that of the last row)
                    constexpr int kPieces = DK / 8;
                    const uint32_t dst = smem_u32(st);
#pragma unroll 4
                    for (int i = lane; i < kBlkTok * kPieces; i += 32) {
                        const int row = i / kPieces, c = i % kPieces;
                        const long long at = static_cast<long long>(b) * kBlkTok + min(row, n - 1);
                        const uint32_t bytes = row < n ? 16u : 0u;
                        cp_async16(dst + row * L::kRow + 16 * c, kp + at * p.k_st + 8 * c, bytes);
                        cp_async16(dst + L::kOffQ + row * L::kRow + 16 * c, qp + at * p.q_st + 8 * c, bytes);
                    }
#pragma unroll
                    for (int i = lane; i < 32 * kGroups; i += 32) {
                        const int row = i / (2 * kGroups);
                        const long long at = static_cast<long long>(b) * kBlkTok + min(row, n - 1);
                        cp_async16(dst + L::kOffV + 16 * i, vp + at * p.v_st + 8 * (i % (2 * kGroups)), row < n ? 16u : 0u);
                    }
                    cp_async_arrive(&full[j]);
                }
                if (b >= 4) {
                    // ---- outputs of block b - 4.  Coefficients of later tokens are left out, not multiplied by zero: an infinite or
                    //      undefined value stays behind its token.
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float* const P = pr + L::kP + (8 * h + i) * 16;
                        const float4 u = *reinterpret_cast<const float4*>(P), w = *reinterpret_cast<const float4*>(P + 4);
                        const float pw[8] = {u.x, u.y, u.z, u.w, w.x, w.y, w.z, w.w};
#pragma unroll
                        for (int q = 0; q < kGroups; ++q) {
#pragma unroll
                            for (int s = 0; s < 8; ++s)
                                if (s <= i || h) o[q][i] = fmaf(pw[s], c0[q][s], o[q][i]);
                        }
                        if (h) {
                            const float4 y = *reinterpret_cast<const float4*>(P + 8), z = *reinterpret_cast<const float4*>(P + 12);
                            const float pz[8] = {y.x, y.y, y.z, y.w, z.x, z.y, z.z, z.w};
#pragma unroll
                            for (int q = 0; q < kGroups; ++q) {
#pragma unroll
                                for (int s = 0; s <= i; ++s) o[q][i] = fmaf(pz[s], c1[q][s], o[q][i]);
                            }
                        }
                    }
                    __syncwarp();
                    const bool good = ok && *static_cast<volatile int*>(&abort_flag) == 0;  // nothing is stored once a wait has given up
                    const long long i0 = static_cast<long long>(b - 4) * kBlkTok + 8 * h;
#pragma unroll
                    for (int q = 0; q < kGroups; ++q) {
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            if (good && i0 + i < ntok) out[(i0 + i) * p.o_st + q * kBlkRows] = __float2bfloat16(o[q][i]);
                    }
                }
                if (!next) break;
                // ---- scalars; tokens past the end: beta 0, decay 1
                float beta = from_bits(b_next, p.beta_f32), gate = from_bits(g_next, p.gate_f32);
                if (p.fused_gating) {
                    // softplus and sigmoid on the fast exponential, logarithm and reciprocal, as in recurrent.cuh
                    const float x = gate + db, e = __expf(x);
                    gate = -al * (x > 20.f ? x : (x < -15.f ? e : __logf(1.f + e)));
                    beta = __fdividef(1.f, 1.f + __expf(-beta));
                }
                const bool real = lane < n;
                const float a = real ? __expf(gate) : 1.f;
                if (!real) beta = 0.f;
                fetch(b + 4);
                float run = 1.f;
#pragma unroll
                for (int i = 0; i < kBlkTok; ++i) {
                    const float ai = __shfl_sync(0xffffffffu, a, i);
                    if (lane == 16 || lane < i) run *= ai;
                    if (lane <= 16) X[i * L::kLdR + lane] = run;  // (entries s > t are not used)
                }
                ok = mbar_wait(&full[j], it & 1u, &abort_flag) && ok;
                // ---- Gram matrices.  kk, qk: tokens 0 .. 15 against tokens 0 .. 7 of k; hh: tokens 8 .. 15 of k and of q against tokens
                //      8 .. 15 of k; qq: the diagonals of q q^T.  The matrix instructions cut their sums off, so only two follow one another.
                float kk[4] = {}, qk[4] = {}, hh[4] = {}, qq0[4] = {}, qq1[4] = {};
                const uint32_t kaddr = smem_u32(st) + lm_row * L::kRow + lm_col * 2, qaddr = kaddr + L::kOffQ;
#pragma unroll 2
                for (int ks = 0; ks < DK / 16; ks += 2) {
                    uint32_t x[2][4], y[2][4];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        ldmatrix_x4(kaddr + 32 * (ks + e), x[e]);
                        ldmatrix_x4(qaddr + 32 * (ks + e), y[e]);
                    }
                    float s0[4] = {}, s1[4] = {}, s2[4] = {};
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const uint32_t h[4] = {x[e][1], y[e][1], x[e][3], y[e][3]};
                        mma_16816(s0, x[e], x[e][0], x[e][2]);
                        mma_16816(s1, y[e], x[e][0], x[e][2]);
                        mma_16816(s2, h, x[e][1], x[e][3]);
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        kk[e] += s0[e];
                        qk[e] += s1[e];
                        hh[e] += s2[e];
                    }
                    if (p.is_qk_norm) {
                        float s3[4] = {}, s4[4] = {};
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            mma_16816(s3, y[e], y[e][0], y[e][2]);
                            mma_16816(s4, y[e], y[e][1], y[e][3]);
                        }
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            qq0[e] += s3[e];
                            qq1[e] += s4[e];
                        }
                    }
                }
                if (t == (g >> 1)) {  // this lane holds the diagonal entries of tokens g and g + 8
                    float r0 = 1.f, r1 = 1.f, r2 = 1.f, r3 = 1.f;
                    if (p.is_qk_norm) {
                        r0 = rsqrtf(((g & 1) ? kk[1] : kk[0]) + 1e-6f);
                        r1 = rsqrtf(((g & 1) ? hh[1] : hh[0]) + 1e-6f);
                        r2 = rsqrtf(((g & 1) ? qq0[1] : qq0[0]) + 1e-6f);
                        r3 = rsqrtf(((g & 1) ? qq1[3] : qq1[2]) + 1e-6f);
                    }
                    X[g * L::kLdR + 17] = r0;
                    X[(g + 8) * L::kLdR + 17] = r1;
                    X[g * L::kLdR + 18] = r2;
                    X[(g + 8) * L::kLdR + 18] = r3;
                }
                __syncwarp();
                const float beta_g = __shfl_sync(0xffffffffu, beta, g), beta_h = __shfl_sync(0xffffffffu, beta, g + 8);
                const float rk_g = X[g * L::kLdR + 17], rk_h = X[(g + 8) * L::kLdR + 17];
                const float rq_g = p.scale * X[g * L::kLdR + 18], rq_h = p.scale * X[(g + 8) * L::kLdR + 18];
                // [s][t] = beta_t Gamma_ts k_s.k_t  and  [t][s] = scale Gamma_ts k_s.q_t (entries s >= t and s > t are not read)
                auto put = [&](int ti, int si, float kkv, float qkv, float bt, float rq) {
                    const float w = X[ti * L::kLdR + si] * X[si * L::kLdR + 17];
                    pr[L::kA + si * 16 + ti] = bt * w * kkv;
                    pr[L::kP + ti * 16 + si] = rq * w * qkv;
                };
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int s0 = 2 * t + e;
                    put(g, s0, kk[e], qk[e], beta_g * rk_g, rq_g);
                    put(g + 8, s0, kk[2 + e], qk[2 + e], beta_h * rk_h, rq_h);
                    put(g + 8, s0 + 8, hh[e], hh[2 + e], beta_h * rk_h, rq_h);
                }
                if (lane < kBlkTok) {
                    const float G = X[lane * L::kLdR + 16], rk = X[lane * L::kLdR + 17], rq = X[lane * L::kLdR + 18];
                    pr[L::kCk + lane] = beta * G * rk;
                    pr[L::kCq + lane] = p.scale * G * rq;
                    pr[L::kW + lane] = real ? X[(n - 1) * L::kLdR + lane] * rk : 0.f;
                    if (lane == n - 1) pr[L::kG] = G;
                }
                __syncwarp();
                // ---- beta v over the decay products
                {
                    const int tk = lane & 15;
                    const float bt = __shfl_sync(0xffffffffu, beta, tk);
#pragma unroll
                    for (int q = 0; q < kGroups; ++q) {
                        const uint4 v = *reinterpret_cast<const uint4*>(st + L::kOffV + tk * L::kRows * 2 + 32 * q + 16 * (lane >> 4));
                        float* const R = X + (kBlkRows * q + 8 * (lane >> 4)) * L::kLdR + tk;
                        const uint32_t vw[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            R[(2 * i) * L::kLdR] = bt * bf16_lo(vw[i]);
                            R[(2 * i + 1) * L::kLdR] = bt * bf16_hi(vw[i]);
                        }
                    }
                }
                __syncwarp();
                if (lane == 0 && ok) mbar_arrive(&ready[j]);  // not handed on once a wait has given up: the other warps' waits end with it
            }
        } else {
            // =============================================================== state
            const int rg = kGroups > 1 ? warp >> 2 : 0, qw = kGroups > 1 ? warp & 3 : warp;  // group of rows, quarter of the columns
            const int col0 = qw * (DK / 4);
            const int r = 4 * qw + (lane >> 3), j2 = 2 * (lane & 7);  // in the solve: row r of the group, tokens j2 and j2 + 1
            float S[2 * NK][4];  // 8 columns each: rows g (0, 1) and g + 8 (2, 3), columns 2t, 2t + 1
            const long long srow = static_cast<long long>(rb * L::kRows + rg * kBlkRows + g) * DK + col0 + 2 * t;
            if (p.state_in) {
                const long long base = static_cast<long long>(slot) * p.si_ss + head * p.si_sh + srow;
#pragma unroll
                for (int i = 0; i < 2 * NK; ++i) {
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const uint32_t w = *reinterpret_cast<const uint32_t*>(static_cast<const __nv_bfloat16*>(p.state_in) + base + 8 * e * DK + 8 * i);
                        S[i][2 * e] = bf16_lo(w);
                        S[i][2 * e + 1] = bf16_hi(w);
                    }
                }
            } else {
#pragma unroll
                for (int i = 0; i < 2 * NK; ++i) S[i][0] = S[i][1] = S[i][2] = S[i][3] = 0.f;
            }
            uint8_t* const sc = smem + L::kOffC + rg * (3 * kBlkRows * L::kRowC);
            auto group_sync = [&]() {
                if (kGroups == 1 || rg == 0)
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                else
                    asm volatile("bar.sync 2, 128;" ::: "memory");
            };
            bool ok = true;  // false once a wait has given up: nothing is stored from then on
            bool ahead = false;  // this lane has seen the next block's preparation complete
            for (int b = 0; b < nblk; ++b) {
                ok = (ahead || mbar_wait(&ready[b & 3], static_cast<uint32_t>((b >> 2) & 1), &abort_flag)) && ok;
                __syncwarp();
                const int n = min(kBlkTok, ntok - b * kBlkTok);
                uint8_t* const st = smem + (b & 3) * L::kStage;
                const float* const pr = prep_of(b);
                const uint32_t kaddr = smem_u32(st) + lm_row * L::kRow + (col0 + lm_col) * 2;
                float* const D = reinterpret_cast<float*>(smem + L::kOffD + rg * L::kDGroup) + (b & 1) * (4 * kBlkRows * L::kLdD);
                // ---- this warp's columns of S_0 [k; q]^T: tokens 0 - 7 and 8 - 15 of k, then of q.  The first terms have sums of their own:
                //      they are the long ones, and the chains are shorter.
                {
                    float dh[4][4], dl[4][4];
                    auto products = [&](auto safe_tag) {
                        constexpr bool kSafe = decltype(safe_tag)::value;
#pragma unroll
                        for (int i = 0; i < 4; ++i)
#pragma unroll
                            for (int e = 0; e < 4; ++e) dh[i][e] = dl[i][e] = 0.f;
                        uint32_t x[2][4], y[2][4];
                        ldmatrix_x4(kaddr, x[0]);
                        ldmatrix_x4(kaddr + L::kOffQ, y[0]);
#pragma unroll
                        for (int kc = 0; kc < NK; ++kc) {
                            if (kc + 1 < NK) {
                                ldmatrix_x4(kaddr + 32 * (kc + 1), x[(kc + 1) & 1]);
                                ldmatrix_x4(kaddr + L::kOffQ + 32 * (kc + 1), y[(kc + 1) & 1]);
                            }
                            const uint32_t* const xk = x[kc & 1];
                            const uint32_t* const yk = y[kc & 1];
                            uint32_t hi[4], mid[4], lo[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const float* s = &S[2 * kc + (e >> 1)][2 * (e & 1)];
                                split3<kSafe>(s[0], s[1], hi[e], mid[e], lo[e]);
                            }
                            mma_16816(dl[0], lo, xk[0], xk[2]);
                            mma_16816(dl[1], lo, xk[1], xk[3]);
                            mma_16816(dl[2], lo, yk[0], yk[2]);
                            mma_16816(dl[3], lo, yk[1], yk[3]);
                            mma_16816(dh[0], hi, xk[0], xk[2]);
                            mma_16816(dh[1], hi, xk[1], xk[3]);
                            mma_16816(dh[2], hi, yk[0], yk[2]);
                            mma_16816(dh[3], hi, yk[1], yk[3]);
                            mma_16816(dl[0], mid, xk[0], xk[2]);
                            mma_16816(dl[1], mid, xk[1], xk[3]);
                            mma_16816(dl[2], mid, yk[0], yk[2]);
                            mma_16816(dl[3], mid, yk[1], yk[3]);
                        }
                    };
                    products(Flag<false>{});
                    // a row of the state with an infinity has undefined low terms in every column: taken again with care
                    const float chk = dl[0][0] + dl[0][2];
                    if (__any_sync(0xffffffffu, chk != chk)) products(Flag<true>{});
                    float* const d = D + (qw * kBlkRows + g) * L::kLdD + 2 * t;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        *reinterpret_cast<float2*>(d + 8 * i) = make_float2(dh[i][0] + dl[i][0], dh[i][1] + dl[i][1]);
                        *reinterpret_cast<float2*>(d + 8 * L::kLdD + 8 * i) = make_float2(dh[i][2] + dl[i][2], dh[i][3] + dl[i][3]);
                    }
                }
                group_sync();
                // ---- c of row r, tokens j2 and j2 + 1: right-hand sides, then forward substitution token by token, a row in eight lanes
                float2 cc;
                {
                    const float* const d = D + r * L::kLdD + j2;
                    float2 x[4];
#pragma unroll
                    for (int w = 0; w < 4; ++w) x[w] = *reinterpret_cast<const float2*>(d + w * (kBlkRows * L::kLdD));
                    const float2 bv = *reinterpret_cast<const float2*>(pr + L::kR0 + (rg * kBlkRows + r) * L::kLdR + j2);
                    const float2 ck = *reinterpret_cast<const float2*>(pr + L::kCk + j2);
                    cc.x = fmaf(-ck.x, (x[0].x + x[1].x) + (x[2].x + x[3].x), bv.x);
                    cc.y = fmaf(-ck.y, (x[0].y + x[1].y) + (x[2].y + x[3].y), bv.y);
                    // (what a token gets from the tokens before it is summed apart from its own, larger, term; those behind it are left out, not
                    // multiplied by zero)
                    float2 acc = make_float2(0.f, 0.f);
                    const float own = pr[L::kA + j2 * 16 + j2 + 1];
#pragma unroll
                    for (int i = 0; i < kBlkTok / 2 - 1; ++i) {
                        const float2 a0 = *reinterpret_cast<const float2*>(pr + L::kA + (2 * i) * 16 + j2);  // columns 2 i, 2 i + 1 of A
                        const float2 a1 = *reinterpret_cast<const float2*>(pr + L::kA + (2 * i + 1) * 16 + j2);
                        const float x0 = cc.x - acc.x, x1 = cc.y - fmaf(own, x0, acc.y);  // c of two tokens, in the lane whose turn it is
                        const float c0 = __shfl_sync(0xffffffffu, x0, (lane & 24) | i), c1 = __shfl_sync(0xffffffffu, x1, (lane & 24) | i);
                        if (j2 > 2 * i) {
                            acc.x = fmaf(a1.x, c1, fmaf(a0.x, c0, acc.x));
                            acc.y = fmaf(a1.y, c1, fmaf(a0.y, c0, acc.y));
                        }
                    }
                    cc.x -= acc.x;
                    cc.y -= fmaf(own, cc.x, acc.y);
                    if (n < kBlkTok) {  // tokens past the end: nothing, whatever the state holds
                        if (j2 >= n) cc.x = 0.f;
                        if (j2 + 1 >= n) cc.y = 0.f;
                    }
                }
                // ---- S <- G S + sum_s (Gamma_ns r_s c_s) k_s^T
                {
                    {
                        const float2 w = *reinterpret_cast<const float2*>(pr + L::kW + j2);
                        uint32_t h, m, l;
                        split3<true>(w.x * cc.x, w.y * cc.y, h, m, l);
                        uint8_t* const o = sc + r * L::kRowC + 2 * j2;
                        *reinterpret_cast<uint32_t*>(o) = h;
                        *reinterpret_cast<uint32_t*>(o + kBlkRows * L::kRowC) = m;
                        *reinterpret_cast<uint32_t*>(o + 2 * kBlkRows * L::kRowC) = l;
                        *reinterpret_cast<float2*>(st + L::kOffC1 + rg * L::kOut + row64_off(r, j2 >> 2) + 4 * (j2 & 2)) = cc;  // for the outputs
                    }
                    group_sync();
                    uint32_t hi[4], mid[4], lo[4];
                    const uint32_t caddr = smem_u32(sc) + lm_row * L::kRowC + lm_col * 2;
                    ldmatrix_x4(caddr, hi);
                    ldmatrix_x4(caddr + kBlkRows * L::kRowC, mid);
                    ldmatrix_x4(caddr + 2 * kBlkRows * L::kRowC, lo);
                    const float G = pr[L::kG];
#pragma unroll
                    for (int kc = 0; kc < NK; ++kc) {
                        uint32_t x[4];
                        ldmatrix_x4_trans(kaddr + 32 * kc, x);  // tokens of k in pairs, columns 0 - 7 and 8 - 15
                        // first terms and the others apart: the matrix instructions cut their sums off, which the short sums of first
                        // terms lose next to nothing by, and an fp32 addition rounds
                        float e0[4] = {0.f, 0.f, 0.f, 0.f}, e1[4] = {0.f, 0.f, 0.f, 0.f}, f0[4] = {0.f, 0.f, 0.f, 0.f}, f1[4] = {0.f, 0.f, 0.f, 0.f};
                        mma_16816(e0, lo, x[0], x[1]);
                        mma_16816(e1, lo, x[2], x[3]);
                        mma_16816(f0, hi, x[0], x[1]);
                        mma_16816(f1, hi, x[2], x[3]);
                        mma_16816(e0, mid, x[0], x[1]);
                        mma_16816(e1, mid, x[2], x[3]);
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            S[2 * kc][e] = fmaf(G, S[2 * kc][e], f0[e] + e0[e]);
                            S[2 * kc + 1][e] = fmaf(G, S[2 * kc + 1][e], f1[e] + e1[e]);
                        }
                    }
                }
                // ---- for the outputs: this warp's quarter of scale G_t (S_0 q_t)
                {
                    const float* const d = D + r * L::kLdD + 16 + j2;
                    float2 x[4];
#pragma unroll
                    for (int w = 0; w < 4; ++w) x[w] = *reinterpret_cast<const float2*>(d + w * (kBlkRows * L::kLdD));
                    const float2 cq = *reinterpret_cast<const float2*>(pr + L::kCq + j2);
                    ahead = b + 1 < nblk && mbar_try_wait(&ready[(b + 1) & 3], static_cast<uint32_t>(((b + 1) >> 2) & 1));
                    *reinterpret_cast<float2*>(st + L::kOffO + rg * L::kOut + row64_off(r, j2 >> 2) + 4 * (j2 & 2)) =
                        make_float2(cq.x * ((x[0].x + x[1].x) + (x[2].x + x[3].x)), cq.y * ((x[0].y + x[1].y) + (x[2].y + x[3].y)));
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&done[b & 3]);
            }
            if (ok && *static_cast<volatile int*>(&abort_flag) == 0) {
                const long long base = static_cast<long long>(slot) * p.so_ss + head * p.so_sh + srow;
#pragma unroll
                for (int i = 0; i < 2 * NK; ++i) {
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        *reinterpret_cast<uint32_t*>(static_cast<__nv_bfloat16*>(p.state_out) + base + 8 * e * DK + 8 * i) = pack_bf16(S[i][2 * e], S[i][2 * e + 1]);
                    }
                }
            }
        }
    };  // run

    if constexpr (kUnits == BlkUnits::kWalk) {
        // (the walk's state is in shared memory: registers are all taken)
        __shared__ long long s_unit;
        __shared__ int s_seq, s_from, s_before;
        if (tid == 0) {
            s_unit = blockIdx.x;
            s_from = s_before = 0;
        }
        while (true) {
            __syncthreads();
            if (tid < 32) {
                int from = s_from, before = s_before;
                const int seq = long_sequence(p.cu_seqlens, p.batch, p.long_run, static_cast<int>(s_unit / (p.vh * rblocks)), from, before);
                __syncwarp();
                if (tid == 0) {
                    s_seq = seq;
                    s_from = from;
                    s_before = before;
                }
            }
            __syncthreads();
            if (s_seq < 0) break;
            const int rem = static_cast<int>(s_unit % (p.vh * rblocks));
            run(s_seq, rem / rblocks, rem % rblocks);
            if (__syncthreads_or(abort_flag)) break;  // no warp waits on the unit's barriers any more
            if (tid == 0) {
                for (int i = 0; i < 4; ++i) {
                    mbar_inval(&full[i]);
                    mbar_inval(&ready[i]);
                    mbar_inval(&done[i]);
                }
                init_barriers();
                s_unit += gridDim.x;
            }
        }
    } else {
        const int unit = static_cast<int>(blockIdx.x) / rblocks, rb = static_cast<int>(blockIdx.x) - unit * rblocks;
        const int seq = unit / p.vh, head = unit - seq * p.vh;
        if (!kPacked || p.cu_seqlens[seq + 1] - p.cu_seqlens[seq] >= p.long_run) run(seq, head, rb);
    }
    if (kPacked) grid_dep_wait();
    __syncthreads();
    if (abort_flag) {
        cp_async_wait_all();  // the copies whose wait gave up
        if (tid == 0 && p.status) atomicExch(p.status, 1);
    }
}

template <int DK, BlkUnits kUnits = BlkUnits::kPadded, int kGroups = 1>
__global__ void __launch_bounds__(blk_threads(kGroups), kGroups == 1 ? 2 : 1) gdn_recurrent_block_kernel(const RecurrentParams p) {
    gdn_recurrent_block_body<DK, kUnits, kGroups>(p);
}

}  // namespace gdn
