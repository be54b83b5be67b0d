// Chunk-parallel stage of the whole-layer chunked prefill (gdn_chunked_forward).
//
// Per (64-token chunk, v-head), with g the chunk-local cumulative gate, g_L its last value and
//     A = tril(diag(beta) K K^T .* exp(g_i - g_j), -1),   X = (I + A)^-1,   T = X diag(beta)
//     P = scale * tril(Q K^T .* exp(g_i - g_j))
// the kernel writes the two matrices the sequential state kernel (prefill_fused.cuh) consumes:
//     Z  = T^T diag(exp(g_L - g)) K      (64 x dk, bf16)
//     PT = P T                           (64 x 64, bf16)
// They fold the WY/UT transform into the chunk-to-chunk recurrence: with R = V - exp(g) .* (K S^T)
//     U_new = T R,   S <- exp(g_L) S + R^T Z,   O = scale * exp(g) .* (Q S^T) + PT R
// so U = T V and W = T (K .* exp(g)) (what the reference's sm90_bf16_compute_u_w writes,
// gdn_cuda/include/gdn_cuda/kernels/sm90_bf16_gdn_compute_u_w.cuh:153-667) never exist, V is not
// read here at all, and the scratch per unit is 24 KB instead of 40 KB.
//
// Work unit = (chunk, k-head): the K and Q tiles are loaded once and K K^T, Q K^T are computed once
// (one M=128 tcgen05 MMA group whose A operand is K stacked on Q) for all the v-heads of the
// k-head group; only beta and the gate differ between them.  A CTA of 256 threads is two teams of
// four warps, each team taking one v-head of the group at a time: A / P pass from tensor memory, inverse row block by row
// block in registers, T and (diag(d) T)^T as bf16 tiles, then M=64 MMAs (Z, and PT) and the bf16 epilogue into a staging
// area that leaves by one bulk copy.
// The inverse: 16x16 diagonal blocks in fp32 (8x8 forward substitution and one TF32 doubling step).  Then warp r owns row
// block r of X and walks it from the diagonal to the left, X_rc = -(sum_{c<m<=r} X_rm A_mc) inv_cc, which needs nothing of
// the other row blocks: the blocks of X stay accumulator fragments, which are the A operands of the next products as they
// lie; A and the inverses are B operands in shared memory.  All of them enter the products as two bf16 terms (16
// significand bits; a doubling scheme on TF32, 11 bits, was here before).
// What bounds it: the latency of a unit's dependent phases (11 200 cycles with four teams per SM, 8 700 with two; before
// 12 100).  The doubling scheme had ten barriers per unit (five now), 5 660 warp instructions (4 990) and 1 808 wavefronts (1 220) of
// shared-memory accesses, besides some 900 of MMA operands and copies, of the 3 000 cycles a unit took an SM.
// Whole calls with the doubling scheme and now, in turn on one GPU: B=4 T=4096, 32 v-heads 215.4 -> 210.3 us; 16 packed sequences of 32768
// tokens 457.6 -> 437.9; B=2 T=131072, 4 v-heads 621.7 -> 599.9.
// Not kept: two of A's seven blocks of warp 1 made by warp 0 from their mirror images and both diagonal blocks of a warp inverted in its 32
// lanes, with a barrier less (the critical path 700 cycles shorter on paper): 206.8 -> 208.3 us.
// Persistent CTAs, two per SM (111 KB of shared memory, 256 tensor-memory columns each).
#pragma once
#include <cuda.h>

#include <type_traits>

#include "prefill_common.cuh"
#include "prefill_uw.cuh"  // uw:: helpers (TF32 block products, packed fp32 pairs)

namespace gdn {

struct ZPParams {
    ChunkMap map;
    ScalarView beta;
    ScalarView gate;  // raw per-token log-decay (the chunk-local cumsum is taken here); ptr == NULL: no decay
    uint8_t* blocks;  // kZPBlockBytes per (global chunk, v-head)
    float p_scale;    // output scale, folded into P
    float* norms;     // kNorm: 128 floats per (global chunk, k-head): rsqrt(sum k^2 + eps)[64], the same for q [64]
    int kh, vh;
    int num_chunks;
    int* status;
};

struct ZPSmem {
    static constexpr int kAtoms = 2;  // 64-column swizzle atoms of a K or Q tile
    // K and Q tiles interleaved atom by atom: [K cols 0-63 | Q cols 0-63 | K cols 64-127 | Q cols 64-127],
    // 8 KB each, so that rows 0-127 of one atom pair are K stacked on Q (the M=128 A operand)
    static constexpr int kOffKQ = 0;
    static constexpr int kTeam = kAtoms * 16384;         // per-team area starts here, two of them
    static constexpr int kOffT = 0, kOffTd = 8192;       // T and dT (8 KB each), later the staged Z
    static constexpr int kOffP = 16384;                  // P tile (8 KB), later the staged PT
    // 16x16 blocks of A below the diagonal, block (r, c) at r (r - 1) / 2 + c, as two bf16 terms
    static constexpr int kOffA = kOffP + 8192;
    // diagonal blocks of A in fp32, 20 floats per row; each makes way for its inverse as two bf16 terms
    static constexpr int kLdD = 20, kDiag = 16 * kLdD * 4;
    static constexpr int kOffDiag = kOffA + 6 * 1024;
    static constexpr int kOffVec = kOffDiag + 4 * kDiag;  // beta[64], d[64], then per warp g log2e[64] and column factors[80]
    static constexpr int kTeamBytes = kOffVec + 3072;    // a multiple of 1024
    static constexpr int kOffNorm = kTeam + 2 * kTeamBytes;  // kNorm: inverse row norms of K [64] and Q [64]
    static constexpr int kOffBar = kOffNorm + 512;
    static constexpr int kUnits = 64;                    // coordinates of this CTA's coming work units, 16 bytes each
    static constexpr int kOffUnits = kOffBar + 128;
    static constexpr int kBytes = kOffUnits + 16 * kUnits + 1024;
    static_assert(kTeamBytes % 1024 == 0, "swizzled tiles need 1024-byte alignment");
    static_assert(kDiag >= 1024 && kDiag % 128 == 0, "the inverse of a diagonal block fits over it");
};

namespace zp {
using namespace ptx;
constexpr int kThreads = 256;
constexpr uint32_t kTmKQ = 0;    // fp32 K K^T (lanes 0-63) and Q K^T (lanes 64-127), 64 columns
constexpr uint32_t kTmPT = 64;   // PT of team 0 (lanes +0) and team 1 (lanes +16), 64 columns
constexpr uint32_t kTmZ = 128;   // Z, 128 columns (lanes +0: team 0, +16: team 1)
// the two warps of a team that write P
__device__ __forceinline__ void pair_sync(int team) { asm volatile("bar.sync %0, 64;" ::"r"(3 + team) : "memory"); }
// TF32 operands of the 8 -> 16 step of the inverse: 8x8 block of `m` at [r0][k0] as the upper half of the A operand (the lower is
// zero), at [k0][n0] as the B operand
__device__ __forceinline__ void load_a8(uint32_t* a, const float* m, int ld, int r0, int k0, int lane) {
    const int g = lane >> 2, t = lane & 3;
    a[0] = uw::to_tf32(m[(r0 + g) * ld + k0 + t]);
    a[1] = 0u;
    a[2] = uw::to_tf32(m[(r0 + g) * ld + k0 + t + 4]);
    a[3] = 0u;
}
__device__ __forceinline__ void load_b8(uint32_t* b, const float* m, int ld, int k0, int n0, int lane) {
    const int g = lane >> 2, t = lane & 3;
    b[0] = uw::to_tf32(m[(k0 + t) * ld + n0 + g]);
    b[1] = uw::to_tf32(m[(k0 + t + 4) * ld + n0 + g]);
}
__device__ __forceinline__ void team_sync(int team) {
    if (team)
        asm volatile("bar.sync 2, 128;" ::: "memory");
    else
        asm volatile("bar.sync 1, 128;" ::: "memory");
}
// A 16x16 block as two bf16 terms: 16 rows of 64 bytes (row64_off), 16-byte pieces { first terms of columns 0-7, 8-15, second terms
// of the same }.
// two fp32 values as two bf16 terms each
__device__ __forceinline__ void split2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
    hi = pack_bf16(x0, x1);
    lo = pack_bf16(x0 - bf16_lo(hi), x1 - bf16_hi(hi));
}
// a 16x16 accumulator fragment (two halves of 8 columns) as the A operand of the next product, two terms
__device__ __forceinline__ void split_frag(const float (*x)[4], uint32_t* hi, uint32_t* lo) {
#pragma unroll
    for (int i = 0; i < 4; ++i) split2(x[i >> 1][2 * (i & 1)], x[i >> 1][2 * (i & 1) + 1], hi[i], lo[i]);
}
// acc += X B for 16x16 blocks: X as fragments of two terms, B in shared memory (`b_lane`: its address plus row64_off(lane & 15,
// lane >> 4)); the product of the second terms is below 2^-16 of the result
__device__ __forceinline__ void mma_blk16(float (*acc)[4], const uint32_t* xh, const uint32_t* xl, uint32_t b_lane) {
    uint32_t bh[4], bl[4];  // { columns 0-7: rows 0-7, 8-15; columns 8-15: the same }
    ldmatrix_x4_trans(b_lane, bh);
    ldmatrix_x4_trans(b_lane ^ 32u, bl);  // (pieces 2, 3 of a row)
    mma_16816(acc[0], xl, bh[0], bh[1]);
    mma_16816(acc[1], xl, bh[2], bh[3]);
    mma_16816(acc[0], xh, bl[0], bl[1]);
    mma_16816(acc[1], xh, bl[2], bl[3]);
    mma_16816(acc[0], xh, bh[0], bh[1]);
    mma_16816(acc[1], xh, bh[2], bh[3]);
}
// Row block R of X = (I + A)^-1 from its diagonal block `x` on, right to left: emit(d, fragment of X_R,R-d).  (Counted by the distance from
// the diagonal, so that one copy of the code serves every R.)
template <class Emit>
__device__ __forceinline__ void row_blocks(int R, const float (*x)[4], uint32_t a_saddr, uint32_t inv_saddr, int lane, Emit emit) {
    const uint32_t lo = row64_off(lane & 15, lane >> 4);
    uint32_t xh[3][4], xl[3][4];
    uint32_t row[3];  // blocks (R - e, 0) of A, then of the present column
#pragma unroll
    for (int e = 0; e < 3; ++e) row[e] = a_saddr + lo + static_cast<uint32_t>((R - e) * (R - e - 1) / 2 + R) * 1024u;
    uint32_t inv = inv_saddr + lo + static_cast<uint32_t>(R * ZPSmem::kDiag);
    split_frag(x, xh[0], xl[0]);
    emit(std::integral_constant<int, 0>{}, x);
    auto step = [&](auto d_tag) {
        constexpr int d = decltype(d_tag)::value;
        float s[2][4] = {};
#pragma unroll
        for (int e = 0; e < d; ++e) {
            row[e] -= e + 1 < d ? 1024u : static_cast<uint32_t>(d) * 1024u;
            mma_blk16(s, xh[e], xl[e], row[e]);
        }
        uint32_t sh[4], sl[4];
        split_frag(s, sh, sl);
        float y[2][4] = {};
        inv -= ZPSmem::kDiag;
        mma_blk16(y, sh, sl, inv);
#pragma unroll
        for (int i = 0; i < 8; ++i) y[i >> 2][i & 3] = -y[i >> 2][i & 3];
        if (d < 3) split_frag(y, xh[d < 3 ? d : 0], xl[d < 3 ? d : 0]);
        emit(d_tag, y);
    };
    if (R >= 1) step(std::integral_constant<int, 1>{});
    if (R >= 2) step(std::integral_constant<int, 2>{});
    if (R >= 3) step(std::integral_constant<int, 3>{});
}
// Raw gates of the tokens `lane` and `lane + 32` -> the chunk's cumulative gate times log2(e) (decay factors are ex2 of differences).
__device__ __forceinline__ void scan_gate(float& g0, float& g1, int lane) {
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
        const float y0 = __shfl_up_sync(0xffffffffu, g0, m), y1 = __shfl_up_sync(0xffffffffu, g1, m);
        if (lane >= m) {
            g0 += y0;
            g1 += y1;
        }
    }
    g1 += __shfl_sync(0xffffffffu, g0, 31);
    g0 *= 1.4426950408889634f;
    g1 *= 1.4426950408889634f;
}
// This warp's tables: g [64], and the decay to the first token of its two row blocks (`upper`: blocks 2 and 3):
// e^{g_32 - g_j} [32], e^{g_48 - g_j} [48], or e^{g_16 - g_j} [16].
__device__ __forceinline__ void decay_tables(float g0, float g1, float* sG, float* sC, bool upper, int lane) {
    using uw::ex2;
    sG[lane] = g0;
    sG[lane + 32] = g1;
    if (upper) {
        const float r2 = __shfl_sync(0xffffffffu, g1, 0), r3 = __shfl_sync(0xffffffffu, g1, 16);
        sC[lane] = ex2(r2 - g0);
        sC[32 + lane] = ex2(r3 - g0);
        if (lane < 16) sC[64 + lane] = ex2(r3 - g1);
    } else {
        const float r1 = __shfl_sync(0xffffffffu, g0, 16);
        if (lane < 16) sC[lane] = ex2(r1 - g0);
    }
}
// Tiles and tables of a team of four warps that works on one (chunk, v-head).
struct TeamTiles {
    uint8_t* p;      // P, bf16, 128-byte rows, swizzled
    uint8_t* a;      // 16x16 blocks of A below the diagonal, block (r, c) at r (r - 1) / 2 + c, as two bf16 terms
    uint8_t* diag;   // its diagonal blocks in fp32, kDiag bytes apart; the inverses go in their place as two bf16 terms
    const float* g;  // this warp's g log2e [64]
    const float* c;  // its column factors
    const float* rn; // kNorm: inverse row norms of K [64] and Q [64]
};
// A = tril(beta_i (k_i.k_j) e^{g_i-g_j}, -1) (warps 0, 1 of the team) and P = scale tril((q_i.k_j) e^{g_i-g_j}) as a bf16 tile
// (warps 2, 3), 16x16 block by block as accumulator fragments: a warp has two rows of blocks and nothing of what lies above the
// diagonal is touched.  A: the diagonal blocks in fp32, the others as two bf16 terms.
// In a block below the diagonal e^{g_i-g_j} = e^{g_i-g_r} e^{g_r-g_j} with r the first of its rows: the column factors come from a
// table, no ex2 is left per element.  Both factors are <= 1 while the cumulative gate falls.  Where it rises they are entries of the
// same matrices (tokens i and r, r and j): neither is infinite unless the exact result is.
// `tm_kq`: column of K K^T (lanes 0-63) and Q K^T (64-127).
// A loop, block by block.  Written out (ten copies of a block, and three of row_blocks) the kernel was 67 KB of code, now 55, and waited for
// instructions in 0.60 of 9.3 warp cycles per issue, now 0.31: B=4 T=4096, 32 v-heads 208.4 -> 206.8 us a call, B=2 T=1000 41.1 -> 40.5 (two runs of
// one side differ by 0.1 to 0.3 %); 16 packed sequences of 32768 tokens 443.7 -> 438.3, within what two runs there differ by (2.5 %).
template <bool kNorm>
__device__ __forceinline__ void ap_pass(uint32_t tm_kq, const TeamTiles& t, int tw, int lane, int n, float g_mine, const float* b_mine,
                                        float p_scale) {
    using namespace uw;
    const bool is_p = tw >= 2;
    const int g = lane >> 2, tq = lane & 3, rb = tw & 1;
    const float bm = rb ? b_mine[1] : b_mine[0];
    const uint32_t pt = smem_u32(t.p) + 128u * (lane & 15);
    // `v`: products of a block, 16 rows; o: its entries [8 columns][row g: two columns, row g + 8: two]
    auto finish = [&](int r, float (*o)[4]) {
        if (n < kChunk) {  // rows past the end: nothing, whatever lies there
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (16 * r + g + 8 * ((i >> 1) & 1) >= n) o[i >> 2][i & 3] = 0.f;
        }
    };
    auto store_p = [&](int r, int c, const float (*o)[4]) {
        stmatrix_x4(pt + 2048u * r + (((2 * c + (lane >> 4)) ^ (lane & 7)) << 4), pack_bf16(o[0][0], o[0][1]), pack_bf16(o[0][2], o[0][3]),
                    pack_bf16(o[1][0], o[1][1]), pack_bf16(o[1][2], o[1][3]));
    };
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        const int r = 2 * rb + h;
        const uint32_t ta = tm_kq + (static_cast<uint32_t>(32 * tw + 16 * h) << 16);
        float gi[2], f[2];  // rows g and g + 8 of the block
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            gi[a] = __shfl_sync(0xffffffffu, g_mine, 16 * h + g + 8 * a);
            f[a] = __shfl_sync(0xffffffffu, bm, 16 * h + g + 8 * a);
            if (is_p) f[a] = p_scale;
            if (kNorm) f[a] *= t.rn[(is_p ? 64 : 0) + 16 * r + g + 8 * a];
        }
        {
            const float gr = t.g[16 * r];
            const float w0 = f[0] * ex2(gi[0] - gr), w1 = f[1] * ex2(gi[1] - gr);
            const f2 fo[2] = {pk(w0, w0), pk(w1, w1)};
            const float* const col = t.c + (rb ? 32 * h : 0) + 2 * tq;
#pragma unroll 1
            for (int c = 0; c < r; ++c) {
                uint32_t v[8];
                tmem_ld_frag16(ta + 16 * c, v);
                f2 cf[2], rn[2];
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    cf[nt] = *reinterpret_cast<const f2*>(col + 16 * c + 8 * nt);
                    if (kNorm) rn[nt] = *reinterpret_cast<const f2*>(t.rn + 16 * c + 8 * nt + 2 * tq);  // the key's norm
                }
                float o[2][4];
                tmem_wait_ld();
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
                    for (int a = 0; a < 2; ++a) {
                        f2 x = pk(__uint_as_float(v[4 * nt + 2 * a]), __uint_as_float(v[4 * nt + 2 * a + 1]));
                        if (kNorm) x = mul2(x, rn[nt]);
                        unpk(mul2(mul2(x, fo[a]), cf[nt]), o[nt][2 * a], o[nt][2 * a + 1]);
                    }
                }
                finish(r, o);
                if (is_p) {
                    store_p(r, c, o);
                } else {
                    uint32_t hi[4], lo[4];
                    split_frag(o, hi, lo);
                    const uint32_t ob = smem_u32(t.a) + static_cast<uint32_t>(r * (r - 1) / 2 + c) * 1024u;
                    stmatrix_x4(ob + row64_off(lane & 15, lane >> 4), hi[0], hi[1], hi[2], hi[3]);
                    stmatrix_x4(ob + row64_off(lane & 15, 2 + (lane >> 4)), lo[0], lo[1], lo[2], lo[3]);
                }
            }
        }
        // the diagonal block: one ex2 per element, selected
        uint32_t v[8];
        tmem_ld_frag16(ta + 16 * r, v);
        float o[2][4], e[2][4];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            const float2 cg = *reinterpret_cast<const float2*>(t.g + 16 * r + 8 * nt + 2 * tq);
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                e[nt][2 * a] = ex2(gi[a] - cg.x);
                e[nt][2 * a + 1] = ex2(gi[a] - cg.y);
            }
        }
        tmem_wait_ld();
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            const int cl = 8 * nt + 2 * tq;  // column within the block
            f2 rn = pk(1.f, 1.f);
            if (kNorm) rn = *reinterpret_cast<const f2*>(t.rn + 16 * r + cl);
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                f2 x = pk(__uint_as_float(v[4 * nt + 2 * a]), __uint_as_float(v[4 * nt + 2 * a + 1]));
                if (kNorm) x = mul2(x, rn);
                const int lim = g + 8 * a - (is_p ? 0 : 1);  // columns kept: cl <= lim
                unpk(mul2(mul2(x, pk(f[a], f[a])), pk(e[nt][2 * a], e[nt][2 * a + 1])), o[nt][2 * a], o[nt][2 * a + 1]);
                if (cl > lim) o[nt][2 * a] = 0.f;
                if (cl + 1 > lim) o[nt][2 * a + 1] = 0.f;
            }
        }
        finish(r, o);
        if (is_p) {
            store_p(r, r, o);
#pragma unroll 1
            for (int c = r + 1; c < 4; ++c) stmatrix_x4(pt + 2048u * r + (((2 * c + (lane >> 4)) ^ (lane & 7)) << 4), 0u, 0u, 0u, 0u);
        } else {
            float* const o2 = reinterpret_cast<float*>(t.diag + r * ZPSmem::kDiag) + g * ZPSmem::kLdD + 2 * tq;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                *reinterpret_cast<float2*>(o2 + (i & 1) * 8 * ZPSmem::kLdD + 8 * (i >> 1)) = make_float2(o[i >> 1][2 * (i & 1)], o[i >> 1][2 * (i & 1) + 1]);
        }
    }
}
// A diagonal block of A (fp32 at `sA`) -> its block of X = (I + A)^-1 as accumulator fragments, and in place of the block as two bf16
// terms.  The two 8x8 diagonal blocks by forward substitution in fp32 (one column per lane, 16 lanes), then X_10 = -X_11 A_10 X_00
// with two TF32 warp MMAs (the intermediate stays in registers).
__device__ __forceinline__ void invert_diagonal(float* const sA, int lane, float (*xd)[4]) {
    using namespace uw;
    const int g = lane >> 2, tq = lane & 3;
    constexpr int LD = ZPSmem::kLdD;
    const int hb = (lane >> 3) & 1, j = lane & 7;
    const int o = 8 * hb;  // first row / column of this lane's 8x8 block
    float xc[8], a[8][8];
#pragma unroll
    for (int i = 1; i < 8; ++i) {
#pragma unroll
        for (int q = 0; q < (i + 3) / 4; ++q) {
            const float4 t = *reinterpret_cast<const float4*>(&sA[(o + i) * LD + o + 4 * q]);
            a[i][4 * q] = t.x; a[i][4 * q + 1] = t.y; a[i][4 * q + 2] = t.z; a[i][4 * q + 3] = t.w;
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) xc[i] = (i == j) ? 1.f : 0.f;
    // x_j = 1, x_i = -sum_{m<i} A_im x_m
#pragma unroll
    for (int i = 1; i < 8; ++i) {
        float acc = 0.f;
#pragma unroll
        for (int m = 0; m + 1 < i; ++m) acc = fmaf(a[i][m], xc[m], acc);
        if (i > j) xc[i] = -fmaf(a[i][i - 1], xc[i - 1], acc);
    }
    __syncwarp();  // the block is private to this warp: every lane has read it
    if (lane < 16) {
#pragma unroll
        for (int i = 0; i < 8; ++i) sA[(o + i) * LD + o + j] = xc[i];
    }
    __syncwarp();
    // 8 -> 16
    float d[4] = {0.f, 0.f, 0.f, 0.f};
    uint32_t bfrag[2], afrag[4];
    load_a8(afrag, sA, LD, 8, 0, lane);
    load_b8(bfrag, sA, LD, 0, 0, lane);
    mma_tf32(d, afrag, bfrag);  // t = A_10 X_00; lane (g, t) holds t[g][2t], t[g][2t+1]
    // t as the B operand of the next product: lane (g, t) needs t[t][g] and t[t + 4][g]
    const float v00 = __shfl_sync(0xffffffffu, d[0], 4 * tq + (g >> 1));
    const float v01 = __shfl_sync(0xffffffffu, d[1], 4 * tq + (g >> 1));
    const float v10 = __shfl_sync(0xffffffffu, d[0], 4 * (tq + 4) + (g >> 1));
    const float v11 = __shfl_sync(0xffffffffu, d[1], 4 * (tq + 4) + (g >> 1));
    bfrag[0] = to_tf32((g & 1) ? v01 : v00);
    bfrag[1] = to_tf32((g & 1) ? v11 : v10);
    load_a8(afrag, sA, LD, 8, 8, lane);
    const float2 c00 = *reinterpret_cast<const float2*>(&sA[g * LD + 2 * tq]);
    const float2 c11 = *reinterpret_cast<const float2*>(&sA[(8 + g) * LD + 8 + 2 * tq]);
    float e[4] = {0.f, 0.f, 0.f, 0.f};
    mma_tf32(e, afrag, bfrag);  // X_11 t
    xd[0][0] = c00.x; xd[0][1] = c00.y; xd[0][2] = -e[0]; xd[0][3] = -e[1];
    xd[1][0] = 0.f; xd[1][1] = 0.f; xd[1][2] = c11.x; xd[1][3] = c11.y;
    __syncwarp();  // the block has been read: its inverse goes in its place, for the row blocks further down
    uint32_t hi[4], lo[4];
    split_frag(xd, hi, lo);
    const uint32_t ia = smem_u32(sA);
    stmatrix_x4(ia + row64_off(lane & 15, lane >> 4), hi[0], hi[1], hi[2], hi[3]);
    stmatrix_x4(ia + row64_off(lane & 15, 2 + (lane >> 4)), lo[0], lo[1], lo[2], lo[3]);
}
}  // namespace zp

// kNorm: q and k are L2-normalised per head (x * rsqrt(sum x^2 + 1e-6)) without touching the tiles:
// (k_i.k_j) r_i r_j and (q_i.k_j) rq_i r_j enter through a row and a column factor of the A / P pass,
// Z = (dT)^T diag(r) K through d_i r_i.  The factors are also written to `norms` for the state kernel.
template <bool kNorm>
__global__ void __launch_bounds__(zp::kThreads, 2) gdn_zp_kernel(const __grid_constant__ CUtensorMap tmK,
                                                                 const __grid_constant__ CUtensorMap tmQ,
                                                                 const ZPParams p) {
    using namespace ptx;
    using namespace uw;
    using namespace zp;
    using L = ZPSmem;
    constexpr int NA = L::kAtoms;
    extern __shared__ uint8_t smem_raw[];
    // aligned by an offset from the array itself, so that the compiler still knows the pointer is shared memory
    uint8_t* smem = smem_raw + ((1024u - (ptx::smem_u32(smem_raw) & 1023u)) & 1023u);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int team = warp >> 2, tw = warp & 3, tt = tid & 127;
    uint8_t* sKQ = smem + L::kOffKQ;
    uint8_t* tbase = smem + L::kTeam + team * L::kTeamBytes;
    uint8_t* sT = tbase + L::kOffT;    // T   = X diag(beta), rows i (128 B), columns j
    uint8_t* sTd = tbase + L::kOffTd;  // dT  = diag(d) T, same layout; read MN-major as (dT)^T
    uint8_t* sP = tbase + L::kOffP;
    float* sBeta = reinterpret_cast<float*>(tbase + L::kOffVec);
    float* sD = sBeta + 64;
    float* sG = sD + 64 + 144 * tw;  // this warp's own copy
    float* sC = sG + 64;
    float* sRn = reinterpret_cast<float*>(smem + L::kOffNorm);  // [128] inverse norms (K rows, then Q rows)
    const TeamTiles tiles{sP, tbase + L::kOffA, tbase + L::kOffDiag, sG, sC, sRn};
    uint64_t* bar_load = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
    uint64_t* bar_kq = bar_load + 1;
    uint64_t* bar_mma = bar_load + 2;  // [2], one per team
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_load + 4);
    int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
    int* teams_done = abort_flag + 1;  // teams that have finished reading the current unit's K tile

    if (tid == 0) {
        *abort_flag = 0;
        *teams_done = 0;
        mbar_init(bar_load, 1);
        mbar_init(bar_kq, 1);
        mbar_init(&bar_mma[0], 1);
        mbar_init(&bar_mma[1], 1);
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(tmem_slot, 256);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    // This kernel is launched as a programmatic dependent of whatever precedes it in the stream: it is placed
    // and set up while that work drains and waits here, before its first read of global memory.
    grid_dep_wait();
    // The state kernel that follows may be placed on SMs as this grid drains (it takes a whole SM, so
    // never beside a CTA of this kernel) and do its set-up there; it reads this kernel's results only
    // after its own grid_dep_wait.  The release comes AFTER the wait above: the state kernel loads its initial
    // state (which the work before this kernel may have produced: a state handed over from the previous call)
    // without waiting, so it must not be able to start before that work has completed.
    if (tid == 0) grid_dep_launch();

    const int rep = p.vh / p.kh;               // v-heads per k-head
    const int rounds = (rep + 1) >> 1;         // head pairs per unit
    const int total_units = p.num_chunks * p.kh;
    // Order of the work units.  Padded mode: the chunks of all sequences from the LAST chunk position to the
    // first (sequences and k-heads inside), so that what this kernel writes last - the blocks of the first
    // chunks - is what the state kernel, which starts right after it, reads first: still in L2.
    // Packed mode: chunk_indices order.
    const int per_pos = p.map.cu_seqlens ? 0 : (p.num_chunks / p.map.chunks_per_seq) * p.kh;  // units per chunk position
    auto unit_chunk = [&](int unit, int& chunk, int& khead) {
        if (per_pos) {
            const int pos = unit / per_pos, rem = unit - pos * per_pos;
            const int seq = rem / p.kh;
            khead = rem - seq * p.kh;
            chunk = seq * p.map.chunks_per_seq + (p.map.chunks_per_seq - 1 - pos);
        } else {
            chunk = unit / p.kh;
            khead = unit - chunk * p.kh;
        }
    };
    // Coordinates of a unit.  They are worked out for 64 of this CTA's units at a time, one thread each, and looked up in
    // shared memory: done in every unit by every thread, the integer divisions (padded) or the two dependent loads (packed)
    // stood in the middle of the unit's chain.
    struct UnitPos {
        int chunk, khead, n, tok0, batch;
        bool valid;
    };
    int4* const sUnits = reinterpret_cast<int4*>(smem + L::kOffUnits);
    auto fill_units = [&](int unit0) {  // entry i: unit0 + i * gridDim.x
        if (tid >= L::kUnits) return;
        const long long unit = unit0 + static_cast<long long>(tid) * gridDim.x;
        int4 e = make_int4(0, 0, 0, 0);
        if (unit < total_units) {
            int chunk, khead;
            unit_chunk(static_cast<int>(unit), chunk, khead);
            const ChunkPos cp = locate_chunk(p.map, chunk);
            // (an entry of chunk_indices may name an empty chunk: the unit is walked all the same, its block is never read)
            e = make_int4(chunk, khead | (max(cp.n, 0) << 16) | (1 << 30), static_cast<int>(cp.tok0), cp.batch);
        }
        sUnits[tid] = e;
    };
    static_assert(L::kUnits <= kThreads, "one entry per thread");
    auto unit_at = [&](int i) {
        const int4 e = sUnits[i];
        UnitPos u;
        u.chunk = e.x;
        u.khead = e.y & 0xFFFF;
        u.n = (e.y >> 16) & 0x7F;
        u.tok0 = e.z;
        u.batch = e.w;
        u.valid = (e.y >> 30) != 0;
        return u;
    };
    fill_units(static_cast<int>(blockIdx.x));
    __syncthreads();
    auto issue_loads = [&](const UnitPos& u) {  // one thread
        mbar_arrive_expect_tx(bar_load, NA * 16384);
        for (int a = 0; a < NA; ++a) {
            tma_load_4d(sKQ + a * 16384, &tmK, bar_load, a * 64, u.khead, u.tok0, u.batch);
            tma_load_4d(sKQ + a * 16384 + 8192, &tmQ, bar_load, a * 64, u.khead, u.tok0, u.batch);
        }
    };
    UnitPos cur = unit_at(0), nxt{};
    int table = 0;  // entry of the present unit
    if (tid == 0 && cur.valid) issue_loads(cur);

    // beta and the raw gate of the tokens `lane` and `lane + 32` for (unit, round), fetched one round ahead, so that
    // their DRAM latency is not in front of every unit
    auto fetch_scalars = [&](const UnitPos& u, int rd, uint32_t* b, uint32_t* g) {
        b[0] = b[1] = g[0] = g[1] = 0u;
        const int hloc = 2 * rd + team;
        if (!u.valid || hloc >= rep) return;
        const int head = u.khead * rep + hloc;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int t = lane + 32 * i;
            if (t < u.n) {
                if (tw < 2) b[i] = p.beta.load_bits(u.batch, u.tok0 + t, head);
                if (p.gate.ptr) g[i] = p.gate.load_bits(u.batch, u.tok0 + t, head);
            }
        }
    };
    uint32_t b_next[2], g_next[2];  // bits, see ScalarView::load_bits
    fetch_scalars(cur, 0, b_next, g_next);

    uint32_t it = 0;      // units done by this CTA (parity of bar_load and bar_kq)
    uint32_t mma_it = 0;  // MMA groups this team has waited for (parity of bar_mma[team])
    bool stores_pending = false;
    for (int unit = blockIdx.x; unit < total_units; unit += gridDim.x, ++it, cur = nxt) {
        const int chunk = cur.chunk, khead = cur.khead;
        const int n = cur.n;
        if (++table == L::kUnits) {  // the next unit is past the table
            __syncthreads();
            fill_units(unit + static_cast<int>(gridDim.x));
            __syncthreads();
            table = 0;
        }
        for (int rd = 0; rd < rounds; ++rd) {
            const int hloc = 2 * rd + team;
            const bool active = hloc < rep;  // team-uniform
            const int head = khead * rep + hloc;
            // ---- beta, chunk-local cumulative gate, decay to the chunk's last token
            float b_mine[2] = {0.f, 0.f}, g_mine = 0.f;
            if (!active) {  // (odd number of v-heads per k-head: team 1 sits the last round out)
                nxt = unit_at(table);
                fetch_scalars(nxt, 0, b_next, g_next);
            } else {
                // (every warp scans the whole chunk for itself: no barrier)
                b_mine[0] = p.beta.value(b_next[0]);
                b_mine[1] = p.beta.value(b_next[1]);
                float g0 = p.gate.value(g_next[0]), g1 = p.gate.value(g_next[1]);
                scan_gate(g0, g1, lane);
                g_mine = (tw & 1) ? g1 : g0;
                decay_tables(g0, g1, sG, sC, tw & 1, lane);
                if (tw == 0) {
                    sBeta[lane] = b_mine[0];
                    sBeta[lane + 32] = b_mine[1];
                } else if (tw == 2) {
                    // tokens past the end had a raw gate of 0: they carry the last valid value
                    const float gl = __shfl_sync(0xffffffffu, g1, 31);
                    sD[lane] = ex2(gl - g0);
                    sD[lane + 32] = ex2(gl - g1);
                }
                __syncwarp();
            }
            // ---- K K^T (lanes 0-63) and Q K^T (lanes 64-127): once per unit, shared by its v-heads
            if (rd == 0) {
                mbar_wait(bar_load, it & 1u, abort_flag);
                if (p.map.cu_seqlens && n < kChunk) {
                    // Keys past the end are another sequence's (in padded mode the copies deliver zeros).  They meet zero rows of dT in Z, and are
                    // cleared all the same, so that no infinity or NaN of a neighbour can enter.
                    for (int i = tid; i < (kChunk - n) * 8 * NA; i += kThreads)
                        *reinterpret_cast<uint4*>(sKQ + (i & (NA - 1)) * 16384 + (n + i / (8 * NA)) * 128 + ((i / NA) & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
                    fence_proxy_async_smem();
                    __syncthreads();
                }
                if (kNorm) {
                    // inverse L2 norm of every row of the stacked K | Q tile: two threads per row, half the columns each
                    const int r = tid >> 1, hf = tid & 1;
                    const uint8_t* rowp = sKQ + hf * (NA / 2) * 16384 + (r >> 6) * 8192 + (r & 63) * 128;
                    float ss = 0.f;
#pragma unroll
                    for (int c = 0; c < 4 * NA; ++c) {
                        // (every row starts with another piece: rows are 128 bytes apart, all in the same banks)
                        const uint4 w = *reinterpret_cast<const uint4*>(rowp + (c >> 3) * 16384 + 16 * ((c + r + 4 * hf) & 7));
                        const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float lo = bf16_lo(ww[e]), hi = bf16_hi(ww[e]);
                            ss = fmaf(lo, lo, ss);
                            ss = fmaf(hi, hi, ss);
                        }
                    }
                    ss += __shfl_xor_sync(0xffffffffu, ss, 1);
                    const float rinv = rsqrtf(ss + 1e-6f);
                    if (hf == 0) {
                        sRn[r] = rinv;
                        if (*abort_flag == 0) p.norms[(static_cast<size_t>(chunk) * p.kh + khead) * 128 + r] = rinv;
                    }
                    __syncthreads();
                }
                if (warp == 0) {
                    tc_fence_after_sync();
                    constexpr uint32_t idesc = make_idesc_bf16(128, 64, false, false);
                    const uint64_t dkq = make_smem_desc_sw128(smem_u32(sKQ), 0, 1024);  // A: 128 rows, B: its first 64
#pragma unroll
                    for (int ks = 0; ks < 4 * NA; ++ks) {
                        const uint32_t off = kmajor_step(ks, 16384);
                        if (ks == 0)
                            mma_ss_w<false>(tmem + kTmKQ, desc_advance(dkq, off), desc_advance(dkq, off), idesc);
                        else
                            mma_ss_w<true>(tmem + kTmKQ, desc_advance(dkq, off), desc_advance(dkq, off), idesc);
                    }
                    mma_commit_w(bar_kq);
                }
                __syncwarp();
                mbar_wait(bar_kq, it & 1u, abort_flag);
                tc_fence_after_sync();
            }
            if (active) {
                if (stores_pending && tw >= 2) {
                    // the previous round's staged Z and PT must have been read out before P (here) and T (past the next
                    // barrier) are written; by now that has long happened and the wait costs nothing
                    if (tt == 64) bulk_wait_read<0>();
                    pair_sync(team);
                }
                // ---- A and P, then X = (I + A)^-1
                ap_pass<kNorm>(tmem + kTmKQ, tiles, tw, lane, n, g_mine, b_mine, p.p_scale);
                tc_fence_before_sync();
                team_sync(team);
                // Every warp owns a 16-row block of X (team 1 in reverse order: the last one is the longest, and warps w of both teams
                // share a scheduler).
                const int rblk = team ? 3 - tw : tw;
                const int g = lane >> 2, tq = lane & 3;
                float xd[2][4];  // its diagonal block as an accumulator fragment
                invert_diagonal(reinterpret_cast<float*>(tiles.diag + rblk * L::kDiag), lane, xd);
                team_sync(team);
                // ---- the row block's other blocks, then T = X diag(beta) and dT = diag(d) T as bf16 swizzled tiles (row = token i,
                //      64 columns j)
                {
                    const uint32_t aa = smem_u32(tiles.a), ia = smem_u32(tiles.diag);
                    const int row = 16 * rblk + g;
                    const float d0 = kNorm ? sD[row] * sRn[row] : sD[row], d1 = kNorm ? sD[row + 8] * sRn[row + 8] : sD[row + 8];
                    const f2 dd[2] = {pk(d0, d0), pk(d1, d1)};
                    const uint32_t tile = smem_u32(sT);
                    row_blocks(rblk, xd, aa, ia, lane, [&](auto d_tag, const float (*x)[4]) {
                        const int c = rblk - decltype(d_tag)::value;
                        uint32_t tv[4], wv[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {  // [8 columns][row g, g + 8]
                            const f2 be = *reinterpret_cast<const f2*>(&sBeta[16 * c + 8 * (i >> 1) + 2 * tq]);
                            const f2 t = mul2(pk(x[i >> 1][2 * (i & 1)], x[i >> 1][2 * (i & 1) + 1]), be);
                            float a, b;
                            unpk(t, a, b);
                            tv[i] = pack_bf16(a, b);
                            unpk(mul2(t, dd[i & 1]), a, b);
                            wv[i] = pack_bf16(a, b);
                        }
                        const uint32_t off = tile_off(16 * rblk + (lane & 15), 2 * c + (lane >> 4));
                        stmatrix_x4(tile + off, tv[0], tv[1], tv[2], tv[3]);
                        stmatrix_x4(tile + 8192 + off, wv[0], wv[1], wv[2], wv[3]);
                    });
#pragma unroll 1
                    for (int c = rblk + 1; c < 4; ++c) {  // above the diagonal
                        const uint32_t off = tile_off(16 * rblk + (lane & 15), 2 * c + (lane >> 4));
                        stmatrix_x4(tile + off, 0u, 0u, 0u, 0u);
                        stmatrix_x4(tile + 8192 + off, 0u, 0u, 0u, 0u);
                    }
                }
                fence_proxy_async_smem();
                team_sync(team);
                // ---- Z = (dT)^T K and PT = P T; team 0 in lanes +0, team 1 in lanes +16 of the same columns
                if (tw == 0) {
                    tc_fence_after_sync();
                    constexpr uint32_t idesc = make_idesc_bf16(64, 64, false, true);   // PT: A K-major, B MN-major
                    constexpr uint32_t idescz = make_idesc_bf16(64, 128, true, true);  // Z: A = (dT)^T read MN-major too
                    const uint64_t dTd = make_smem_desc_sw128(smem_u32(sTd), 8192, 1024);       // A, read MN-major
                    const uint64_t dPa = make_smem_desc_sw128(smem_u32(sP), 0, 1024);           // A, K-major
                    const uint64_t dTb = make_smem_desc_sw128(smem_u32(sT), 8192, 1024);        // B, read MN-major
                    const uint64_t dK = make_smem_desc_sw128(smem_u32(sKQ), 16384, 1024);       // B, K, MN-major: two 64-column atoms
                    const uint32_t tZ = tmem + kTmZ + (team ? (16u << 16) : 0u);
                    const uint32_t tPT = tmem + kTmPT + (team ? (16u << 16) : 0u);
                    mma_ss_w<false>(tZ, dTd, dK, idescz);
#pragma unroll
                    for (int ks = 1; ks < 4; ++ks) mma_ss_w<true>(tZ, desc_advance(dTd, ks * 2048), desc_advance(dK, ks * 2048), idescz);
                    mma_ss_w<false>(tPT, dPa, dTb, idesc);
#pragma unroll
                    for (int ks = 1; ks < 4; ++ks) mma_ss_w<true>(tPT, desc_advance(dPa, ks * 32), desc_advance(dTb, ks * 2048), idesc);
                    mma_commit_w(&bar_mma[team]);
                }
                __syncwarp();
                // the next round's scalars, requested in front of a long wait: anywhere else other loads that share their
                // scoreboard wait for DRAM with them (the substitution took 700 cycles instead of 250 behind them)
                if (rd + 1 < rounds) {
                    fetch_scalars(cur, rd + 1, b_next, g_next);
                } else {
                    nxt = unit_at(table);
                    fetch_scalars(nxt, 0, b_next, g_next);
                }
                mbar_wait(&bar_mma[team], mma_it & 1u, abort_flag);
                ++mma_it;
                tc_fence_after_sync();
            }
            if (rd == rounds - 1 && tt == 0) {
                // This team's MMAs have read the K tile (or it sat the round out).  The team that gets here second
                // knows that both are done with the tiles and requests the next unit's, which land while the
                // epilogues run; the teams do not wait for one another.
                if (atomicAdd(teams_done, 1) == 1) {
                    *teams_done = 0;
                    if (nxt.valid) issue_loads(nxt);
                }
            }
            if (active) {
                const int row = 16 * tw + (lane & 15);
                const uint32_t tl = static_cast<uint32_t>(32 * tw + 16 * team) << 16;
                // ---- accumulators -> bf16 -> staged tiles (Z over T / dT, PT over P) -> one bulk copy.  As fragments: 16 lanes of
                //      tensor memory are one team's.
#pragma unroll
                for (int cb = 0; cb < 6; cb += 2) {  // 32 columns each: four of Z, two of PT
                    uint32_t r[2][16];
                    const uint32_t col = cb < 4 ? kTmZ + 32 * cb : kTmPT;
                    tmem_ld_frag32(tmem + col + tl, r[0]);
                    tmem_ld_frag32(tmem + col + 32 + tl, r[1]);
                    tmem_wait_ld();
                    const uint32_t tile = smem_u32(cb < 4 ? sT : sP);
#pragma unroll
                    for (int h = 0; h < 4; ++h) {  // 16 columns
                        uint32_t w[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {  // [8 columns][row l/4, l/4 + 8]
                            const uint32_t* const v = &r[h >> 1][8 * (h & 1) + 2 * i];
                            w[i] = pack_bf16(__uint_as_float(v[0]), __uint_as_float(v[1]));
                        }
                        stmatrix_x4(tile + tile_off(row, 4 * (cb & 3) + 2 * h + (lane >> 4)), w[0], w[1], w[2], w[3]);
                    }
                }
                fence_proxy_async_smem();
                tc_fence_before_sync();
                team_sync(team);
                if (tt == 64 && *abort_flag == 0) {  // nothing is written once a wait has given up
                    // the state kernel reads these blocks back soon: ask L2 to hold on to them
                    bulk_store_hint(p.blocks + (static_cast<size_t>(chunk) * p.vh + head) * kZPBlockBytes, sT, kZPBlockBytes,
                                    l2_policy_evict_last());
                    bulk_commit();
                }
                stores_pending = true;
            }
        }  // head pairs
    }      // units
    if (stores_pending && tt == 64) bulk_wait_read<0>();
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 256);
    if (tid == 0 && *abort_flag && p.status) atomicExch(p.status, 2);
}

}  // namespace gdn
