// k_crt16.cu -- the last four stages of the inverse transform and the CRT straight to mod q in one
// kernel, for the 16-row split: residues after the inverse row pass in, result limbs out, so that
// the inverse column pass does not go through memory.
//
// A tile is 128 coefficients, 16 rows x 8 columns of the 4-step matrix.  Producers hold a column
// of one prime in registers (16 rows; a warp's 4 primes x 8 columns of a row are halves of two
// lines of the pair layout), run the four inverse stages as a radix-16 network, and write the 16
// results -- y_j, in [0, 2p), since one operand was decomposed times the CRT's per-prime factor --
// straight into the tcgen05 A operand
// (K-major bytes: a residue is the 4 K bytes 4j .. 4j + 3 of its coefficient's row).  The GEMM is
// that of k_tc.cu,
//   D[m][v] = sum_{j,t} byte_t(y_j) byte_(v-t)(Q_j),
// with 6 more result bytes for the CRT's quotient: sum_j y_j floor(2^53 / p_j), exact in integers,
// is 2^53 sum_j y_j / p_j to within K 2^31 (relative to 2^53: below 2^-14, under the rounding
// error of the fp32 sum of up to 128 terms below 2 that the other forms use).  The epilogue takes
// v = round of it, adds v T_1 limb by limb while it carries bytes into limbs, folds and reduces.
//
// What bounds it: per tile and SM sub-partition the integer multiply-add pipe (236 butterflies and
// 14 x 5 wide products per thread pair, ~3300 clocks at K = 118, L = 55) beside the HBM time of
// the tile's bytes (~3800 clocks); producers and epilogue run on different tiles.  Measured: 11,000
// clocks a tile, 20.0 us a multiply at N = 65536, W = 1747 in launches of 32 (an inverse column pass and
// a CRT of their own: 26); the multiply-add pipe at 49%, issue slots at 51%.
#include "pm_crt.cuh"
#include "pm_ntt.cuh"
#include "pm_tc.cuh"

namespace pm {

// ----------------------------------------------------------------------------------------
// Persistent, 896 threads, one CTA per SM.
//   producers (warps 0-15): warp w takes prime groups g = w, w + 16, ... (4 primes x 8 columns a
//     round); the next round's 16 residues are loaded while this round's network runs.  The K bytes
//     form two blocks (the rounds' first and second half): a block is written once the previous
//     tile's MMAs over it are complete, and its MMAs run while the next block is computed.
//   epilogue (warps 16-23): two threads per coefficient (low and high limbs), one of two TMEM
//     accumulators per tile.  The two warps of a TMEM lane quarter hold whole rows of the tile and
//     synchronise only with one another;
//   warp 24 issues the MMAs.
// smem: [B image nrows x kb][A 128 x kb][z 128 x zs][T_1 L][twiddles 15 x KP][bars][slot][abort]
// ----------------------------------------------------------------------------------------
namespace {
__host__ __device__ inline int crt16_t1_words(int L) { return (L + 4 + 3) & ~3; }
constexpr int C16_PROD = 32 * CRT16_PROD_WARPS;
constexpr int C16_EPI = 32 * CRT16_EPI_WARPS;
// registers per thread: 896 threads start with 72; the producers (four warpgroups) and the MMA
// warpgroup give theirs to the epilogue (two): 4 x 64 + 2 x 104 + 40 = 7 x 72
constexpr int C16_PROD_REGS = 64, C16_EPI_REGS = 104, C16_MMA_REGS = 40;
static_assert(CRT16_PROD_WARPS / 4 * C16_PROD_REGS + CRT16_EPI_WARPS / 4 * C16_EPI_REGS + C16_MMA_REGS <=
              (CRT16_PROD_WARPS + CRT16_EPI_WARPS + 4) / 4 * 72, "a warp's share of its SM sub-partition");
}

// LN >= 0: log2 of the row length N / 16 at compile time (row addresses become immediates).
template <int LN>
__global__ void __launch_bounds__(CRT16_THREADS, 1) k_crt16(const __grid_constant__ Crt16Args A) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int kb = A.kb, L = A.L, zl = crt_zl(L), zs = crt_zstride(L);
    unsigned char* b_s = smem_raw;
    unsigned char* a_s = b_s + (size_t)A.nrows * kb;
    uint32_t* z_s = reinterpret_cast<uint32_t*>(a_s + (size_t)TC_M * kb);
    uint32_t* t1_s = z_s + (size_t)TC_M * zs;
    uint2* tw_s = reinterpret_cast<uint2*>(t1_s + crt16_t1_words(L));  // [15][KP], then [KP] {p, -}
    uint64_t* bars = reinterpret_cast<uint64_t*>(tw_s + 16 * A.KP);
    uint64_t *bar_b = bars, *a_free = bars + 1, *mma_done = bars + 3, *acc_empty = bars + 5, *a_full = bars + 7;
    uint32_t* slot = reinterpret_cast<uint32_t*>(bars + 9);
    volatile int* abort_f = reinterpret_cast<volatile int*>(slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t tiles_x = A.cw / 8;
    const uint32_t ntiles = tiles_x * A.nbatch;

    if (threadIdx.x == 0) {
        mbar_init(bar_b, 1);
        for (int k = 0; k < 2; ++k) {
            mbar_init(a_free + k, 1);
            mbar_init(mma_done + k, 1);
            mbar_init(acc_empty + k, C16_EPI);
            mbar_init(a_full + k, C16_PROD);
        }
        *abort_f = 0;
        bulk_g2s_all(b_s, A.img, (uint32_t)((size_t)A.nrows * kb), bar_b);
    }
    // (T_1 padded with zero limbs to whole 4-limb steps)
    for (int l = threadIdx.x; l < crt16_t1_words(L); l += blockDim.x) t1_s[l] = l < L ? __ldg(A.t1 + l) : 0u;
    for (int x = threadIdx.x; x < 15 * A.KP; x += blockDim.x) tw_s[x] = __ldg(A.tw16 + x);
    for (int x = threadIdx.x; x < A.KP; x += blockDim.x) tw_s[15 * A.KP + x] = make_uint2(__ldg(A.p + x), 0u);
    if (warp == 0) tmem_alloc(slot, 512);
    pdl_wait();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_trigger();  // after this block's TMEM allocation
    const uint32_t tmem = *slot;
    const uint32_t sbo = 8u * (uint32_t)kb;
    const int G = A.KP / 4, nr = (G + CRT16_PROD_WARPS - 1) / CRT16_PROD_WARPS;
    const int nr0 = (nr + 1) / 2;                              // rounds of block 0
    const int nblk = nr > 1 ? 2 : 1;
    const int kk0 = min(kb / 32, nr0 * CRT16_PROD_WARPS / 2);  // MMA steps (32 K bytes: 2 groups) of block 0

    if (warp < CRT16_PROD_WARPS) {
        // ---------------- producers ----------------
        regs_dec<C16_PROD_REGS>();
        const int c = lane & 7, jj = lane >> 3;
        const size_t N = LN >= 0 ? (size_t)16 << (LN >= 0 ? LN : 0) : A.N;
        const size_t step = N / 16 * 2;  // words between rows
        // the lane's prime in a group, and in the last one, where lanes past the last pair of primes read
        // that pair's residues
        const size_t lane_off = residue_base(0, 4, jj, N) + c;
        const size_t last_off = residue_base(0, 4, A.K2 % 4 ? jj & 1 : jj, N) + c;
        auto load = [&](uint32_t tile, int rd, uint32_t (&x)[16]) {
            const int g = rd * CRT16_PROD_WARPS + warp;
            if (tile >= ntiles || g >= G) return;
            const uint32_t b = tile / tiles_x, cx = tile - b * tiles_x;
            const uint32_t* s = A.R + residue_base(b, A.K2, 4 * g, N) + (g + 1 < G ? lane_off : last_off) +
                                residue_off(A.col0 + 8 * cx);
#pragma unroll
            for (int e = 0; e < 16; ++e) x[e] = s[e * step];
        };
        uint32_t tile = blockIdx.x, i = 0;
        int rd = 0;
        // one round: the next round's residues into y, this round's (x) through the network into A,
        // and after a block's last round its MMAs; false after the last tile or on an abort
        auto round = [&](uint32_t (&x)[16], uint32_t (&y)[16]) -> bool {
            const int blk = rd >= nr0;
            if (rd + 1 < nr) load(tile, rd + 1, y);
            else load(tile + gridDim.x, 0, y);
            const int g = rd * CRT16_PROD_WARPS + warp;
            if ((rd == 0 || rd == nr0) && i > 0)  // the previous tile's MMAs have read this block
                wait_or_abort(a_free + blk, (i - 1) & 1, abort_f, A.wait_clocks);
            if (g < G) {
                // (primes K .. KP - 1: whatever comes out, against zero B columns)
                const uint2* tw = tw_s + 4 * g + jj;
                const uint32_t p = tw[15 * A.KP].x;
                auto stw = [&](int t) { return StrideTw<true>{tw + ((1 << t) - 1) * A.KP, A.KP, 1 << t}; };
                radix_inv<4, 0>(x, stw, p);
                unsigned char* d = a_s + (size_t)g * 128 + c * 16 + jj * 4;
#pragma unroll
                for (int e = 0; e < 16; ++e) *reinterpret_cast<uint32_t*>(d + e * sbo) = x[e];
            }
            if (rd == nr0 - 1 || rd == nr - 1) {  // the block is complete
                fence_smem_to_async();
                mbar_arrive(a_full + blk);
                if (*abort_f) return false;
            }
            if (++rd == nr) {
                rd = 0;
                tile += gridDim.x;
                ++i;
            }
            return tile < ntiles;
        };
        if (tile < ntiles) {
            uint32_t u[16], w[16];
            load(tile, 0, u);
            while (round(u, w) && round(w, u)) {
            }
        }
    } else if (warp >= CRT16_PROD_WARPS + CRT16_EPI_WARPS) {
        // ---------------- MMA issue ----------------
        regs_dec<C16_MMA_REGS>();
        if (warp == CRT16_PROD_WARPS + CRT16_EPI_WARPS) {
        const uint32_t mine = elect_one();
        const uint32_t idesc = idesc_u8(A.nrows);
        const uint64_t ad0 = sdesc(smem_addr(a_s), 128u, sbo), bd0 = sdesc(smem_addr(b_s), 128u, sbo);
        const bool b_seen = wait_or_abort(bar_b, 0, abort_f, A.wait_clocks);
        bool ok = __all_sync(0xffffffffu, b_seen);
        uint32_t i = 0, blocks[2] = {0, 0};
        for (uint32_t tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, ++i) {
            const int b = (int)(i & 1);
            // tile i - 2's epilogue has read this accumulator
            if (i >= 2) ok = wait_or_abort(acc_empty + b, ((i >> 1) - 1) & 1, abort_f, A.wait_clocks);
            for (int blk = 0; blk < nblk; ++blk) {
                ok = ok && wait_or_abort(a_full + blk, i & 1, abort_f, A.wait_clocks);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                const int k0 = blk ? kk0 : 0, k1 = blk + 1 == nblk ? kb / 32 : kk0;
                uint64_t ad = ad0 + 16u * k0, bd = bd0 + 16u * k0;
#pragma unroll 4
                for (int kk = k0; kk < k1; ++kk, ad += 16, bd += 16)
                    umma_u8_if(mine, tmem + 256u * b, ad, bd, idesc, kk > 0 ? 1u : 0u);
                ++blocks[blk];
                if (mine) {
                    umma_commit(a_free + blk);
                    if (blk + 1 == nblk) umma_commit(mma_done + b);
                }
                __syncwarp();
            }
        }
        // copies and MMAs still in flight must land before this CTA's memory goes away
        if (mine) {
            if (!b_seen) mbar_wait_bounded(bar_b, 0, A.wait_clocks);
            for (int blk = 0; blk < 2; ++blk)
                if (blocks[blk]) mbar_wait_bounded(a_free + blk, (blocks[blk] - 1) & 1, A.wait_clocks);
        }
        __syncwarp();
        }
    } else {
        // ---------------- epilogue ----------------
        regs_inc<C16_EPI_REGS>();
        const int hf = (warp - CRT16_PROD_WARPS) >> 2, quarter = warp & 3;
        const int m = quarter * 32 + lane;
        const int nl = A.nz / 4;                    // limbs under the result-byte columns (L + 1)
        const int lh = ((nl + 1) / 2 + 3) / 4 * 4;  // limbs of half 0 (whole 16-column loads)
        uint32_t* z = z_s + (size_t)m * zs;
        uint32_t i = 0;
        for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++i) {
            // (also: the previous tile's rows have been stored)
            if (named_sync_or(2 + quarter, 64, *abort_f != 0)) break;
            const int b = (int)(i & 1);
            const bool got =
                __all_sync(0xffffffffu, wait_or_abort(mma_done + b, (i >> 1) & 1, abort_f, A.wait_clocks));
            tc_fence_after();
            const uint32_t tacc = tmem + 256u * b + ((uint32_t)(quarter * 32) << 16);
            // S = 2^53 sum y_j / p_j; v = round(S / 2^53): |x| < M/8 puts the sum within 1/8 of an
            // integer, further than 1/4 is a failed check
            uint32_t sv[8];
            if (got) {
                tmem_ld8_async(tacc + (uint32_t)A.nz, sv);
                tmem_wait_ld_8(sv);
            } else {
#pragma unroll
                for (int k = 0; k < 8; ++k) sv[k] = 0u;
            }
            uint64_t S = 0;
#pragma unroll
            for (int k = 0; k < 6; ++k) S += (uint64_t)sv[k] << (8 * k);
            const uint32_t v = (uint32_t)((S + (1ull << 52)) >> 53);
            const int64_t frac = (int64_t)(S - ((uint64_t)v << 53));
            if (hf == 0 && (frac > (1ll << 51) || frac < -(1ll << 51))) flag_error(A.status, DEV_ERR_CRT_BOUND);
            // bytes -> limbs with carries, + v T_1 (T_1 = (-M) mod q; v T_1 == -v M)
            uint64_t carry = 0;
            const int l0 = hf ? lh : 0, l1 = hf ? nl : min(lh, nl);
            int l = l0;
            // four limbs: independent sums, then the carry chain
            auto limbs4 = [&](const uint32_t* r, const uint32_t* t1, uint64_t (&t)[4]) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    t[k] = (uint64_t)v * t1[k] + r[4 * k] + (uint64_t)r[4 * k + 1] * 256u +
                           (uint64_t)r[4 * k + 2] * 65536u + (uint64_t)r[4 * k + 3] * 16777216u;
            };
            uint32_t ra[16], rn[16];
            if (got && l < l1) tmem_ld16_async(tacc + (uint32_t)(4 * l), rn);
            // four limbs from x, loaded before; the next step's load (y) runs under them
            auto step = [&](uint32_t (&x)[16], uint32_t (&y)[16]) {
                if (got) tmem_wait_ld_16(x);
                if (got && l + 4 < l1) tmem_ld16_async(tacc + (uint32_t)(4 * l + 16), y);
                const uint4 q1 = *reinterpret_cast<const uint4*>(t1_s + l);
                const uint32_t t1[4] = {q1.x, q1.y, q1.z, q1.w};
                uint64_t t[4];
                limbs4(x, t1, t);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    t[k] += carry;
                    z[l + k] = (uint32_t)t[k];
                    carry = t[k] >> 32;
                }
                l += 4;
            };
            while (l + 8 <= l1) {
                step(rn, ra);
                step(ra, rn);
            }
            if (l + 4 <= l1) {
                step(rn, ra);
                if (got && l < l1) tmem_wait_ld_16(ra);  // a load in flight may not be copied
#pragma unroll
                for (int k = 0; k < 16; ++k) rn[k] = ra[k];
            }
            if (l < l1) {  // the last limbs: the loaded columns past them belong to the quotient
                if (got) tmem_wait_ld_16(rn);
                uint64_t t[4];
                limbs4(rn, t1_s + l, t);
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    if (l + k < l1) {
                        t[k] += carry;
                        z[l + k] = (uint32_t)t[k];
                        carry = t[k] >> 32;
                    }
            }
            tc_fence_before();
            mbar_arrive(acc_empty + b);  // the accumulator is free for tile i + 2
            if (hf) {
                for (int x = l1; x < zl; ++x) {
                    z[x] = (uint32_t)carry;
                    carry >>= 32;
                }
            }
            named_sync(2 + quarter, 64);
            if (hf == 0) {
                for (int x = l1; carry && x < zl; ++x) {  // half 0's carry-out into half 1's limbs
                    const uint64_t t = (uint64_t)z[x] + carry;
                    z[x] = (uint32_t)t;
                    carry = t >> 32;
                }
                crt_reduce_fast(z, zl, A);
            }
            named_sync(2 + quarter, 64);
            // the quarter's rows of the tile: 4 runs of 8 coefficients, contiguous in the result; warp
            // hf stores runs 2 hf and 2 hf + 1
            const uint32_t bt = tile / tiles_x, cx = tile - bt * tiles_x;
            for (int rr = 0; rr < 2; ++rr) {
                const int row = quarter * 4 + 2 * hf + rr;
                uint32_t* o = A.out + (((size_t)bt * 16 + row) * A.cw + 8 * cx) * L;
                const uint32_t* zr = z_s + (size_t)(8 * row) * zs;
                if (L > 16) {  // 32 limbs of each of the 8 coefficients at a time
                    for (int w = lane; w < L; w += 32) {
                        uint32_t x[8];
#pragma unroll
                        for (int cc = 0; cc < 8; ++cc) x[cc] = zr[cc * zs + w];
#pragma unroll
                        for (int cc = 0; cc < 8; ++cc) o[cc * L + w] = x[cc];
                    }
                } else {
                    for (int w = lane; w < 8 * L; w += 32) {
                        const int cc = w / L;
                        o[w] = zr[cc * zs + (w - cc * L)];
                    }
                }
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && *abort_f) flag_error(A.status, DEV_ERR_WAIT);
    if (warp == 0) tmem_dealloc(tmem, 512);
}

size_t crt16_smem(const Crt16Args& A) {
    return (size_t)A.nrows * A.kb + (size_t)TC_M * A.kb + (size_t)TC_M * crt_zstride(A.L) * 4 +
           (size_t)crt16_t1_words(A.L) * 4 + (size_t)16 * A.KP * 8 + 9 * 8 + 16;
}

namespace {
using Crt16Kernel = void (*)(Crt16Args);
Crt16Kernel crt16_kernel(uint32_t N) {
    switch (N) {
        case 1u << 12: return k_crt16<8>;
        case 1u << 13: return k_crt16<9>;
        case 1u << 14: return k_crt16<10>;
        case 1u << 15: return k_crt16<11>;
        case 1u << 16: return k_crt16<12>;
        default: return k_crt16<-1>;
    }
}
}  // namespace

void launch_crt16(const Crt16Args& A, uint32_t grid, cudaStream_t s, bool pdl) {
    const cudaError_t e = launch_kernel(crt16_kernel(A.N), dim3(grid), dim3(CRT16_THREADS), crt16_smem(A), s, pdl, A);
    if (e != cudaSuccess) throw_cuda(e, "launch k_crt16");
}

void crt16_set_smem_limit(int bytes) {
    for (uint32_t N : {1u << 12, 1u << 13, 1u << 14, 1u << 15, 1u << 16, 0u}) {
        const cudaError_t e =
            cudaFuncSetAttribute((const void*)crt16_kernel(N), cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) throw_cuda(e, "k_crt16 attribute");
    }
}

}  // namespace pm
