// k_dec16.cu -- RNS decomposition and the first four stages of the forward transform in one
// kernel, for the 16-row split (nrows = 16, ncols = N / 16): limbs of the operand in, residues
// after the whole column pass out, so that neither the plain residues nor a column pass go
// through memory.
//
// The decomposition is the byte-sliced tcgen05 kind::i8 GEMM of k_tc.cu turned on its side: the
// constants are the M operand (one TMEM lane per prime, one 128-lane block per constant byte t)
// and a tile of 128 coefficients -- 16 rows x 8 columns of the 4-step matrix -- the N operand:
//   D_t[j][n] = sum_s byte_t(2^(8s) mod p_j) byte_s(a_n)          (< 4L 255^2 < 2^25)
//   a_n mod p_j = sum_t D_t[j][n] 2^(8t)  (< 2^50), reduced once in the epilogue.
// With a prime per thread the epilogue holds all 16 rows of a column in registers: p, its
// reduction constant and the pass's 15 twiddles depend on the thread alone, the 4 column stages
// are a radix-16 network between registers, and a row's 8 columns leave as one 32-byte store,
// next to the same 8 columns of the neighbouring prime (the pair layout, pm_device.cuh).
//
// What bounds it: per 128-coefficient tile and SM sub-partition, the integer multiply-add pipe
// (128 reductions of 1 high + 1 low product, 256 butterflies of 1 high + 2 low: ~3200 clocks) is
// next to the HBM time of the tile's bytes (128 x (4L + 4K) at 6.5 TB/s: ~3800 clocks at
// L = 55, K = 118); the tensor pipe runs beside them.
#include "pm_ntt.cuh"
#include "pm_tc.cuh"

namespace pm {

// 32 consecutive bytes, 32-byte aligned
__device__ __forceinline__ void st_global_v8(uint32_t* p, const uint32_t (&r)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}

namespace {
// Residue of one coefficient from its four byte sums: x = r0 + r1 2^8 + r2 2^16 + r3 2^24, which
// lies below 2^50; q = hi(x >> 16) * floor(2^48 / p) >> 32 is at most two below floor(x / p), so
// x - q p is in [0, 2p + 2^16) -- the forward butterflies take inputs below 4p.  (4L <= 256: t0 is
// below 257 255^2 4L < 2^32.)
__device__ __forceinline__ uint32_t dec_reduce(uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3, uint32_t p,
                                               uint32_t wsh) {
    const uint32_t t0 = r0 + (r1 << 8), t1 = r2 + (r3 << 8);
    const uint32_t th = t1 + (t0 >> 16);
    return t0 + (t1 << 16) - (uint32_t)(((uint64_t)th * wsh) >> 32) * p;
}
}  // namespace

// ----------------------------------------------------------------------------------------
// Persistent, warp-specialised, 384 threads, one CTA per SM.
//   warps 0-7: two epilogue groups of 4 warps (one warp per TMEM lane quarter); group g takes the
//     CTA's tiles i = g, g + 2, ...: columns 0-3 from accumulator half 0, columns 4-7 from half 1
//     (64 coefficients, 256 TMEM columns each), releasing a half as soon as its last TMEM load is
//     done, so that the next tile's MMAs of that half run under this tile's butterflies;
//   warp 8 issues the MMAs of the two halves, each once the epilogue has released it;
//   warp 9 keeps a ring of raw pieces filled: the row segments of `npo` row octets of the super-tile
//     (8 columns x L limbs each, contiguous in the operand), one bulk copy per row;
//   warps 10-11 re-lay each piece out as the K-major operand, in one of `nb_buf` buffers.
// The four hand work to one another through mbarriers only, and the helpers' roles are apart because
// their warps get the issue slots and the instruction cache that the epilogue leaves.
// Measured 25.8 us for both operands of a multiply at N = 65536, W = 1747 in launches of 32 (separate
// decompositions and column passes: 48): the epilogue is the limit, two warps an SM sub-partition with
// 224 registers, which cannot cover one another's waits (issue 51%, multiply-add pipe 56%).  It stays
// at two groups because three, with 152 registers each, can hold half a row's 8 columns and would
// store half sectors, which do not merge in L2: 44.5 us.
// A CTA works for one operand (blockIdx.x mod nops), so that its constant image is loaded once and
// both operands of a multiply share a launch.
// Few primes (K <= 32 or 64): q = 4 or 2 tiles share an accumulator.  Lanes are split into q groups
// of 128 / q; the constants sit between zero rows, so that an MMA whose A window starts 128 / q
// rows earlier lands its residues in the next lane group and adds zeros to the others.
// All waits are bounded (wait_or_abort); the kernel reports DEV_ERR_WAIT.
// smem: [A image 4 x a_rows x kb][B buffers nb_buf x q x 128 x kb][raw ring][twiddles 15 x KP][bars][slot][abort]
// ----------------------------------------------------------------------------------------
constexpr int D16_EPI_THREADS = 256;
constexpr int D16_RELAY_THREADS = 64;
// registers per thread: 384 threads start with 168; the other four warps give up 112 each (56 + 2 x 224 = 3 x 168)
constexpr int D16_LOAD_REGS = 56, D16_EPI_REGS = 224;
static_assert(D16_LOAD_REGS + 2 * D16_EPI_REGS <= 3 * 168, "a warp's share of its SM sub-partition");

// LV: words per aligned load of a coefficient's limbs (4, 2 or 1 as L mod 4 is 0, 2 or odd); 0: an
// operand off the 16-byte alignment of bulk copies, read limb by limb.  The re-layout has to be
// short and branch-free: its warps get the instruction cache and the issue slots that the epilogue
// leaves, and with these cases chosen at run time it took 6,400 clocks a tile (L = 55).
template <int LV>
__global__ void __launch_bounds__(DEC16_THREADS, 1) k_dec16(const __grid_constant__ Dec16Args A) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int kb = A.kb, q = A.q, qrun = A.qrun, L = A.L;
    const uint32_t op = blockIdx.x % A.nops, me = blockIdx.x / A.nops;
    const uint32_t mates = (gridDim.x - op + A.nops - 1) / A.nops;  // CTAs of this operand
    const uint32_t* src = A.src[op];
    const uint32_t tiles_x = A.cw / 8;  // tiles per batch entry
    const uint32_t ntiles = tiles_x * A.nbatch;
    const uint32_t nsuper = (ntiles + qrun - 1) / qrun;

    unsigned char* a_s = smem_raw;
    unsigned char* b_s = a_s + A.a_bytes;
    const size_t b_bytes = (size_t)q * TC_M * kb;
    uint32_t* raw_s = reinterpret_cast<uint32_t*>(b_s + A.nb_buf * b_bytes);
    const int segw = A.segw;                     // words between a piece's row segments
    const int npo = A.npo;                       // row octets of a piece
    const size_t piece_words = (size_t)A.piece_octets * 8 * segw;
    const int tws = A.KP;                         // entries per row of the twiddle table
    uint2* tw_s = reinterpret_cast<uint2*>(raw_s + A.ring * piece_words);
    uint64_t* bars = reinterpret_cast<uint64_t*>(tw_s + 15 * tws);
    uint64_t *bar_a = bars, *mma_done = bars + 1 /* [group][half] */, *acc_empty = bars + 5 /* [half] */,
             *b_full = bars + 7 /* [buffer] */, *raw_full = bars + 9, *raw_empty = raw_full + DEC16_MAX_RING;
    uint32_t* slot = reinterpret_cast<uint32_t*>(raw_empty + DEC16_MAX_RING);
    volatile int* abort_f = reinterpret_cast<volatile int*>(slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // super-tiles me, me + mates, ... of the operand; their row octets (two a tile) in pieces of npo
    const int npieces = 2 * qrun / npo;  // of a super-tile
    const uint32_t my_super = me < nsuper ? (nsuper - me + mates - 1) / mates : 0;

    if (threadIdx.x == D16_EPI_THREADS) {
        mbar_init(bar_a, 1);
        for (int k = 0; k < 4; ++k) mbar_init(mma_done + k, 1);
        for (int k = 0; k < 2; ++k) {
            mbar_init(acc_empty + k, 128);
            mbar_init(b_full + k, D16_RELAY_THREADS);
        }
        for (int k = 0; k < A.ring; ++k) {
            mbar_init(raw_full + k, 1);
            mbar_init(raw_empty + k, D16_RELAY_THREADS);
        }
        *abort_f = 0;
        bulk_g2s_all(a_s, A.img[A.ra_op == op ? 1 : 0], A.a_bytes, bar_a);
    }
    if (warp == 0) tmem_alloc(slot, 512);
    for (int x = threadIdx.x; x < 15 * tws; x += blockDim.x) tw_s[x] = __ldg(A.tw16 + x);
    // the prologue above reads only the plan's constant tables
    pdl_wait();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_trigger();  // after this block's TMEM allocation
    const uint32_t tmem = *slot;
    if (threadIdx.x >= D16_EPI_THREADS) {
        regs_dec<D16_LOAD_REGS>();
        const uint32_t sbo = 8u * (uint32_t)kb;
        if (warp == 8) {
            // ---------------- MMA issue ----------------
            const uint32_t mine = elect_one();
            const uint32_t idesc = idesc_u8(64);
            const uint64_t ad0 = sdesc(smem_addr(a_s) + (uint32_t)(A.a_zero >> 3) * sbo, 128u, sbo);
            const uint64_t bd0 = sdesc(smem_addr(b_s), 128u, sbo);
            // descriptor steps (16-byte units) of a constant-byte block, a lane group, a tile of the
            // super-tile, a half of it, an operand buffer
            const uint32_t a_blk = (uint32_t)(A.a_rows * kb) >> 4, a_grp = (uint32_t)((16 / q) * 8 * kb) >> 4;
            const uint32_t b_tile = (uint32_t)(TC_M * kb) >> 4, b_half = b_tile / 2, b_buf = (uint32_t)(b_bytes >> 4);
            const int nk = kb / 32;
            const bool a_seen = wait_or_abort(bar_a, 0, abort_f, A.wait_clocks);
            bool ok = __all_sync(0xffffffffu, a_seen);
            uint32_t i = 0;
            for (; i < my_super && ok; ++i) {
                const uint32_t buf = A.nb_buf == 2 ? (i & 1) : 0u;
                ok = wait_or_abort(b_full + buf, (A.nb_buf == 2 ? i >> 1 : i) & 1, abort_f, A.wait_clocks);
                for (int h = 0; h < 2; ++h) {
                    if (i > 0) ok = ok && wait_or_abort(acc_empty + h, (i - 1) & 1, abort_f, A.wait_clocks);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    tc_fence_after();
                    for (int t = 0; t < 4; ++t) {
                        const uint32_t d = tmem + 256u * h + 64u * t;
                        uint32_t acc = 0;
                        for (int s = 0; s < qrun; ++s) {
                            uint64_t ad = ad0 + a_blk * t - a_grp * s;
                            uint64_t bd = bd0 + b_buf * buf + b_tile * s + b_half * h;
#pragma unroll 4
                            for (int kk = 0; kk < nk; ++kk, ad += 16, bd += 16) {
                                umma_u8_if(mine, d, ad, bd, idesc, acc);
                                acc = 1;
                            }
                        }
                    }
                    if (mine) umma_commit(mma_done + 2 * (i & 1) + h);
                    __syncwarp();
                }
            }
            // MMAs and the image copy must land before this CTA's memory goes away, also where the
            // epilogue, which waits for every MMA, has given up: whatever was issued, behind one more commit
            if (mine) {
                if (!a_seen) mbar_wait_bounded(bar_a, 0, A.wait_clocks);
                if (i > 0) {
                    umma_commit(bar_a);
                    mbar_wait_bounded(bar_a, 1, A.wait_clocks);
                }
            }
            __syncwarp();
        } else if (warp == 9) {
            // ---------------- raw copies ----------------
            if constexpr (LV > 0) {
                uint32_t k = 0;
                bool ok = true;
                for (uint32_t i = 0; i < my_super && ok; ++i) {
                    const uint32_t t0 = (me + i * mates) * (uint32_t)qrun;
                    for (int pc = 0; pc < npieces && ok; ++pc) {
                        const int o0 = pc * npo;  // the piece's first octet
                        const int no = min(npo, 2 * (int)min((uint32_t)qrun, ntiles - t0) - o0);  // with tiles
                        if (no <= 0) break;
                        const uint32_t sl = k % A.ring, use = k / A.ring;
                        if (use > 0) ok = wait_or_abort(raw_empty + sl, (use - 1) & 1, abort_f, A.wait_clocks);
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) break;
                        if (lane == 0) mbar_arrive_expect_tx(raw_full + sl, 32u * L * 8u * no);
                        __syncwarp();
                        for (int x = lane; x < 8 * no; x += 32) {
                            const int row = 8 * o0 + x;  // row of the super-tile
                            const uint32_t tile = t0 + (row >> 4), b = tile / tiles_x, cx = tile - b * tiles_x;
                            bulk_g2s(raw_s + sl * piece_words + x * segw,
                                     src + (((size_t)b * 16 + (row & 15)) * A.cw + 8 * cx) * L, 32u * L, raw_full + sl);
                        }
                        ++k;
                    }
                }
                // every copy issued lands before the CTA exits (the latest per slot)
                __syncwarp();
                if (lane == 0)
                    for (uint32_t x = k > (uint32_t)A.ring ? k - A.ring : 0; x < k; ++x)
                        mbar_wait_bounded(raw_full + x % A.ring, (x / A.ring) & 1, A.wait_clocks);
                __syncwarp();
            }
        } else {
            // ---------------- re-layout ----------------
            const int tid = threadIdx.x - D16_EPI_THREADS - 64;
            const int groups = (L + 3) / 4;  // (K bytes past a row's L limbs meet zero constants: whatever is there)
            // a coefficient of an octet (8 rows x 8 columns) each; consecutive threads take consecutive
            // rows of one column, so that their 16-byte stores (rows of a core matrix) and, by the raw
            // rows' pitch, their loads fall on different banks
            const int r = tid & 7, c = tid >> 3;
            const int row_off = r * segw + c * L;
            uint32_t k = 0;
            bool ok = true;
            for (uint32_t i = 0; i < my_super && ok; ++i) {
                const int buf = A.nb_buf == 2 ? (int)(i & 1) : 0;
                const uint32_t t0 = (me + i * mates) * (uint32_t)qrun;
                // the MMAs that last read this buffer (super-tile i - nb_buf) are complete
                if (i >= (uint32_t)A.nb_buf) {
                    const uint32_t o = i - A.nb_buf;
                    ok = wait_or_abort(mma_done + 2 * (o & 1) + 1, (o >> 1) & 1, abort_f, A.wait_clocks);
                }
                // octet o's rows of column c: operand rows 16 c + 8 (o & 1) + r of tile o / 2
                unsigned char* bt = b_s + buf * b_bytes + (size_t)(2 * c) * sbo + r * 16;
                for (int pc = 0; pc < npieces && ok; ++pc) {
                    const int o0 = pc * npo;
                    const int no = min(npo, 2 * (int)min((uint32_t)qrun, ntiles - t0) - o0);
                    if (no <= 0) break;
                    const uint32_t sl = k % A.ring;
                    if constexpr (LV > 0) {
                        ok = wait_or_abort(raw_full + sl, (k / A.ring) & 1, abort_f, A.wait_clocks);
                        if (!ok) break;
                    }
                    ++k;
#pragma unroll 1
                    for (int oc = 0; oc < no; ++oc) {
                        const int o = o0 + oc;
                        unsigned char* dst = bt + (size_t)(16 * (o >> 1) + (o & 1)) * sbo;
                        const uint32_t* row = raw_s + sl * piece_words + (8 * oc) * segw + row_off;
                        if constexpr (LV == 0) {
                            const uint32_t tile = t0 + (o >> 1), b = tile / tiles_x, cx = tile - b * tiles_x;
                            row = src + (((size_t)b * 16 + 8 * (o & 1) + r) * A.cw + 8 * cx + c) * L;
                        }
                        // a batch's loads before its stores: the compiler must assume that they alias
#pragma unroll 1
                        for (int g = 0; g < groups; g += 4) {
                            uint4 v[4];
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                // (past the row's end: its first group, not stored)
                                const int l = g + u < groups ? 4 * (g + u) : 0;
                                if constexpr (LV == 4) {
                                    v[u] = *reinterpret_cast<const uint4*>(row + l);
                                } else if constexpr (LV == 2) {
                                    const uint2 u0 = *reinterpret_cast<const uint2*>(row + l);
                                    const uint2 u1 = *reinterpret_cast<const uint2*>(row + l + 2);
                                    v[u] = make_uint4(u0.x, u0.y, u1.x, u1.y);
                                } else if constexpr (LV == 1) {
                                    v[u] = make_uint4(row[l], row[l + 1], row[l + 2], row[l + 3]);
                                } else {
                                    v[u] = make_uint4(row[l], row[min(l + 1, L - 1)], row[min(l + 2, L - 1)],
                                                      row[min(l + 3, L - 1)]);
                                }
                            }
#pragma unroll
                            for (int u = 0; u < 4; ++u)
                                if (g + u < groups) *reinterpret_cast<uint4*>(dst + (g + u) * 128) = v[u];
                        }
                    }
                    if constexpr (LV > 0) {
                        fence_smem_to_async();  // the reads above, before the slot's next copy
                        mbar_arrive(raw_empty + sl);
                    }
                }
                fence_smem_to_async();
                if (ok) mbar_arrive(b_full + buf);
            }
        }
    } else {
        // ---------------- epilogue ----------------
        regs_inc<D16_EPI_REGS>();
        const int grp = warp >> 2, quarter = warp & 3;
        const int glanes = 128 / q;
        const int ln = quarter * 32 + lane;
        const int s = ln / glanes, jl = ln % glanes;  // tile of the super-tile, prime
        const bool warp_used = s < qrun && (quarter * 32) % glanes < A.K;  // warp-uniform
        const bool mine = s < qrun && jl < A.K;
        const int j = min(jl, A.K - 1);
        const uint32_t p = A.p[j], wsh = A.wsh[j];
        const uint2* tw = tw_s + j;
        const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16);
        const size_t N = A.N, ncols = A.N / 16;
        for (uint32_t i = (uint32_t)grp; i < my_super; i += 2) {
            if (*abort_f) break;
            const uint32_t tile = (me + i * mates) * (uint32_t)qrun + (uint32_t)s;
            uint64_t* done = mma_done + 2 * grp;
            const uint32_t par = (i >> 1) & 1;
            // columns 0-3 and 4-7 of the tile, [column][row].  The two halves run through one copy
            // of the code: unrolled, its 58 KB passed the instruction cache (measured: up to 32 KB
            // run at full rate) and fetching took more time than issuing.
            uint32_t lo[4][16], hi[4][16];
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int e = 0; e < 16; ++e) lo[c][e] = hi[c][e];
                const bool got = __all_sync(0xffffffffu, wait_or_abort(done + h, par, abort_f, A.wait_clocks));
                tc_fence_after();
                if (!got || !warp_used) {
                    tc_fence_before();
                    mbar_arrive(acc_empty + h);
                    continue;
                }
                // 8 chunks of 8 rows (column k / 2, rows 8 (k % 2) ..): the next chunk's TMEM loads
                // run under this chunk's reductions
                uint32_t r[2][4][8];
                const uint32_t ta = taddr + 256u * h;
                auto load = [&](int k, uint32_t (&x)[4][8]) {
#pragma unroll
                    for (int t = 0; t < 4; ++t) tmem_ld8_async(ta + 8u * k + 64u * t, x[t]);
                };
                load(0, r[0]);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    uint32_t(&x)[4][8] = r[k & 1];
                    tmem_wait_ld_4x8(x[0], x[1], x[2], x[3]);
                    if (k < 7) load(k + 1, r[(k + 1) & 1]);
                    else {  // the half's last loads are done: it is free for the next tile
                        tc_fence_before();
                        mbar_arrive(acc_empty + h);
                    }
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        hi[k >> 1][8 * (k & 1) + e] = dec_reduce(x[0][e], x[1][e], x[2][e], x[3][e], p, wsh);
                }
                auto stw = [&](int t) { return StrideTw<false>{tw + ((1 << t) - 1) * tws, tws, 1 << t}; };
                radix_fwd2<4, 0>(hi[0], hi[1], stw, p);  // pairs of columns share their twiddle reads
                radix_fwd2<4, 0>(hi[2], hi[3], stw, p);
            }
            if (mine && tile < ntiles && *abort_f == 0) {
                const uint32_t b = tile / tiles_x, cx = tile - b * tiles_x;
                uint32_t* o = A.R[op] + residue_base(b, A.K2, j, N) + residue_off(A.col0 + 8 * cx);
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const uint32_t w[8] = {lo[0][e], lo[1][e], lo[2][e], lo[3][e], hi[0][e], hi[1][e], hi[2][e], hi[3][e]};
                    st_global_v8(o + e * (2 * ncols), w);
                }
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && *abort_f) flag_error(A.status, DEV_ERR_WAIT);
    if (warp == 0) tmem_dealloc(tmem, 512);
}

size_t dec16_smem(const Dec16Args& A) {
    return (size_t)A.a_bytes + (size_t)A.nb_buf * A.q * TC_M * A.kb + (size_t)A.ring * A.piece_octets * 8 * A.segw * 4 +
           (size_t)15 * A.KP * 8 + (9 + 2 * DEC16_MAX_RING) * 8 + 16;
}

void launch_dec16(const Dec16Args& A, uint32_t grid, size_t smem, cudaStream_t s, bool pdl) {
    const bool bulk = (uintptr_t)A.src[0] % 16 == 0 && (A.nops == 1 || (uintptr_t)A.src[1] % 16 == 0);
    const cudaError_t e = launch_kernel(!bulk ? k_dec16<0> : A.L % 4 == 0 ? k_dec16<4> : A.L % 2 == 0 ? k_dec16<2> : k_dec16<1>,
                                        dim3(grid), dim3(DEC16_THREADS), smem, s, pdl, A);
    if (e != cudaSuccess) throw_cuda(e, "launch k_dec16");
}

void dec16_set_smem_limit(int bytes) {
    for (auto f : {k_dec16<0>, k_dec16<1>, k_dec16<2>, k_dec16<4>}) {
        const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) throw_cuda(e, "k_dec16 attribute");
    }
}

}  // namespace pm
