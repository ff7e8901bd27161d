// hbg_mixed_kernels.cuh -- kernels of the mixed-precision form.
//
// Storage: every matrix of a frequency is two FP32 planes (real, imaginary), Np x Np with Np the
// panel count rounded up to a multiple of 128, column-major as the assembly writes it: entry (k, n)
// of A at n Np + k.  Read row-major, that buffer is M = A^T, and the LU runs on M without pivoting
// (in panels of PW = 256 columns): M = L U, so A = U^T L^T and A x = b is U^T y = b, L^T x = y.
// Up to LU_Q panels form a super-step, after which the trailing matrix is updated once: its FP32 entries pass
// through DRAM N / (256 q) times instead of N / 256.  Panel j of a super-step (columns k0 .. k0 + 255):
//   update    its columns, then its rows to their right, by the super-step's panels before it (FP16 operands)
//   diag      the 256 x 256 block: two 128 blocks factored and inverted in shared memory, the products
//             between them in FP32 (k_mid); X = L^-1 and Y = U^-1 of the whole block
//   L, U      L = M Y below the block (in place), U = X M to its right (from a transposed copy), TF32
// and after the last panel the trailing matrix -= [L of the super-step] [U of the super-step] (FP16 copies
// of L and U, FP32 accumulation); the refinement in FP64 restores the accuracy of the solution
// (iterative refinement against the stored complex64 matrix).
#pragma once
#include <cuda_fp16.h>

#include "hbg_tc.cuh"

namespace hbg {

constexpr int NBL = 128;    // order of the diagonal blocks
constexpr int PW = 2 * NBL;  // columns of a panel
constexpr int LU_Q = 4;      // panels of a super-step, at most
constexpr int GBM = 128, GBN = 128, GBK = 32, GSTAGES = 3;  // rows, complex columns; FP32 complex entries of a chunk
constexpr int GNBOX = 2;     // ring of 32-column output boxes in shared memory

enum CgemmTri { CG_FULL, CG_RIGHT_UPPER, CG_LEFT_LOWER };
struct CgemmArgs {
    int mt, nt;            // row tiles and column tiles (128 complex columns) of a matrix
    int K;                 // complex inner length
    int tri;               // CG_RIGHT_UPPER: C = A Y with Y upper triangular, K = 256: column tile 1 first, then tile 0 with
                           // its 128 k alone, by the same CTA (C may lie over A); CG_LEFT_LOWER: C = X B with X lower
                           // triangular, K = 256: row tile 0 with its 128 k alone
    int a_k0, a_row0;      // A's first k and row in its map
    int b_n0;              // B's first column (K-major: row) in its map
    int subtract;          // C -= A B by a reduction at L2, else C = A B
    int o_row0, o_col0;    // C's first row and column in the planar matrix
    int batch, b0;         // matrices of the launch, the first one's index in the maps
    // an FP16 copy of C (or null): planes of h_plane halves, row o_row0 + i at i + h_row0, column o_col0 + j at j + h_col0
    __half* h16;
    size_t h_bstride, h_plane;
    int h_ld, h_row0, h_col0;
    int* err;
};

__device__ __forceinline__ uint8_t* align1024(uint8_t* p) {
    return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~uintptr_t(1023));
}

constexpr int GEMM_THREADS = 192;  // warp 0 TMA, warp 1 MMA, warps 2..5 epilogue
constexpr size_t GEMM_TILE_BYTES = (size_t)GBM * GBK * 4;        // one plane of one operand's chunk
constexpr size_t GEMM_STAGE_BYTES = 4 * GEMM_TILE_BYTES;         // Ar, Ai, Br, Bi
constexpr size_t GEMM_BOX_BYTES = (size_t)GBM * 32 * 4;  // one 32-column box of the output tile
constexpr size_t gemm_smem_bytes() { return 1024 + GSTAGES * GEMM_STAGE_BYTES + GNBOX * GEMM_BOX_BYTES + 256; }

// Persistent, warp-specialized complex product of the mixed LU, C = A B or C -= A B on planar operands:
// tiles of 128 rows x 128 complex columns taken round-robin over (row tile, column tile, matrix).  A k-chunk
// is the four planes Ar, Ai, Br, Bi (128-byte rows: 32 FP32 or 64 FP16 entries), streamed by warp 0 through a
// three-stage TMA ring; warp 1 issues per 32 bytes of k the four M 128, N 128 products Cr += Ar Br,
// Ci += Ar Bi, Cr += (-Ai) Bi (the descriptor's negation), Ci += Ai Br into one of two TMEM accumulators [Cr | Ci].
// Each operand byte is loaded once for two products: 64 KB from L2 per 128 x 128 x 64 complex chunk against
// 96 KB for the real product on the doubled operand [[Br, Bi], [-Bi, Br]], which also had to be stored.
// F16: FP16 operands (kind::f16), B in its natural row-major form (k rows, N contiguous: MN-major); otherwise
// FP32 read as TF32, B given transposed (K-major).  Warps 2..5 read the accumulator (tcgen05.ld) in 32-column
// chunks, place each chunk in a ring of shared-memory boxes (128-byte swizzle, conflict-free 16-byte accesses) and
// write it out by TMA: a store, or for an update a TMA reduction that adds -acc to C in L2 (so C never
// passes through the SM).  The epilogue of one tile overlaps the main loop of the next.
// Bound by the tensor pipe and, over a whole LU, the power cap: the first trailing update of five systems of
// order 18560 (K = 1024) runs at 1231 TFLOP/s (10.2 ms) where cuBLAS bf16 reaches 1361 sustained; the doubled real
// product at K = 256 a step ran at 530 on 88 SMs, its C passing through DRAM four times as often.
template <bool F16>
__global__ void __launch_bounds__(GEMM_THREADS, 1) k_cgemm(const __grid_constant__ CUtensorMap mapA,
                                                           const __grid_constant__ CUtensorMap mapB,
                                                           const __grid_constant__ CUtensorMap mapC, CgemmArgs g) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = align1024(smem_raw);
    float* sBox = reinterpret_cast<float*>(base + GSTAGES * GEMM_STAGE_BYTES);  // [GNBOX][128 rows][32]
    uint64_t* full = reinterpret_cast<uint64_t*>(sBox + GNBOX * GBM * 32);
    uint64_t* empty = full + GSTAGES;
    uint64_t* tfull = empty + GSTAGES;  // [2]
    uint64_t* tempty = tfull + 2;       // [2]
    uint64_t* drain = tempty + 2;       // the MMA warp's last commit (every issued MMA complete)
    uint32_t* tslot = reinterpret_cast<uint32_t*>(drain + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int KE = F16 ? 2 * GBK : GBK;  // entries per chunk row (128 bytes either way)
    if (threadIdx.x == 0) {
        for (int s = 0; s < GSTAGES; s++) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            tc::mbar_init(&tfull[b], 1);
            tc::mbar_init(&tempty[b], 4);  // one arrival per epilogue warp
        }
        tc::mbar_init(drain, 1);
        tc::fence_barrier_init();
        tc::prefetch_tensormap(&mapA);
        tc::prefetch_tensormap(&mapB);
        tc::prefetch_tensormap(&mapC);
    }
    if (warp == 0) tc::tmem_alloc(tslot, 4 * GBN);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = *tslot;
    // the CTA's it-th tile: row and column tile, matrix, chunks of k; false beyond the last
    auto tile = [&](int it, int& m, int& n, int& f, int& nk) -> bool {
        int u = it, sub = -1;
        if (g.tri == CG_RIGHT_UPPER) u = it >> 1, sub = 1 - (it & 1);  // units of one row tile
        const int per = sub < 0 ? g.mt * g.nt : g.mt, t = blockIdx.x + u * gridDim.x;
        if (t >= per * g.batch) return false;
        f = t / per;
        const int r = t - f * per;
        n = sub < 0 ? r / g.mt : sub;  // row tiles fastest: consecutive CTAs share the B block
        m = r % g.mt;
        const bool half = (g.tri == CG_RIGHT_UPPER && n == 0) || (g.tri == CG_LEFT_LOWER && m == 0);
        nk = (half ? NBL : g.K) / KE;
        return true;
    };
    int m, n, f, nk;
    if (warp == 0) {
        if (lane == 0) {
            int kc_global = 0;
            bool bad = false;
            for (int it = 0; !bad && tile(it, m, n, f, nk); it++) {
                for (int kc = 0; kc < nk; kc++, kc_global++) {
                    const int s = kc_global % GSTAGES;
                    if (kc_global >= GSTAGES && !tc::mbar_wait(&empty[s], ((kc_global / GSTAGES) - 1) & 1)) {
                        atomicExch(g.err, 1);
                        bad = true;
                        break;
                    }
                    tc::mbar_arrive_expect_tx(&full[s], (uint32_t)GEMM_STAGE_BYTES);
                    uint8_t* st = base + s * GEMM_STAGE_BYTES;
                    const int kk = kc * KE;
#pragma unroll
                    for (int p = 0; p < 2; p++)
                        tc::tma_load_4d(st + p * GEMM_TILE_BYTES, &mapA, &full[s], g.a_k0 + kk, g.a_row0 + m * GBM, p,
                                        g.b0 + f);
#pragma unroll
                    for (int p = 0; p < 2; p++) {
                        uint8_t* sb = st + (2 + p) * GEMM_TILE_BYTES;
                        if constexpr (F16) {
#pragma unroll
                            for (int h = 0; h < 2; h++)  // 64 columns a box
                                tc::tma_load_4d(sb + h * (GEMM_TILE_BYTES / 2), &mapB, &full[s], g.b_n0 + n * GBN + 64 * h,
                                                kk, p, g.b0 + f);
                        } else {
                            tc::tma_load_4d(sb, &mapB, &full[s], kk, g.b_n0 + n * GBN, p, g.b0 + f);
                        }
                    }
                }
            }
            // every load still in flight lands before the CTA leaves (also after an error): the last
            // phase armed on each stage completes (bounded)
            for (int k = kc_global > GSTAGES ? kc_global - GSTAGES : 0; k < kc_global; k++)
                if (!tc::mbar_wait(&full[k % GSTAGES], (k / GSTAGES) & 1)) {
                    atomicExch(g.err, 6);
                    break;
                }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = F16 ? (tc::idesc_f16(GBM, GBN) | tc::IDESC_B_MN) : tc::idesc_tf32(GBM, GBN);
            constexpr uint32_t TB_ = (uint32_t)GEMM_TILE_BYTES;
            int kc_global = 0;
            for (int it = 0; tile(it, m, n, f, nk); it++) {
                const int b = it & 1;
                // the accumulator buffer must have been drained by the epilogue of tile it - 2
                if (it >= 2 && !tc::mbar_wait(&tempty[b], ((it >> 1) - 1) & 1)) {
                    atomicExch(g.err, 5);
                    break;
                }
                tc::tc_fence_after();
                const uint32_t cr = tmem + b * 2 * GBN, ci = cr + GBN;
                bool bad = false;
                for (int kc = 0; kc < nk; kc++, kc_global++) {
                    const int s = kc_global % GSTAGES;
                    if (!tc::mbar_wait(&full[s], (kc_global / GSTAGES) & 1)) {
                        atomicExch(g.err, 2);
                        bad = true;
                        break;
                    }
                    tc::tc_fence_after();
                    const uint32_t a0 = tc::smem_u32(base + s * GEMM_STAGE_BYTES), b0 = a0 + 2 * TB_;
                    // four k-steps per 128-byte row: K = 8 (tf32) or 16 (f16); in the MN-major B, 16 rows of 128 bytes
#pragma unroll
                    for (int ks = 0; ks < 4; ks++) {
                        const uint64_t ar = tc::desc_kmajor_sw128(a0 + 32 * ks), ai = tc::desc_kmajor_sw128(a0 + TB_ + 32 * ks);
                        uint64_t br, bi;
                        if constexpr (F16) {
                            br = tc::desc_mnmajor_sw128(b0 + 2048 * ks, TB_ / 2);
                            bi = tc::desc_mnmajor_sw128(b0 + TB_ + 2048 * ks, TB_ / 2);
                        } else {
                            br = tc::desc_kmajor_sw128(b0 + 32 * ks);
                            bi = tc::desc_kmajor_sw128(b0 + TB_ + 32 * ks);
                        }
                        const uint32_t acc = (kc | ks) != 0;
                        if constexpr (F16) {
                            tc::mma_f16(cr, ar, br, idesc, acc);
                            tc::mma_f16(ci, ar, bi, idesc, acc);
                            tc::mma_f16(cr, ai, bi, idesc | tc::IDESC_NEG_A, 1);
                            tc::mma_f16(ci, ai, br, idesc, 1);
                        } else {
                            tc::mma_tf32(cr, ar, br, idesc, acc);
                            tc::mma_tf32(ci, ar, bi, idesc, acc);
                            tc::mma_tf32(cr, ai, bi, idesc | tc::IDESC_NEG_A, 1);
                            tc::mma_tf32(ci, ai, br, idesc, 1);
                        }
                    }
                    tc::mma_commit(&empty[s]);
                }
                tc::mma_commit(&tfull[b]);
                if (bad) break;
            }
            // every issued MMA completes before TMEM is freed (also after an error; bounded)
            tc::mma_commit(drain);
            if (!tc::mbar_wait(drain, 0)) atomicExch(g.err, 7);
        }
    } else {
        // epilogue warps 2..5: TMEM lane quadrant (warp % 4), rows 32 (warp % 4) .. + 32 of the tile;
        // thread 64 (warp 2, lane 0) issues the box writes and tracks their bulk groups
        const int quad = warp & 3;
        const int r = quad * 32 + lane;  // row within the tile
        const bool issuer = threadIdx.x == 64;
        int bx = 0;
        for (int it = 0; tile(it, m, n, f, nk); it++) {
            const int b = it & 1;
            const bool ok = tc::mbar_wait(&tfull[b], (it >> 1) & 1);
            // one decision for the four epilogue warps, so none waits at a barrier the others left
            __syncwarp();
            if (!tc::bar_and(ok, 1, 128)) {
                if (issuer) atomicExch(g.err, 3);
                break;
            }
            tc::tc_fence_after();
            const int hr = m * GBM + r + g.h_row0;  // the row of the FP16 copy
            const float sg = g.subtract ? -1.f : 1.f;
            for (int q = 0; q < 2 * GBN / 32; q++, bx++) {
                float v[32];
                tc::tmem_ld32(tmem + b * 2 * GBN + ((uint32_t)(quad * 32) << 16) + q * 32, v);
                const int plane = q / (GBN / 32), col = n * GBN + 32 * (q % (GBN / 32));
                // the box slot is free once the write issued GNBOX boxes ago has read it
                if (issuer && bx >= GNBOX) tc::bulk_wait_read_n<GNBOX - 1>();
                asm volatile("bar.sync 1, 128;" ::: "memory");
                float* row = sBox + (bx % GNBOX) * GBM * 32 + r * 32;  // 128 B, 16-byte chunks swizzled by r % 8
#pragma unroll
                for (int j = 0; j < 8; j++)
                    *reinterpret_cast<float4*>(row + 4 * (j ^ (r & 7))) =
                        make_float4(sg * v[4 * j], sg * v[4 * j + 1], sg * v[4 * j + 2], sg * v[4 * j + 3]);
                if (g.h16) {
                    __half* h = g.h16 + (size_t)(g.b0 + f) * g.h_bstride + (size_t)plane * g.h_plane +
                                (size_t)hr * g.h_ld + g.h_col0 + col;
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        __half2 hv[4];
#pragma unroll
                        for (int e = 0; e < 4; e++) hv[e] = __floats2half2_rn(v[8 * j + 2 * e], v[8 * j + 2 * e + 1]);
                        *reinterpret_cast<uint4*>(h + 8 * j) = *reinterpret_cast<const uint4*>(hv);
                    }
                }
                tc::fence_proxy_async_smem();
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (issuer) {
                    const float* box = sBox + (bx % GNBOX) * GBM * 32;
                    if (g.subtract)
                        tc::tma_reduce_add_4d(&mapC, box, g.o_col0 + col, g.o_row0 + m * GBM, plane, g.b0 + f);
                    else
                        tc::tma_store_4d(&mapC, box, g.o_col0 + col, g.o_row0 + m * GBM, plane, g.b0 + f);
                    tc::bulk_commit();  // one group per box
                }
            }
            // the accumulator buffer is free for the MMA of tile it + 2
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&tempty[b]);
        }
        if (issuer) tc::bulk_wait_all();
    }
    tc::tc_fence_before();
    __syncthreads();
    // freed even when a drain wait above gave up (err set, the results discarded): a CTA that left
    // holding TMEM would stall every later allocation on its SM
    if (warp == 0) tc::tmem_dealloc(tmem, 4 * GBN);
}

// ---- the diagonal block: M11 = L11 U11 (no pivoting), then L11^-1 and U11^-1.  Two CTAs per matrix
// (blockIdx.x = 2 f + side, one cluster, so that they run at once) factor the same block in their own
// shared memory; side 0 then forms L^-1 (and writes the factors back to W, once side 1 has read the block
// too: a cluster barrier, arrived at after the load), side 1 U^-1.  Outputs: PX (rows of L^-1, the A operand of
// the U product) and PY (columns of U^-1 as rows, the B operand of the L product), the 128 blocks at
// (koff, koff) of [F][2 planes][PW][PW], and DINV (U^-1 on and above the diagonal, L^-1 below it, two planes
// a block, for the triangular solves).  A pivot of modulus below 1e-15 sets err (the mixed form then reports the
// frequency; the FP64 form pivots).
constexpr int DF_THREADS = 512, DF_LD = NBL + 1, DF_BLK = 32, DF_NB = NBL / DF_BLK, DF_SLD = DF_BLK + 1;

__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// complex multiply-adds as four FMA instructions (no separate product and sum)
__device__ __forceinline__ void cfma_sub(float2& x, float2 a, float2 b) {  // x -= a b
    x.x = fmaf(-a.x, b.x, x.x);
    x.x = fmaf(a.y, b.y, x.x);
    x.y = fmaf(-a.x, b.y, x.y);
    x.y = fmaf(-a.y, b.x, x.y);
}
__device__ __forceinline__ void cfma_add(float2& x, float2 a, float2 b) {  // x += a b
    x.x = fmaf(a.x, b.x, x.x);
    x.x = fmaf(-a.y, b.y, x.x);
    x.y = fmaf(a.x, b.y, x.y);
    x.y = fmaf(a.y, b.x, x.y);
}

// LU by 16-column panels: the 16 x 16 diagonal block by one warp in registers (lane = row, the pivot
// row published through shared memory, no CTA barrier per pivot), then L21 = A21 U11^-1 (a lane per
// row) and U12 = L11^-1 A12 (a lane per column) by independent substitutions, then A22 -= L21 U12 by
// all warps in register tiles.  Inverses: the eight 16 x 16 diagonal blocks inverted in registers and
// put in place, then the off-diagonal blocks by the block recursion inv([[A, 0], [C, B]]) =
// [[A^-1, 0], [-B^-1 C A^-1, B^-1]] (16 -> 32 -> 64 -> 128; for U the transposed pattern), each level
// two products of block-triangular operands through a shared scratch.  (Fully unrolled code run by a
// single warp, and per-pivot shuffles, were measured slower than these short register recursions.)
constexpr int DF3_TLD = 2 * DF_BLK + 1, DF3_P = 16;  // DF3_P: LU panel width
constexpr int DF3_TSZ = DF_NB * DF_BLK * DF_SLD;  // the scratch: 4 blocks of 32 x DF_SLD (>= 64 x DF3_TLD)
static_assert(DF3_TSZ >= 2 * DF_BLK * DF3_TLD, "scratch holds the 64 x 64 product");
constexpr size_t df_smem_bytes() { return (size_t)(NBL * DF_LD + DF3_TSZ + NBL) * sizeof(float2); }

__device__ __forceinline__ float2 crecip(float2 d) {  // 1 / d by one reciprocal of |d|^2
    const float r = __frcp_rn(d.x * d.x + d.y * d.y);
    return make_float2(d.x * r, -d.y * r);
}

// A22 -= L21 U12 over rows and columns b0 .. NBL - 1 (n2 = NBL - b0 = 16 TR = 32 TC), k over the panel
// c0 .. c0 + 31: warp w the rows b0 + 16 a + w, lane the columns b0 + 32 b + lane.
template <int TR, int TC>
__device__ __forceinline__ void df3_trailing(float2* blk, int c0, int b0) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float2 acc[TR][TC];
#pragma unroll
    for (int a = 0; a < TR; a++)
#pragma unroll
        for (int b = 0; b < TC; b++) acc[a][b] = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int k = 0; k < DF3_P; k++) {
        float2 l[TR], u[TC];
#pragma unroll
        for (int a = 0; a < TR; a++) l[a] = blk[(b0 + 16 * a + warp) * DF_LD + c0 + k];
#pragma unroll
        for (int b = 0; b < TC; b++) u[b] = blk[(c0 + k) * DF_LD + min(b0 + 32 * b + lane, NBL - 1)];
#pragma unroll
        for (int a = 0; a < TR; a++)
#pragma unroll
            for (int b = 0; b < TC; b++) cfma_add(acc[a][b], l[a], u[b]);
    }
#pragma unroll
    for (int a = 0; a < TR; a++)
#pragma unroll
        for (int b = 0; b < TC; b++)
            if (b0 + 32 * b + lane < NBL) {
                float2& x = blk[(b0 + 16 * a + warp) * DF_LD + b0 + 32 * b + lane];
                x = make_float2(x.x - acc[a][b].x, x.y - acc[a][b].y);
            }
}

// Step J of a 16 x 16 LU by lanes 0..15 of a warp (lane = row, a = the lane's row; lanes 16..31 hold
// zeros): the pivot row published through shared memory (row, 16 entries), rcp[J] = 1 / U(J, J), ok
// false on a pivot of modulus below 1e-15.  Recursion keeps every register index constant; no
// branch around the updates (lanes at or above the pivot subtract zero).
template <int J>
__device__ __forceinline__ void df3_lu16_step(float2 (&a)[DF3_P], int lane, float2* row, float2* rcp, bool& ok) {
    if constexpr (J < DF3_P) {
        if (lane == J)
#pragma unroll
            for (int k = J; k < DF3_P; k++) row[k] = a[k];
        __syncwarp();
        const float2 d = row[J];
        ok = ok && d.x * d.x + d.y * d.y > 1e-30f;
        const float2 inv = crecip(d);
        if (lane == 0) rcp[J] = inv;
        const float2 l = cmulf(a[J], inv);
        const float2 lm = lane > J ? l : make_float2(0.f, 0.f);
#pragma unroll
        for (int k = J + 1; k < DF3_P; k++) cfma_sub(a[k], lm, row[k]);
        if (lane > J) a[J] = l;
        __syncwarp();
        df3_lu16_step<J + 1>(a, lane, row, rcp, ok);
    }
}

// x = x U^-1 for the upper 16 x 16 block at Ub (leading dimension DF_LD; rcp[k] = 1 / U(k, k)): step K
// finishes x[K] and removes it from the later unknowns.
template <int K>
__device__ __forceinline__ void df3_urow16_step(float2 (&x)[DF3_P], const float2* Ub, const float2* rcp) {
    if constexpr (K < DF3_P) {
        x[K] = cmulf(x[K], rcp[K]);
#pragma unroll
        for (int j = K + 1; j < DF3_P; j++) cfma_sub(x[j], x[K], Ub[K * DF_LD + j]);
        df3_urow16_step<K + 1>(x, Ub, rcp);
    }
}

// x = x L^-1 for the unit lower 16 x 16 block at Lb, from the last column: step K (x[K] final) removes
// x[K] from the earlier unknowns.
template <int K>
__device__ __forceinline__ void df3_lrow16_back_step(float2 (&x)[DF3_P], const float2* Lb) {
    if constexpr (K > 0) {
#pragma unroll
        for (int j = 0; j < K; j++) cfma_sub(x[j], x[K], Lb[K * DF_LD + j]);
        df3_lrow16_back_step<K - 1>(x, Lb);
    }
}

// y = L^-1 y for the unit lower 16 x 16 block at Lb, step K removing y[K] from the later unknowns.
template <int K>
__device__ __forceinline__ void df3_lcol16_step(float2 (&y)[DF3_P], const float2* Lb) {
    if constexpr (K < DF3_P - 1) {
#pragma unroll
        for (int j = K + 1; j < DF3_P; j++) cfma_sub(y[j], Lb[j * DF_LD + K], y[K]);
        df3_lcol16_step<K + 1>(y, Lb);
    }
}

// Block-triangular operand patterns of df3_product (block = 32 x 32): which k of the sum are nonzero
// for the output tile in block row ib, block column jb of C.
enum Df3Tri { DF3_B_LOWER, DF3_A_LOWER, DF3_B_UPPER, DF3_A_UPPER };

// C(m x m) = sgn A(m x m) B(m x m), m = 32 or 64, A and B of leading dimensions lda, ldb, C of ldc;
// threads tid0 .. tid0 + nthr - 1, each a 2 x 2 tile: rows 2 ri + {0, 1}, columns cj + {0, 16} of a
// 32 x 32 output block (consecutive lanes read consecutive columns of B).
__device__ __forceinline__ void df3_product(const float2* A, int lda, const float2* B, int ldb, float2* C, int ldc,
                                            int m, Df3Tri tri, float sgn, int tid, int nthr) {
    const int nbk = m / DF_BLK, tiles = nbk * nbk * 256;
    for (int t = tid; t < tiles; t += nthr) {
        const int blkid = t / 256, w = t % 256, ib = blkid / nbk, jb = blkid % nbk;
        const int i0 = ib * DF_BLK + 2 * (w / 16), j0 = jb * DF_BLK + (w % 16);
        int klo = 0, khi = m;
        if (tri == DF3_B_LOWER) klo = jb * DF_BLK;
        if (tri == DF3_A_LOWER) khi = (ib + 1) * DF_BLK;
        if (tri == DF3_B_UPPER) khi = (jb + 1) * DF_BLK;
        if (tri == DF3_A_UPPER) klo = ib * DF_BLK;
        float2 c00 = make_float2(0.f, 0.f), c01 = c00, c10 = c00, c11 = c00;
#pragma unroll 4
        for (int k = klo; k < khi; k++) {
            const float2 a0 = A[i0 * lda + k], a1 = A[(i0 + 1) * lda + k];
            const float2 b0 = B[k * ldb + j0], b1 = B[k * ldb + j0 + 16];
            cfma_add(c00, a0, b0);
            cfma_add(c01, a0, b1);
            cfma_add(c10, a1, b0);
            cfma_add(c11, a1, b1);
        }
        C[i0 * ldc + j0] = make_float2(sgn * c00.x, sgn * c00.y);
        C[i0 * ldc + j0 + 16] = make_float2(sgn * c01.x, sgn * c01.y);
        C[(i0 + 1) * ldc + j0] = make_float2(sgn * c10.x, sgn * c10.y);
        C[(i0 + 1) * ldc + j0 + 16] = make_float2(sgn * c11.x, sgn * c11.y);
    }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(DF_THREADS) k_diag_factor(float* __restrict__ W, int Np, size_t bstride, int k0,
                                                              int koff, float* __restrict__ PX, float* __restrict__ PY,
                                                              float* __restrict__ DINV, int* __restrict__ err) {
    extern __shared__ float2 df_smem[];
    float2* blk = df_smem;                   // [NBL][DF_LD]: the block, then its factors, then the inverse
    float2* T = blk + NBL * DF_LD;  // scratch: the diagonal-block inverses, then the products of the recursion
    float2* rcp = T + DF3_TSZ;      // [NBL]: 1 / U(j, j)
    const int f = blockIdx.x >> 1, side = blockIdx.x & 1;
    const bool upper = side == 1;
    float* Wr = W + (size_t)f * bstride;
    float* Wi = Wr + (size_t)Np * Np;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the block in 16-byte loads (rows of 128 entries, k0 and Np multiples of 128), 16 in flight a thread
#pragma unroll 8
    for (int t = threadIdx.x; t < NBL * NBL / 4; t += DF_THREADS) {
        const int r = t / (NBL / 4), c = 4 * (t % (NBL / 4));
        const size_t o = (size_t)(k0 + r) * Np + k0 + c;
        const float4 re = *reinterpret_cast<const float4*>(Wr + o), im = *reinterpret_cast<const float4*>(Wi + o);
        float2* d = blk + r * DF_LD + c;
        d[0] = make_float2(re.x, im.x);
        d[1] = make_float2(re.y, im.y);
        d[2] = make_float2(re.z, im.z);
        d[3] = make_float2(re.w, im.w);
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // this CTA has read the block
    __syncthreads();
#pragma unroll 1
    for (int pb = 0; pb < NBL / DF3_P; pb++) {
        const int c0 = pb * DF3_P, b0 = c0 + DF3_P, n2 = NBL - b0;
        if (warp == 0) {  // the 16 x 16 diagonal block: lane = row (lanes 16..31 carry zeros, write nothing)
            float2* P = blk + c0 * DF_LD + c0;
            float2 a[DF3_P];
#pragma unroll
            for (int k = 0; k < DF3_P; k++) a[k] = lane < DF3_P ? P[lane * DF_LD + k] : make_float2(0.f, 0.f);
            bool ok = true;
            df3_lu16_step<0>(a, lane, T, rcp + c0, ok);
            if (lane == 0 && !ok) atomicExch(err, 10);
            if (lane < DF3_P)
#pragma unroll
                for (int k = 0; k < DF3_P; k++) P[lane * DF_LD + k] = a[k];
        }
        __syncthreads();
        if (n2 == 0) break;
        const int nw = (n2 + 31) / 32;  // warps of each substitution
        if (warp >= 1 && warp <= nw) {  // L21 = A21 U11^-1: lane = row
            const int i = b0 + 32 * (warp - 1) + lane;
            if (i < NBL) {
                float2 x[DF3_P];
#pragma unroll
                for (int k = 0; k < DF3_P; k++) x[k] = blk[i * DF_LD + c0 + k];
                df3_urow16_step<0>(x, blk + c0 * DF_LD + c0, rcp + c0);
#pragma unroll
                for (int k = 0; k < DF3_P; k++) blk[i * DF_LD + c0 + k] = x[k];
            }
        } else if (warp >= 5 && warp < 5 + nw) {  // U12 = L11^-1 A12: lane = column
            const int cc = b0 + 32 * (warp - 5) + lane;
            if (cc < NBL) {
                float2 y[DF3_P];
#pragma unroll
                for (int k = 0; k < DF3_P; k++) y[k] = blk[(c0 + k) * DF_LD + cc];
                df3_lcol16_step<0>(y, blk + c0 * DF_LD + c0);
#pragma unroll
                for (int k = 0; k < DF3_P; k++) blk[(c0 + k) * DF_LD + cc] = y[k];
            }
        }
        __syncthreads();
        switch (n2 / DF3_P) {  // A22 -= L21 U12 (k over the 16 panel columns)
            case 7: df3_trailing<7, 4>(blk, c0, b0); break;
            case 6: df3_trailing<6, 3>(blk, c0, b0); break;
            case 5: df3_trailing<5, 3>(blk, c0, b0); break;
            case 4: df3_trailing<4, 2>(blk, c0, b0); break;
            case 3: df3_trailing<3, 2>(blk, c0, b0); break;
            case 2: df3_trailing<2, 1>(blk, c0, b0); break;
            default: df3_trailing<1, 1>(blk, c0, b0); break;
        }
        __syncthreads();
    }
    // ---- the factors back to W (side 0), the other CTA's reads of the block done
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (side == 0)
#pragma unroll 8
        for (int t = threadIdx.x; t < NBL * NBL / 4; t += DF_THREADS) {
            const int r = t / (NBL / 4), c = 4 * (t % (NBL / 4));
            const size_t o = (size_t)(k0 + r) * Np + k0 + c;
            const float2* d = blk + r * DF_LD + c;
            *reinterpret_cast<float4*>(Wr + o) = make_float4(d[0].x, d[1].x, d[2].x, d[3].x);
            *reinterpret_cast<float4*>(Wi + o) = make_float4(d[0].y, d[1].y, d[2].y, d[3].y);
        }
    __syncthreads();
    // ---- the inverse of this side's factor, in place in blk
    // the eight 16 x 16 diagonal blocks (warp w: block w, lane = row of its inverse, in registers)
    constexpr int P = DF3_P, PL16 = DF3_P + 1;
    if (warp < NBL / P) {
        const float2* Ab = blk + warp * P * DF_LD + warp * P;
        float2 x[P];
#pragma unroll
        for (int k = 0; k < P; k++) x[k] = make_float2(k == lane ? 1.f : 0.f, 0.f);
        if (!upper)
            df3_lrow16_back_step<P - 1>(x, Ab);
        else
            df3_urow16_step<0>(x, Ab, rcp + warp * P);
        if (lane < P)
#pragma unroll
            for (int k = 0; k < P; k++) T[(warp * P + lane) * PL16 + k] = x[k];
    }
    __syncthreads();
    // ... into place, with zeros in the other triangle's 16-block of each 32 x 32 diagonal block
    for (int t = threadIdx.x; t < NBL * P; t += DF_THREADS) {
        const int w = t / (P * P), i = (t / P) % P, k = t % P;
        blk[(w * P + i) * DF_LD + w * P + k] = T[(w * P + i) * PL16 + k];
        const int z = w ^ 1;  // the partner block of the 32-block
        if ((z > w) == !upper) blk[(w * P + i) * DF_LD + z * P + k] = make_float2(0.f, 0.f);
    }
    __syncthreads();
    // 32-level: the four pairs at once (128 threads each); lower X(I, J) = -X(I, I) L(I, J) X(J, J) for
    // (I, J) = (2q + 1, 2q), upper Y(I, J) = -Y(I, I) U(I, J) Y(J, J) for (2q, 2q + 1) (16-blocks)
    {
        const int q = threadIdx.x / 128, tq = threadIdx.x % 128;
        const int I = (upper ? 2 * q : 2 * q + 1) * P, J = (upper ? 2 * q + 1 : 2 * q) * P;
        float2* Tq = T + q * P * PL16;
        // T = L(I, J) X(J, J), then X(I, J) = -X(I, I) T: two 16 x 16 outputs a thread
#pragma unroll
        for (int pass = 0; pass < 2; pass++) {
            const float2* A = pass == 0 ? blk + I * DF_LD + J : blk + I * DF_LD + I;
            const int lda = DF_LD;
            const float2* B = pass == 0 ? blk + J * DF_LD + J : Tq;
            const int ldb = pass == 0 ? DF_LD : PL16;
            const int r = tq / 8, c0 = (tq % 8) * 2;  // rows 0..15, column pairs
            float2 c00 = make_float2(0.f, 0.f), c01 = c00;
#pragma unroll 4
            for (int k = 0; k < P; k++) {
                const float2 a = A[r * lda + k];
                cfma_add(c00, a, B[k * ldb + c0]);
                cfma_add(c01, a, B[k * ldb + c0 + 1]);
            }
            __syncthreads();  // (pass 0) every thread's reads of L(I, J) done; (pass 1) of T
            if (pass == 0) {
                Tq[r * PL16 + c0] = c00;
                Tq[r * PL16 + c0 + 1] = c01;
            } else {
                blk[(I + r) * DF_LD + J + c0] = make_float2(-c00.x, -c00.y);
                blk[(I + r) * DF_LD + J + c0 + 1] = make_float2(-c01.x, -c01.y);
            }
            __syncthreads();
        }
    }
    // 64-level: the two pairs of 32-blocks at once (256 threads each); lower: X(I, J) = -X(I, I) L(I, J)
    // X(J, J) for (I, J) = (1, 0), (3, 2); upper: Y(I, J) = -Y(I, I) U(I, J) Y(J, J) for (0, 1), (2, 3)
    {
        const int q = threadIdx.x / 256, tq = threadIdx.x % 256;
        const int d0 = 2 * q * DF_BLK, d1 = d0 + DF_BLK;  // the pair's two diagonal blocks
        const int I = upper ? d0 : d1, J = upper ? d1 : d0;
        float2* Tq = T + q * DF_BLK * DF3_TLD;  // [32][DF3_TLD] rows of the pair's scratch
        df3_product(blk + I * DF_LD + J, DF_LD, blk + J * DF_LD + J, DF_LD, Tq, DF3_TLD, DF_BLK,
                    upper ? DF3_B_UPPER : DF3_B_LOWER, 1.f, tq, 256);
        __syncthreads();
        df3_product(blk + I * DF_LD + I, DF_LD, Tq, DF3_TLD, blk + I * DF_LD + J, DF_LD, DF_BLK,
                    upper ? DF3_A_UPPER : DF3_A_LOWER, -1.f, tq, 256);
    }
    __syncthreads();
    // 128-level: lower X21 = -X22 (L21 X11), upper Y12 = -Y11 (U12 Y22), 64 x 64 blocks
    {
        const int h = 2 * DF_BLK;
        const int I = upper ? 0 : h, J = upper ? h : 0;
        df3_product(blk + I * DF_LD + J, DF_LD, blk + J * DF_LD + J, DF_LD, T, DF3_TLD, h,
                    upper ? DF3_B_UPPER : DF3_B_LOWER, 1.f, threadIdx.x, DF_THREADS);
        __syncthreads();
        df3_product(blk + I * DF_LD + I, DF_LD, T, DF3_TLD, blk + I * DF_LD + J, DF_LD, h,
                    upper ? DF3_A_UPPER : DF3_A_LOWER, -1.f, threadIdx.x, DF_THREADS);
    }
    __syncthreads();
    // ---- outputs: this side's triangle of the inverse
    {
        float* D = DINV + ((size_t)f * (Np / NBL) + k0 / NBL) * 2 * NBL * NBL;
        for (int t = threadIdx.x; t < NBL * NBL; t += DF_THREADS) {
            const int i = t / NBL, c = t % NBL;
            if ((i > c) == !upper) {
                const float2 v = blk[i * DF_LD + c];
                D[t] = v.x;
                D[NBL * NBL + t] = v.y;
            }
        }
    }
    float* Pf = (upper ? PY : PX) + (size_t)f * 2 * PW * PW + (size_t)koff * PW + koff;
    for (int t = threadIdx.x; t < NBL * NBL; t += DF_THREADS) {
        const int a = t / NBL, b = t % NBL, i = upper ? b : a, c = upper ? a : b;  // PX: row i, PY: row c (b fastest)
        const float2 v = (upper ? i <= c : i > c) ? blk[i * DF_LD + c] : make_float2(!upper && i == c ? 1.f : 0.f, 0.f);
        Pf[(size_t)a * PW + b] = v.x;
        Pf[(size_t)PW * PW + (size_t)a * PW + b] = v.y;
    }
}

// The products between the two 128 blocks of a panel's diagonal block, in FP32, a launch a stage (two problems
// each, blockIdx.z = 2 f + problem, but for stage 1).  The chain of a panel waits for them, so each is spread over
// 16 CTAs of 32 x 32 output tiles (13-14 us a launch).  X = L^-1 and Y = U^-1 of the blocks from DINV.
//   stage 0: T0 = L21 = M21 Y11, T1 = U12 = X11 M12    stage 1: M22 -= T0 T1; T0, T1 into W
//   stage 2: T0 = X22 L21, T1 = U12 Y22                stage 3: X21 = -T0 X11, Y12 = -Y11 T1 (into PX, PY)
__global__ void __launch_bounds__(256) k_mid(int stage, float* __restrict__ W, int Np, size_t bstride, int k0,
                                             const float* __restrict__ DINV, size_t dstride, float2* __restrict__ TXY,
                                             float* __restrict__ PX, float* __restrict__ PY) {
    constexpr int KC = 32, LD = 33;
    __shared__ float2 As[32 * LD], Bs[KC * LD];
    const int prob = stage == 1 ? 0 : blockIdx.z & 1, f = stage == 1 ? blockIdx.z : blockIdx.z >> 1;
    float* Wr = W + (size_t)f * bstride + (size_t)k0 * Np + k0;
    float* Wi = Wr + (size_t)Np * Np;
    const float* D = DINV + (size_t)f * dstride + (size_t)(k0 / NBL) * 2 * NBL * NBL;  // the two blocks' inverses
    float2* T = TXY + ((size_t)f * 2 + prob) * NBL * NBL;
    const int i0 = blockIdx.y * 32, j0 = blockIdx.x * 32, tid = threadIdx.x;
    auto w = [&](int r, int c) { const size_t o = (size_t)r * Np + c; return make_float2(Wr[o], Wi[o]); };
    auto dv = [&](int b, int r, int c) {
        const int o = b * 2 * NBL * NBL + r * NBL + c;
        return make_float2(D[o], D[o + NBL * NBL]);
    };
    auto xi = [&](int b, int r, int c) { return r > c ? dv(b, r, c) : make_float2(r == c ? 1.f : 0.f, 0.f); };  // L^-1
    auto yi = [&](int b, int r, int c) { return r <= c ? dv(b, r, c) : make_float2(0.f, 0.f); };                // U^-1
    // entry (i, k) of the left and (k, j) of the right operand; the triangular operands' zero blocks are left out
    auto left = [&](int i, int k) {
        switch (2 * stage + prob) {
            case 0: return w(NBL + i, k);
            case 1: return xi(0, i, k);
            case 2: return T[i * NBL + k];
            case 4: return xi(1, i, k);
            case 5: return w(i, NBL + k);
            case 6: return T[i * NBL + k];
            default: return yi(0, i, k);
        }
    };
    auto right = [&](int k, int j) {
        switch (2 * stage + prob) {
            case 0: return yi(0, k, j);
            case 1: return w(k, NBL + j);
            case 2: return T[NBL * NBL + k * NBL + j];
            case 4: return w(NBL + k, j);
            case 5: return yi(1, k, j);
            case 6: return xi(0, k, j);
            default: return T[k * NBL + j];
        }
    };
    int klo = 0, khi = NBL;
    if ((stage == 0 && prob == 1) || (stage == 2 && prob == 0)) khi = i0 + 32;  // lower on the left
    if ((stage == 0 && prob == 0) || (stage == 2 && prob == 1)) khi = j0 + 32;  // upper on the right
    if (stage == 3) klo = prob == 0 ? j0 : i0;                                 // lower right, upper left
    const int tr = tid / 16, tc_ = tid % 16;  // outputs (tr, tr + 16) x (tc, tc + 16)
    float2 acc[2][2];
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int b = 0; b < 2; b++) acc[a][b] = make_float2(0.f, 0.f);
    float2 la[4], lb[4];
    auto load = [&](int kc) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int t = tid + 256 * q, r = t / 32, c = t % 32;
            la[q] = left(i0 + r, kc + c);
            lb[q] = right(kc + r, j0 + c);
        }
    };
    load(klo);
    for (int kc = klo; kc < khi; kc += KC) {
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int t = tid + 256 * q, r = t / 32, c = t % 32;
            As[r * LD + c] = la[q];
            Bs[r * LD + c] = lb[q];
        }
        __syncthreads();
        if (kc + KC < khi) load(kc + KC);  // in flight during the products
#pragma unroll 8
        for (int k = 0; k < KC; k++) {
            const float2 a0 = As[tr * LD + k], a1 = As[(tr + 16) * LD + k];
            const float2 b0 = Bs[k * LD + tc_], b1 = Bs[k * LD + tc_ + 16];
            cfma_add(acc[0][0], a0, b0);
            cfma_add(acc[0][1], a0, b1);
            cfma_add(acc[1][0], a1, b0);
            cfma_add(acc[1][1], a1, b1);
        }
    }
    float* Pf = (prob == 0 ? PX : PY) + (size_t)f * 2 * PW * PW + (size_t)NBL * PW;
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const int i = i0 + tr + 16 * a, j = j0 + tc_ + 16 * b;
            const float2 v = acc[a][b];
            if (stage == 1) {
                const size_t o = (size_t)(NBL + i) * Np + NBL + j, ol = (size_t)(NBL + i) * Np + j,
                             ou = (size_t)i * Np + NBL + j;
                Wr[o] -= v.x;
                Wi[o] -= v.y;
                const float2 l = T[i * NBL + j], u = T[NBL * NBL + i * NBL + j];
                Wr[ol] = l.x;
                Wi[ol] = l.y;
                Wr[ou] = u.x;
                Wi[ou] = u.y;
            } else if (stage == 0 || stage == 2) {
                T[i * NBL + j] = v;
            } else {  // PX row 128 + i, column j; PY row 128 + j (the column of Y), entry i
                const size_t o = prob == 0 ? (size_t)i * PW + j : (size_t)j * PW + i;
                Pf[o] = -v.x;
                Pf[(size_t)PW * PW + o] = -v.y;
            }
        }
}

// The panel's rows k0 .. k0 + PW, columns c0 .. c0 + n, transposed (32 x 32 tiles through shared memory): row j
// of P2 [F][2 planes][Np][PW] holds column c0 + j, the K-major B operand of the U product.
__global__ void k_prep_block_row(const float* __restrict__ W, int Np, size_t bstride, int k0, int c0,
                                 float* __restrict__ P2) {
    __shared__ float t[32][33];
    const int f = blockIdx.z >> 1, p = blockIdx.z & 1;
    const int j0 = blockIdx.x * 32, kk0 = blockIdx.y * 32;
    const float* Wp = W + (size_t)f * bstride + (size_t)p * Np * Np;
    const int tx = threadIdx.x, ty = threadIdx.y;
#pragma unroll
    for (int r = 0; r < 32; r += 8) t[ty + r][tx] = Wp[(size_t)(k0 + kk0 + ty + r) * Np + c0 + j0 + tx];
    __syncthreads();
    float* Pf = P2 + ((size_t)f * 2 + p) * Np * PW;
#pragma unroll
    for (int r = 0; r < 32; r += 8) Pf[(size_t)(j0 + ty + r) * PW + kk0 + tx] = t[tx][ty + r];
}

// Packed FP32 pairs (fma.rn.f32x2: two FP32 FMAs per instruction), here over two right-hand sides.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 f2pack(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 f2unpack(f32x2 r) {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(r));
    return v;
}
__device__ __forceinline__ f32x2 ffma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

constexpr int GV_ROWS = 256, GV_COLS = 16, GV_STAGES = 3, GV_CHUNK = 1024;
constexpr int GV_WORKERS = GV_ROWS / 2;

// Partial products of y = M x over column chunks: part[z][f][c][k] = sum_{n in chunk z} M(k, n) x[f][c][n], M
// column-major planar FP32 (entry (k, n) at n Np + k), x FP64 complex [F][nrhs][ldx], FP64 accumulation;
// k_gemv_reduce or k_residual_reduce then forms bias - sum_z part[z] in a fixed order (deterministic).  On the
// FP64 tensor cores (mma.sync m8n8k4): the matrix and vector tiles streamed by TMA (16 columns a stage, both FP32 planes of 256 rows, 32 KB, and the 16 complex entries of every right-hand side) from a
// producer warp, eight warps of 32 rows each.  Real columns 2 c and 2 c + 1 of the product are the real and imaginary
// part of right-hand side c: C += Mr [Xr, Xi] + Mi [-Xi, Xr].  Lane (i, k) of a warp reads rows 4 i .. 4 i + 3 of column
// k by one 16-byte load, row tile t taking rows 4 i + t, and each pair of vector entries serves four row tiles; all
// right-hand sides in one pass over the matrix.  Bound by the FP64 pipe (4 FMA an entry and right-hand side at 37
// TFLOP/s, NT tiles of 4 right-hand sides); the FMA form before it (a thread two rows, at most 16 right-hand sides a
// pass) spent as long on its shared-memory loads.  Measured, ms, before / now: 40 matrices of order 4096 and 10
// right-hand sides 2.39 / 2.03, 4 of order 12288 and 19 5.4 / 3.0, 5 of order 18496 and 14 12.1 / 6.7.  The steps of a
// stage unrolled four times up to five tiles, not at all beyond (ms, 16 matrices of order 4096, unrolled / not: 8
// right-hand sides 0.60 / 0.62, 12 0.87 / 0.91, 20 1.367 / 1.373, 24 1.66 / 1.63, 32 2.23 / 2.18).
constexpr int GD_THREADS = GV_ROWS + 32;  // eight MMA warps of 32 rows, the producer
template <int NT>
struct GdCfg {  // NT: tiles of four right-hand sides
    static constexpr size_t TX = (size_t)2 * GV_COLS * GV_ROWS * 4 + (size_t)4 * NT * GV_COLS * 16;  // bytes of a stage
    static constexpr size_t STAGE = (TX + 1023) / 1024 * 1024;
    static constexpr int STAGES = NT <= 2 ? 3 : 4;  // two CTAs an SM, or one
    static constexpr size_t SMEM = 1024 + STAGES * STAGE + 128;
};
template <int NT>
__global__ void __launch_bounds__(GD_THREADS, NT <= 2 ? 2 : 1) k_cgemv_dmma(const __grid_constant__ CUtensorMap mapM,
                                                              const __grid_constant__ CUtensorMap mapX, int N,
                                                              int nrhs, double2* __restrict__ part, int F,
                                                              int* __restrict__ err) {
    using C = GdCfg<NT>;
    extern __shared__ uint8_t gv_raw[];
    uint8_t* base = align1024(gv_raw);
    uint64_t* full = reinterpret_cast<uint64_t*>(base + C::STAGES * C::STAGE);
    uint64_t* empty = full + C::STAGES;
    const int f = blockIdx.y, z = blockIdx.z;
    const int k0 = blockIdx.x * GV_ROWS;
    const int nbeg = z * GV_CHUNK, nend = min(N, nbeg + GV_CHUNK);
    const int nst = (nend - nbeg + GV_COLS - 1) / GV_COLS;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; s++) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], GV_ROWS / 32);
        }
        tc::fence_barrier_init();
    }
    __syncthreads();
    if (warp == GV_ROWS / 32) {
        if (lane == 0) {
            tc::prefetch_tensormap(&mapM);
            tc::prefetch_tensormap(&mapX);
            int si = 0;
            for (; si < nst; si++) {
                const int s = si % C::STAGES;
                if (si >= C::STAGES && !tc::mbar_wait(&empty[s], ((si / C::STAGES) - 1) & 1)) {
                    atomicExch(err, 6);
                    break;
                }
                uint8_t* st = base + s * C::STAGE;
                const int n0 = nbeg + si * GV_COLS;
                tc::mbar_arrive_expect_tx(&full[s], (uint32_t)C::TX);
                tc::tma_load_4d(st, &mapM, &full[s], k0, n0, 0, f);
                tc::tma_load_4d(st + GV_COLS * GV_ROWS * 4, &mapM, &full[s], k0, n0, 1, f);
                tc::tma_load_4d(st + 2 * GV_COLS * GV_ROWS * 4, &mapX, &full[s], 2 * n0, 0, f, 0);
            }
            // every load still in flight lands before the CTA leaves, also after an error (bounded)
            for (int q = max(0, si - C::STAGES); q < si; q++)
                if (!tc::mbar_wait(&full[q % C::STAGES], (q / C::STAGES) & 1)) {
                    atomicExch(err, 6);
                    break;
                }
        }
        return;
    }
    const int i = lane >> 2, kq = lane & 3;  // row group (and column of B), k of a step
    double acc[4][NT][2];
#pragma unroll
    for (int t = 0; t < 4; t++)
#pragma unroll
        for (int c = 0; c < NT; c++) acc[t][c][0] = acc[t][c][1] = 0.0;
    for (int si = 0; si < nst; si++) {
        const int s = si % C::STAGES;
        // (the vote: one answer for the warp, each lane leaves the wait by itself)
        if (!__all_sync(0xffffffffu, tc::mbar_wait(&full[s], (si / C::STAGES) & 1))) {
            atomicExch(err, 7);
            break;
        }
        // The stage before is handed back: every lane orders its reads of it before the TMA writes that refill it
        // (another proxy), the warp barrier orders those fences before lane 0's arrival, and the second one brings the
        // lanes together for the mma.  It stands behind the wait for this stage because the fence alone is not what was
        // measured: an arrival at the end of the stage's own unrolled loop, with a warp barrier but no fence before
        // it, let entries be overwritten (a product done twice differed in 1.1e6 entries of 1210 calls; in none with a
        // pause before the arrival, or with the arrival here).
        tc::fence_proxy_async_smem();
        __syncwarp();
        if (si > 0 && lane == 0) tc::mbar_arrive(&empty[(si - 1) % C::STAGES]);
        __syncwarp();
        const uint8_t* st = base + s * C::STAGE;
        const float* sM = reinterpret_cast<const float*>(st) + 32 * warp + 4 * i;
        const double2* sx = reinterpret_cast<const double2*>(st + 2 * GV_COLS * GV_ROWS * 4);  // [4 NT][GV_COLS]
        // columns beyond N take no part (the padding may hold anything)
        const int lim = nend - (nbeg + si * GV_COLS);
#pragma unroll(NT <= 5 ? 4 : 1)
        for (int ks = 0; ks < GV_COLS / 4; ks++) {
            const int k = 4 * ks + kq;
            float4 mr = *reinterpret_cast<const float4*>(sM + k * GV_ROWS);
            float4 mi = *reinterpret_cast<const float4*>(sM + (GV_COLS + k) * GV_ROWS);
            if (k >= lim) mr = mi = make_float4(0.f, 0.f, 0.f, 0.f);
            const double ar[4] = {mr.x, mr.y, mr.z, mr.w}, ai[4] = {mi.x, mi.y, mi.z, mi.w};
#pragma unroll
            for (int c = 0; c < NT; c++) {
                const double2 v = sx[(4 * c + (i >> 1)) * GV_COLS + k];  // right-hand side 4 c + i / 2
                const double b1 = i & 1 ? v.y : v.x, b2 = i & 1 ? v.x : -v.y;
#pragma unroll
                for (int t = 0; t < 4; t++)
                    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                                 : "+d"(acc[t][c][0]), "+d"(acc[t][c][1])
                                 : "d"(ar[t]), "d"(b1));
#pragma unroll
                for (int t = 0; t < 4; t++)
                    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                                 : "+d"(acc[t][c][0]), "+d"(acc[t][c][1])
                                 : "d"(ai[t]), "d"(b2));
            }
        }
    }
    // lane (i, kq) holds right-hand sides 4 c + kq of rows 4 i + t
    const int row = k0 + 32 * warp + 4 * i;
#pragma unroll
    for (int c = 0; c < NT; c++)
        if (4 * c + kq < nrhs) {
            double2* o = part + (((size_t)z * F + f) * nrhs + 4 * c + kq) * N + row;
#pragma unroll
            for (int t = 0; t < 4; t++)
                if (row + t < N) o[t] = make_double2(acc[t][c][0], acc[t][c][1]);
        }
}

// The same product with a complex64 vector d (a refinement correction): part = M d over column chunks,
// each product and each 16-column sum in FP32, the sums added into FP64.  For a correction d that is
// small against the solution (|d| ~ 1e-3 |x| after the first), FP32 products put errors of ~1e-10 of
// |A x| into the residual r - M d, far below what the refinement converges to.
// The complex64 vectors of the refinement are kept by column pairs, [F][pairs][Np] of {re, re', im, im'}, so that a
// 16-byte load of shared memory feeds the packed FMAs of two columns as it is.
template <int NR>
__host__ __device__ constexpr size_t gv32_tx_bytes() {
    return (size_t)2 * GV_COLS * GV_ROWS * 4 + (size_t)(NR / 2) * GV_COLS * 16;
}
template <int NR>
__host__ __device__ constexpr size_t gv32_stage_bytes() {
    return (gv32_tx_bytes<NR>() + 1023) / 1024 * 1024;
}
template <int NR>
__host__ __device__ constexpr size_t gv32_smem_bytes() {
    return 1024 + GV_STAGES * gv32_stage_bytes<NR>() + 128;
}

// HV = 2: two groups of workers, each half of the columns of the same rows (the FP64 sums of 12 or 16 columns of two
// rows take 128 registers and more, which left one CTA of four warps an SM).  ms of three products, one group / two: 5
// matrices of order 18496 and 14 columns 10.1 / 6.7, 4 of order 12288 and 19 columns (chunks of 16 and 4) 3.3 / 2.9.
template <int NR>
__host__ __device__ constexpr int gv32_halves() {
    return NR >= 12 ? 2 : 1;
}
template <int NR>
__host__ __device__ constexpr int gv32_threads() {
    return gv32_halves<NR>() * GV_WORKERS + 32;
}
template <int NR>
__global__ void __launch_bounds__(gv32_threads<NR>()) k_cgemv32_tma(const __grid_constant__ CUtensorMap mapM,
                                                               const __grid_constant__ CUtensorMap mapD, int N,
                                                               int nrhs, int c0, double2* __restrict__ part, int F,
                                                               int* __restrict__ err) {
    constexpr int HV = gv32_halves<NR>(), NH = NR / HV, WARPS = HV * GV_WORKERS / 32;
    extern __shared__ uint8_t gv_raw[];
    uint8_t* base = align1024(gv_raw);
    uint64_t* full = reinterpret_cast<uint64_t*>(base + GV_STAGES * gv32_stage_bytes<NR>());
    uint64_t* empty = full + GV_STAGES;
    const int f = blockIdx.y, z = blockIdx.z;
    const int k0 = blockIdx.x * GV_ROWS;
    const int nbeg = z * GV_CHUNK, nend = min(N, nbeg + GV_CHUNK);
    const int nst = (nend - nbeg + GV_COLS - 1) / GV_COLS;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < GV_STAGES; s++) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], WARPS);
        }
        tc::fence_barrier_init();
    }
    __syncthreads();
    if (warp == WARPS) {
        if (lane == 0) {
            tc::prefetch_tensormap(&mapM);
            tc::prefetch_tensormap(&mapD);
            int si = 0;
            for (; si < nst; si++) {
                const int s = si % GV_STAGES;
                if (si >= GV_STAGES && !tc::mbar_wait(&empty[s], ((si / GV_STAGES) - 1) & 1)) {
                    atomicExch(err, 6);
                    break;
                }
                uint8_t* st = base + s * gv32_stage_bytes<NR>();
                const int n0 = nbeg + si * GV_COLS;
                tc::mbar_arrive_expect_tx(&full[s], (uint32_t)gv32_tx_bytes<NR>());
                tc::tma_load_4d(st, &mapM, &full[s], k0, n0, 0, f);
                tc::tma_load_4d(st + GV_COLS * GV_ROWS * 4, &mapM, &full[s], k0, n0, 1, f);
                tc::tma_load_4d(st + 2 * GV_COLS * GV_ROWS * 4, &mapD, &full[s], 4 * n0, c0 / 2, f, 0);
            }
            // every load still in flight lands before the CTA leaves, also after an error (bounded)
            for (int q = max(0, si - GV_STAGES); q < si; q++)
                if (!tc::mbar_wait(&full[q % GV_STAGES], (q / GV_STAGES) & 1)) {
                    atomicExch(err, 6);
                    break;
                }
        }
        return;
    }
    double2 acc[NH], acd[NH];  // rows k0 + t and k0 + t + GV_WORKERS
#pragma unroll
    for (int c = 0; c < NH; c++) acc[c] = acd[c] = make_double2(0.0, 0.0);
    const int t = threadIdx.x % GV_WORKERS, h0 = threadIdx.x / GV_WORKERS * NH;  // row, first column
    for (int si = 0; si < nst; si++) {
        const int s = si % GV_STAGES;
        if (!tc::mbar_wait(&full[s], (si / GV_STAGES) & 1)) {
            atomicExch(err, 7);
            break;
        }
        const uint8_t* st = base + s * gv32_stage_bytes<NR>();
        const float* sMr = reinterpret_cast<const float*>(st);
        const float* sMi = sMr + GV_COLS * GV_ROWS;
        const float4* sd = reinterpret_cast<const float4*>(st + 2 * GV_COLS * GV_ROWS * 4) + h0 / 2 * GV_COLS;  // [pair][GV_COLS]
        const int lim = min(GV_COLS, nend - (nbeg + si * GV_COLS));
        f32x2 r0[NH / 2], i0[NH / 2], r1[NH / 2], i1[NH / 2];
#pragma unroll
        for (int c = 0; c < NH / 2; c++) r0[c] = i0[c] = r1[c] = i1[c] = f2pack(0.f, 0.f);
#pragma unroll 4
        for (int j = 0; j < lim; j++) {
            const float mr = sMr[j * GV_ROWS + t], mi = sMi[j * GV_ROWS + t];
            const float nr = sMr[j * GV_ROWS + t + GV_WORKERS], ni = sMi[j * GV_ROWS + t + GV_WORKERS];
            const f32x2 a0 = f2pack(mr, mr), b0 = f2pack(mi, mi), e0 = f2pack(-mi, -mi);
            const f32x2 a1 = f2pack(nr, nr), b1 = f2pack(ni, ni), e1 = f2pack(-ni, -ni);
#pragma unroll
            for (int c = 0; c < NH / 2; c++) {
                const float4 v = sd[c * GV_COLS + j];
                const f32x2 vr = f2pack(v.x, v.y), vi = f2pack(v.z, v.w);
                r0[c] = ffma2(e0, vi, ffma2(a0, vr, r0[c]));
                i0[c] = ffma2(b0, vr, ffma2(a0, vi, i0[c]));
                r1[c] = ffma2(e1, vi, ffma2(a1, vr, r1[c]));
                i1[c] = ffma2(b1, vr, ffma2(a1, vi, i1[c]));
            }
        }
#pragma unroll
        for (int c = 0; c < NH; c++) {
            const float2 x0 = f2unpack(r0[c / 2]), y0 = f2unpack(i0[c / 2]), x1 = f2unpack(r1[c / 2]), y1 = f2unpack(i1[c / 2]);
            acc[c].x += (double)(c & 1 ? x0.y : x0.x);
            acc[c].y += (double)(c & 1 ? y0.y : y0.x);
            acd[c].x += (double)(c & 1 ? x1.y : x1.x);
            acd[c].y += (double)(c & 1 ? y1.y : y1.x);
        }
        tc::fence_proxy_async_smem();  // (the reads before the TMA writes that refill the stage)
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&empty[s]);
    }
    const int k = k0 + t, kd = k + GV_WORKERS;
#pragma unroll
    for (int c = 0; c < NH; c++)
        if (c0 + h0 + c < nrhs) {
            if (k < N) part[(((size_t)z * F + f) * nrhs + c0 + h0 + c) * N + k] = acc[c];
            if (kd < N) part[(((size_t)z * F + f) * nrhs + c0 + h0 + c) * N + kd] = acd[c];
        }
}

// out = bias - sum of the partial products (fixed order), FP64 [F][nrhs][ldo]
__global__ void k_gemv_reduce(int N, int nrhs, int F, int nz, const double2* __restrict__ part,
                              const double2* __restrict__ bias, int ldb, double2* __restrict__ out, int ldo) {
    const int f = blockIdx.y;
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (size_t)nrhs * N) return;
    const int c = (int)(t / N), k = (int)(t % N);
    double sr = 0.0, si = 0.0;
    for (int z = 0; z < nz; z++) {
        double2 v = part[(((size_t)z * F + f) * nrhs + c) * N + k];
        sr += v.x;
        si += v.y;
    }
    double2 b = bias ? bias[((size_t)f * nrhs + c) * ldb + k] : make_double2(0.0, 0.0);
    out[((size_t)f * nrhs + c) * ldo + k] = make_double2(b.x - sr, b.y - si);
}

// The residual bias - sum of the partial products as complex64 column pairs; the bias is FP64 [F][nrhs][Np]
// (the right-hand sides) or, PAIRS, the residual before the correction in the pairs' layout.
template <bool PAIRS>
__global__ void k_residual_reduce(int N, int Np, int nrhs, int F, int nz, const double2* __restrict__ part,
                                  const void* __restrict__ bias, float4* __restrict__ out) {
    const int f = blockIdx.y, np = (nrhs + 1) / 2;
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (size_t)np * N) return;
    const int q = (int)(t / N), k = (int)(t % N);
    const size_t o = ((size_t)f * np + q) * Np + k;
    double2 v[2];
    float4 b4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (PAIRS) b4 = static_cast<const float4*>(bias)[o];
#pragma unroll
    for (int e = 0; e < 2; e++) {
        const int c = 2 * q + e;
        v[e] = make_double2(0.0, 0.0);
        if (c >= nrhs) continue;
        double sr = 0.0, si = 0.0;
        for (int z = 0; z < nz; z++) {
            const double2 p = part[(((size_t)z * F + f) * nrhs + c) * N + k];
            sr += p.x;
            si += p.y;
        }
        const double2 b = PAIRS ? make_double2((double)(e ? b4.y : b4.x), (double)(e ? b4.w : b4.z))
                                : static_cast<const double2*>(bias)[((size_t)f * nrhs + c) * Np + k];
        v[e] = make_double2(b.x - sr, b.y - si);
    }
    out[o] = make_float4((float)v[0].x, (float)v[1].x, (float)v[0].y, (float)v[1].y);
}

// d = A^-1 r with the factors of M = A^T = L U (FP32 planar, row-major in W): U^T y = r, then
// L^T d = y, in FP32 (the correction only needs the accuracy of the TF32 factors; the residual that
// sets the attainable accuracy is formed in FP64), complex64 column pairs in place, in blocks of TB = 128 rows:
// one persistent launch a direction.  The columns are split into groups that are solved independently, v = (matrix,
// group) the systems; the work items are (k, v), block k in solve order of system v, handed out by a ticket counter in
// the order k nv + v.  An item streams the block row of the factor against the blocks 0 .. k-1 as their solutions
// are published (ctrl[1 + v] = blocks of system v done), subtracts the sum, solves its diagonal block by the
// stored inverse and publishes it.  An item waits only on items of smaller ticket, which running CTAs
// hold and work on in order, so the sweep cannot deadlock; every wait is bounded (error 8: from then on nothing
// waits, the results are discarded).  ctrl = [ticket, done[nv]], zero at launch.
//
// One CTA an SM.  Warp 8 takes the tickets and streams the factor by TMA (32 rows of the solved block x 128 rows, both
// planes, 32 KB a stage) without waiting for solutions, the item's diagonal inverse after its last block and then the
// next item's blocks; warp 9 waits for the solutions and copies them (cp.async) beside them; warps 0 .. 7 multiply:
// four rows a lane, a part of each stage's k and (KS = 4) half of the column pairs a warp, so that one 16-byte load
// of a pair's solution feeds 16 packed FMAs and the k-parts are summed through shared memory only at an item's end.
// A chain step is the last block's product, the diagonal's product (each 0.52 us a column pair on one SM's FP32 pipe)
// and about 6 us of waiting, copying and summing; the whole is bound by the chain with few matrices and by the FP32 pipe with
// many.  A sweep measured, ms before / now: 40 matrices of order 4096, 10 columns 1.31 / 0.72; 4 of order 12288, 19
// columns 4.4 / 1.42; 5 of order 18560, 14 columns 7.2 / 3.2.  What it replaces (two rows a thread, the factor loaded into registers after the wait, one CTA doing
// everything in turn) spent 25-45 us a chain step, its shared-memory loads twice the FMAs' time.
constexpr int TB = 128;
constexpr int TRI_THREADS = 320, TRI_SK = 32;  // k rows of a stage
constexpr size_t TRI_STAGE = (size_t)2 * TRI_SK * TB * 4;
template <int NQ>  // column pairs of a group
struct TriCfg {
    static constexpr int KS = NQ <= 5 ? 8 : 4, NH = KS == 8 ? NQ : NQ / 2;  // k-parts, pairs of a warp
    static constexpr int NST = NQ <= 4 ? 4 : 3;                             // factor stages
    static constexpr size_t VEC = (size_t)NQ * TB * 16;                     // one block's vectors
    static constexpr size_t SMEM = 1024 + NST * TRI_STAGE + (2 + 1 + KS) * VEC + 256;
    static_assert(SMEM <= 227 * 1024, "shared memory of a CTA");
    static_assert(NH * 8 / KS == NQ, "the warps cover the pairs");
};
constexpr int TRI_MAXQ = 8;  // pairs of a group, at most
constexpr uint32_t TRI_WAIT_LIMIT = 1u << 20;

__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_gpu(int* p, int v) {
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void cp_async_f4(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tc::smem_u32(smem)), "l"(gmem) : "memory");
}
// this thread's arrival on the barrier once its cp.async so far have landed
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}

// acc (4 rows x NH pairs, real and imaginary sums) += the warp's k-part of a stage times the vectors at v
// ([pair][128], from the stage's first k on); MASK: the diagonal inverse, of which entry (p, row) counts where
// p <= row (upper) or p > row
template <int KS, int NH, bool MASK>
__device__ __forceinline__ void tri_stage(const float* sF, const float4* v, int k0, int lane, int p0, bool upper,
                                          f32x2 (&ar)[4][NH], f32x2 (&ai)[4][NH]) {
#pragma unroll(NH <= 5 ? 4 : 2)
    for (int kk = 0; kk < TRI_SK / KS; kk++) {
        const int k = k0 + kk;
        float4 fr = *reinterpret_cast<const float4*>(sF + k * TB + 4 * lane);
        float4 fi = *reinterpret_cast<const float4*>(sF + (TRI_SK + k) * TB + 4 * lane);
        if (MASK) {
            const int p = p0 + k, r = 4 * lane;
            if (upper != (p <= r)) fr.x = fi.x = 0.f;
            if (upper != (p <= r + 1)) fr.y = fi.y = 0.f;
            if (upper != (p <= r + 2)) fr.z = fi.z = 0.f;
            if (upper != (p <= r + 3)) fr.w = fi.w = 0.f;
        }
        const float fre[4] = {fr.x, fr.y, fr.z, fr.w}, fim[4] = {fi.x, fi.y, fi.z, fi.w};
#pragma unroll
        for (int c = 0; c < NH; c++) {
            const float4 y = v[c * TB + k];
            const f32x2 yr = f2pack(y.x, y.y), yi = f2pack(y.z, y.w);
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const f32x2 a = f2pack(fre[r], fre[r]), b = f2pack(fim[r], fim[r]), bn = f2pack(-fim[r], -fim[r]);
                ar[r][c] = ffma2(bn, yi, ffma2(a, yr, ar[r][c]));
                ai[r][c] = ffma2(b, yr, ffma2(a, yi, ai[r][c]));
            }
        }
    }
}

template <int NQ>
__global__ void __launch_bounds__(TRI_THREADS, 1) k_tri_sweep(const __grid_constant__ CUtensorMap mapF,
                                                              const __grid_constant__ CUtensorMap mapD, int Np,
                                                              int npair, float4* __restrict__ Xall, int nb, int ngroup,
                                                              int upper_t,
                                                              int* __restrict__ ctrl, int* __restrict__ err) {
    using C = TriCfg<NQ>;
    constexpr int NH = C::NH, KS = C::KS, NYB = 2;
    extern __shared__ uint8_t tri_raw[];
    uint8_t* base = align1024(tri_raw);
    float4* ys = reinterpret_cast<float4*>(base + C::NST * TRI_STAGE);  // [NYB][NQ][TB]
    float4* rb = ys + NYB * NQ * TB;                              // [NQ][TB]: the item's right-hand side
    float4* pt = rb + NQ * TB;                                       // [KS][NQ][TB]: partial sums
    uint64_t* full = reinterpret_cast<uint64_t*>(pt + KS * NQ * TB);
    uint64_t* empty = full + C::NST;
    uint64_t* yfull = empty + C::NST;
    uint64_t* yempty = yfull + NYB;
    uint64_t* rfull = yempty + NYB;  // then rempty, the item ring's full[2] and empty[2]
    uint64_t* rempty = rfull + 1;
    uint64_t* ifull = rempty + 1;
    uint64_t* iempty = ifull + 2;
    int* s_item = reinterpret_cast<int*>(iempty + 2);  // [2]
    const int nblk = Np / TB, nv = nb * ngroup, items = nblk * nv;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < C::NST; i++) {
            tc::mbar_init(&full[i], 1);
            tc::mbar_init(&empty[i], 8);
        }
        for (int i = 0; i < NYB; i++) {
            tc::mbar_init(&yfull[i], 32);
            tc::mbar_init(&yempty[i], 8);
        }
        tc::mbar_init(rfull, 32);
        tc::mbar_init(rempty, 8);
        for (int i = 0; i < 2; i++) {
            tc::mbar_init(&ifull[i], 1);
            tc::mbar_init(&iempty[i], 9);
        }
        tc::fence_barrier_init();
    }
    // (a group's missing pairs hold zeros, or an earlier item's values: their results are not stored)
    for (int t = threadIdx.x; t < (NYB + 1) * NQ * TB; t += TRI_THREADS) ys[t] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    auto wait = [&](uint64_t* bar, uint32_t parity) {  // bounded; after an error the protocol runs on, its results discarded
        if (!tc::mbar_wait(bar, parity)) atomicExch(err, 8);
    };
    if (warp == 8) {
        if (lane == 0) {
            tc::prefetch_tensormap(&mapF);
            tc::prefetch_tensormap(&mapD);
            int st = 0;  // stages issued
            for (int n = 0;; n++) {
                if (n >= 2) wait(&iempty[n & 1], ((n >> 1) - 1) & 1);
                const int t = atomicAdd(ctrl, 1);
                s_item[n & 1] = t;
                tc::mbar_arrive(&ifull[n & 1]);
                if (t >= items) break;
                const int k = t / nv, f = t % nv / ngroup, blk = upper_t ? k : nblk - 1 - k;
                for (int q = 0; q < 4 * (k + 1); q++, st++) {
                    const int s = st % C::NST, kk = q >> 2, sub = q & 3;
                    if (st >= C::NST) wait(&empty[s], ((st / C::NST) - 1) & 1);
                    tc::mbar_arrive_expect_tx(&full[s], (uint32_t)TRI_STAGE);
                    uint8_t* d = base + s * TRI_STAGE;
                    for (int p = 0; p < 2; p++)
                        if (kk < k)
                            tc::tma_load_4d(d + p * (TRI_STAGE / 2), &mapF, &full[s], blk * TB,
                                            (upper_t ? kk : nblk - 1 - kk) * TB + sub * TRI_SK, p, f);
                        else
                            tc::tma_load_4d(d + p * (TRI_STAGE / 2), &mapD, &full[s], 0, sub * TRI_SK, p, f * nblk + blk);
                }
            }
        }
    } else if (warp == 9) {
        int yb = 0;  // solutions loaded
        for (int n = 0;; n++) {
            wait(&ifull[n & 1], (n >> 1) & 1);
            const int t = s_item[n & 1];
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&iempty[n & 1]);
            if (t >= items) break;
            const int k = t / nv, v = t % nv, f = v / ngroup, p0 = (v % ngroup) * NQ, nq = min(NQ, npair - p0);
            const int blk = upper_t ? k : nblk - 1 - k;
            const float4* X = Xall + ((size_t)f * npair + p0) * Np;
            const int* done = ctrl + 1 + v;
            if (n > 0) wait(rempty, (n - 1) & 1);
            for (int q = 0; q < nq; q++)
#pragma unroll
                for (int e = 0; e < TB / 32; e++)
                    cp_async_f4(rb + q * TB + 32 * e + lane, X + (size_t)q * Np + blk * TB + 32 * e + lane);
            cp_async_arrive(rfull);
            int have = 0;
            for (int kk = 0; kk < k; kk++, yb++) {
                const int b = yb % NYB;
                if (yb >= NYB) wait(&yempty[b], ((yb / NYB) - 1) & 1);
                if (have <= kk) {
                    if (lane == 0) {
                        uint32_t polls = 0;
                        while ((have = ld_acquire_gpu(done)) <= kk && *(volatile int*)err == 0)
                            if (++polls > TRI_WAIT_LIMIT) atomicExch(err, 8);
                    }
                    __syncwarp();
                    have = __shfl_sync(0xffffffffu, have, 0);
                }
                const float4* xs = X + (size_t)(upper_t ? kk : nblk - 1 - kk) * TB;
                float4* yd = ys + b * NQ * TB;
                for (int q = 0; q < nq; q++)
#pragma unroll
                    for (int e = 0; e < TB / 32; e++)
                        cp_async_f4(yd + q * TB + 32 * e + lane, xs + (size_t)q * Np + 32 * e + lane);
                cp_async_arrive(&yfull[b]);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        const int ks = warp % KS, k0 = ks * (TRI_SK / KS), q0 = warp / KS * NH;  // first k of a stage, first pair
        f32x2 ar[4][NH], ai[4][NH];
        auto clear = [&]() {
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int c = 0; c < NH; c++) ar[r][c] = ai[r][c] = f2pack(0.f, 0.f);
        };
        auto barrier = [&]() { asm volatile("bar.sync 1, 256;" ::: "memory"); };
        // the k-parts' sums, each thread its entries (pair q, row) passed to put
        auto reduce = [&](auto put) {
#pragma unroll
            for (int c = 0; c < NH; c++)
#pragma unroll
                for (int r = 0; r < 4; r++) {  // (row 4 lane + r at 32 r + lane: consecutive 16-byte accesses)
                    const float2 a = f2unpack(ar[r][c]), b = f2unpack(ai[r][c]);
                    pt[(ks * NQ + q0 + c) * TB + 32 * r + lane] = make_float4(a.x, a.y, b.x, b.y);
                }
            barrier();
#pragma unroll
            for (int e = threadIdx.x; e < NQ * TB; e += 256) {
                float4 a = pt[e];
#pragma unroll
                for (int h = 1; h < KS; h++) {
                    const float4 v = pt[h * NQ * TB + e];
                    a = make_float4(a.x + v.x, a.y + v.y, a.z + v.z, a.w + v.w);
                }
                const int slot = e % TB;
                put(e / TB, 4 * (slot % 32) + slot / 32, a);
            }
            barrier();  // the partial sums are consumed, the entries written
        };
        int st = 0, yb = 0;
        for (int n = 0;; n++) {
            wait(&ifull[n & 1], (n >> 1) & 1);
            const int t = s_item[n & 1];
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&iempty[n & 1]);
            if (t >= items) break;
            const int k = t / nv, v = t % nv, f = v / ngroup, p0 = (v % ngroup) * NQ, nq = min(NQ, npair - p0);
            const int blk = upper_t ? k : nblk - 1 - k;
            clear();
            for (int kk = 0; kk < k; kk++, yb++) {
                const int b = yb % NYB;
                wait(&yfull[b], (yb / NYB) & 1);
                const float4* y = ys + (b * NQ + q0) * TB;
#pragma unroll 1
                for (int sub = 0; sub < 4; sub++, st++) {
                    const int s = st % C::NST;
                    wait(&full[s], (st / C::NST) & 1);
                    tri_stage<KS, NH, false>(reinterpret_cast<const float*>(base + s * TRI_STAGE), y + sub * TRI_SK, k0, lane, 0,
                                         false, ar, ai);
                    tc::fence_proxy_async_smem();  // (the reads before the TMA writes that refill the stage)
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&empty[s]);
                }
                if (lane == 0) tc::mbar_arrive(&yempty[b]);
            }
            wait(rfull, n & 1);
            if (k > 0) {
                reduce([&](int q, int row, float4 a) {
                    float4& u = rb[q * TB + row];
                    u = make_float4(u.x - a.x, u.y - a.y, u.z - a.z, u.w - a.w);
                });
                clear();
            }
#pragma unroll 1
            for (int sub = 0; sub < 4; sub++, st++) {
                const int s = st % C::NST;
                wait(&full[s], (st / C::NST) & 1);
                tri_stage<KS, NH, true>(reinterpret_cast<const float*>(base + s * TRI_STAGE), rb + q0 * TB + sub * TRI_SK, k0, lane,
                                    sub * TRI_SK, upper_t != 0, ar, ai);
                tc::fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&empty[s]);
            }
            float4* X = Xall + ((size_t)f * npair + p0) * Np + (size_t)blk * TB;
            reduce([&](int q, int row, float4 a) {
                if (!upper_t) {  // the unit diagonal of L^-1
                    const float4 u = rb[q * TB + row];
                    a = make_float4(a.x + u.x, a.y + u.y, a.z + u.z, a.w + u.w);
                }
                if (q < nq) X[(size_t)q * Np + row] = a;
                __threadfence();
            });
            if (threadIdx.x == 0) st_release_gpu(ctrl + 1 + v, k + 1);
            if (lane == 0) tc::mbar_arrive(rempty);
        }
    }
}

// FP64 right-hand sides to complex64 column pairs (entering the first correction).
__global__ void k_to_pairs(int Np, int nrhs, const double2* __restrict__ b, float4* __restrict__ r) {
    const int f = blockIdx.z, q = blockIdx.y, np = (nrhs + 1) / 2, k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= Np) return;
    const double2 v0 = b[((size_t)f * nrhs + 2 * q) * Np + k];
    const double2 v1 = 2 * q + 1 < nrhs ? b[((size_t)f * nrhs + 2 * q + 1) * Np + k] : make_double2(0.0, 0.0);
    r[((size_t)f * np + q) * Np + k] = make_float4((float)v0.x, (float)v1.x, (float)v0.y, (float)v1.y);
}

// x += d; per matrix the largest |d| and |x| (for the refinement's stopping test) into norms [F][2], zero before
// (bits of non-negative doubles order as the values do).  A correction or solution that is not finite counts as an
// infinite |d|: fmax drops a NaN, and a system of NaNs would pass for converged.  A CTA per 256 rows of a column pair:
// one CTA a matrix took 94 us for 40 matrices of order 4096 and 10 columns.
__global__ void __launch_bounds__(256) k_ir_update(int Np, int nrhs, double2* __restrict__ x, const float4* __restrict__ d,
                                                   unsigned long long* __restrict__ norms) {
    __shared__ double sd[8], sx[8];
    const int f = blockIdx.z, q = blockIdx.y, np = (nrhs + 1) / 2, k = blockIdx.x * blockDim.x + threadIdx.x;
    double md = 0.0, mx = 0.0;
    if (k < Np) {
        const float4 v = d[((size_t)f * np + q) * Np + k];
#pragma unroll
        for (int e = 0; e < 2; e++)
            if (2 * q + e < nrhs) {
                const size_t o = ((size_t)f * nrhs + 2 * q + e) * Np + k;
                const double dx = (double)(e ? v.y : v.x), dy = (double)(e ? v.w : v.z);
                double2 a = x[o];
                a.x += dx;
                a.y += dy;
                x[o] = a;
                md = isfinite(a.x) && isfinite(a.y) ? fmax(md, fmax(fabs(dx), fabs(dy))) : INFINITY;
                mx = fmax(mx, fmax(fabs(a.x), fabs(a.y)));
            }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        md = fmax(md, __shfl_xor_sync(0xffffffffu, md, o));
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0) sd[threadIdx.x >> 5] = md, sx[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int w = 1; w < 8; w++) {
            md = fmax(md, sd[w]);
            mx = fmax(mx, sx[w]);
        }
        atomicMax(norms + 2 * f, (unsigned long long)__double_as_longlong(md));
        atomicMax(norms + 2 * f + 1, (unsigned long long)__double_as_longlong(mx));
    }
}

// The padding rows and columns N..Np of the planar matrices A and W: identity (zero elsewhere).
__global__ void k_pad_identity(float* __restrict__ A, float* __restrict__ W, int N, int Np, size_t bstride) {
    const int f = blockIdx.y;
    float* Mr[2] = {A + (size_t)f * bstride, W + (size_t)f * bstride};
    const size_t npad = (size_t)(Np - N);
    const size_t total = 2 * npad * Np;  // the last npad columns and the last npad rows
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        size_t r, c;
        if (t < npad * Np) {
            c = N + t / Np;
            r = t % Np;
        } else {
            size_t u = t - npad * Np;
            r = N + u / Np;
            c = u % Np;
        }
        size_t o = c * Np + r;
#pragma unroll
        for (int m = 0; m < 2; m++) {
            Mr[m][o] = (r == c) ? 1.f : 0.f;
            Mr[m][o + (size_t)Np * Np] = 0.f;
        }
    }
}

}  // namespace hbg
