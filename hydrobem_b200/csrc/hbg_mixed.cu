// hbg_mixed.cu -- the mixed-precision form of the frequency solve: the pair kernels in FP64 as in
// the FP64 form, the matrices stored as complex64 (two FP32 planes), the LU on the tensor cores
// (tcgen05 kind::tf32 and kind::f16, FP32 accumulation, no pivoting), the right-hand sides and the residuals
// accumulated in FP64, and iterative refinement until the predicted error is below 1e-9 of the solution (IR_TOL).
// The result is the solution of the complex64-rounded system (the reference's production path
// stores its matrices in complex64 too, lo_frequency.rs:1-6).
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "hbg_mixed.h"
#include "hbg_mixed_kernels.cuh"

namespace hbg {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static const EncodeTiledFn fn = [] {  // resolved once, thread-safe (the pipelines of a batch share it)
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return reinterpret_cast<EncodeTiledFn>(p);
        return (EncodeTiledFn) nullptr;
    }();
    return fn;
}

// A 4-D FP32 tensor map (x innermost) with a {32, box_rows, 1, 1} box in the 128-byte swizzle.
static bool make_map(CUtensorMap* m, void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t d3, uint64_t s1,
                     uint64_t s2, uint64_t s3, uint32_t box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[4] = {d0, d1, d2, d3};
    cuuint64_t strides[3] = {s1, s2, s3};
    cuuint32_t box[4] = {32, box_rows, 1, 1};
    cuuint32_t es[4] = {1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
           CUDA_SUCCESS;
}

// The same for FP16 rows: box {64, box_rows} (128 bytes a row, 128-byte swizzle).
static bool make_map16(CUtensorMap* m, void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t d3, uint64_t s1,
                       uint64_t s2, uint64_t s3, uint32_t box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[4] = {d0, d1, d2, d3};
    cuuint64_t strides[3] = {s1, s2, s3};
    cuuint32_t box[4] = {64, box_rows, 1, 1};
    cuuint32_t es[4] = {1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
           CUDA_SUCCESS;
}

// A 4-D tensor map with an arbitrary box, no swizzle (plain row-major tiles in shared memory).
static bool make_map_box(CUtensorMap* m, CUtensorMapDataType dt, void* base, const uint64_t dims[4],
                         const uint64_t strides[3], const uint32_t box[4]) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t d[4] = {dims[0], dims[1], dims[2], dims[3]};
    cuuint64_t st[3] = {strides[0], strides[1], strides[2]};
    cuuint32_t bx[4] = {box[0], box[1], box[2], box[3]};
    cuuint32_t es[4] = {1, 1, 1, 1};
    return fn(m, dt, 4, base, d, st, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct MixedBuffers {
    void* p[24] = {};
    int n = 0;
    ~MixedBuffers() {
        for (int i = 0; i < n; i++)
            if (p[i]) cudaFree(p[i]);
    }
    template <class T>
    T* get(size_t count) {
        void* q = nullptr;
        if (cudaMalloc(&q, count * sizeof(T)) != cudaSuccess) return nullptr;
        p[n++] = q;
        return reinterpret_cast<T*>(q);
    }
};

// Refinement stops when the error left after the last correction d_k is predicted below IR_TOL of
// the largest solution entry: rho |d_k|, rho = |d_k| / |d_{k-1}| being the observed contraction (about
// 1e-3 with the TF32 factors).  The corrections still to come add up to rho / (1 - rho) |d_k| while they
// contract by rho: at a contraction of 0.5, the limit for a system to stay with these factors, twice that.
// The solution is then that of the complex64 system to ~1e-9 (2e-9), far inside its ~1e-7 distance from the
// FP64 system's solution (the rounding of the stored matrix).
constexpr double IR_TOL = 1e-9;
constexpr int IR_MAX_IT = 30;

// Corrections run back to back before the host first looks at their norms: the count the previous
// batch of the same problem needed, IR_GUESS_START at a problem's first batch, at least 2.  Every problem
// starts from the same count, so its corrections -- and the frequencies it hands to the FP64 form --
// do not depend on what the host thread solved before (the pipelines of a batch take the problems in
// an order that varies from call to call).
constexpr int IR_GUESS_START = 3;  // the benchmark workload's count
inline int& ir_guess() {
    static thread_local int g = IR_GUESS_START;
    return g;
}

// The partial products of the FP64 product M x by TMA and DMMA, its maps covering exactly the nb matrices (planar FP32,
// leading dimension Np) and vectors ([nb][nrhs][ldx]), nz column chunks; false if a map cannot be encoded.
template <int NT>
static void launch_cgemv_dmma_tiles(const CUtensorMap& mM, const CUtensorMap& mX, dim3 g, int N, int nrhs, double2* part,
                                    int nb, int* err, cudaStream_t s) {
    cudaFuncSetAttribute(k_cgemv_dmma<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GdCfg<NT>::SMEM);
    k_cgemv_dmma<NT><<<g, GD_THREADS, GdCfg<NT>::SMEM, s>>>(mM, mX, N, nrhs, part, nb, err);
}
static bool launch_cgemv_dmma(const float* M, int N, int Np, const double2* x, int ldx, int nrhs, int nb, int nz,
                              double2* part, int* err, cudaStream_t s) {
    CUtensorMap mM, mX;
    const uint64_t plane = (uint64_t)Np * Np;
    const uint64_t dm[4] = {(uint64_t)Np, (uint64_t)Np, 2, (uint64_t)nb};
    const uint64_t sm[3] = {(uint64_t)Np * 4, plane * 4, 2 * plane * 4};
    const uint32_t bm[4] = {GV_ROWS, GV_COLS, 1, 1};
    const int nt = std::max(2, (nrhs + 3) / 4);  // (one tile: padded to two, zeros beyond nrhs)
    const uint64_t dx[4] = {2 * (uint64_t)ldx, (uint64_t)nrhs, (uint64_t)nb, 1};
    const uint64_t sx[3] = {(uint64_t)ldx * 16, (uint64_t)nrhs * ldx * 16, (uint64_t)nb * nrhs * ldx * 16};
    const uint32_t bx[4] = {2 * GV_COLS, (uint32_t)(4 * nt), 1, 1};
    if (!make_map_box(&mM, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, (void*)M, dm, sm, bm) ||
        !make_map_box(&mX, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, (void*)x, dx, sx, bx))
        return false;
    const dim3 g((N + GV_ROWS - 1) / GV_ROWS, nb, nz);
    switch (nt) {
        case 2: launch_cgemv_dmma_tiles<2>(mM, mX, g, N, nrhs, part, nb, err, s); break;
        case 3: launch_cgemv_dmma_tiles<3>(mM, mX, g, N, nrhs, part, nb, err, s); break;
        case 4: launch_cgemv_dmma_tiles<4>(mM, mX, g, N, nrhs, part, nb, err, s); break;
        case 5: launch_cgemv_dmma_tiles<5>(mM, mX, g, N, nrhs, part, nb, err, s); break;
        case 6: launch_cgemv_dmma_tiles<6>(mM, mX, g, N, nrhs, part, nb, err, s); break;
        case 7: launch_cgemv_dmma_tiles<7>(mM, mX, g, N, nrhs, part, nb, err, s); break;
        default: launch_cgemv_dmma_tiles<8>(mM, mX, g, N, nrhs, part, nb, err, s); break;
    }
    return true;
}

// Side streams for the LU of LU_GROUPS groups of a batch and their fork/join events, per device and
// host thread (kept across solves).
constexpr int LU_GROUPS = 4;  // at most (the streams kept)
static std::atomic<int> g_lu_groups_override{0};
void mixed_lu_groups(int groups) { g_lu_groups_override = std::max(0, std::min(groups, LU_GROUPS)); }
// the groups of a batch of ns systems of order Np: about eight systems a group, at most LU_GROUPS (a group's
// launches cover its systems, so a group of a few small systems leaves its products and factors too
// short to fill the device); fewer than eight large systems in up to two groups, from order 5120 in up to three, so that
// one group's chain of diagonal blocks (217 us a panel) runs beside the products of the others: with smaller orders the
// products are too short to hide much of it.  LU measured, ms with 1 / 2 / 3 / 4 groups: 40 systems of order 4096 17.1 /
// 16.2 / 15.8 / 15.5; six bodies of 16 systems of orders 1792-3840 on two pipelines 48.3 / 45.8 / 49.2 / 49.6; 10 of
// order 512 0.47 with any; of order 2176, 3 systems 2.27 / 2.27 / 2.34, 7 2.51 / 2.44 / 2.45 / 2.49; of order 4096, 3
// 4.71 / 4.59 / 4.70, 5 5.25 / 5.07 / 5.07 / 5.12, 7 5.87 / 5.62 / 5.54 / 5.53; of order 6144, 3 8.19 / 7.99 / 7.93, 5
// 9.80 / 9.41 / 9.21 / 9.17; of order 12288, 3 26.7 / 25.7 / 25.1, 4 31.7 / 29.7 / 29.9 / 29.6; 5 of order 18560 114 /
// 114 / 109 / 110.
static int lu_groups_for(int Np, int ns) {
    const int o = g_lu_groups_override.load();
    const int g = ns >= 8 || Np < 2048 ? std::min(LU_GROUPS, ns / 8) : Np < 5120 ? 2 : 3;
    return std::max(1, std::min(o > 0 ? o : g, ns));
}
// The panels of a super-step of the LU: its trailing matrix (8 bytes an entry, read and written by the
// reduction) passes through DRAM once for 256 q columns.  LU measured, ms with q = 1 / 2 / 4: 40 systems of order
// 4096 19.2 / 16.6 / 15.5, 4 of order 12288 46.0 / 37.2 / 33.8, 5 of order 18560 167 / 122 / 110, 160 of order
// 1024 4.50 / 4.45 / 4.43 (a short matrix has no more panels; its buffers stay half as large).
static int lu_super(int Np) { return Np >= 2048 ? LU_Q : 2; }
// The column pairs of a group of the triangular sweeps, for npair pairs, nblk blocks and nb matrices: the smallest of
// the larger of two times, the dependency chain of a system (a step: two products of one block, 0.52 us a pair each,
// and 6 us) and the blocks' products over the SMs (their factor tiles loaded anew for every group: 1.4 us at least).
static int tri_group_pairs(int npair, int nblk, int nb, int n_sm) {
    int best = TRI_MAXQ;
    double tbest = 1e300;
    for (int q : {8, 6, 5, 4, 3, 2, 1}) {
        const int groups = (npair + q - 1) / q;
        const double t = std::max(1.4, 0.52 * q + 0.4), chain = nblk * (2.0 * (0.52 * q + 0.4) + 6.0);
        const double work = nb * groups * (0.5 * nblk * (nblk - 1) * t + nblk * (t + 4.0)) / n_sm;
        const double all = std::max(chain, work) + 0.25 * std::min(chain, work);
        if (all < tbest) tbest = all, best = q;
    }
    return best;
}
struct SideStreams {
    cudaStream_t s[LU_GROUPS + 1] = {};  // the LU groups, then the right-hand sides
    cudaEvent_t fork = nullptr, join[LU_GROUPS + 1] = {};
    bool ok = false;
};
static SideStreams& side_streams() {
    static thread_local SideStreams t[16];
    int d = 0;
    cudaGetDevice(&d);
    if (d < 0 || d >= 16) d = 0;
    SideStreams& x = t[d];
    if (!x.ok) {
        bool ok = true;
        for (int i = 0; i <= LU_GROUPS; i++) {
            ok = ok && cudaStreamCreateWithFlags(&x.s[i], cudaStreamNonBlocking) == cudaSuccess;
            ok = ok && cudaEventCreateWithFlags(&x.join[i], cudaEventDisableTiming) == cudaSuccess;
        }
        x.ok = ok && cudaEventCreateWithFlags(&x.fork, cudaEventDisableTiming) == cudaSuccess;
    }
    return x;
}

#define MIXED_FAIL(code, text, fq) \
    do {                           \
        *msg = text;               \
        *freq = fq;                \
        return code;               \
    } while (0)

int mixed_solve_frequencies(const PanelsView& pv, const double* st, const HbgProblem& pr, const HbgOptions& opt,
                            bool fin, double depth, cudaStream_t s, double* prof, int64_t* launches, const char** msg,
                            int64_t* freq, const std::function<void()>& start, const double* motion,
                            const FieldArgs& field, std::vector<int64_t>* fallback) {
    KernelProfiler& P = profiler();
    ir_guess() = IR_GUESS_START;
    // N panels; with symmetry sectors G systems of Nm = N / G unknowns per frequency (one of N otherwise)
    const int N = pv.N, G = pv.G, Nm = N / G, F = (int)pr.n_omega, H = (int)pr.n_heading, D = 6 * pv.nbod,
              nrhs = D + H;
    const int Np = (Nm + NBL - 1) / NBL * NBL;
    const size_t NP2 = (size_t)Np * Np, MB = 2 * NP2;  // floats per matrix (two planes)
    if (nrhs > 32) MIXED_FAIL(HB_ERR_UNSUPPORTED, "more than 32 right-hand sides (6 per body and one per heading)", -1);
    if (!encode_fn()) MIXED_FAIL(HB_ERR_UNSUPPORTED, "the driver offers no tensor-map encoder (TMA)", -1);
    // ---- batch size from free memory
    // the LU's operands of a system: the transposed block row (FP32), the FP16 copies of a super-step's L and U,
    // the panel's inverses (FP32), the products between its diagonal blocks
    const int Q = lu_super(Np), SW = Q * PW;  // panels and columns of a super-step
    const size_t prep = 2 * (size_t)Np * PW, op16 = 2 * (size_t)Np * SW, inv = 2 * (size_t)PW * PW,
                 midsz = 2 * (size_t)NBL * NBL;
    const size_t nblk = (size_t)Np / NBL, dinv = nblk * 2 * NBL * NBL;
    const int npair = (nrhs + 1) / 2;  // complex64 vectors by column pairs
    const int nz = (Nm + GV_CHUNK - 1) / GV_CHUNK;  // column chunks of the products
    const int nfp = field.P;
    // A, B [D][D], X, FK, SC, motions, Haskind [H][D], field values [P][D] and 3 x [P][H] per frequency
    // the Kochin functions kr, krt [TK][D], kd, kdt [TK][H] and the drift [H][H][3] after them
    const int TK = pr.kochin_angles > 0 && H > 0 ? pr.kochin_angles : 0;
    const size_t kochin_per = ((size_t)TK * 2 * (D + H) + (TK ? (size_t)3 * H * H : 0)) * 2;
    const size_t out_per = 2 * (size_t)D * D + 5 * (size_t)H * 2 * D + (size_t)nfp * 2 * (D + 3 * H) + kochin_per,
                 DD = (size_t)D * D;
    // the device buffers of a batch of nf frequencies
    auto needs = [&](int nf) {
        const size_t n = (size_t)nf * G, f = (size_t)nf;  // systems, frequencies
        Workspace::Needs v = {
            {WS_S32, MB * n * 4}, {WS_A32, MB * n * 4}, {WS_W, MB * n * 4}, {WS_P2, prep * n * 4},
            {WS_L16, op16 * n * 2}, {WS_U16, op16 * n * 2}, {WS_PX, inv * n * 4}, {WS_PY, inv * n * 4},
            {WS_TXY, midsz * n * sizeof(float2)}, {WS_DINV, dinv * n * 4},
            {WS_U, (size_t)nrhs * N * f * 16}, {WS_PHII, (size_t)std::max(H, 1) * N * f * 16},
            {WS_B, (size_t)nrhs * Np * n * 16}, {WS_XM, (size_t)nrhs * Np * n * 16},
            {WS_R, (size_t)npair * Np * n * 16}, {WS_RS, (size_t)npair * Np * n * 16},
            {WS_PART, (size_t)nz * n * nrhs * Nm * 16},
            {WS_NORMS, IR_MAX_IT * 2 * n * 8}, {WS_TRI_CTRL, sizeof(int) * (1 + n * npair)},
            {WS_FI, sizeof(FreqInfo) * f}, {WS_FD, sizeof(FdParams) * f}, {WS_OUT, sizeof(double) * out_per * f}};
        if (G > 1) {
            v.push_back({WS_UP, (size_t)nrhs * Nm * n * 16});
            v.push_back({WS_PHI, (size_t)nrhs * N * f * 16});
        }
        if (fin) {
            v.push_back({WS_TILES, sizeof(double) * (T1_SIZE + T2_SIZE) * f});
            v.push_back({WS_TILES_F, sizeof(float) * (T1F_SIZE + T2F_SIZE) * f});
            v.push_back({WS_SCR, sizeof(double) * 6912 * 3 * f});
            v.push_back({WS_FPT, sizeof(double) * FP_PLANES * N * f});
            if (nfp) v.push_back({WS_FQ, sizeof(double) * FP_PLANES * (size_t)(N + nfp) * f});
        }
        return v;
    };
    size_t per = 0;  // bytes a frequency
    for (const auto& q : needs(1)) per += q.second;
    // The batch size: all frequencies while the buffers held hold every one of them (the same problem again, or a smaller
    // one of a batch), else from free memory.  cudaMemGetInfo can take milliseconds, so that decision is kept per thread
    // and device for the same problem shape while the workspace still holds its buffers.
    Workspace& ws = workspace();
    int B = 0;
    {
        struct BatchChoice {
            int N = -1, G = -1, nrhs = -1, fin = -1, F = -1, B = 0;
            int64_t max_batch = -2;
            size_t budget = 0;
        };
        static thread_local BatchChoice last[16];
        int dev_b = 0;
        cudaGetDevice(&dev_b);
        BatchChoice& c = last[dev_b < 0 || dev_b >= 16 ? 0 : dev_b];
        const int most = opt.max_batch > 0 ? std::min(F, (int)opt.max_batch) : F;
        if (ws.holds(needs(most))) {
            B = most;
        } else {
            const size_t budget = hbm_budget()();
            const bool same = c.N == N && c.G == G && c.nrhs == nrhs && c.fin == (int)fin && c.F == F &&
                              c.max_batch == opt.max_batch && c.budget == budget;
            if (same && c.B > 0 && ws.holds(needs(c.B))) {
                B = c.B;
            } else {
                size_t freeb = 0, totalb = 0;
                if (cudaMemGetInfo(&freeb, &totalb) != cudaSuccess)
                    MIXED_FAIL(HB_ERR_INTERNAL, "cudaMemGetInfo failed", -1);
                freeb += ws.bytes[WS_S32] + ws.bytes[WS_A32] + ws.bytes[WS_W] + ws.bytes[WS_DINV];
                size_t avail = (size_t)(0.85 * (double)freeb);
                if (budget > 0) avail = std::min(avail, budget);
                B = (int)std::min<size_t>(most, std::max<size_t>(1, avail / per));
            }
            // buffers that cannot be had beside what else is held: all given back, half the frequencies
            while (!ws.take(needs(B))) {
                ws.drop(needs(B));
                if (B == 1) MIXED_FAIL(HB_ERR_INTERNAL, "device memory allocation failed for the mixed form", -1);
                B = (B + 1) / 2;
            }
            c = BatchChoice{N, G, nrhs, (int)fin, F, B, opt.max_batch, budget};
        }
    }
    const int BS = B * G;  // systems per batch
    bool okb = true;
    auto get = [&](int slot, size_t bytes) -> void* {
        void* q = ws.get(slot, bytes);
        okb = okb && q != nullptr;
        return q;
    };
    // (of the batch: taken above)
    float *S32 = (float*)ws.p[WS_S32], *A32 = (float*)ws.p[WS_A32], *W = (float*)ws.p[WS_W], *P2 = (float*)ws.p[WS_P2];
    __half* L16 = (__half*)ws.p[WS_L16];  // [BS][2 planes][Np rows][SW]
    __half* U16 = (__half*)ws.p[WS_U16];  // [BS][2 planes][SW rows][Np]
    float *PX = (float*)ws.p[WS_PX], *PY = (float*)ws.p[WS_PY], *DINV = (float*)ws.p[WS_DINV];
    float2* TXY = (float2*)ws.p[WS_TXY];
    double2 *u = (double2*)ws.p[WS_U], *phiI = (double2*)ws.p[WS_PHII];
    // symmetry sectors: the right-hand sides projected on the sectors, the potentials of every panel
    double2 *up = (double2*)ws.p[WS_UP], *phi = (double2*)ws.p[WS_PHI];
    double2 *b = (double2*)ws.p[WS_B], *x = (double2*)ws.p[WS_XM], *part = (double2*)ws.p[WS_PART];
    float4* r = (float4*)ws.p[WS_R];
    float4* rs = (float4*)ws.p[WS_RS];        // a residual kept for r - A d
    double* norms = (double*)ws.p[WS_NORMS];  // [iteration][batch][2]
    int* tctrl = (int*)ws.p[WS_TRI_CTRL];     // the triangular sweeps' tickets
    FreqInfo* dfi = (FreqInfo*)ws.p[WS_FI];
    FdParams* dfd = (FdParams*)ws.p[WS_FD];
    double *tiles = (double*)ws.p[WS_TILES], *scr = (double*)ws.p[WS_SCR], *fpt = (double*)ws.p[WS_FPT];
    float* tiles_f = (float*)ws.p[WS_TILES_F];
    double *dout = (double*)ws.p[WS_OUT], *fq = (double*)ws.p[WS_FQ];
    int* err = (int*)get(WS_ERR, sizeof(int));
    double* dheads = (double*)get(WS_HEADS, sizeof(double) * std::max(H, 1));
    // the wave-term network (optional): its parameters, the packed BF16 image the assembly loads, and
    // the count of pairs it served
    const bool sg = opt.surrogate != nullptr;
    float* sg_params = sg ? (float*)get(WS_SG_PARAMS, sizeof(float) * SURROGATE_FLOATS) : nullptr;
    uint8_t* sg_img = sg ? (uint8_t*)get(WS_SG_IMG, sg_image_bytes()) : nullptr;
    unsigned long long* sg_count = sg ? (unsigned long long*)get(WS_SG_COUNT, sizeof(unsigned long long)) : nullptr;
    if (!okb) MIXED_FAIL(HB_ERR_INTERNAL, "device memory allocation failed for the mixed form", -1);
    last_surrogate_pairs() = 0;
    // ---- tensor maps (whole batch; the batch index is the 4th coordinate)
    CUtensorMap mapW, mapPX, mapPY, mapP2, mapL16, mapU16;
    const uint64_t fb = 4;  // bytes per float
    bool okm = make_map(&mapW, W, Np, Np, 2, BS, Np * fb, NP2 * fb, MB * fb, GBM) &&
               make_map(&mapPX, PX, PW, PW, 2, BS, PW * fb, (uint64_t)PW * PW * fb, inv * fb, GBM) &&
               make_map(&mapPY, PY, PW, PW, 2, BS, PW * fb, (uint64_t)PW * PW * fb, inv * fb, GBN) &&
               make_map(&mapP2, P2, PW, Np, 2, BS, PW * fb, (uint64_t)Np * PW * fb, prep * fb, GBN) &&
               make_map16(&mapL16, L16, SW, Np, 2, BS, SW * 2, (uint64_t)Np * SW * 2, op16 * 2, GBM) &&
               make_map16(&mapU16, U16, Np, SW, 2, BS, Np * 2, (uint64_t)Np * SW * 2, op16 * 2, 2 * GBK);
    CUtensorMap mapF, mapD;  // the sweeps' factor and diagonal-inverse tiles
    {
        const uint64_t df[4] = {(uint64_t)Np, (uint64_t)Np, 2, (uint64_t)BS}, sf[3] = {Np * fb, NP2 * fb, MB * fb};
        const uint64_t dd[4] = {TB, TB, 2, nblk * BS}, sd[3] = {TB * fb, TB * TB * fb, 2 * TB * TB * fb};
        const uint32_t bx[4] = {TB, TRI_SK, 1, 1};
        okm = okm && make_map_box(&mapF, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, W, df, sf, bx) &&
              make_map_box(&mapD, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, DINV, dd, sd, bx);
    }
    if (!okm) MIXED_FAIL(HB_ERR_INTERNAL, "tensor-map encoding failed", -1);
    const int smem = (int)gemm_smem_bytes();
    cudaFuncSetAttribute(k_cgemm<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    cudaFuncSetAttribute(k_cgemm<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    int dev = 0, n_sm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
    const int dsmem = (int)df_smem_bytes();
    cudaFuncSetAttribute(k_diag_factor, cudaFuncAttributeMaxDynamicSharedMemorySize, dsmem);
    std::vector<double> heads(std::max(H, 1));
    for (int h = 0; h < H; h++) heads[h] = pr.headings_deg[h] * PI / 180.0;
    std::vector<FreqInfo> fi(B);
    std::vector<FdParams> fdh(B);
    // page-locked: the reads of norms, outputs and the error flag queue behind the work, no host wait
    double* hout = (double*)ws.host(HS_OUT, sizeof(double) * (out_per * B + 1));
    double* hn = (double*)ws.host(HS_NORMS, sizeof(double) * IR_MAX_IT * 2 * (size_t)BS);
    if (!hout || !hn) MIXED_FAIL(HB_ERR_INTERNAL, "page-locked host memory could not be allocated", -1);
    int* herr = reinterpret_cast<int*>(hout + out_per * B);
    // the column width of a chunk of w right-hand sides of the FP32 product (its padded columns cost as much as real ones)
    auto chunk_width = [](int w) { return w <= 4 ? 4 : w <= 8 ? 8 : w <= 10 ? 10 : w <= 12 ? 12 : 16; };
    for (auto fn : {(const void*)k_cgemv32_tma<4>, (const void*)k_cgemv32_tma<8>, (const void*)k_cgemv32_tma<10>,
                    (const void*)k_cgemv32_tma<12>, (const void*)k_cgemv32_tma<16>})
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gv32_smem_bytes<16>());
    // r = rk - M d with the complex64 correction d (FP32 products, FP64 sums; beyond 16 columns in chunks):
    // the residual after a correction that is small against the solution
    auto gemv32 = [&](const float* Mm, const float4* dv, const float4* rk, float4* out, int nb) {
        CUtensorMap mM, mD;
        const uint64_t dm[4] = {(uint64_t)Np, (uint64_t)Np, 2, (uint64_t)nb};
        const uint64_t sm[3] = {(uint64_t)Np * 4, NP2 * 4, MB * 4};
        const uint32_t bm[4] = {GV_ROWS, GV_COLS, 1, 1};
        const uint64_t dd[4] = {4 * (uint64_t)Np, (uint64_t)npair, (uint64_t)nb, 1};
        const uint64_t sd[3] = {(uint64_t)Np * 16, (uint64_t)npair * Np * 16, (uint64_t)nb * npair * Np * 16};
        if (!make_map_box(&mM, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, (void*)Mm, dm, sm, bm)) return false;
        CUtensorMap mDc[2];  // the map of each chunk width (a full chunk, the last one)
        const int nrc[2] = {chunk_width(std::min(16, nrhs)), chunk_width(nrhs - (nrhs - 1) / 16 * 16)};
        for (int q = 0; q < 2; q++) {
            const uint32_t bd[4] = {4 * GV_COLS, (uint32_t)nrc[q] / 2, 1, 1};
            if (!make_map_box(&mDc[q], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, (void*)dv, dd, sd, bd)) return false;
        }
        P.begin(s);
        dim3 g((Nm + GV_ROWS - 1) / GV_ROWS, nb, nz);
        for (int c0 = 0; c0 < nrhs; c0 += 16) {
            const bool last = c0 + 16 >= nrhs;
            const int nr = nrc[last];
            mD = mDc[last];
            if (nr == 4)
                k_cgemv32_tma<4><<<g, gv32_threads<4>(), gv32_smem_bytes<4>(), s>>>(mM, mD, Nm, nrhs, c0, part, nb, err);
            else if (nr == 8)
                k_cgemv32_tma<8><<<g, gv32_threads<8>(), gv32_smem_bytes<8>(), s>>>(mM, mD, Nm, nrhs, c0, part, nb, err);
            else if (nr == 10)
                k_cgemv32_tma<10><<<g, gv32_threads<10>(), gv32_smem_bytes<10>(), s>>>(mM, mD, Nm, nrhs, c0, part, nb, err);
            else if (nr == 12)
                k_cgemv32_tma<12><<<g, gv32_threads<12>(), gv32_smem_bytes<12>(), s>>>(mM, mD, Nm, nrhs, c0, part, nb, err);
            else
                k_cgemv32_tma<16><<<g, gv32_threads<16>(), gv32_smem_bytes<16>(), s>>>(mM, mD, Nm, nrhs, c0, part, nb, err);
        }
        k_residual_reduce<true><<<dim3((unsigned)(((size_t)npair * Nm + 255) / 256), nb), 256, 0, s>>>(
            Nm, Np, nrhs, nb, nz, part, rk, out);
        P.end(KF_MIXED_RESIDUAL, 8.0 * (double)Nm * Nm * nb, s);
        *launches += 2;
        return true;
    };
    // out = bias - M x over the batch (M column-major planar FP32), FP64 accumulation
    bool maps_ok = true;  // the FP64 product's maps were encoded: looked at once the batch has run
    auto gemv = [&](const float* Mm, const double2* xv, int ldx, const double2* bias, auto* out, int nb, int fam,
                    cudaStream_t s) {
        P.begin(s);
        maps_ok = launch_cgemv_dmma(Mm, Nm, Np, xv, ldx, nrhs, nb, nz, part, err, s) && maps_ok;
        if constexpr (std::is_same_v<decltype(out), float4*>)  // a residual, for the sweeps
            k_residual_reduce<false><<<dim3((unsigned)(((size_t)npair * Nm + 255) / 256), nb), 256, 0, s>>>(
                Nm, Np, nrhs, nb, nz, part, bias, out);
        else
            k_gemv_reduce<<<dim3((unsigned)(((size_t)nrhs * Nm + 255) / 256), nb), 256, 0, s>>>(Nm, nrhs, nb, nz, part,
                                                                                               bias, Np, out, Np);
        P.end(fam, 8.0 * (double)Nm * Nm * nb, s);
        *launches += 2;
    };
    // d = A^-1 d in place (complex64) with the FP32 factors in W: U^T y = d, then L^T d = y, the
    // diagonal blocks by the products with their inverses (stored by the LU)
    auto sweep = [&](auto nq, float4* xv, int nb, int groups, int up) {
        constexpr int NQ = decltype(nq)::value;
        cudaFuncSetAttribute(k_tri_sweep<NQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TriCfg<NQ>::SMEM);
        k_tri_sweep<NQ><<<std::min((int)nblk * nb * groups, n_sm), TRI_THREADS, TriCfg<NQ>::SMEM, s>>>(
            mapF, mapD, Np, npair, xv, nb, groups, up, tctrl, err);
    };
    auto trisolve = [&](float4* xv, int nb) {  // one persistent sweep per direction
        P.begin(s);
        const int nq = tri_group_pairs(npair, (int)nblk, nb, n_sm), groups = (npair + nq - 1) / nq;
        for (int up = 1; up >= 0; up--) {
            cudaMemsetAsync(tctrl, 0, sizeof(int) * (1 + (size_t)nb * groups), s);
            switch (nq) {
                case 1: sweep(std::integral_constant<int, 1>(), xv, nb, groups, up); break;
                case 2: sweep(std::integral_constant<int, 2>(), xv, nb, groups, up); break;
                case 3: sweep(std::integral_constant<int, 3>(), xv, nb, groups, up); break;
                case 4: sweep(std::integral_constant<int, 4>(), xv, nb, groups, up); break;
                case 5: sweep(std::integral_constant<int, 5>(), xv, nb, groups, up); break;
                case 6: sweep(std::integral_constant<int, 6>(), xv, nb, groups, up); break;
                default: sweep(std::integral_constant<int, 8>(), xv, nb, groups, up); break;
            }
            (*launches)++;
        }
        P.end(KF_LU_SOLVE, 8.0 * (double)NP2 * nb, s);  // the factors read once
    };
    // matrices f0 .. f0 + nb of the batch on stream st, at most cap persistent CTAs
    auto gemm = [&](const CUtensorMap& mA, const CUtensorMap& mB, CgemmArgs g, int f0, int nb, cudaStream_t st,
                    int cap, bool f16) {
        g.batch = nb;
        g.b0 = f0;
        const int units = g.mt * (g.tri == CG_RIGHT_UPPER ? 1 : g.nt) * nb;
        if (units <= 0) return;
        P.begin(st);
        if (f16)
            k_cgemm<true><<<std::min(units, cap), GEMM_THREADS, smem, st>>>(mA, mB, mapW, g);
        else
            k_cgemm<false><<<std::min(units, cap), GEMM_THREADS, smem, st>>>(mA, mB, mapW, g);
        const double k_all = g.tri == CG_FULL ? (double)g.K * g.mt * g.nt : 1.5 * NBL * g.mt * g.nt;
        P.end(KF_MIXED_GEMM, 8.0 * GBM * GBN * k_all * nb, st);
        (*launches)++;
    };
    SideStreams& side = side_streams();
    if (!side.ok) MIXED_FAIL(HB_ERR_INTERNAL, "CUDA streams for the LU could not be created", -1);
    // ---- the device work: statics, then per batch assembly, LU, refinement, forces
    start();
    cudaMemcpyAsync(dheads, heads.data(), sizeof(double) * heads.size(), cudaMemcpyHostToDevice, s);
    if (sg) {
        cudaMemcpyAsync(sg_params, opt.surrogate, sizeof(float) * SURROGATE_FLOATS, cudaMemcpyHostToDevice, s);
        launch_sg_pack(sg_params, sg_img, s);
        cudaMemsetAsync(sg_count, 0, sizeof(unsigned long long), s);
        (*launches)++;
    }
    for (int f0 = 0; f0 < F; f0 += B) {
        if (opt.cancel && *opt.cancel) MIXED_FAIL(HB_ERR_CANCELLED, "the solve was cancelled", f0);
        const int nb = std::min(B, F - f0), ns = nb * G;  // frequencies, systems
        for (int i = 0; i < nb; i++) {
            double w = pr.omegas[f0 + i], K = w * w / opt.gravity;
            fi[i].omega = w;
            fi[i].K = K;
            fi[i].k = fin ? dispersion_x0(K * depth) / depth : K;
            fi[i].logc = opt.logarithmic ? 1.0 : 0.0;
            if (fin) make_fd_params(depth, K, fdh[i]);
        }
        cudaMemcpyAsync(dfi, fi.data(), sizeof(FreqInfo) * nb, cudaMemcpyHostToDevice, s);
        if (fin) cudaMemcpyAsync(dfd, fdh.data(), sizeof(FdParams) * nb, cudaMemcpyHostToDevice, s);
        cudaMemsetAsync(err, 0, sizeof(int), s);
        // ---- assembly, boundary values, right-hand sides
        {
            EventTimer t(s, &prof[1]);
            if (fin) {
                P.begin(s);
                launch_fd_tiles(nb, dfd, tiles, scr, s);
                launch_tiles_f32(nb, tiles, tiles_f, s);
                launch_fin_points(pv, nb, dfd, fpt, s);
                if (nfp) launch_field_fin(pv, field.pts, nfp, nb, dfd, fq, s);
                P.end(KF_FD_TILES, 0.0, s);
                *launches += 4 + (nfp > 0);
            }
            P.begin(s);
            if (sg)
                launch_assemble_f32_sg(pv, st, nb, dfi, dfd, tiles_f, fpt, fin, S32, A32, Np, sg_img, sg_count, err, s);
            else
                launch_assemble_f32(pv, st, nb, dfi, dfd, tiles_f, fpt, fin, S32, A32, G > 1 ? nullptr : W, Np, s);
            if (G > 1) {
                launch_sectors_f32(S32, A32, W, nb, G, Nm, Np, s);
                (*launches)++;
            }
            // algorithmic bytes per pair: 4 FP64 statics read (32 B), S and A written as complex64 (16 B)
            P.end(KF_ASSEMBLE, 48.0 * (double)Nm * N * nb, s);
            if (Np > Nm) k_pad_identity<<<dim3(64, ns), 256, 0, s>>>(A32, W, Nm, Np, MB);
            if (sg && G == 1)  // (the others write the LU's working copy of A beside it)
                cudaMemcpyAsync(W, A32, MB * ns * 4, cudaMemcpyDeviceToDevice, s);
            P.begin(s);
            launch_boundary(pv, nb, dfi, H, dheads, depth, opt.gravity, u, phiI, s);
            P.end(KF_BOUNDARY, 0.0, s);
            *launches += 2 + (Np > Nm);  // the assembly, the boundary values, the identity padding
            t.stop();
        }
        // ---- LU of M = A^T without pivoting, blocked by NBL, the products on the tensor cores
        {
            EventTimer t(s, &prof[2]);
            // The LU of LU_GROUPS groups of the batch on side streams: the chain of a panel's diagonal block of
            // one group runs beside the tensor-core products of the others, whose persistent grids leave it SMs.
            struct Half {
                cudaStream_t st;
                int f0, nb, cap;
            };
            auto diag = [&](const Half& h, int k0, int koff) {
                P.begin(h.st);
                k_diag_factor<<<2 * h.nb, DF_THREADS, dsmem, h.st>>>(
                    W + (size_t)h.f0 * MB, Np, MB, k0, koff, PX + (size_t)h.f0 * inv, PY + (size_t)h.f0 * inv,
                    DINV + (size_t)h.f0 * dinv, err);
                P.end(KF_LU_PANEL, 8.0 * NBL * (double)NBL * NBL * h.nb, h.st);
                (*launches)++;
            };
            auto mid = [&](const Half& h, int k0, int stage) {
                P.begin(h.st);
                k_mid<<<dim3(NBL / 32, NBL / 32, stage == 1 ? h.nb : 2 * h.nb), 256, 0, h.st>>>(
                    stage, W + (size_t)h.f0 * MB, Np, MB, k0, DINV + (size_t)h.f0 * dinv, dinv,
                    TXY + (size_t)h.f0 * midsz, PX + (size_t)h.f0 * inv, PY + (size_t)h.f0 * inv);
                P.end(KF_LU_PANEL, (stage == 1 ? 8.0 : 16.0) * NBL * (double)NBL * NBL * h.nb, h.st);
                (*launches)++;
            };
            auto prep_row = [&](const Half& h, int k0, int c0, int ncols) {  // rows k0..k0+PW, columns c0..c0+ncols
                P.begin(h.st);
                k_prep_block_row<<<dim3(ncols / 32, PW / 32, 2 * h.nb), dim3(32, 8), 0, h.st>>>(
                    W + (size_t)h.f0 * MB, Np, MB, k0, c0, P2 + (size_t)h.f0 * prep);
                P.end(KF_MIXED_CONVERT, 2.0 * PW * (double)ncols * 8 * h.nb, h.st);
                (*launches)++;
            };
            CgemmArgs g0{};
            g0.err = err;
            // W(rows r0 .. , mt tiles; columns c0 .. , nt tiles) -= [L of the super-step's first k columns] [U of its
            // first k rows], S0 its first column, FP16 operands, FP32 accumulation and reduction into W
            auto update = [&](const Half& h, int r0, int mt, int c0, int nt, int k) {
                CgemmArgs g = g0;
                g.mt = mt;
                g.nt = nt;
                g.K = k;
                g.a_row0 = r0;
                g.b_n0 = c0;
                g.subtract = 1;
                g.o_row0 = r0;
                g.o_col0 = c0;
                gemm(mapL16, mapU16, g, h.f0, h.nb, h.st, h.cap, true);
            };
            // L(rows k0 + PW ..) = M(., columns k0 .. k0 + PW) Y in place, and into L16 at column koff
            auto gemm_l = [&](const Half& h, int k0, int koff) {
                CgemmArgs g = g0;
                g.mt = (Np - k0 - PW) / GBM;
                g.nt = 2;
                g.K = PW;
                g.tri = CG_RIGHT_UPPER;
                g.a_k0 = k0;
                g.a_row0 = k0 + PW;
                g.o_row0 = k0 + PW;
                g.o_col0 = k0;
                g.h16 = L16;
                g.h_bstride = op16;
                g.h_plane = (size_t)Np * SW;
                g.h_ld = SW;
                g.h_row0 = k0 + PW;
                g.h_col0 = koff;
                gemm(mapW, mapPY, g, h.f0, h.nb, h.st, h.cap, false);
            };
            // U(rows k0 .. k0 + PW, columns k0 + PW ..) = X M (transposed in P2), and into U16 at row koff
            auto gemm_u = [&](const Half& h, int k0, int koff) {
                CgemmArgs g = g0;
                g.mt = 2;
                g.nt = (Np - k0 - PW) / GBN;
                g.K = PW;
                g.tri = CG_LEFT_LOWER;
                g.o_row0 = k0;
                g.o_col0 = k0 + PW;
                g.h16 = U16;
                g.h_bstride = op16;
                g.h_plane = (size_t)Np * SW;
                g.h_ld = Np;
                g.h_row0 = koff;
                g.h_col0 = k0 + PW;
                gemm(mapPX, mapP2, g, h.f0, h.nb, h.st, h.cap, false);
            };
            // the panel at column k0 of the super-step that begins at S0
            auto panel = [&](const Half& h, int S0, int k0) {
                const int w = std::min(PW, Np - k0), c2 = k0 + w, n = Np - c2, koff = k0 - S0;
                if (koff > 0) {
                    update(h, k0, (Np - k0) / GBM, k0, w / GBN, koff);
                    if (n > 0) update(h, k0, w / GBM, c2, n / GBN, koff);
                }
                diag(h, k0, 0);
                if (w < PW) return;  // an odd last block
                mid(h, k0, 0);
                mid(h, k0, 1);
                diag(h, k0 + NBL, NBL);
                if (n == 0) return;
                mid(h, k0, 2);
                mid(h, k0, 3);
                prep_row(h, k0, c2, n);
                gemm_l(h, k0, koff);
                gemm_u(h, k0, koff);
                if (koff + PW == SW)
                    update(h, c2, n / GBM, c2, n / GBN, koff + PW);
            };
            const int nh = lu_groups_for(Np, ns);
            Half hs[LU_GROUPS];
            for (int i = 0, f0 = 0; i < nh; i++) {
                const int ni = ns / nh + (i < ns % nh ? 1 : 0);
                // the diagonal factors of the other groups' matrices take two CTAs each: as many SMs are left to
                // them, but a product keeps half of the device at least (with 160 systems of order 1024 the first
                // rule alone left it one CTA: LU 50.5 ms, with the half 4.4 ms, with all SMs 4.6; the 40 systems of
                // order 4096: 22.6 with 88 CTAs, 23.7 with all)
                hs[i] = Half{side.s[i], f0, ni, std::max(n_sm - 2 * (ns - ni), n_sm / 2)};
                f0 += ni;
            }
            cudaEventRecord(side.fork, s);
            for (int i = 0; i < nh; i++) cudaStreamWaitEvent(hs[i].st, side.fork, 0);
            // the right-hand sides b = -S u on their own stream, beside the LU (the refinement needs them)
            cudaStream_t srhs = side.s[LU_GROUPS];
            cudaStreamWaitEvent(srhs, side.fork, 0);
            cudaMemsetAsync(b, 0, sizeof(double2) * nrhs * Np * ns, srhs);
            if (G > 1) {  // projected on the sectors first
                launch_project(u, up, nb, G, Nm, nrhs, Nm, srhs);
                (*launches)++;
            }
            gemv(S32, G > 1 ? up : u, Nm, nullptr, b, ns, KF_RHS, srhs);
            cudaEventRecord(side.join[LU_GROUPS], srhs);
            for (int S0 = 0; S0 < Np; S0 += SW)
                for (int k0 = S0; k0 < std::min(S0 + SW, Np); k0 += PW)
                    for (int i = 0; i < nh; i++) panel(hs[i], S0, k0);
            for (int i = 0; i < nh; i++) {
                cudaEventRecord(side.join[i], hs[i].st);
                cudaStreamWaitEvent(s, side.join[i], 0);
            }
            cudaStreamWaitEvent(s, side.join[LU_GROUPS], 0);
            t.stop();
        }
        // ---- refinement: x_{i+1} = x_i + A^-1 (b - A x_i), A^-1 by the TF32 factors, residuals in FP64
        int it = 0;
        bool converged = false;
        {
            EventTimer t(s, &prof[3]);
            cudaMemsetAsync(x, 0, sizeof(double2) * nrhs * Np * ns, s);
            k_to_pairs<<<dim3((Np + 255) / 256, npair, ns), 256, 0, s>>>(Np, nrhs, b, r);
            cudaMemsetAsync(norms, 0, sizeof(double) * IR_MAX_IT * 2 * ns, s);
            (*launches)++;
            IrHistory& hist = last_ir_history();
            hist.n = 0;
            // the largest relative correction over the batch at iteration i (norms of slot i)
            auto worst_at = [&](int i) {
                double worst = 0.0;
                for (int f = 0; f < ns; f++) {
                    double ratio = hn[(size_t)i * 2 * ns + 2 * f] / std::max(hn[(size_t)i * 2 * ns + 2 * f + 1], 1e-300);
                    if (!std::isfinite(ratio)) ratio = INFINITY;
                    worst = std::max(worst, ratio);
                }
                return worst;
            };
            auto correction = [&](int i) {  // d = A^-1 r (FP32), x += d, norms into slot i
                trisolve(r, ns);
                k_ir_update<<<dim3((Np + 255) / 256, npair, ns), 256, 0, s>>>(
                    Np, nrhs, x, r, reinterpret_cast<unsigned long long*>(norms) + (size_t)i * 2 * ns);
                *launches += 1;
            };
            // the forces and the readback of outputs, norms and the error flag (one wait for all)
            auto forces = [&]() {
                EventTimer tf(s, &prof[4]);
                double* dA = dout;
                double* dB = dout + DD * nb;
                double2* dX = reinterpret_cast<double2*>(dout + 2 * DD * nb);
                double2* dFK = dX + (size_t)H * D * nb;
                double2* dSC = dFK + (size_t)H * D * nb;
                if (G > 1) {  // the potentials of every panel from the sector solutions
                    launch_recombine(x, phi, nb, G, Nm, nrhs, Np, s);
                    (*launches)++;
                }
                P.begin(s);
                launch_forces(pv, nb, dfi, H, G > 1 ? phi : x, G > 1 ? N : Np, phiI, opt.density, dA, dB, dX, dFK, dSC, s);
                P.end(KF_FORCES, 16.0 * (double)N * (nrhs + H) * nb, s);
                launch_haskind(pv, nb, dfi, H, G > 1 ? phi : x, G > 1 ? N : Np, u, phiI, opt.density,
                               dSC + 2 * (size_t)H * D * nb + (size_t)nfp * (D + 3 * H) * nb, s);
                *launches += 1 + (H > 0);
                if (motion && H > 0) {  // the motion equation of every frequency (motion.rs:121-158)
                    launch_motions(nb, D, H, dfi, dA, dB, dX, motion, motion + DD, motion + 2 * DD,
                                   dSC + (size_t)H * D * nb, err, s);
                    (*launches)++;
                }
                if (nfp) {  // the field points from the potentials of every panel
                    double2* fr = dSC + 2 * (size_t)H * D * nb;
                    double2* fi_ = fr + (size_t)nfp * D * nb;
                    launch_field(pv, field.pts, nfp, field.stp, nb, dfi, dfd, tiles, fq, fin, H, dheads, depth,
                                 opt.gravity, G > 1 ? phi : x, G > 1 ? N : Np, u, phiI, fr, fi_, fi_ + (size_t)nfp * H * nb,
                                 fi_ + 2 * (size_t)nfp * H * nb, s);
                    (*launches)++;
                }
                if (TK) {  // the Kochin functions, then the momentum drift (with the motions when computed)
                    double2* kr = dSC + 3 * (size_t)H * D * nb + (size_t)nfp * (D + 3 * H) * nb;
                    double2* krt = kr + (size_t)TK * D * nb;
                    double2* kd = krt + (size_t)TK * D * nb;
                    double2* kdt = kd + (size_t)TK * H * nb;
                    launch_kochin(pv, nb, dfi, TK, H, depth, G > 1 ? phi : x, G > 1 ? N : Np, u, phiI, kr, krt, kd, kdt, s);
                    launch_drift(nb, D, H, TK, dfi, depth, opt.gravity, opt.density, dheads, kr, krt, kd, kdt,
                                 motion ? dSC + (size_t)H * D * nb : nullptr, kdt + (size_t)TK * H * nb, s);
                    *launches += 2;
                }
                cudaMemcpyAsync(hout, dout, sizeof(double) * out_per * nb, cudaMemcpyDeviceToHost, s);
                cudaMemcpyAsync(herr, err, sizeof(int), cudaMemcpyDeviceToHost, s);
                tf.stop();
                solve_end().record(s);
            };
            // the first `guess` corrections and the forces without waiting on the host, then one look
            // at all the norms; further corrections (and the forces again) only when they fall short.
            // The residual after the first correction is b - A x with FP64 products; after a later one
            // (|d| ~ 1e-3 |x| and smaller) it is r - A d with FP32 products (the r before the
            // correction kept in rs); the host-driven corrections beyond `guess` use b - A x again.
            const int guess = std::min(std::max(ir_guess(), 2), IR_MAX_IT);
            for (int i = 0; i < guess; i++) {
                const bool more = i + 1 < guess, inc = more && i >= 1 && rs;
                if (inc) cudaMemcpyAsync(rs, r, sizeof(float4) * npair * Np * ns, cudaMemcpyDeviceToDevice, s);
                correction(i);
                if (more && !(inc && gemv32(A32, r, rs, r, ns))) gemv(A32, x, Np, b, r, ns, KF_MIXED_RESIDUAL, s);
            }
            cudaMemcpyAsync(hn, norms, sizeof(double) * 2 * ns * guess, cudaMemcpyDeviceToHost, s);
            t.stop();
            forces();
            cudaStreamSynchronize(s);
            double prev = INFINITY;
            bool stalled = false;
            for (it = 0; it < guess; it++) {
                const double worst = worst_at(it);
                hist.ratio[hist.n++] = worst;
                const double rho = it > 0 ? std::min(1.0, worst / prev) : 1.0;
                if (worst * rho <= IR_TOL) {  // the error left is negligible
                    converged = true;
                    break;
                }
                if (it >= 3 && !(worst < 0.5 * prev)) stalled = true;  // stalled or diverging
                prev = worst;
            }
            if (converged) {
                ir_guess() = it + 1;
                it = guess;  // the corrections that ran (a later one only refines further)
            } else if (!stalled && *herr == 0) {
                // further corrections, one host look each: no residual after the one that meets the test
                EventTimer t2(s, &prof[3]);
                for (it = guess; it < IR_MAX_IT; it++) {
                    gemv(A32, x, Np, b, r, ns, KF_MIXED_RESIDUAL, s);
                    correction(it);
                    cudaMemcpyAsync(hn + (size_t)it * 2 * ns, norms + (size_t)it * 2 * ns, sizeof(double) * 2 * ns,
                                    cudaMemcpyDeviceToHost, s);
                    cudaStreamSynchronize(s);
                    const double worst = worst_at(it);
                    hist.ratio[hist.n++] = worst;
                    const double rho = std::min(1.0, worst / prev);
                    if (worst * rho <= IR_TOL) {
                        converged = true;
                        ir_guess() = it + 1;
                        it++;
                        break;
                    }
                    if (it >= 3 && !(worst < 0.5 * prev)) break;
                    prev = worst;
                }
                t2.stop();
                // the outputs read back so far are those of the iterate after `guess` corrections; the
                // keep-or-redo test below looks at the last correction, so the outputs must be its
                // iterate's, converged or not
                if (hist.n > guess) {
                    forces();
                    cudaStreamSynchronize(s);
                }
            }
        }
        P.flush();
        {
            const cudaError_t ce = cudaGetLastError();
            if (ce != cudaSuccess) {
                static thread_local std::string why;
                why = std::string("CUDA error in the mixed-precision solve: ") + cudaGetErrorString(ce);
                MIXED_FAIL(HB_ERR_INTERNAL, why.c_str(), f0);
            }
        }
        if (!maps_ok) MIXED_FAIL(HB_ERR_INTERNAL, "tensor-map encoding failed", f0);
        if (*herr == 8) MIXED_FAIL(HB_ERR_INTERNAL, "a triangular sweep wait timed out", f0);
        if (*herr == 11) MIXED_FAIL(HB_ERR_NUMERICAL, "singular motion equation", f0);
        if (*herr != 0 && *herr != 10) MIXED_FAIL(HB_ERR_INTERNAL, "a tensor-core pipeline wait timed out", f0);
        // Frequencies the reduced-precision factors cannot solve (a zero pivot of the unpivoted LU: the whole
        // batch; a system whose corrections do not contract, as near an irregular frequency) go to the FP64
        // form; a system counts as solved when its own predicted error, as the batch test, is below IR_TOL.
        std::vector<char> redo(nb, 0);
        if (*herr == 10) {
            std::fill(redo.begin(), redo.end(), 1);
        } else if (!converged) {
            const int last = last_ir_history().n - 1;
            for (int q = 0; q < ns; q++) {
                auto ratio = [&](int i) {
                    const double r = hn[(size_t)i * 2 * ns + 2 * q] / std::max(hn[(size_t)i * 2 * ns + 2 * q + 1], 1e-300);
                    return std::isfinite(r) ? r : INFINITY;
                };
                const double rl = last >= 0 ? ratio(last) : INFINITY;
                const double rho = last >= 1 ? std::min(1.0, rl / std::max(ratio(last - 1), 1e-300)) : 1.0;
                if (!(rl * rho <= IR_TOL)) redo[q / G] = 1;
            }
        }
        if (!fallback) {
            for (int i = 0; i < nb; i++)
                if (redo[i])
                    MIXED_FAIL(HB_ERR_NUMERICAL, "iterative refinement of the mixed-precision solve did not converge", f0 + i);
        }
        const double* hA = hout;
        const double* hB = hA + DD * nb;
        const double* hX = hA + 2 * DD * nb;
        const double* hFK = hX + (size_t)H * 2 * D * nb;
        const double* hSC = hFK + (size_t)H * 2 * D * nb;
        const double* hMo = hSC + (size_t)H * 2 * D * nb;
        const double* hFr = hMo + (size_t)H * 2 * D * nb;
        const double* hFi = hFr + (size_t)nfp * 2 * D * nb;
        const double* hHK = hFi + (size_t)nfp * 2 * 3 * H * nb;
        const double* hKr = hHK + (size_t)H * 2 * D * nb;
        for (int i = 0; i < nb; i++) {
            const size_t fo = (size_t)(f0 + i), hx = (size_t)H * 2 * D;
            if (redo[i]) {
                fallback->push_back((int64_t)fo);
                continue;
            }
            for (size_t q = 0; q < DD; q++)
                if (!std::isfinite(hA[DD * i + q]) || !std::isfinite(hB[DD * i + q]))
                    MIXED_FAIL(HB_ERR_NUMERICAL, "non-finite solution", f0 + i);
            if (pr.out.added_mass) memcpy(pr.out.added_mass + fo * DD, hA + DD * i, DD * sizeof(double));
            if (pr.out.radiation_damping) memcpy(pr.out.radiation_damping + fo * DD, hB + DD * i, DD * sizeof(double));
            if (pr.out.excitation) memcpy(pr.out.excitation + fo * hx, hX + hx * i, hx * sizeof(double));
            if (pr.out.froude_krylov) memcpy(pr.out.froude_krylov + fo * hx, hFK + hx * i, hx * sizeof(double));
            if (pr.out.scattering) memcpy(pr.out.scattering + fo * hx, hSC + hx * i, hx * sizeof(double));
            if (motion && pr.out.motions) memcpy(pr.out.motions + fo * hx, hMo + hx * i, hx * sizeof(double));
            if (pr.out.haskind) memcpy(pr.out.haskind + fo * hx, hHK + hx * i, hx * sizeof(double));
            if (TK) copy_kochin(pr.out, hKr, TK, D, H, nb, i, fo);
            if (nfp) {
                const size_t pd = (size_t)nfp * 2 * D, ph = (size_t)nfp * 2 * H;
                if (pr.out.field_radiation) memcpy(pr.out.field_radiation + fo * pd, hFr + pd * i, pd * sizeof(double));
                double* dst3[3] = {pr.out.field_incident, pr.out.field_scattering, pr.out.field_diffraction};
                for (int q = 0; q < 3; q++)
                    if (dst3[q]) memcpy(dst3[q] + fo * ph, hFi + ph * ((size_t)q * nb + i), ph * sizeof(double));
            }
        }
        last_ir_iterations() = it;
    }
    if (sg) {
        unsigned long long used = 0;
        cudaMemcpyAsync(&used, sg_count, sizeof used, cudaMemcpyDeviceToHost, s);
        cudaStreamSynchronize(s);
        last_surrogate_pairs() = (long long)used;
    }
    return 0;
}

// Test support: C (M x N, row-major FP32) = A (M x K, row-major) B^T where B is given N x K
// (K-major), or C -= A B^T, on the tcgen05 TF32 path of the mixed LU (its complex product, the imaginary planes
// zero).  M, N, K multiples of 128, 128, 32.
int debug_gemm_tf32(int M, int N, int K, const float* A, const float* B, float* C, bool subtract, const char** msg) {
    if (M % GBM || N % GBN || K % GBK || M <= 0 || N <= 0 || K <= 0) {
        *msg = "debug GEMM shape: M % 128, N % 128, K % 32";
        return HB_ERR_VALUE;
    }
    if (!encode_fn()) {
        *msg = "no tensor-map encoder";
        return HB_ERR_UNSUPPORTED;
    }
    MixedBuffers mb;
    const size_t nA = (size_t)M * K, nB = (size_t)N * K, nC = (size_t)M * N;
    float* dA = mb.get<float>(2 * nA);
    float* dB = mb.get<float>(2 * nB);
    float* dC = mb.get<float>(2 * nC);
    int* err = mb.get<int>(1);
    if (!dA || !dB || !dC || !err) {
        *msg = "allocation failed";
        return HB_ERR_INTERNAL;
    }
    cudaMemset(dA + nA, 0, sizeof(float) * nA);
    cudaMemset(dB + nB, 0, sizeof(float) * nB);
    cudaMemset(dC, 0, sizeof(float) * 2 * nC);
    cudaMemcpy(dA, A, sizeof(float) * nA, cudaMemcpyHostToDevice);
    cudaMemcpy(dB, B, sizeof(float) * nB, cudaMemcpyHostToDevice);
    if (subtract) cudaMemcpy(dC, C, sizeof(float) * nC, cudaMemcpyHostToDevice);
    cudaMemset(err, 0, sizeof(int));
    CUtensorMap mA, mB, mC;
    if (!make_map(&mA, dA, K, M, 2, 1, (uint64_t)K * 4, nA * 4, 2 * nA * 4, GBM) ||
        !make_map(&mB, dB, K, N, 2, 1, (uint64_t)K * 4, nB * 4, 2 * nB * 4, GBN) ||
        !make_map(&mC, dC, N, M, 2, 1, (uint64_t)N * 4, nC * 4, 2 * nC * 4, GBM)) {
        *msg = "tensor-map encoding failed";
        return HB_ERR_INTERNAL;
    }
    CgemmArgs g{};
    g.mt = M / GBM;
    g.nt = N / GBN;
    g.K = K;
    g.subtract = subtract;
    g.batch = 1;
    g.err = err;
    const int smem = (int)gemm_smem_bytes();
    cudaFuncSetAttribute(k_cgemm<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    int dev = 0, n_sm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
    // fewer CTAs than tiles, so that the persistent loop and both accumulator buffers are exercised
    const int tiles = g.mt * g.nt;
    k_cgemm<false><<<std::max(1, std::min(tiles / 3, n_sm)), GEMM_THREADS, smem>>>(mA, mB, mC, g);
    int herr = 0;
    cudaMemcpy(&herr, err, sizeof(int), cudaMemcpyDeviceToHost);
    cudaMemcpy(C, dC, sizeof(float) * nC, cudaMemcpyDeviceToHost);
    if (cudaGetLastError() != cudaSuccess) {
        *msg = "CUDA error";
        return HB_ERR_INTERNAL;
    }
    if (herr) {
        *msg = "pipeline wait timed out";
        return HB_ERR_INTERNAL;
    }
    return 0;
}

// Test support: y [batch][nrhs][n] = M x by the FP64 product of the mixed form (M planar FP32 [batch][2][n][n],
// column-major, its padding to a multiple of 128 filled with NaNs here; x [batch][nrhs][n]), repeated `repeats` times:
// *differ counts the entries of the later results that are not those of the first to the bit.
int debug_cgemv(int n, int batch, int nrhs, const float* M, const double2* x, double2* y, int repeats, long long* differ,
                const char** msg) {
    if (n <= 0 || batch <= 0 || batch > 65535 || nrhs <= 0 || nrhs > 32 || repeats <= 0) {
        *msg = "debug product: n, repeats > 0, 0 < batch <= 65535, 0 < nrhs <= 32";
        return HB_ERR_VALUE;
    }
    if (!encode_fn()) {
        *msg = "no tensor-map encoder";
        return HB_ERR_UNSUPPORTED;
    }
    MixedBuffers mb;
    const int Np = (n + NBL - 1) / NBL * NBL, nz = (n + GV_CHUNK - 1) / GV_CHUNK;
    const size_t nM = (size_t)2 * Np * Np * batch, nx = (size_t)n * nrhs * batch;
    float* dM = mb.get<float>(nM);
    double2* dx = mb.get<double2>(nx);
    double2* dy = mb.get<double2>(nx);
    double2* part = mb.get<double2>(nx * nz);
    int* err = mb.get<int>(1);
    if (!dM || !dx || !dy || !part || !err) {
        *msg = "allocation failed";
        return HB_ERR_INTERNAL;
    }
    cudaMemset(dM, 0xff, nM * sizeof(float));
    for (size_t p = 0; p < 2 * (size_t)batch; p++)
        cudaMemcpy2D(dM + p * Np * Np, sizeof(float) * Np, M + p * n * n, sizeof(float) * n, sizeof(float) * n, n,
                     cudaMemcpyHostToDevice);
    cudaMemcpy(dx, x, nx * sizeof(double2), cudaMemcpyHostToDevice);
    cudaMemset(err, 0, sizeof(int));
    std::vector<double2> again(repeats > 1 ? nx : 0);
    *differ = 0;
    for (int r = 0; r < repeats; r++) {
        if (!launch_cgemv_dmma(dM, n, Np, dx, n, nrhs, batch, nz, part, err, nullptr)) {
            *msg = "tensor-map encoding failed";
            return HB_ERR_INTERNAL;
        }
        k_gemv_reduce<<<dim3((unsigned)((nx / batch + 255) / 256), batch), 256>>>(n, nrhs, batch, nz, part, nullptr, n, dy, n);
        double2* to = r ? again.data() : y;
        cudaMemcpy(to, dy, nx * sizeof(double2), cudaMemcpyDeviceToHost);
        if (r)
            for (size_t i = 0; i < nx; i++) *differ += memcmp(&again[i], &y[i], sizeof(double2)) != 0;
    }
    for (size_t i = 0; i < nx; i++) y[i] = make_double2(-y[i].x, -y[i].y);  // (the reduction forms bias - M x)
    int herr = 0;
    cudaMemcpy(&herr, err, sizeof(int), cudaMemcpyDeviceToHost);
    if (cudaGetLastError() != cudaSuccess || herr) {
        *msg = herr ? "a tensor-core pipeline wait timed out" : "CUDA error";
        return HB_ERR_INTERNAL;
    }
    return 0;
}

}  // namespace hbg
