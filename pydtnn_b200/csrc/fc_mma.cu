// Fully connected layers of float32 whose passes are too short for the convolution engine: forward in one launch, both
// gradients in another (reference: pydtnn/backends/gpu/layers/fc_gpu.py:54-94, three cuBLAS calls and a bias kernel).
//
// Such a pass as a split 1x1 convolution is a few microseconds of products between 7 of set-up (tensor memory, barriers, tensor
// maps) and a second stage that adds the splits.  Here a block multiplies a 64-column tile with warp-level tf32 products out of a
// cp.async ring; the blocks of a cluster share the K loop of a tile and add their sums through distributed shared memory, so no
// partial sum touches global memory.  Forward / both gradients in us, before -> now: 64 x 256 x 256 8.8 / 16.5 -> 5.1 / 5.2;
// 64 x 333 x 777 (pixels of no 16 bytes) 17.3 / 35.4 -> 7.5 / 9.6; 1 x 2048 x 1000 11.0 / 16.2 -> 7.8 / 8.8; gradients of
// 64 x 4096 x 10 25.4 -> 6.1; forward 32 x 40 x 512 (FMAs) 12.5 -> 3.4.  Bound by instructions: 387 a warp for a step of
// 64 x 64 x 32 (460 while the split looked at each hi half), 0.8 us of which the products take 0.4; what the
// convolution engine does faster is left to it (fc_mma_takes).
//
// Precision: both operands are split by rounding, a = hi + lo.  hi * hi is summed by the tensor core over 32 products at most and
// then added in float32 (its own additions truncate); the sums of lo * hi and hi * lo are 2^-11 of that and stay there.
// Against float64 (2-norms) 1.0 to 1.5e-7, as the convolution engine's fine sums; fewer than 48 products are plain FMAs, and so are
// sums that do not come out finite.
#include "b2c_common.cuh"
#include <cooperative_groups.h>
#include <float.h>

namespace b2c {

namespace cg = cooperative_groups;

enum { FC_FWD = 0, FC_DX = 1, FC_DW = 2 };
#define FC_BN 64
#define FC_BK 32
#define FC_STAGES 4
#define FC_THREADS 256
#define FC_SHORT 48
#define FC_CLUSTER 8

// C[M][N] (pitch N) = A B.  The operands' rows lie lda and ldb floats apart:
//   FWD  A = x  [M = batch][K = in]        B = w  [K = in][N = out]      C = y + bias
//   DX   A = dy [M = batch][K = out]       B = w  [N = in][K = out]      C = dx
//   DW   A = x  [K = batch][M = in]        B = dy [K = batch][N = out]   C = dw, and the column sums of dy: db
struct FcProblem {
    const float *a, *b, *bias;
    float *c, *db;
    int M, N, K, lda, ldb;
    int mt, nt, ks, kper;       // row and column tiles, blocks that share a tile's K loop, K per block (a multiple of FC_BK)
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const float* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const float* src, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(in ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// hi = v rounded to tf32, lo = v - hi.  Of an infinity, a NaN, or a value that rounds to an infinity one half is NaN, or they are
// infinities of either sign: no sum that such a value is part of comes out finite, and such sums are then taken from FMAs.
__device__ __forceinline__ void split_tf32(float v, uint32_t& hi, uint32_t& lo) {
    const float h = __uint_as_float((__float_as_uint(v) + 0x1000u) & 0xFFFFE000u);
    hi = __float_as_uint(h); lo = __float_as_uint(v - h);
}

// Shared-memory pitch of a tile whose rows run along K (36: a fragment's eight rows x four k fall into 32 banks) or across it.
template <bool KROWS, int EXT> constexpr int fc_pitch() { return KROWS ? FC_BK + 4 : EXT + 8; }
template <int KIND, int BM> constexpr int fc_a_floats() { return KIND == FC_DW ? FC_BK * (BM + 8) : BM * (FC_BK + 4); }
template <int KIND> constexpr int fc_b_floats() { return KIND == FC_DX ? FC_BN * (FC_BK + 4) : FC_BK * (FC_BN + 8); }
template <int KIND, int BM> constexpr int fc_smem_bytes() { return FC_STAGES * (fc_a_floats<KIND, BM>() + fc_b_floats<KIND>()) * 4; }

// One operand tile of EXT rows or columns x 32 k to shared memory; what lies outside reads as zeros.
template <bool KROWS, int EXT, bool VEC>
__device__ __forceinline__ void fc_load(uint32_t dst, const float* __restrict__ src, int ld, int e0, int ext, int k0, int k_end)
{
    constexpr int W = VEC ? 4 : 1, INNER = KROWS ? FC_BK : EXT, CHUNKS = EXT * FC_BK / W, P = fc_pitch<KROWS, EXT>();
#pragma unroll
    for (int i = 0; i < (CHUNKS + FC_THREADS - 1) / FC_THREADS; i++) {
        const int q = threadIdx.x + i * FC_THREADS;
        if (CHUNKS % FC_THREADS && q >= CHUNKS) break;
        const int o = q / (INNER / W), n = (q - o * (INNER / W)) * W;         // outer and inner index inside the tile
        const int e = e0 + (KROWS ? o : n), k = k0 + (KROWS ? n : o);
        const bool in = e < ext && k < k_end;
        const float* s = in ? src + (KROWS ? (int64_t)e * ld + k : (int64_t)k * ld + e) : src;
        if (VEC) cp_async16(dst + (uint32_t)(o * P + n) * 4u, s, in); else cp_async4(dst + (uint32_t)(o * P + n) * 4u, s, in);
    }
}

// Up to four stored outputs again where they are not finite, as chains of FMAs in the order of k: steps of sa and sb floats, columns
// `next` apart in b.  hi * lo + lo * hi + hi * hi of an infinity has an infinity times a zero, or two infinities of either sign, where
// the product itself has one value.  (A call after the store: with the chains in the epilogue passes of 5 us took 0.4 longer.)
__device__ __noinline__ void fc_redo(const float* a, int64_t sa, const float* b, int64_t sb, int64_t next, int K, const float* bias, float* d, int count)
{
#pragma unroll 1
    for (int e = 0; e < count; e++) {
        if (fabsf(d[e]) <= FLT_MAX) continue;
        float acc = 0.f;
#pragma unroll 4
        for (int k = 0; k < K; k++) acc = fmaf(__ldg(a + k * sa), __ldg(b + e * next + k * sb), acc);
        d[e] = bias ? acc + bias[e] : acc;
    }
}

// Sums of fewer than 48 products, in all three kinds: 4 columns x BM / 16 rows a thread in float32 FMAs in the order of k (the
// split would cost more precision than it is worth there: 2.5e-8 against 8e-8 for one row).  K is at most two steps, the tile is
// one block's.
template <int KIND, int BM, bool VEC>
__device__ void fc_tile_short(const FcProblem& p, int tile, float* smem)
{
    constexpr bool A_KROWS = KIND != FC_DW, B_KROWS = KIND == FC_DX;
    constexpr int AF = fc_a_floats<KIND, BM>(), BF = fc_b_floats<KIND>(), AP = fc_pitch<A_KROWS, BM>(), BP = fc_pitch<B_KROWS, FC_BN>();
    constexpr int TM = BM / 16;                                   // rows per thread
    const int mi = tile / p.nt, ni = tile - mi * p.nt, m0 = mi * BM, n0 = ni * FC_BN, steps = (p.K + FC_BK - 1) / FC_BK;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem);
    for (int i = 0; i < steps; i++) {
        const uint32_t st = base + (uint32_t)(i * (AF + BF)) * 4u;
        fc_load<A_KROWS, BM, VEC>(st, p.a, p.lda, m0, p.M, i * FC_BK, p.K);
        fc_load<B_KROWS, FC_BN, VEC>(st + AF * 4u, p.b, p.ldb, n0, p.N, i * FC_BK, p.K);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    const int c = (threadIdx.x & 15) * 4, r = (threadIdx.x >> 4) * TM;
    float acc[TM][4];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
    for (int k = 0; k < p.K; k++) {
        const float* as = smem + (k / FC_BK) * (AF + BF);
        const float* bs = as + AF;
        const int kk = k % FC_BK;
        float a[TM], b[4];
#pragma unroll
        for (int i = 0; i < TM; i++) a[i] = A_KROWS ? as[(r + i) * AP + kk] : as[kk * AP + r + i];
#pragma unroll
        for (int j = 0; j < 4; j++) b[j] = B_KROWS ? bs[(c + j) * BP + kk] : bs[kk * BP + c + j];
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
#pragma unroll
    for (int i = 0; i < TM; i++) {
        const int m = m0 + r + i, n = n0 + c;
        if (m >= p.M || n >= p.N) continue;
        float* d = p.c + (int64_t)m * p.N + n;
        if (KIND == FC_FWD && p.bias)
#pragma unroll
            for (int j = 0; j < 4; j++) if (n + j < p.N) acc[i][j] += __ldg(p.bias + n + j);
        if (VEC && p.N % 4 == 0) *reinterpret_cast<float4*>(d) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        else
#pragma unroll
            for (int j = 0; j < 4; j++) if (n + j < p.N) d[j] = acc[i][j];
    }
    if (KIND == FC_DW && p.db && mi == 0 && threadIdx.x < FC_BN && n0 + (int)threadIdx.x < p.N) {
        double col = 0.0;
        for (int k = 0; k < p.K; k++) col += (double)(smem + (k / FC_BK) * (AF + BF) + AF)[(k % FC_BK) * BP + threadIdx.x];
        p.db[n0 + threadIdx.x] = (float)col;
    }
}

// One tile: block `rank` of the tile's cluster takes k in [rank * kper, (rank + 1) * kper).
// BM = 64: 2 x 4 warps of 32 x 16 outputs; BM = 32 or 16 (small batches): 1 x 4 warps, two of them share a tile's k steps.
template <int KIND, int BM, bool VEC>
__device__ void fc_tile(const FcProblem& p, int tile, int rank, float* smem)
{
    constexpr bool A_KROWS = KIND != FC_DW, B_KROWS = KIND == FC_DX;
    constexpr int AF = fc_a_floats<KIND, BM>(), BF = fc_b_floats<KIND>(), AP = fc_pitch<A_KROWS, BM>(), BP = fc_pitch<B_KROWS, FC_BN>();
    constexpr int WM = BM < 32 ? BM : 32, MW = BM / WM, KZ = 8 / (MW * 4), MT = WM / 16, STEPS = FC_BK / 8 / KZ;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int wn = warp & 3, wm = MW == 2 ? (warp >> 2) : 0, wz = KZ == 2 ? (warp >> 2) : 0;
    const int mi = tile / p.nt, ni = tile - mi * p.nt, m0 = mi * BM, n0 = ni * FC_BN;
    const int kb = rank * p.kper, ke = kb + p.kper < p.K ? kb + p.kper : p.K;
    const int blocks = ke > kb ? (ke - kb + FC_BK - 1) / FC_BK : 0;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem);
    auto load = [&](int i) {
        if (i < blocks) {
            const uint32_t st = base + (uint32_t)((i % FC_STAGES) * (AF + BF)) * 4u;
            fc_load<A_KROWS, BM, VEC>(st, p.a, p.lda, m0, p.M, kb + i * FC_BK, ke);
            fc_load<B_KROWS, FC_BN, VEC>(st + AF * 4u, p.b, p.ldb, n0, p.N, kb + i * FC_BK, ke);
        }
        cp_async_commit();
    };
    float sum[MT][2][4], small[MT][2][4];
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) sum[i][j][e] = small[i][j][e] = 0.f;
    const bool do_db = KIND == FC_DW && p.db && mi == 0;
    double col = 0.0;
#pragma unroll
    for (int i = 0; i < FC_STAGES - 1; i++) load(i);
    for (int i = 0; i < blocks; i++) {
        cp_async_wait<FC_STAGES - 2>();
        __syncthreads();
        load(i + FC_STAGES - 1);
        const float* as = smem + (i % FC_STAGES) * (AF + BF);
        const float* bs = as + AF;
        float large[MT][2][4];
#pragma unroll
        for (int a = 0; a < MT; a++)
#pragma unroll
            for (int b = 0; b < 2; b++)
#pragma unroll
                for (int e = 0; e < 4; e++) large[a][b][e] = 0.f;
#pragma unroll
        for (int s = 0; s < STEPS; s++) {
            const int k = (wz * STEPS + s) * 8 + t;
            uint32_t ah[MT][4], al[MT][4], bh[2][2], bl[2][2];
#pragma unroll
            for (int a = 0; a < MT; a++)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int m = wm * WM + a * 16 + g + (e & 1) * 8, kk = k + (e >> 1) * 4;
                    split_tf32(A_KROWS ? as[m * AP + kk] : as[kk * AP + m], ah[a][e], al[a][e]);
                }
#pragma unroll
            for (int b = 0; b < 2; b++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int n = wn * 16 + b * 8 + g, kk = k + e * 4;
                    split_tf32(B_KROWS ? bs[n * BP + kk] : bs[kk * BP + n], bh[b][e], bl[b][e]);
                }
            // neighbours in the issue order go to different sums (one after the other on one sum they wait for it)
#pragma unroll
            for (int q = 0; q < 3; q++)
#pragma unroll
                for (int a = 0; a < MT; a++)
#pragma unroll
                    for (int b = 0; b < 2; b++) {
                        if (q == 0) mma_tf32(small[a][b], al[a], bh[b]);
                        if (q == 1) mma_tf32(large[a][b], ah[a], bh[b]);
                        if (q == 2) mma_tf32(small[a][b], ah[a], bl[b]);
                    }
        }
#pragma unroll
        for (int a = 0; a < MT; a++)
#pragma unroll
            for (int b = 0; b < 2; b++)
#pragma unroll
                for (int e = 0; e < 4; e++) sum[a][b][e] += large[a][b][e];
        if (KIND == FC_DW && do_db && threadIdx.x < FC_BN)
#pragma unroll 8
            for (int k = 0; k < FC_BK; k++) col += (double)bs[k * BP + threadIdx.x];      // rows past the batch are zeros
    }
    if (KIND == FC_DW && do_db && threadIdx.x < FC_BN && n0 + (int)threadIdx.x < p.N) p.db[n0 + threadIdx.x] = (float)col;
    cp_async_wait<0>();
    __syncthreads();
    // the block's sums to shared memory (over the operand ring), [KZ][BM][64 + 4]
    constexpr int OP = FC_BN + 4;
    static_assert(KZ * BM * OP * 4 <= fc_smem_bytes<KIND, BM>(), "the sums fit where the operands were");
#pragma unroll
    for (int a = 0; a < MT; a++)
#pragma unroll
        for (int b = 0; b < 2; b++)
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
                float* d = smem + (wz * BM + wm * WM + a * 16 + g + (e >> 1) * 8) * OP + wn * 16 + b * 8 + 2 * t;
                *reinterpret_cast<float2*>(d) = make_float2(sum[a][b][e] + small[a][b][e], sum[a][b][e + 1] + small[a][b][e + 1]);
            }
    cg::cluster_group cluster = cg::this_cluster();
    if (p.ks > 1) cluster.sync(); else __syncthreads();
    // rows of the tile shared out among the blocks of the cluster; every sum is taken in block order
    constexpr int Q = FC_BN / 4;
    const int rows = BM / p.ks, r0 = p.ks > 1 ? rank * rows : 0;
    for (int i = threadIdx.x; i < rows * Q; i += FC_THREADS) {
        const int r = r0 + i / Q, c4 = (i % Q) * 4, m = m0 + r, n = n0 + c4;
        if (m >= p.M || n >= p.N) continue;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int q = 0; q < p.ks; q++) {
            const float* peer = p.ks > 1 ? cluster.map_shared_rank(smem, q) : smem;
#pragma unroll
            for (int z = 0; z < KZ; z++) {
                const float4 u = *reinterpret_cast<const float4*>(peer + (z * BM + r) * OP + c4);
                v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
            }
        }
        float o[4] = {v.x, v.y, v.z, v.w};
        float* d = p.c + (int64_t)m * p.N + n;
        if (KIND == FC_FWD && p.bias)
#pragma unroll
            for (int e = 0; e < 4; e++) if (n + e < p.N) o[e] += __ldg(p.bias + n + e);
        if (VEC && p.N % 4 == 0) *reinterpret_cast<float4*>(d) = make_float4(o[0], o[1], o[2], o[3]);
        else
#pragma unroll
            for (int e = 0; e < 4; e++) if (n + e < p.N) d[e] = o[e];
        if (0.f * o[0] + 0.f * o[1] + 0.f * o[2] + 0.f * o[3] != 0.f)              // NaN where one of them is not finite
            fc_redo(p.a + (A_KROWS ? (int64_t)m * p.lda : m), A_KROWS ? 1 : p.lda, p.b + (B_KROWS ? (int64_t)n * p.ldb : n), B_KROWS ? 1 : p.ldb,
                    B_KROWS ? p.ldb : 1, p.K, KIND == FC_FWD && p.bias ? p.bias + n : nullptr, d, p.N - n < 4 ? p.N - n : 4);
    }
    if (p.ks > 1) cluster.sync();                        // nobody leaves while another block reads its sums
}

template <int BM, bool VEC>
__global__ void __launch_bounds__(FC_THREADS, 2) fc_mma_forward_kernel(FcProblem p)
{
    pdl_prologue();
    extern __shared__ __align__(16) float smem[];
    if (p.K < FC_SHORT) fc_tile_short<FC_FWD, BM, VEC>(p, blockIdx.x, smem);
    else fc_tile<FC_FWD, BM, VEC>(p, blockIdx.x / p.ks, blockIdx.x % p.ks, smem);
}
// dx tiles first (their K loops are the long ones), then the tiles of dw.
template <int BM, bool VEC>
__global__ void __launch_bounds__(FC_THREADS, 2) fc_mma_backward_kernel(FcProblem dx, FcProblem dw, int dx_blocks)
{
    pdl_prologue();
    extern __shared__ __align__(16) float smem[];
    const int b = blockIdx.x;
    if (b < dx_blocks) {
        if (dx.K < FC_SHORT) fc_tile_short<FC_DX, BM, VEC>(dx, b, smem);
        else fc_tile<FC_DX, BM, VEC>(dx, b / dx.ks, b % dx.ks, smem);
    } else if (b - dx_blocks < dw.mt * dw.nt) {
        if (dw.K < FC_SHORT) fc_tile_short<FC_DW, 64, VEC>(dw, b - dx_blocks, smem);
        else fc_tile<FC_DW, 64, VEC>(dw, b - dx_blocks, 0, smem);
    }
}

template <auto KERNEL, typename... Args>
static int launch_cluster(const char* what, int blocks, int ks, size_t smem, cudaStream_t st, const Args&... args)
{
    static PerDeviceOnce attr_set;             // a kernel's shared memory is the same at every launch
    const cudaError_t e = attr_set.run([smem] { return cudaFuncSetAttribute((const void*)KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); });
    if (e != cudaSuccess) { set_cuda_error(e, what); return B2C_ERR_CUDA; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = blocks; cfg.blockDim = FC_THREADS; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = ks; attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, KERNEL, args...);
    return check_launch(what);
}

// Row tile, and the blocks that share a tile's K loop: up to eight (a portable cluster; four were 1.1 to 2 times slower), until
// there are two blocks for each SM or a block would be left with fewer than two steps of 32.
static int fc_bm(int batch) { return batch <= 16 ? 16 : batch <= 32 ? 32 : 64; }
static void fc_split(FcProblem& p, int bm)
{
    p.mt = (p.M + bm - 1) / bm; p.nt = (p.N + FC_BN - 1) / FC_BN;
    int ks = 1;
    while (ks < FC_CLUSTER && (int64_t)p.mt * p.nt * ks * 2 <= 2 * (int64_t)tc_sm_count() && p.K >= ks * 2 * 2 * FC_BK) ks *= 2;
    p.ks = ks;
    p.kper = ((p.K + ks - 1) / ks + FC_BK - 1) / FC_BK * FC_BK;
}

// A pass is taken where it costs less than as convolutions, in microseconds.  One step of 32 products takes an SM 0.43, 0.67 or 1.05
// with tiles of 16, 32 or 64 rows, 0.6 in FMAs, and 2.5 come before the first and after the last.  Many clusters of eight leave SMs
// idle (a GPU part of 16 SMs and a few more holds two of them): 1.6 times.  The convolutions' side is a fit to nine layers of 41 000 to
// 38 million weights at 1 to 256 rows: forward 7 to 14, gradients 10 to 36; looked at again on 28 layers at 14 batch sizes.
static double fc_step_us(int bm) { return bm == 16 ? 0.43 : bm == 32 ? 0.67 : 1.05; }
static double fc_chain_us(const FcProblem& p, int bm)
{
    const int blocks = p.mt * p.nt * p.ks, per_sm = (blocks + tc_sm_count() - 1) / tc_sm_count();
    return (p.K < FC_SHORT ? 0.6 : fc_step_us(bm)) * (p.kper / FC_BK) * per_sm * (p.ks == 8 && 2 * blocks > tc_sm_count() ? 1.6 : 1.1);
}
bool fc_mma_takes(int dtype, int engine, int batch, int in_f, int out_f, bool backward)
{
    if (dtype != B2C_F32 || engine != B2C_ENGINE_AUTO || batch > 256 || (int64_t)in_f * out_f > (1 << 25)) return false;
    const int bm = fc_bm(batch);
    const double weights = (double)in_f * out_f * 1e-6, lim = weights < 2.1 ? weights : 2.1, limb = weights < 4.1 ? weights : 4.1;
    FcProblem p{};
    p.M = batch;
    if (!backward) {
        p.N = out_f; p.K = in_f;
        fc_split(p, bm);
        return 2.5 + fc_chain_us(p, bm) < 0.9 * (6.6 + 1.9 * lim);
    }
    p.N = in_f; p.K = out_f;
    fc_split(p, bm);
    const int steps_x = (out_f + FC_BK - 1) / FC_BK, steps_w = (batch + FC_BK - 1) / FC_BK;
    const double dx = (double)p.mt * p.nt * steps_x * (out_f < FC_SHORT ? 0.6 : fc_step_us(bm));
    const double dw = (double)((in_f + 63) / 64) * ((out_f + FC_BN - 1) / FC_BN) * steps_w * (batch < FC_SHORT ? 0.6 : fc_step_us(64));
    if (batch > 128) {
        // More rows than a weight gradient's blocks get through quickly: 1.3 a step (1.35 to 1.5 times that where two blocks share an SM),
        // and the blocks past two an SM wait for most of the dx blocks.  The convolutions no longer use fine sums where in and out are whole blocks of 32:
        // 256 x 512 x 512 21 us against 22 here, 256 x 1024 x 256 18 / 21, 256 x 100 x 4000 25 / 29; 256 x 256 x 256 15.5 / 13.0, 192 x 512 x 512 19 / 13.
        const int blocks = p.mt * p.nt * p.ks + (in_f + 63) / 64 * ((out_f + FC_BN - 1) / FC_BN);
        const double share = blocks > 2 * tc_sm_count() ? 1.5 : blocks > tc_sm_count() ? 1.35 : 1.0;
        const double x = 1.1 * (out_f < FC_SHORT ? 0.6 : fc_step_us(bm)) * (p.kper / FC_BK) * share, w = 1.3 * steps_w * share;
        const double here = 2.5 + (blocks > 2 * tc_sm_count() ? 0.8 * x + w : x > w ? x : w);
        const double work = 1.25 * (dx + dw) / tc_sm_count() + 2.5;
        const double there = in_f % 32 == 0 && out_f % 32 == 0 ? (out_f > 64 ? 12.5 : 10.3) + 14.0 * (weights < 1.0 ? weights : 1.0) + 0.012 * (batch - 128)
                                                               : 10.0 + 3.5 * limb + 0.05 * batch;
        if ((here > work ? here : work) >= there) return false;
    }
    double t = 1.25 * (dx + dw) / tc_sm_count();
    const double chain_x = fc_chain_us(p, bm), chain_w = 2.1 * steps_w;        // the blocks that also sum the bias gradient take twice as long
    t = t > chain_x ? t : chain_x;
    t = t > chain_w ? t : chain_w;
    return 1.1 * (2.5 + t) < 10.0 + 3.5 * limb + 0.05 * batch;
}

template <int BM>
static int forward(const FcProblem& p, bool vec, cudaStream_t st)
{
    constexpr size_t smem = fc_smem_bytes<FC_FWD, BM>();
    const int blocks = p.mt * p.nt * p.ks;
    return vec ? launch_cluster<fc_mma_forward_kernel<BM, true>>("fc_mma_forward_kernel", blocks, p.ks, smem, st, p)
               : launch_cluster<fc_mma_forward_kernel<BM, false>>("fc_mma_forward_kernel", blocks, p.ks, smem, st, p);
}
int fc_mma_forward(int batch, int in_f, int out_f, const void* x, const void* w, const void* bias, void* y, cudaStream_t st)
{
    FcProblem p{(const float*)x, (const float*)w, (const float*)bias, (float*)y, nullptr, batch, out_f, in_f, in_f, out_f};
    const int bm = fc_bm(batch);
    fc_split(p, bm);
    const bool vec = in_f % 4 == 0 && out_f % 4 == 0 && !(((uintptr_t)x | (uintptr_t)w | (uintptr_t)y) & 15);
    return bm == 16 ? forward<16>(p, vec, st) : bm == 32 ? forward<32>(p, vec, st) : forward<64>(p, vec, st);
}

template <int BM>
static int backward(const FcProblem& px, const FcProblem& pw, bool vec, cudaStream_t st)
{
    constexpr size_t smem_w = fc_smem_bytes<FC_DW, 64>(), smem_x = fc_smem_bytes<FC_DX, 64>(), smem = smem_w > smem_x ? smem_w : smem_x;
    const int dx_blocks = px.mt * px.nt * px.ks, blocks = dx_blocks + (pw.mt * pw.nt + px.ks - 1) / px.ks * px.ks;      // whole clusters
    return vec ? launch_cluster<fc_mma_backward_kernel<BM, true>>("fc_mma_backward_kernel", blocks, px.ks, smem, st, px, pw, dx_blocks)
               : launch_cluster<fc_mma_backward_kernel<BM, false>>("fc_mma_backward_kernel", blocks, px.ks, smem, st, px, pw, dx_blocks);
}
// dw with db, or dx, or all three (db alone is a column sum of dy and not for this).
int fc_mma_backward(int batch, int in_f, int out_f, const void* x, const void* dy, const void* w, void* dw, void* db, void* dx, cudaStream_t st)
{
    FcProblem px{(const float*)dy, (const float*)w, nullptr, (float*)dx, nullptr, batch, in_f, out_f, out_f, out_f};
    FcProblem pw{(const float*)x, (const float*)dy, nullptr, (float*)dw, (float*)db, in_f, out_f, batch, in_f, out_f};
    const int bm = fc_bm(batch);
    px.ks = 1;
    if (dx) fc_split(px, bm); else px.mt = px.nt = 0;
    pw.mt = dw ? (in_f + 63) / 64 : 0; pw.nt = (out_f + FC_BN - 1) / FC_BN; pw.ks = 1; pw.kper = (batch + FC_BK - 1) / FC_BK * FC_BK;
    const bool vec = in_f % 4 == 0 && out_f % 4 == 0 && !(((uintptr_t)x | (uintptr_t)dy | (uintptr_t)w | (uintptr_t)dw | (uintptr_t)dx) & 15);
    return bm == 16 ? backward<16>(px, pw, vec, st) : bm == 32 ? backward<32>(px, pw, vec, st) : backward<64>(px, pw, vec, st);
}

}  // namespace b2c
