// Generic FMA engine: implicit-GEMM convolution (fprop / dgrad / wgrad) for float32 and float64,
// NHWC and NCHW, any filter layout, stride, padding and dilation.  The lowered matrix is never
// written to memory: each CTA gathers its A tile straight from the activation tensor using the
// same tap arithmetic the index-map kernel exposes for the bit-exact check.
//
//   fprop : C[pixel(n,ho,wo)][co] = sum_tap  x[pixel + tap] * w[co][tap]
//   dgrad : C[pixel(n,h,w)][ci]   = sum_tap  dy[(pixel + pad - tap) / stride] * w[tap.co][ci][tap.r][tap.s]
//   wgrad : C[tap(ci,r,s)][co]    = sum_pixel x[pixel + tap] * dy[pixel][co]      (split over pixels)
//
// float32 uses FP32 FMA, float64 the FP64 tensor pipe.  This engine is the one every shape can run on; the tensor-core engine (conv_tc.cu) takes over the shapes it supports.
#include "b2c_common.cuh"
#include <atomic>
#include <type_traits>

namespace b2c {

enum { MODE_FPROP = 0, MODE_DGRAD = 1, MODE_WGRAD = 2 };

// Decoded pixel or tap. For a pixel: a_off = image base in the gathered tensor, (d0,d1) = the
// pixel's origin in gathered coordinates, b_off = its offset in the pixel-indexed second tensor.
// For a tap: a_off = channel offset, (d0,d1) = (r*vdil, s*hdil), b_off = offset in the filter tensor.
struct Info { int64_t a_off; int64_t b_off; int d0, d1; };

#define B2C_SENTINEL (1 << 29)

struct IgemmParams {
    int M, N, K;
    int P, Q, PQ;                 // pixel grid the pixel index runs over
    int C, R, S, tap_c_fast;      // tap space; tap_c_fast: index = (r*S+s)*C + c, else (c*R + r)*S + s
    int H, W;                     // extent of the gathered tensor
    int64_t a_sn, a_sh, a_sw, a_sc;
    int vstr, hstr, vpad, hpad, vdil, hdil;
    int64_t pb_sn, pb_sh, pb_sw;  // b_off of a pixel
    int64_t tb_sc, tb_sr, tb_ss;  // b_off of a tap
    int64_t b_sn;                 // B(k, n) = Bsrc[kinfo.b_off + n*b_sn]
    int64_t c_sn;                 // C(m, n) = Cdst[rowinfo.b_off + n*c_sn]
    int a_lanes_k, b_lanes_k;     // which index runs fastest across lanes when loading A / B
    int k_chunk, splits, bn;      // bn: columns of a tile
    int whole, m_whole;           // float64: tiles, and the rows they cover, that take no part in the split
    int relu;
    // Sub-lattices (strided dgrad runs one launch per residue class of the output pixels, each with the taps that
    // reach it): pixel (pp, qq) of the grid is row pix_h0 + pp*pix_hs, column pix_w0 + qq*pix_ws of the tensor;
    // tap (r, s) of the (R, S) grid is filter tap (tap_r0 + r*tap_rs, tap_s0 + s*tap_ss).  Identity elsewhere.
    int pix_h0, pix_hs, pix_w0, pix_ws;
    int tap_r0, tap_rs, tap_s0, tap_ss;
    bool small;                   // x (dx), y (dy) with a window's overhang and the filter have fewer than 2^31 elements each
    int lin_h, lin_w;             // dgrad: how far one tap of the (R, S) grid moves the gathered row and column
    FastDiv f_pq, f_q, f_c, f_s, f_rs;       // float64 kernel (launch_igemm): PQ, Q, C, S, R * S
};

template <typename T> struct Epilogue { const T *bias, *mean, *inv_std, *gamma, *beta; int relu; };
// The same of one output channel, whose values are loaded once.
template <typename T> struct ChannelEpilogue {
    T bias, mean, inv_std, gamma, beta;
    bool has_bias, has_bn, relu;
    __device__ __forceinline__ ChannelEpilogue(const Epilogue<T>& ep, int n)
        : bias(ep.bias ? ep.bias[n] : T(0)), mean(ep.mean ? ep.mean[n] : T(0)), inv_std(ep.mean ? ep.inv_std[n] : T(0)),
          gamma(ep.mean ? ep.gamma[n] : T(0)), beta(ep.mean ? ep.beta[n] : T(0)), has_bias(ep.bias), has_bn(ep.mean), relu(ep.relu) {}
    __device__ __forceinline__ T operator()(T v) const {
        if (has_bias) v += bias;
        if (has_bn) { T t = (v - mean) * inv_std; v = t * gamma + beta; }
        if (relu) v = v > T(0) ? v : T(0);
        return v;
    }
};

template <int MODE> __device__ __forceinline__ Info decode_pix(const IgemmParams& p, int idx, int limit) {
    Info f;
    if (idx >= limit) { f.a_off = 0; f.b_off = 0; f.d0 = -B2C_SENTINEL; f.d1 = 0; return f; }
    int n = idx / p.PQ; int rem = idx - n * p.PQ; int pp = rem / p.Q; int qq = rem - pp * p.Q;
    pp = p.pix_h0 + pp * p.pix_hs; qq = p.pix_w0 + qq * p.pix_ws;
    f.a_off = (int64_t)n * p.a_sn;
    f.b_off = (int64_t)n * p.pb_sn + (int64_t)pp * p.pb_sh + (int64_t)qq * p.pb_sw;
    if (MODE == MODE_DGRAD) { f.d0 = pp + p.vpad; f.d1 = qq + p.hpad; }
    else { f.d0 = pp * p.vstr - p.vpad; f.d1 = qq * p.hstr - p.hpad; }
    return f;
}

template <int MODE> __device__ __forceinline__ Info decode_tap(const IgemmParams& p, int idx, int limit) {
    Info f;
    if (idx >= limit) { f.a_off = 0; f.b_off = 0; f.d0 = (MODE == MODE_DGRAD) ? B2C_SENTINEL : -B2C_SENTINEL; f.d1 = 0; return f; }
    int c, r, s;
    if (p.tap_c_fast) { c = idx % p.C; int rs = idx / p.C; r = rs / p.S; s = rs - r * p.S; }
    else { int RS = p.R * p.S; c = idx / RS; int rs = idx - c * RS; r = rs / p.S; s = rs - r * p.S; }
    r = p.tap_r0 + r * p.tap_rs; s = p.tap_s0 + s * p.tap_ss;
    f.a_off = (int64_t)c * p.a_sc;
    f.b_off = (int64_t)c * p.tb_sc + (int64_t)r * p.tb_sr + (int64_t)s * p.tb_ss;
    f.d0 = r * p.vdil; f.d1 = s * p.hdil;
    return f;
}

__device__ __forceinline__ bool info_valid(const Info& f) { return f.d0 > -(B2C_SENTINEL >> 1) && f.d0 < (B2C_SENTINEL >> 1); }

// The tap arithmetic shared by every pass and by the index-map kernel: where in the gathered
// tensor does (pixel, tap) read, and is that inside the tensor?
template <int MODE>
__device__ __forceinline__ bool gather_off(const IgemmParams& p, const Info& pix, const Info& tap, int64_t& off) {
    int ih, iw;
    if (MODE == MODE_DGRAD) {
        int th = pix.d0 - tap.d0, tw = pix.d1 - tap.d1;
        if (th < 0 || tw < 0) return false;
        if (p.vstr != 1) { ih = th / p.vstr; if (ih * p.vstr != th) return false; } else ih = th;
        if (p.hstr != 1) { iw = tw / p.hstr; if (iw * p.hstr != tw) return false; } else iw = tw;
    } else {
        ih = pix.d0 + tap.d0; iw = pix.d1 + tap.d1;
    }
    if ((unsigned)ih >= (unsigned)p.H || (unsigned)iw >= (unsigned)p.W) return false;
    off = pix.a_off + tap.a_off + (int64_t)ih * p.a_sh + (int64_t)iw * p.a_sw;
    return true;
}

__device__ __forceinline__ void lds4(const float* p, float (&o)[4]) {
    float4 v = *reinterpret_cast<const float4*>(p); o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
}

template <typename T> __device__ __forceinline__ T apply_epilogue(T v, int n, const Epilogue<T>& ep) {
    if (ep.bias) v += ep.bias[n];
    if (ep.mean) { T t = (v - ep.mean[n]) * ep.inv_std[n]; v = t * ep.gamma[n] + ep.beta[n]; }
    if (ep.relu) v = v > T(0) ? v : T(0);
    return v;
}

constexpr int FMA_BK = 16;

template <int MODE, int BN, int TN>
__global__ void __launch_bounds__(256)
igemm_kernel(IgemmParams p, const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C,
             float* __restrict__ partial, Epilogue<float> ep)
{
    using T = float;
    pdl_prologue();
    constexpr int BM = 128, NT = 256, BK = FMA_BK;
    constexpr int A_PER = BM * BK / NT, B_PER = BN * BK / NT;
    constexpr int PADW = 16 / sizeof(T);
    __shared__ __align__(16) T As[2][BK][BM + PADW];
    __shared__ __align__(16) T Bs[2][BK][BN + PADW];
    __shared__ Info rowinfo[BM];
    __shared__ Info kinfo[2][BK];

    const int tid = threadIdx.x;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const int kbeg = blockIdx.z * p.k_chunk;
    const int kend = min(p.K, kbeg + p.k_chunk);
    const int nslice = (kend - kbeg + BK - 1) / BK;

    if (tid < BM)
        rowinfo[tid] = (MODE == MODE_WGRAD) ? decode_tap<MODE>(p, m0 + tid, p.M) : decode_pix<MODE>(p, m0 + tid, p.M);
    if (tid >= BM && tid < BM + BK) {
        int k = kbeg + (tid - BM);
        kinfo[0][tid - BM] = (MODE == MODE_WGRAD) ? decode_pix<MODE>(p, k, kend) : decode_tap<MODE>(p, k, kend);
    }
    __syncthreads();

    T ra[A_PER], rb[B_PER];
    auto fetch = [&](int buf) {
#pragma unroll
        for (int i = 0; i < A_PER; i++) {
            int e = tid + i * NT;
            int k = p.a_lanes_k ? (e % BK) : (e / BM);
            int m = p.a_lanes_k ? (e / BK) : (e % BM);
            const Info& ri = rowinfo[m];
            const Info& ki = kinfo[buf][k];
            int64_t off;
            bool ok = (MODE == MODE_WGRAD) ? gather_off<MODE>(p, ki, ri, off) : gather_off<MODE>(p, ri, ki, off);
            ra[i] = ok ? A[off] : T(0);
        }
#pragma unroll
        for (int i = 0; i < B_PER; i++) {
            int e = tid + i * NT;
            int k = p.b_lanes_k ? (e % BK) : (e / BN);
            int n = p.b_lanes_k ? (e / BK) : (e % BN);
            const Info& ki = kinfo[buf][k];
            bool ok = info_valid(ki) && (n0 + n) < p.N;
            rb[i] = ok ? B[ki.b_off + (int64_t)(n0 + n) * p.b_sn] : T(0);
        }
    };
    auto stash = [&](int buf) {
#pragma unroll
        for (int i = 0; i < A_PER; i++) {
            int e = tid + i * NT;
            int k = p.a_lanes_k ? (e % BK) : (e / BM);
            int m = p.a_lanes_k ? (e / BK) : (e % BM);
            As[buf][k][m] = ra[i];
        }
#pragma unroll
        for (int i = 0; i < B_PER; i++) {
            int e = tid + i * NT;
            int k = p.b_lanes_k ? (e % BK) : (e / BN);
            int n = p.b_lanes_k ? (e / BK) : (e % BN);
            Bs[buf][k][n] = rb[i];
        }
    };

    T acc[8][TN];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = T(0);

    const int tx = tid & 15, ty = tid >> 4;

    if (nslice > 0) {
        fetch(0);
        stash(0);
        if (tid < BK) {
            int k = kbeg + BK + tid;
            kinfo[1][tid] = (MODE == MODE_WGRAD) ? decode_pix<MODE>(p, k, kend) : decode_tap<MODE>(p, k, kend);
        }
    }
    __syncthreads();

    for (int s = 0; s < nslice; s++) {
        const int cur = s & 1;
        if (s + 1 < nslice) fetch(cur ^ 1);
#pragma unroll
        for (int k = 0; k < BK; k++) {
            T a[8], b[TN];
            T t4[4];
            lds4(&As[cur][k][ty * 4], t4);
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = t4[i];
            lds4(&As[cur][k][BM / 2 + ty * 4], t4);
#pragma unroll
            for (int i = 0; i < 4; i++) a[4 + i] = t4[i];
            {
                lds4(&Bs[cur][k][tx * 4], t4);
#pragma unroll
                for (int j = 0; j < 4; j++) b[j] = t4[j];
                if (TN == 8) {
                    lds4(&Bs[cur][k][BN / 2 + tx * 4], t4);
#pragma unroll
                    for (int j = 0; j < 4; j++) b[(TN == 8 ? 4 : 0) + j] = t4[j];
                }
            }
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
        if (s + 1 < nslice) {
            stash(cur ^ 1);
            if (tid < BK) {
                int k = kbeg + (s + 2) * BK + tid;
                kinfo[cur][tid] = (MODE == MODE_WGRAD) ? decode_pix<MODE>(p, k, kend) : decode_tap<MODE>(p, k, kend);
            }
        }
        __syncthreads();
    }

    // epilogue
#pragma unroll
    for (int i = 0; i < 8; i++) {
        int rl = (i < 4) ? (ty * 4 + i) : (BM / 2 + ty * 4 + i - 4);
        int m = m0 + rl;
        if (m >= p.M) continue;
        const int64_t row_off = rowinfo[rl].b_off;
#pragma unroll
        for (int j = 0; j < TN; j++) {
            int cl = (j < 4) ? (tx * 4 + j) : (BN / 2 + tx * 4 + j - 4);
            int n = n0 + cl;
            if (n >= p.N) continue;
            if (p.splits > 1) partial[((int64_t)blockIdx.z * p.M + m) * p.N + n] = acc[i][j];
            else C[row_off + (int64_t)n * p.c_sn] = apply_epilogue<T>(acc[i][j], n, ep);
        }
    }
}

// Forward pass of sums so short that gathering them is the work (a 3x3 filter on one channel): a thread owns a pixel and NC output
// channels, its operands come through L1 and the filter from shared memory.  The products of an output are added in the order of
// igemm_kernel, whose 128 x 64 tiles spend a slice of 16 on nine products and several block barriers: the first layer of a digit
// classifier (64 images of 28x28, 1 -> 16 channels) 13.0 -> 5.5 us.  Taken where short_fprop_pays.
constexpr int SHORT_K = 64;
template <int NC>
__global__ void __launch_bounds__(256)
short_fprop_kernel(IgemmParams p, const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C, Epilogue<float> ep, bool vec)
{
    pdl_prologue();
    __shared__ __align__(16) float w[SHORT_K][NC];
    __shared__ Info taps[SHORT_K];
    const int n0 = blockIdx.y * NC;
    for (int k = threadIdx.x; k < p.K; k += 256) taps[k] = decode_tap<MODE_FPROP>(p, k, p.K);
    __syncthreads();
    for (int i = threadIdx.x; i < p.K * NC; i += 256) {
        const int k = i / NC, n = n0 + i % NC;
        w[k][i % NC] = n < p.N ? B[taps[k].b_off + (int64_t)n * p.b_sn] : 0.f;
    }
    __syncthreads();
    const int m = blockIdx.x * 256 + threadIdx.x;
    if (m >= p.M) return;
    const Info pix = decode_pix<MODE_FPROP>(p, m, p.M);
    float acc[NC];
#pragma unroll
    for (int j = 0; j < NC; j++) acc[j] = 0.f;
#pragma unroll 4
    for (int k = 0; k < p.K; k++) {
        int64_t off;
        const float a = gather_off<MODE_FPROP>(p, pix, taps[k], off) ? __ldg(A + off) : 0.f;
#pragma unroll
        for (int j = 0; j < NC; j += 4) {
            const float4 q = *reinterpret_cast<const float4*>(&w[k][j]);
            acc[j] = fmaf(a, q.x, acc[j]); acc[j + 1] = fmaf(a, q.y, acc[j + 1]); acc[j + 2] = fmaf(a, q.z, acc[j + 2]); acc[j + 3] = fmaf(a, q.w, acc[j + 3]);
        }
    }
    float* d = C + pix.b_off + (int64_t)n0 * p.c_sn;
#pragma unroll
    for (int j = 0; j < NC; j++) if (n0 + j < p.N) acc[j] = apply_epilogue<float>(acc[j], n0 + j, ep);
    if (vec) {
#pragma unroll
        for (int j = 0; j < NC; j += 4) if (n0 + j < p.N) *reinterpret_cast<float4*>(d + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
    } else {
#pragma unroll
        for (int j = 0; j < NC; j++) if (n0 + j < p.N) d[j * p.c_sn] = acc[j];
    }
}

// ---- float64: the same implicit GEMM on the double-precision tensor pipe ----------------------------
// mma.m16n8k8 keeps the full FP64 rate (measured 37.0 TFLOP/s on register-resident chains, 35 with the fragment reads of
// this kernel; the FMA pipe reaches 33) with a sixteenth of the operand reads of 8 x 8 register blocks, which is what held
// the FMA form of this kernel to 14 TFLOP/s.  One CTA per SM = a 128 x BN tile: eight warps of 64 x 32 (BN = 128) or
// 32 x 32 (BN = 64) only read fragments and multiply, four more gather k-slices of 16 into a ring of stages with cp.async,
// zero-filled where a tap or an index is out of range.  The roles are separate because a warp issues in order: with the
// gather's address arithmetic between the products of the same warps the pipe stood idle 30 to 40 % of the time.
// An address is the sum of a row's and a k's offset, a bound check the sum of their coordinates (DInfo), and pairs of
// doubles go as one 16-byte copy where the channel count and the pointers allow: a slice of a 128-column tile is 16 copies
// a thread under 4096 cycles of products.
// Tiles in shared memory are [index][k] with rows of 20 or [k][index] with rows of 132 or 68 doubles, whichever way the
// source is contiguous: a row pitch of 4 modulo 16 doubles makes the fragments' (8 x 4) reads conflict-free either way.
// Consecutive warps lie along M so that a narrow N (whose unused 8-column steps are skipped) still feeds all four
// sub-partitions.
constexpr int DG_BK = 16, DG_KP = DG_BK + 4, DG_MMA = 256, DG_GATHER = 128, DG_THREADS = DG_MMA + DG_GATHER;

// A GEMM row or a k index: element (row, k) of A lies at off + off and is inside the tensor when the summed coordinates
// are; boff is a k's offset in B or a row's in C.  With 32-bit offsets it is one 16-byte read.
template <typename OFF> struct __align__(16) DInfo { OFF off; int d0, d1; OFF boff; };

template <int BN> constexpr int dg_tile_doubles() {
    return (128 * DG_KP > DG_BK * 132 ? 128 * DG_KP : DG_BK * 132) + (BN * DG_KP > DG_BK * (BN + 4) ? BN * DG_KP : DG_BK * (BN + 4));
}
// Stages of the ring: one is multiplied, one has landed, the others are on their way.  More than these leave less of the SM's memory to
// the L1 that copies of single doubles want (64 columns, six stages: 7x25x25 512->64 3x3 108 -> 112 us).
template <int BN> constexpr int dg_stages() { return BN == 128 ? 5 : 4; }
// The k's of DG_AHEAD slices are decoded at once, one by each gathering thread (slice by slice, by 16 of them with the others waiting, that
// was half of the 1.3 us a slice of a small launch took), into one of two places in turn.
constexpr int DG_AHEAD = DG_GATHER / DG_BK;
// The ring of slices, whose place the output tile takes on its way out: [row][32] of each warp's 32 columns, rows of DG_OUT doubles.
constexpr int DG_OUT = 34;
template <int BN> constexpr int dg_ring_doubles() {
    return dg_stages<BN>() * dg_tile_doubles<BN>() > 128 * (BN / 32) * DG_OUT ? dg_stages<BN>() * dg_tile_doubles<BN>() : 128 * (BN / 32) * DG_OUT;
}
template <int BN, typename OFF> constexpr size_t dg_smem_bytes() {
    return dg_ring_doubles<BN>() * sizeof(double) + (2 * DG_GATHER + 128) * sizeof(DInfo<OFF>);
}
template <int N> __device__ __forceinline__ void cp_async_doubles(uint32_t d, const double* src, bool ok) {
    if (N == 2) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(ok ? 16 : 0) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(ok ? 8 : 0) : "memory");
}
__device__ __forceinline__ void dmma_16x8x8(double (&c)[4], const double (&a)[4], const double (&b)[2]) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3]) : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// A strided input gradient runs per residue class (dgrad_class_params), inside which the division by the stride is exact:
// the row takes the quotient at the class's first tap and every further tap lowers it by lin_h.
template <typename OFF>
__device__ __forceinline__ DInfo<OFF> dinfo_pix(const IgemmParams& p, int mode, int idx, int limit) {
    DInfo<OFF> f{0, -B2C_SENTINEL, 0, 0};
    if (idx >= limit) return f;
    const int n = p.f_pq.div(idx), rem = idx - n * p.PQ;
    int pp = p.f_q.div(rem), qq = rem - pp * p.Q;
    pp = p.pix_h0 + pp * p.pix_hs; qq = p.pix_w0 + qq * p.pix_ws;
    if (mode == MODE_DGRAD) { f.d0 = (pp + p.vpad - p.tap_r0 * p.vdil) / p.vstr; f.d1 = (qq + p.hpad - p.tap_s0 * p.hdil) / p.hstr; }
    else { f.d0 = pp * p.vstr - p.vpad; f.d1 = qq * p.hstr - p.hpad; }
    f.off = (OFF)(n * p.a_sn + f.d0 * p.a_sh + f.d1 * p.a_sw);
    f.boff = (OFF)(n * p.pb_sn + pp * p.pb_sh + qq * p.pb_sw);
    return f;
}
template <typename OFF>
__device__ __forceinline__ DInfo<OFF> dinfo_tap(const IgemmParams& p, int mode, int idx, int limit) {
    DInfo<OFF> f{0, -B2C_SENTINEL, 0, 0};
    if (idx >= limit) return f;
    int c, r, s;
    int rs;
    if (p.tap_c_fast) { rs = p.f_c.div(idx); c = idx - rs * p.C; }
    else { c = p.f_rs.div(idx); rs = idx - c * (p.R * p.S); }
    r = p.f_s.div(rs); s = rs - r * p.S;
    if (mode == MODE_DGRAD) { f.d0 = -r * p.lin_h; f.d1 = -s * p.lin_w; }
    else { f.d0 = r * p.vdil; f.d1 = s * p.hdil; }
    f.off = (OFF)(c * p.a_sc + f.d0 * p.a_sh + f.d1 * p.a_sw);
    f.boff = (OFF)(c * p.tb_sc + (p.tap_r0 + r * p.tap_rs) * p.tb_sr + (p.tap_s0 + s * p.tap_ss) * p.tb_ss);
    return f;
}

// Named barriers: DG_FULL + stage (slice landed), DG_EMPTY + stage (slice read), DG_KS (among the gathering warps), DG_DONE (among
// the multiplying warps, behind the last slice).  The
// gathering warps wait for DG_EMPTY of slice s - stages before they refill its stage and report slice s - LAG = s - stages + 2 only
// after that; the multiplying warps need slices up to s - stages for it, all of them reported before: no cycle.  They have slice
// s - stages + 1 to multiply meanwhile (with the report one slice later they stood while slice s was issued: 28x28 256->256 3x3
// 1005 -> 1422 us forward).
enum { DG_FULL = 1, DG_EMPTY = 7, DG_KS = 13, DG_DONE = 14 };
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
// what this thread wrote or read before it is done when the barrier completes
__device__ __forceinline__ void bar_arrive(int id, int n) {
    __threadfence_block();
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// AK, BK_: the tile of A (B) is contiguous along k, else along its other index.  V doubles per copy.  OFF: offsets in A, B, C.
// TAIL: only the tiles past whole rounds of the chip are split (split_last_round_f64).  A form of its own: with its index arithmetic
// in the launches of a few microseconds a small float64 network took 755 us a step for 697.
template <int BN, bool AK, bool BK_, int V, typename OFF, bool TAIL>
__global__ void __launch_bounds__(DG_THREADS, 1)
dgemm_kernel(IgemmParams p, int mode, const double* __restrict__ A, const double* __restrict__ B,
             double* __restrict__ C, double* __restrict__ partial, Epilogue<double> ep)
{
    constexpr int BM = 128, BK = DG_BK, KP = DG_KP, NP = DG_GATHER, DG_STAGES = dg_stages<BN>(), LAG = DG_STAGES - 2;
    static_assert(LAG >= 1 && LAG <= 3 && DG_STAGES <= DG_EMPTY - DG_FULL && DG_STAGES <= DG_KS - DG_EMPTY, "a named barrier each way for every stage");
    constexpr int A_SIZE = 128 * KP > BK * 132 ? 128 * KP : BK * 132, TILE = dg_tile_doubles<BN>();
    constexpr int WM = BN == 128 ? 64 : 32, MI = WM / 16, WARPS_M = BM / WM;     // warp tile WM x 32
    constexpr int A_SI = AK ? KP : 1, A_SK = AK ? 1 : 132, B_SI = BK_ ? KP : 1, B_SK = BK_ ? 1 : BN + 4;   // strides of (index, k)
    extern __shared__ __align__(16) uint8_t dg_smem[];
    double* tiles = reinterpret_cast<double*>(dg_smem);
    DInfo<OFF>* kinfo = reinterpret_cast<DInfo<OFF>*>(dg_smem + dg_ring_doubles<BN>() * sizeof(double));
    DInfo<OFF>* rowinfo = kinfo + 2 * DG_GATHER;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int m_tile = blockIdx.x, n_tile = blockIdx.y, z = blockIdx.z;
    bool split = p.splits > 1;
    if constexpr (TAIL) {
        // one row of blocks over the tiles in row order, column tiles fastest: the first p.whole tiles are one block's, of the
        // others a block takes one of p.splits shares of the K loop
        const int nt = (p.N + BN - 1) / BN, rest = (p.M + BM - 1) / BM * nt - p.whole;
        split = m_tile >= p.whole;
        z = split ? (m_tile - p.whole) / rest : 0;
        const int tile = m_tile - z * rest;
        m_tile = tile / nt; n_tile = tile - m_tile * nt;
    }
    const int m0 = m_tile * BM, n0 = n_tile * BN;
    const int kbeg = z * p.k_chunk, kend = TAIL && !split ? p.K : min(p.K, kbeg + p.k_chunk);
    const int nslice = (kend - kbeg + BK - 1) / BK;
    if (tid < BM) rowinfo[tid] = mode == MODE_WGRAD ? dinfo_tap<OFF>(p, mode, m0 + tid, p.M) : dinfo_pix<OFF>(p, mode, m0 + tid, p.M);
    __syncthreads();

    if (warp >= DG_MMA / 32) {
        // ---------------- gather ----------------
        const int t = tid - DG_MMA;
        const int H = p.H, W = p.W, N = p.N;
        // copy e of a tile: V doubles from index (e % FAST) * V along memory, at index e / FAST of the other axis
        constexpr int A_FAST = (AK ? BK : BM) / V, A_CNT = BM * BK / V / NP, B_FAST = (BK_ ? BK : BN) / V, B_CNT = BN * BK / V / NP;
        const uint32_t tiles_s = (uint32_t)__cvta_generic_to_shared(tiles);
        int st = 0;
        bool first = true;
#pragma unroll 1
        for (int s = 0; s < nslice; s++) {
            DInfo<OFF>* block = kinfo + (s / DG_AHEAD & 1) * DG_GATHER;
            if (s % DG_AHEAD == 0) {                      // every thread is past the k's that lie there: it has met the barrier since
                const int k = kbeg + s * BK + t;
                block[t] = mode == MODE_WGRAD ? dinfo_pix<OFF>(p, mode, k, kend) : dinfo_tap<OFF>(p, mode, k, kend);
                bar_sync(DG_KS, NP);
            }
            if (first) { pdl_prologue(); first = false; }      // rows and k's are decoded while the kernel in front ends
            if (s >= DG_STAGES) bar_sync(DG_EMPTY + st, DG_THREADS);
            const DInfo<OFF>* kis = block + s % DG_AHEAD * BK;
            const uint32_t as = tiles_s + st * TILE * 8, bs = as + A_SIZE * 8;
#pragma unroll 8
            for (int i = 0; i < A_CNT; i++) {
                const int e = t + i * NP, f = e % A_FAST * V, x = e / A_FAST;
                const DInfo<OFF> &u = AK ? kis[f] : rowinfo[f], &w = AK ? rowinfo[x] : kis[x];
                const bool ok = (unsigned)(u.d0 + w.d0) < (unsigned)H && (unsigned)(u.d1 + w.d1) < (unsigned)W;
                cp_async_doubles<V>(as + 8 * (x * (AK ? KP : 132) + f), A + (ok ? u.off + w.off : 0), ok);
            }
#pragma unroll 8
            for (int i = 0; i < B_CNT; i++) {
                const int e = t + i * NP, f = e % B_FAST * V, x = e / B_FAST, n = n0 + (BK_ ? x : f);
                const DInfo<OFF>& ki = kis[BK_ ? f : x];
                const bool ok = ki.d0 > -(B2C_SENTINEL >> 1) && n < N;
                cp_async_doubles<V>(bs + 8 * (x * (BK_ ? KP : BN + 4) + f), B + (ok ? ki.boff + n * (OFF)p.b_sn : 0), ok);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            const int nxt = st + 1 == DG_STAGES ? 0 : st + 1, landed = st + 2 >= DG_STAGES ? st + 2 - DG_STAGES : st + 2;      // stage of slice s - LAG
            if (s >= LAG) {
                asm volatile("cp.async.wait_group %0;" ::"n"(LAG) : "memory");
                bar_arrive(DG_FULL + landed, DG_THREADS);
            }
            st = nxt;
        }
        // the last LAG slices one by one; st is the stage of the slice behind the last one
        auto rest = [&](auto left_c) {
            constexpr int left = decltype(left_c)::value;          // slices behind this one
            if (nslice > left) {
                asm volatile("cp.async.wait_group %0;" ::"n"(left) : "memory");
                int at = st - 1 - left;
                if (at < 0) at += DG_STAGES;
                bar_arrive(DG_FULL + at, DG_THREADS);
            }
        };
        if (LAG > 2) rest(std::integral_constant<int, 2>{}); rest(std::integral_constant<int, 1>{}); rest(std::integral_constant<int, 0>{});
        return;
    }

    // ---------------- products ----------------
    pdl_prologue();
    const int wm = (warp % WARPS_M) * WM, wn = (warp / WARPS_M) * 32;
    const int g = lane >> 2, t = lane & 3;
    int nj = (p.N - n0 - wn + 7) / 8;            // 8-column steps of this warp that hold columns of the output
    nj = nj < 0 ? 0 : nj > 4 ? 4 : nj;
    double acc[MI][4][4];
#pragma unroll
    for (int i = 0; i < MI; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[i][j][e] = 0.0;
    // k of a thread's two operand slots in an 8-step: t and t + 4, or with both tiles along k the pair 2t, 2t + 1 (one
    // 16-byte read; any assignment serves as long as A and B agree)
    constexpr bool PAIR = AK && BK_;
    const double* a_src = tiles + (wm + g) * A_SI + (PAIR ? 2 * t : t) * A_SK;
    const double* b_src = tiles + A_SIZE + (wn + g) * B_SI + (PAIR ? 2 * t : t) * B_SK;
    int st = 0;
#pragma unroll 1
    for (int s = 0; s < nslice; s++) {
        bar_sync(DG_FULL + st, DG_THREADS);
        const double *as = a_src + st * TILE, *bs = b_src + st * TILE;
        if (nj > 0) {
#pragma unroll
            for (int kk = 0; kk < BK; kk += 8) {
                double a[MI][4], b[4][2];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const double* q = bs + j * 8 * B_SI + kk * B_SK;
                    if (PAIR) { const double2 u = *reinterpret_cast<const double2*>(q); b[j][0] = u.x; b[j][1] = u.y; }
                    else { b[j][0] = q[0]; b[j][1] = q[4 * B_SK]; }
                }
#pragma unroll
                for (int i = 0; i < MI; i++) {
                    const double *q = as + i * 16 * A_SI + kk * A_SK, *q8 = q + 8 * A_SI;
                    if (PAIR) {
                        const double2 u = *reinterpret_cast<const double2*>(q), w = *reinterpret_cast<const double2*>(q8);
                        a[i][0] = u.x; a[i][2] = u.y; a[i][1] = w.x; a[i][3] = w.y;
                    } else { a[i][0] = q[0]; a[i][1] = q8[0]; a[i][2] = q[4 * A_SK]; a[i][3] = q8[4 * A_SK]; }
                }
#pragma unroll
                for (int i = 0; i < MI; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        if (j < nj) dmma_16x8x8(acc[i][j], a[i], b[j]);
            }
        }
        // the last DG_STAGES slices are not refilled: nobody waits for their stages
        if (s + DG_STAGES < nslice) bar_arrive(DG_EMPTY + st, DG_THREADS);
        st = st + 1 == DG_STAGES ? 0 : st + 1;
    }

    // The way out: the tile goes through shared memory to a loop of few instructions.  Written from the registers, 64 values a
    // thread with the epilogue's steps beside each, it was 30 KB of code that a launch runs through once, and a small one waited
    // for instructions most of its time (32x4x4 32->128 1x1: 18.7 us, of which 4.2 are products).  A store's lanes lie along
    // whichever of rows and columns is contiguous.
    bar_sync(DG_DONE, DG_MMA);                   // nobody reads the ring any more
    double* out = tiles + warp * (WM * DG_OUT);
#pragma unroll
    for (int i = 0; i < MI; i++)
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int j = 0; j < 4; j++)
                *reinterpret_cast<double2*>(out + (i * 16 + h * 8 + g) * DG_OUT + j * 8 + 2 * t) = make_double2(acc[i][j][2 * h], acc[i][j][2 * h + 1]);
    __syncwarp();
    const bool part = TAIL ? split : p.splits > 1;
    const int n_end = min(32, p.N - n0 - wn), m_end = min(WM, p.M - m0 - wm);       // what the warp has of columns and rows
    const DInfo<OFF>* rows = rowinfo + wm;
    if (part || p.c_sn == 1) {
        if (lane >= n_end) return;
        const int n = n0 + wn + lane;
        if (part) {
            double* d = partial + ((TAIL ? (int64_t)z * (p.M - p.m_whole) - p.m_whole : (int64_t)z * p.M) + m0 + wm) * p.N + n;
#pragma unroll 8
            for (int r = 0; r < m_end; r++) d[(int64_t)r * p.N] = out[r * DG_OUT + lane];
        } else {
            const ChannelEpilogue<double> own(ep, n);
#pragma unroll 8
            for (int r = 0; r < m_end; r++) C[rows[r].boff + n] = own(out[r * DG_OUT + lane]);
        }
    } else {
        for (int r = lane; r < m_end; r += 32) {
            double* d = C + rows[r].boff + (int64_t)(n0 + wn) * p.c_sn;
#pragma unroll 4
            for (int c = 0; c < n_end; c++) d[c * p.c_sn] = apply_epilogue<double>(out[r * DG_OUT + c], n0 + wn + c, ep);
        }
    }
}

// Second stage of split-K: fixed-order sum over the splits, epilogue, scatter to the output.  Block (32, ROWS): the thread
// rows share the splits (row y adds splits y, y + ROWS, .. in order, then the rows are added in order).  ROWS = 8 for many
// splits: a thread's chain of loads is one L2 round trip instead of eight (11 -> 4 us on a 144 x 16 filter cut 128 times).
template <typename T, int MODE, int ROWS>
__global__ void __launch_bounds__(256) splitk_reduce_kernel(IgemmParams p, const T* __restrict__ partial, T* __restrict__ C, Epilogue<T> ep)
{
    constexpr int COLS = 256 / ROWS;
    __shared__ T part[ROWS][COLS];
    const int64_t idx = (int64_t)blockIdx.x * COLS + threadIdx.x, total = (int64_t)(p.M - p.m_whole) * p.N;
    // where the sum goes is worked out while the kernel in front ends
    int64_t to = 0;
    int n = 0;
    if (idx < total && threadIdx.y == 0) {
        const int row = (int)(idx / p.N), m = p.m_whole + row;
        n = (int)(idx - (int64_t)row * p.N);
        const Info ri = (MODE == MODE_WGRAD) ? decode_tap<MODE>(p, m, p.M) : decode_pix<MODE>(p, m, p.M);
        to = ri.b_off + (int64_t)n * p.c_sn;
    }
    pdl_prologue();
    T v = T(0);
    if (idx < total) {
        int z = threadIdx.y;
        for (; z + 7 * ROWS < p.splits; z += 8 * ROWS) {          // eight independent loads
            T q[8];
#pragma unroll
            for (int u = 0; u < 8; u++) q[u] = partial[(int64_t)(z + u * ROWS) * total + idx];
#pragma unroll
            for (int u = 0; u < 8; u++) v += q[u];
        }
        for (; z < p.splits; z += ROWS) v += partial[(int64_t)z * total + idx];
    }
    if (ROWS > 1) {
        part[threadIdx.y][threadIdx.x] = v;
        __syncthreads();
        if (threadIdx.y != 0) return;
#pragma unroll
        for (int y = 1; y < ROWS; y++) v += part[y][threadIdx.x];
    }
    if (idx >= total) return;
    C[to] = apply_epilogue<T>(v, n, ep);
}

// Index map of the lowering, numbered as the reference numbers rows and columns.
__global__ void index_map_kernel(IgemmParams p, int64_t* __restrict__ map, int nchw)
{
    pdl_prologue();
    int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t total = (int64_t)p.M * p.K;
    if (idx >= total) return;
    int m, t;
    if (nchw) { t = (int)(idx / p.M); m = (int)(idx - (int64_t)t * p.M); }
    else { m = (int)(idx / p.K); t = (int)(idx - (int64_t)m * p.K); }
    Info pix = decode_pix<MODE_FPROP>(p, m, p.M);
    Info tap = decode_tap<MODE_FPROP>(p, t, p.K);
    int64_t off;
    bool ok = gather_off<MODE_FPROP>(p, pix, tap, off);
    map[idx] = ok ? off : -1;
}

// ---- fully connected layer: weight gradient as an outer-product sum ---------------------------------
// dw[i][o] = sum_b x[b][i] * dy[b][o] for a (batch, in) input, a (batch, out) output gradient and an (in, out)
// row-major weight matrix (pydtnn/backends/cpu/layers/fc_cpu.py:66-71).  The sum is over the batch only (32-64
// terms), so the pass is bound by writing dw; the general kernel above spends its time on gather arithmetic that a
// dense matrix does not need.  One CTA = one 128 x 128 tile of dw, all of the batch, 8 x 8 outputs per thread.
__device__ __forceinline__ void ldg4(const float* p, float (&o)[4]) {
    float4 v = __ldg(reinterpret_cast<const float4*>(p)); o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
}
__device__ __forceinline__ void sts4(float* p, const float (&v)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}

__global__ void __launch_bounds__(256)
fc_wgrad_kernel(const float* __restrict__ x, const float* __restrict__ dy, float* __restrict__ dw, int batch, int in_f, int out_f)
{
    using T = float;
    pdl_prologue();
    constexpr int BT = 128, KC = FMA_BK, PER = KC * BT / 4 / 256;     // 4-element vectors per thread per tile
    __shared__ __align__(16) T xs[2][KC][BT];
    __shared__ __align__(16) T ds[2][KC][BT];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int o0 = blockIdx.x * BT, i0 = blockIdx.y * BT;
    T rx[PER][4], rd[PER][4];
    auto fetch = [&](int b0) {
#pragma unroll
        for (int j = 0; j < PER; j++) {
            const int v = tid + j * 256, k = v / (BT / 4), col = (v % (BT / 4)) * 4;
            const bool row_ok = b0 + k < batch;
            if (row_ok && i0 + col < in_f) ldg4(x + (int64_t)(b0 + k) * in_f + i0 + col, rx[j]);
            else { rx[j][0] = rx[j][1] = rx[j][2] = rx[j][3] = T(0); }
            if (row_ok && o0 + col < out_f) ldg4(dy + (int64_t)(b0 + k) * out_f + o0 + col, rd[j]);
            else { rd[j][0] = rd[j][1] = rd[j][2] = rd[j][3] = T(0); }
        }
    };
    auto stash = [&](int buf) {
#pragma unroll
        for (int j = 0; j < PER; j++) {
            const int v = tid + j * 256, k = v / (BT / 4), col = (v % (BT / 4)) * 4;
            sts4(&xs[buf][k][col], rx[j]);
            sts4(&ds[buf][k][col], rd[j]);
        }
    };
    T acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = T(0);
    const int nchunk = (batch + KC - 1) / KC;
    fetch(0);
    stash(0);
    __syncthreads();
    for (int c = 0; c < nchunk; c++) {
        const int cur = c & 1;
        if (c + 1 < nchunk) fetch((c + 1) * KC);
#pragma unroll
        for (int k = 0; k < KC; k++) {
            T a[8], b[8], t4[4];
            lds4(&xs[cur][k][ty * 4], t4);
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = t4[i];
            lds4(&xs[cur][k][BT / 2 + ty * 4], t4);
#pragma unroll
            for (int i = 0; i < 4; i++) a[4 + i] = t4[i];
            lds4(&ds[cur][k][tx * 4], t4);
#pragma unroll
            for (int j = 0; j < 4; j++) b[j] = t4[j];
            lds4(&ds[cur][k][BT / 2 + tx * 4], t4);
#pragma unroll
            for (int j = 0; j < 4; j++) b[4 + j] = t4[j];
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
        if (c + 1 < nchunk) stash(cur ^ 1);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int row = i0 + ((i < 4) ? (ty * 4 + i) : (BT / 2 + ty * 4 + i - 4));
        if (row >= in_f) continue;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int col = o0 + h * (BT / 2) + tx * 4;
            if (col >= out_f) continue;
            const T v[4] = {acc[i][4 * h], acc[i][4 * h + 1], acc[i][4 * h + 2], acc[i][4 * h + 3]};
            sts4(dw + (int64_t)row * out_f + col, v);
        }
    }
}

// ---- fully connected layers with a small weight matrix ------------------------------------------------
// The last layer of a small classifier (128 x 10 and the like): a GEMM kernel's start-up, its second stage and the separate
// bias sum are all there is to such a layer, so each direction is one launch of plain dot products whose operands stay in L1.
// Weights up to 16 K elements; with more, re-reading them per batch row costs more than the launches saved.
// Sums are in double and rounded once: a float32 sum in eight parts is up to 1.3 times further from float64 than one chain of
// FMAs (5 rows), and the bias gradient of every other route is a sum in double.
bool fc_tiny(int batch, int in_f, int out_f) { return batch <= 512 && (int64_t)in_f * out_f <= (1 << 14); }

// y[b][o]: block = 32 outputs x 8 parts of the sum over the inputs, one batch row.
template <typename T>
__global__ void __launch_bounds__(256) fc_tiny_forward_kernel(const T* __restrict__ x, const T* __restrict__ w, const T* __restrict__ bias,
                                                              T* __restrict__ y, int in_f, int out_f)
{
    pdl_prologue();
    __shared__ double part[8][33];
    const int o = blockIdx.x * 32 + threadIdx.x;
    const T* xr = x + (int64_t)blockIdx.y * in_f;
    double v = 0.0;
    if (o < out_f) {
#pragma unroll 8
        for (int i = threadIdx.y; i < in_f; i += 8) v = fma((double)__ldg(xr + i), (double)__ldg(w + (int64_t)i * out_f + o), v);
    }
    part[threadIdx.y][threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.y != 0 || o >= out_f) return;
#pragma unroll
    for (int k = 1; k < 8; k++) v += part[k][threadIdx.x];
    y[(int64_t)blockIdx.y * out_f + o] = (T)(bias ? v + (double)bias[o] : v);
}

// The first dw_blocks blocks: dw[i][o] and db[o] (the row i = in_f), 32 outputs x 8 parts of the sum over the batch; the
// rest: dx[b][i], a thread each.
template <typename T>
__global__ void __launch_bounds__(256) fc_tiny_backward_kernel(const T* __restrict__ x, const T* __restrict__ dy, const T* __restrict__ w,
                                                               T* __restrict__ dw, T* __restrict__ db, T* __restrict__ dx, int batch, int in_f, int out_f,
                                                               int dw_blocks)
{
    pdl_prologue();
    __shared__ double part[8][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    if ((int)blockIdx.x < dw_blocks) {
        const int nt = (out_f + 31) / 32, i = blockIdx.x / nt, o = (blockIdx.x - i * nt) * 32 + tx;
        double v = 0.0;
        if (o < out_f) {
            if (i < in_f) {
#pragma unroll 8
                for (int b = ty; b < batch; b += 8) v = fma((double)__ldg(x + (int64_t)b * in_f + i), (double)__ldg(dy + (int64_t)b * out_f + o), v);
            } else {
#pragma unroll 8
                for (int b = ty; b < batch; b += 8) v += (double)__ldg(dy + (int64_t)b * out_f + o);
            }
        }
        part[ty][tx] = v;
        __syncthreads();
        if (ty != 0 || o >= out_f) return;
#pragma unroll
        for (int k = 1; k < 8; k++) v += part[k][tx];
        if (i < in_f) { if (dw) dw[(int64_t)i * out_f + o] = (T)v; }
        else if (db) db[o] = (T)v;
        return;
    }
    const int64_t e = (int64_t)(blockIdx.x - dw_blocks) * 256 + threadIdx.x;
    if (e >= (int64_t)batch * in_f) return;
    const int b = (int)(e / in_f), i = (int)(e - (int64_t)b * in_f);
    const T *d = dy + (int64_t)b * out_f, *wr = w + (int64_t)i * out_f;
    double v = 0.0;
#pragma unroll 8
    for (int o = 0; o < out_f; o++) v = fma((double)__ldg(d + o), (double)__ldg(wr + o), v);
    dx[e] = (T)v;
}

template <typename T>
static int fc_tiny_forward_t(int batch, int in_f, int out_f, const void* x, const void* w, const void* bias, void* y, cudaStream_t st)
{
    launch_pdl(fc_tiny_forward_kernel<T>, dim3((out_f + 31) / 32, batch), dim3(32, 8), 0, st, (const T*)x, (const T*)w, (const T*)bias, (T*)y, in_f, out_f);
    return check_launch("fc_tiny_forward_kernel");
}
int fc_tiny_forward(int dtype, int batch, int in_f, int out_f, const void* x, const void* w, const void* bias, void* y, cudaStream_t st)
{
    return dtype == B2C_F32 ? fc_tiny_forward_t<float>(batch, in_f, out_f, x, w, bias, y, st) : fc_tiny_forward_t<double>(batch, in_f, out_f, x, w, bias, y, st);
}
template <typename T>
static int fc_tiny_backward_t(int batch, int in_f, int out_f, const void* x, const void* dy, const void* w, void* dw, void* db, void* dx, cudaStream_t st)
{
    const int dw_blocks = dw ? (in_f + (db ? 1 : 0)) * ((out_f + 31) / 32) : 0;
    const int dx_blocks = dx ? (int)(((int64_t)batch * in_f + 255) / 256) : 0;
    if (dw_blocks + dx_blocks == 0) return B2C_OK;
    launch_pdl(fc_tiny_backward_kernel<T>, dw_blocks + dx_blocks, 256, 0, st, (const T*)x, (const T*)dy, (const T*)w, (T*)dw, (T*)db, (T*)dx, batch, in_f, out_f, dw_blocks);
    return check_launch("fc_tiny_backward_kernel");
}
int fc_tiny_backward(int dtype, int batch, int in_f, int out_f, const void* x, const void* dy, const void* w, void* dw, void* db, void* dx, cudaStream_t st)
{
    return dtype == B2C_F32 ? fc_tiny_backward_t<float>(batch, in_f, out_f, x, dy, w, dw, db, dx, st)
                            : fc_tiny_backward_t<double>(batch, in_f, out_f, x, dy, w, dw, db, dx, st);
}

static bool is_dense_fc(const Geo& g)
{
    return g.layout == B2C_LAYOUT_NHWC && g.w_layout == B2C_W_CRSK && g.h == 1 && g.w == 1 && g.kh == 1 && g.kw == 1 &&
           g.vpad == 0 && g.hpad == 0 && g.ci % 4 == 0 && g.co % 4 == 0 && g.dtype == B2C_F32;
}

// ---- host side ----------------------------------------------------------------------------

static IgemmParams make_params(const Geo& g, int mode)
{
    IgemmParams p{};
    ActStride xs = act_stride(g.layout, g.h, g.w, g.ci);
    ActStride ys = act_stride(g.layout, g.ho, g.wo, g.co);
    WStride ws = w_stride(g.w_layout, g.ci, g.co, g.kh, g.kw);
    const bool nhwc = g.layout == B2C_LAYOUT_NHWC;
    p.R = g.kh; p.S = g.kw;
    p.vstr = g.vstr; p.hstr = g.hstr; p.vpad = g.vpad; p.hpad = g.hpad; p.vdil = g.vdil; p.hdil = g.hdil;
    p.relu = 0; p.splits = 1;
    p.pix_h0 = 0; p.pix_hs = 1; p.pix_w0 = 0; p.pix_ws = 1;
    p.tap_r0 = 0; p.tap_rs = 1; p.tap_s0 = 0; p.tap_ss = 1; p.lin_h = g.vdil; p.lin_w = g.hdil;
    if (mode == MODE_FPROP) {
        p.M = (int)g.M; p.N = g.co; p.K = (int)g.K;
        p.P = g.ho; p.Q = g.wo; p.C = g.ci; p.H = g.h; p.W = g.w;
        p.a_sn = xs.sn; p.a_sh = xs.sh; p.a_sw = xs.sw; p.a_sc = xs.sc;
        p.pb_sn = ys.sn; p.pb_sh = ys.sh; p.pb_sw = ys.sw; p.c_sn = ys.sc;
        p.tb_sc = ws.sc; p.tb_sr = ws.sr; p.tb_ss = ws.ss; p.b_sn = ws.sk;
        p.tap_c_fast = nhwc; p.a_lanes_k = nhwc;
        p.b_lanes_k = (g.w_layout != B2C_W_CRSK);
    } else if (mode == MODE_DGRAD) {
        p.M = g.n * g.h * g.w; p.N = g.ci; p.K = g.co * g.kh * g.kw;
        p.P = g.h; p.Q = g.w; p.C = g.co; p.H = g.ho; p.W = g.wo;
        p.a_sn = ys.sn; p.a_sh = ys.sh; p.a_sw = ys.sw; p.a_sc = ys.sc;
        p.pb_sn = xs.sn; p.pb_sh = xs.sh; p.pb_sw = xs.sw; p.c_sn = xs.sc;
        p.tb_sc = ws.sk; p.tb_sr = ws.sr; p.tb_ss = ws.ss; p.b_sn = ws.sc;
        p.tap_c_fast = nhwc; p.a_lanes_k = nhwc;
        p.b_lanes_k = (g.w_layout != B2C_W_KRSC);
    } else {
        p.M = (int)g.K; p.N = g.co; p.K = (int)g.M;
        p.P = g.ho; p.Q = g.wo; p.C = g.ci; p.H = g.h; p.W = g.w;
        p.a_sn = xs.sn; p.a_sh = xs.sh; p.a_sw = xs.sw; p.a_sc = xs.sc;
        p.pb_sn = ys.sn; p.pb_sh = ys.sh; p.pb_sw = ys.sw; p.b_sn = ys.sc;
        p.tb_sc = ws.sc; p.tb_sr = ws.sr; p.tb_ss = ws.ss; p.c_sn = ws.sk;
        p.tap_c_fast = nhwc;          // rows run over taps: channel fastest keeps NHWC loads contiguous
        p.a_lanes_k = !nhwc;          // NCHW: pixels are contiguous
        p.b_lanes_k = !nhwc;
    }
    p.PQ = p.P * p.Q;
    // a row's offset alone may lie a window outside the tensor
    const int64_t over_h = (int64_t)g.kh * g.vdil + g.vpad, over_w = (int64_t)g.kw * g.hdil + g.hpad;
    p.small = (int64_t)g.n * (g.h + 2 * over_h) * (g.w + 2 * over_w) * g.ci < (1LL << 31) && (int64_t)g.n * (g.ho + 2 * over_h) * (g.wo + 2 * over_w) * g.co < (1LL << 31) &&
              g.K * g.co < (1LL << 31);
    return p;
}

static int tile_bn(int N) { return N <= 64 ? 64 : 128; }

// Number of K splits: enough CTAs to fill the 148 SMs about twice, each split at least 8 slices.
static int choose_splits(const IgemmParams& p, int bk)
{
    int64_t ctas = (int64_t)((p.M + 127) / 128) * ((p.N + tile_bn(p.N) - 1) / tile_bn(p.N));
    if (ctas >= tc_sm_count()) return 1;
    int64_t want = (2 * tc_sm_count() + ctas - 1) / ctas;
    int64_t max_by_k = p.K / (8 * bk);
    if (max_by_k < 1) max_by_k = 1;
    int64_t s = want < max_by_k ? want : max_by_k;
    if (s > 128) s = 128;
    return (int)s;
}

// The float64 tensor kernel holds one CTA per SM: the split count that needs the least time by rounds of the chip x (slices of a
// split + about three for its start and its drain, six with its share of the second stage).  Tiles of 128 columns that leave half of the
// chip idle may be two of 64, whose slices take two thirds of the time (1.4 us of 2.1, 1.8 where doubles are copied one by one; the starts half as long): 32x4x4 32->128
// 1x1 15.6 -> 8.4 us, while 5x7x48 256->512 3x3, 144 slices, is 166 us by 128 columns and 210 by 64.
struct F64Plan { int bn, splits; };
static F64Plan plan_f64(const IgemmParams& p, int bk)
{
    F64Plan best{};
    double cost = 0.0;
    const int64_t room = tc_sm_count(), slices = (p.K + bk - 1) / bk;
    for (int bn = p.N <= 64 ? 64 : 128; bn >= 64; bn -= 64) {
        const int64_t ctas = (int64_t)((p.M + 127) / 128) * ((p.N + bn - 1) / bn);
        if (best.bn && ctas > room) break;
        const double slice = bn == 128 || !best.bn ? 1.0 : p.tap_c_fast && p.C % 2 == 0 ? 0.67 : 0.85, start = best.bn ? 0.5 : 1.0;
        for (int64_t s = 1; s <= 128 && s <= slices && (s == 1 || ctas * s <= 2 * room); s++) {
            const double c = (double)((ctas * s + room - 1) / room) * ((double)((slices + s - 1) / s) * slice + (s > 1 ? 6.0 : 3.0) * start);
            if (!best.bn || c < (bn == best.bn ? 1.0 : 0.95) * cost) { best = F64Plan{bn, (int)s}; cost = c; }
        }
    }
    return best;
}

// More than one round of whole float64 tiles: the 392 of a 28x28 256->256 3x3 layer, batch 32, are 2.65 rounds on 148 SMs that ran as
// three.  Row tiles that fill whole rounds stay whole, the K loops of the others are split so that they fill the chip too (that
// layer, three passes: 3168 -> 2987 us).  Costs in slices of 128 columns (2.1 us) as in plan_f64; a whole tile takes a
// twentieth longer in the form with a tail, and a MB of partial sums 0.2 (0.4 of the narrow tiles' slices).  Without these two a tail saved
// nothing where K loops are short: 1x1 512->128 of 7040 pixels 66 us whole, 76 with a tail.  By this rule 1716 of 1979 passes
// measured (5 to 300 slices) have one, 1.27 times as fast on average; 48 of them are slower than whole by more than 1 %.
static void split_last_round_f64(IgemmParams& p, int bk)
{
    const int64_t nt = (p.N + tile_bn(p.N) - 1) / tile_bn(p.N), ctas = (int64_t)((p.M + 127) / 128) * nt, room = tc_sm_count(), slices = (p.K + bk - 1) / bk;
    const int64_t rows = ctas / room * room / nt, whole = rows * nt, rest = ctas - whole;         // row tiles that fill whole rounds
    if (ctas <= room || !rows || !rest) return;
    int64_t best = 1;
    double cost = (double)((ctas + room - 1) / room * (slices + 3));
    const double split_mb = (double)(p.M - rows * 128) * p.N * 8e-6 * (tile_bn(p.N) == 64 ? 0.4 : 0.2);
    for (int64_t s = 2; s <= 16 && s <= slices; s++) {
        const double c = (double)((whole + room - 1) / room) * (1.05 * (double)slices + 3.0) +
                         (double)((rest * s + room - 1) / room * ((slices + s - 1) / s + 6)) + (double)s * split_mb;
        if (c < cost) { best = s; cost = c; }
    }
    if (best == 1) return;
    p.k_chunk = (int)(((slices + best - 1) / best) * bk);
    p.splits = (p.K + p.k_chunk - 1) / p.k_chunk;
    p.whole = (int)whole; p.m_whole = (int)(rows * 128);
}

static void finish_params(IgemmParams& p, int dtype)
{
    const int bk = 16;
    static_assert(FMA_BK == 16 && DG_BK == 16, "k-chunks are whole slices of either kernel");
    p.bn = tile_bn(p.N);
    if (p.K <= 0) { p.splits = 1; p.k_chunk = bk; return; }        // no taps reach these pixels: the launch writes zeros
    if (dtype == B2C_F32) p.splits = choose_splits(p, bk);
    else { const F64Plan plan = plan_f64(p, bk); p.splits = plan.splits; p.bn = plan.bn; }
    int chunk = (p.K + p.splits - 1) / p.splits;
    chunk = (chunk + bk - 1) / bk * bk;
    p.k_chunk = chunk;
    p.splits = (p.K + chunk - 1) / chunk;
    p.whole = p.m_whole = 0;
    if (p.splits == 1 && dtype != B2C_F32 && p.bn == tile_bn(p.N)) split_last_round_f64(p, bk);
}
static size_t partial_bytes(const IgemmParams& p, size_t es) { return p.splits > 1 ? (size_t)p.splits * (p.M - p.m_whole) * p.N * es : 0; }

// Strided dgrad: input pixel (h, w) only receives taps with r * vdil = h + vpad, s * hdil = w + hpad (mod the strides).
// Class (a, b) of those residues is a dense problem over its own pixels and taps; gathering all taps for all pixels instead
// would spend (vstr*hstr - 1) / (vstr*hstr) of the inner loop on zeros.
static bool dgrad_by_class(const Geo& g) { return g.vstr > 1 || g.hstr > 1; }

// The taps r < k with r * dil = a (mod str): first, step and count; one step moves the gathered position by lin.
static void class_taps(int a, int str, int dil, int k, int& first, int& step, int& count, int& lin)
{
    int x = dil, y = str;
    while (y) { const int t = x % y; x = y; y = t; }
    step = str / x; lin = dil / x;
    first = 0; count = 0;
    for (int r = 0; r < k && r < str; r++)
        if ((int64_t)r * dil % str == a) { first = r; count = (k - r + step - 1) / step; break; }
}

static IgemmParams dgrad_class_params(const Geo& g, int a, int b)
{
    IgemmParams p = make_params(g, MODE_DGRAD);
    const int h0 = ((a - g.vpad) % g.vstr + g.vstr) % g.vstr, w0 = ((b - g.hpad) % g.hstr + g.hstr) % g.hstr;
    p.pix_h0 = h0; p.pix_hs = g.vstr; p.pix_w0 = w0; p.pix_ws = g.hstr;
    p.P = h0 < g.h ? (g.h - h0 + g.vstr - 1) / g.vstr : 0;
    p.Q = w0 < g.w ? (g.w - w0 + g.hstr - 1) / g.hstr : 0;
    p.PQ = p.P * p.Q;
    p.M = g.n * p.PQ;
    class_taps(a, g.vstr, g.vdil, g.kh, p.tap_r0, p.tap_rs, p.R, p.lin_h);
    class_taps(b, g.hstr, g.hdil, g.kw, p.tap_s0, p.tap_ss, p.S, p.lin_w);
    p.K = g.co * p.R * p.S;
    return p;
}

size_t fma_workspace_bytes(const Geo& g, int pass)
{
    size_t es = g.dtype == B2C_F32 ? 4 : 8;
    if (pass == B2C_PASS_DGRAD && dgrad_by_class(g)) {
        size_t most = 0;
        for (int a = 0; a < g.vstr; a++)
            for (int b = 0; b < g.hstr; b++) {
                IgemmParams p = dgrad_class_params(g, a, b);
                if (p.M == 0) continue;
                finish_params(p, g.dtype);
                size_t bytes = partial_bytes(p, es);
                if (bytes > most) most = bytes;
            }
        return most;
    }
    IgemmParams p = make_params(g, pass);
    finish_params(p, g.dtype);
    size_t bytes = partial_bytes(p, es);
    if (pass == B2C_PASS_WGRAD) bytes = align_up(bytes, 256) + channel_sum_workspace_bytes(g.n, g.co, g.ho * g.wo);
    return bytes;
}

template <int BN, bool AK, bool BK_, int V, typename OFF, bool TAIL = false>
static int launch_dgemm_v(const IgemmParams& p, int mode, dim3 grid, const double* A, const double* B, double* C, double* ws, const Epilogue<double>& ep, cudaStream_t st)
{
    // once per device: the attribute belongs to the device's copy of the kernel
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev > 63) dev = 63;
    if (dev == 63 || !(done.load() >> dev & 1)) {
        const cudaError_t e = cudaFuncSetAttribute(dgemm_kernel<BN, AK, BK_, V, OFF, TAIL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dg_smem_bytes<BN, OFF>());
        if (e != cudaSuccess) { set_cuda_error(e, "cudaFuncSetAttribute(dgemm_kernel)"); return B2C_ERR_CUDA; }
        done.fetch_or(1ull << dev);
    }
    launch_pdl(dgemm_kernel<BN, AK, BK_, V, OFF, TAIL>, grid, DG_THREADS, dg_smem_bytes<BN, OFF>(), st, p, mode, A, B, C, ws, ep);
    return B2C_OK;          // the caller checks the launch
}

template <int BN>
static int launch_dgemm(const IgemmParams& p, int mode, dim3 grid, const double* A, const double* B, double* C, double* ws, const Epilogue<double>& ep, cudaStream_t st)
{
    // Pairs of doubles per copy: the index that runs along memory must step by one element, keep a pair inside one tap and
    // one bound (an even channel count), and every other stride and the pointer must be even.
    const bool a_pair = p.a_sc == 1 && p.tap_c_fast && p.C % 2 == 0 && ((p.a_sn | p.a_sh | p.a_sw) & 1) == 0 && ((uintptr_t)A & 15) == 0;
    // B(k, n): along k it is a filter's channel axis, along n the output channels of a filter or of dy
    bool b_pair = ((uintptr_t)B & 15) == 0;
    if (p.b_lanes_k) b_pair = b_pair && mode != MODE_WGRAD && p.tap_c_fast && p.tb_sc == 1 && p.C % 2 == 0 && ((p.tb_sr | p.tb_ss | p.b_sn) & 1) == 0;
    else b_pair = b_pair && p.b_sn == 1 && p.N % 2 == 0 &&
                  ((mode == MODE_WGRAD ? (p.pb_sn | p.pb_sh | p.pb_sw) : (p.tb_sc | p.tb_sr | p.tb_ss)) & 1) == 0;
    const bool pairs = a_pair && b_pair && p.small;         // small: every offset fits 31 bits
#define B2C_DG(AK, BK_) (p.whole ? (pairs ? launch_dgemm_v<BN, AK, BK_, 2, int, true>(p, mode, grid, A, B, C, ws, ep, st) : launch_dgemm_v<BN, AK, BK_, 1, int64_t, true>(p, mode, grid, A, B, C, ws, ep, st)) \
                         : pairs ? launch_dgemm_v<BN, AK, BK_, 2, int>(p, mode, grid, A, B, C, ws, ep, st) : launch_dgemm_v<BN, AK, BK_, 1, int64_t>(p, mode, grid, A, B, C, ws, ep, st))
    if (p.a_lanes_k && p.b_lanes_k) return B2C_DG(true, true);
    if (p.a_lanes_k) return B2C_DG(true, false);
    if (!p.b_lanes_k) return B2C_DG(false, false);
#undef B2C_DG
    return p.whole ? launch_dgemm_v<BN, false, true, 1, int64_t, true>(p, mode, grid, A, B, C, ws, ep, st)
                   : launch_dgemm_v<BN, false, true, 1, int64_t>(p, mode, grid, A, B, C, ws, ep, st);
}

// Which of the two kernels takes a forward pass of at most SHORT_K products an output, in microseconds.  Both are fits (7 to 12 %) to
// 1728 layers: 784 to 100 352 pixels, 8 to 512 outputs, 8 to 64 products, both layouts.  A tile costs igemm_kernel by slices of 16; a
// thread of short_fprop_kernel pays for each product in latency (more where a product is a channel of one tap, and so a line
// of its own), gathers its pixel again for every 32 outputs and is slow to store outputs that are no float4 runs.  16x28x28 40->512 1x1
// 39 us in tiles, 46 by threads (NHWC); 44->47 10 / 18; 1->16 3x3 13 / 6; 17->64 1x1 of 56x56, 32 images, 39 / 25 (NCHW).  Lines of a warp's
// pixels 192 bytes and more apart do not stay in L1 until their last channel: 64->512 29 / 53.  In place (1x1) is for the tiles, which
// read a whole row before they store it.
static bool short_fprop_pays(const IgemmParams& p, bool vec, bool in_place)
{
    const bool nhwc = p.c_sn == 1;
    if (in_place || (nhwc && p.C >= 48)) return false;
    const int slices = (p.K + 15) / 16, narrow = p.N <= 16;
    auto rounds_past_one = [](int64_t blocks) { const double r = (double)blocks / tc_sm_count() - 1.0; return r > 0.0 ? r : 0.0; };
    const double t = rounds_past_one((int64_t)((p.M + 127) / 128) * ((p.N + tile_bn(p.N) - 1) / tile_bn(p.N)));
    const double b = rounds_past_one((int64_t)((p.M + 255) / 256) * (narrow ? 1 : (p.N + 31) / 32));
    const double tiles_us = tile_bn(p.N) == 64 ? 5.1 + 1.9 * slices + t * (2.3 + 1.5 * slices)
                          : nhwc ? 9.4 + 2.8 * slices + t * (5.0 + 2.2 * slices) : 12.8 + 2.8 * slices + t * (8.0 + 2.2 * slices);
    const double latency = (p.R * p.S == 1 && p.K >= 24 ? 0.22 : 0.15) * p.K;
    const double threads_us = narrow ? 3.6 + latency + b * (1.3 + 0.12 * p.K)
                            : nhwc && !vec ? 11.0 + latency + b * (4.5 + 0.107 * p.K) : 6.5 + latency + b * ((nhwc ? 2.5 : 1.5) + 0.105 * p.K);
    return 1.05 * threads_us < tiles_us;
}

template <typename T, int MODE>
static int launch_igemm(IgemmParams& p, const void* A, const void* B, void* C, void* ws, size_t ws_bytes,
                        Epilogue<T> ep, cudaStream_t st)
{
    finish_params(p, sizeof(T) == 4 ? B2C_F32 : B2C_F64);
    size_t need = partial_bytes(p, sizeof(T));
    if (p.whole && (need > ws_bytes || !ws)) { p.splits = 1; p.k_chunk = (p.K + 15) / 16 * 16; p.whole = p.m_whole = 0; need = 0; }    // whole tiles need none
    if (need > ws_bytes || (need && !ws)) return B2C_ERR_WORKSPACE_TOO_SMALL;
    const int bn = p.bn;
    const bool vec = p.c_sn == 1 && p.N % 4 == 0 && ((p.pb_sn | p.pb_sh | p.pb_sw) & 3) == 0 && ((uintptr_t)C & 15) == 0;
    dim3 grid((p.M + 127) / 128, (p.N + bn - 1) / bn, p.splits);
    if (grid.y > 65535 || grid.z > 65535) return B2C_ERR_TOO_LARGE;
    if constexpr (sizeof(T) == 8) {
        p.f_pq = FastDiv(p.PQ); p.f_q = FastDiv(p.Q);
        if (p.K > 0) { p.f_c = FastDiv(p.C); p.f_s = FastDiv(p.S); p.f_rs = FastDiv(p.R * p.S); }
        if (p.whole) {
            const int64_t blocks = p.whole + ((int64_t)grid.x * grid.y - p.whole) * p.splits;
            if (blocks > 0x7fffffffLL) return B2C_ERR_TOO_LARGE;
            grid = dim3((unsigned)blocks);
        }
        const int rc = bn == 64 ? launch_dgemm<64>(p, MODE, grid, (const double*)A, (const double*)B, (double*)C, (double*)ws, ep, st)
                                : launch_dgemm<128>(p, MODE, grid, (const double*)A, (const double*)B, (double*)C, (double*)ws, ep, st);
        if (rc) return rc;
    } else if (MODE == MODE_FPROP && p.K <= SHORT_K && p.splits == 1 && (p.N + 31) / 32 <= 65535 && short_fprop_pays(p, vec, A == C)) {
        if (p.N <= 16) launch_pdl(short_fprop_kernel<16>, dim3((p.M + 255) / 256), 256, 0, st, p, (const float*)A, (const float*)B, (float*)C, ep, vec);
        else launch_pdl(short_fprop_kernel<32>, dim3((p.M + 255) / 256, (p.N + 31) / 32), 256, 0, st, p, (const float*)A, (const float*)B, (float*)C, ep, vec);
    } else if (bn == 64)
        launch_pdl(igemm_kernel<MODE, 64, 4>, grid, 256, 0, st, p, (const float*)A, (const float*)B, (float*)C, (float*)ws, ep);
    else
        launch_pdl(igemm_kernel<MODE, 128, 8>, grid, 256, 0, st, p, (const float*)A, (const float*)B, (float*)C, (float*)ws, ep);
    int rc = check_launch("igemm_kernel");
    if (rc) return rc;
    if (p.splits > 1) {
        int64_t total = (int64_t)(p.M - p.m_whole) * p.N;
        if (p.splits >= 16) launch_pdl(splitk_reduce_kernel<T, MODE, 8>, (unsigned)((total + 31) / 32), dim3(32, 8), 0, st, p, (const T*)ws, (T*)C, ep);
        else launch_pdl(splitk_reduce_kernel<T, MODE, 1>, (unsigned)((total + 255) / 256), dim3(256, 1), 0, st, p, (const T*)ws, (T*)C, ep);
        rc = check_launch("splitk_reduce_kernel");
    }
    return rc;
}

template <typename T>
static Epilogue<T> make_epilogue(const void* bias, const b2c_bn_params* bn, int relu)
{
    Epilogue<T> ep{};
    ep.bias = (const T*)bias;
    if (bn) { ep.mean = (const T*)bn->mean; ep.inv_std = (const T*)bn->inv_std; ep.gamma = (const T*)bn->gamma; ep.beta = (const T*)bn->beta; }
    ep.relu = relu;
    return ep;
}

int fma_fprop(const Geo& g, const void* x, const void* w, const void* bias, const b2c_bn_params* bn, int relu,
              void* y, void* ws, size_t ws_bytes, cudaStream_t st)
{
    IgemmParams p = make_params(g, MODE_FPROP);
    if (g.dtype == B2C_F32) return launch_igemm<float, MODE_FPROP>(p, x, w, y, ws, ws_bytes, make_epilogue<float>(bias, bn, relu), st);
    return launch_igemm<double, MODE_FPROP>(p, x, w, y, ws, ws_bytes, make_epilogue<double>(bias, bn, relu), st);
}

int fma_dgrad(const Geo& g, const void* dy, const void* w, void* dx, void* ws, size_t ws_bytes, cudaStream_t st)
{
    if (dgrad_by_class(g)) {
        for (int a = 0; a < g.vstr; a++)
            for (int b = 0; b < g.hstr; b++) {
                IgemmParams p = dgrad_class_params(g, a, b);
                if (p.M == 0) continue;
                int rc = g.dtype == B2C_F32
                    ? launch_igemm<float, MODE_DGRAD>(p, dy, w, dx, ws, ws_bytes, Epilogue<float>{}, st)
                    : launch_igemm<double, MODE_DGRAD>(p, dy, w, dx, ws, ws_bytes, Epilogue<double>{}, st);
                if (rc) return rc;
            }
        return B2C_OK;
    }
    IgemmParams p = make_params(g, MODE_DGRAD);
    if (g.dtype == B2C_F32) return launch_igemm<float, MODE_DGRAD>(p, dy, w, dx, ws, ws_bytes, Epilogue<float>{}, st);
    return launch_igemm<double, MODE_DGRAD>(p, dy, w, dx, ws, ws_bytes, Epilogue<double>{}, st);
}

int fma_wgrad(const Geo& g, const void* x, const void* dy, void* dw, void* db, void* ws, size_t ws_bytes,
              cudaStream_t st)
{
    if (is_dense_fc(g) && !(((uintptr_t)x | (uintptr_t)dy | (uintptr_t)dw) & 15)) {
        dim3 grid((g.co + 127) / 128, (g.ci + 127) / 128);
        if (grid.y > 65535) return B2C_ERR_TOO_LARGE;
        launch_pdl(fc_wgrad_kernel, grid, 256, 0, st, (const float*)x, (const float*)dy, (float*)dw, g.n, g.ci, g.co);
        int rc = check_launch("fc_wgrad_kernel");
        if (rc || !db) return rc;
        size_t cs = channel_sum_workspace_bytes(g.n, g.co, 1);
        if (!ws || ws_bytes < cs) return B2C_ERR_WORKSPACE_TOO_SMALL;
        return channel_sum(g.dtype, g.layout, g.n, g.co, 1, dy, db, ws, cs, st);
    }
    IgemmParams p = make_params(g, MODE_WGRAD);
    finish_params(p, g.dtype);
    size_t es = g.dtype == B2C_F32 ? 4 : 8;
    size_t part = align_up(partial_bytes(p, es), 256), gemm_bytes = ws_bytes;
    if (p.whole && ws_bytes < part + (db ? channel_sum_workspace_bytes(g.n, g.co, g.ho * g.wo) : 0)) part = gemm_bytes = 0;      // whole tiles only
    int rc;
    if (g.dtype == B2C_F32) rc = launch_igemm<float, MODE_WGRAD>(p, x, dy, dw, ws, gemm_bytes, Epilogue<float>{}, st);
    else rc = launch_igemm<double, MODE_WGRAD>(p, x, dy, dw, ws, gemm_bytes, Epilogue<double>{}, st);
    if (rc || !db) return rc;
    size_t cs = channel_sum_workspace_bytes(g.n, g.co, g.ho * g.wo);
    if (!ws || ws_bytes < part + cs) return B2C_ERR_WORKSPACE_TOO_SMALL;
    return channel_sum(g.dtype, g.layout, g.n, g.co, g.ho * g.wo, dy, db, (char*)ws + part, cs, st);
}

int fma_index_map(const Geo& g, int64_t* map, cudaStream_t st)
{
    Geo gr = g;
    IgemmParams p = make_params(gr, MODE_FPROP);
    p.tap_c_fast = 0;  // the reference numbers taps channel-slowest: col = cc*kh*kw + ii*kw + jj
    int64_t total = (int64_t)p.M * p.K;
    if (total > (int64_t)0x7fffffff * 256) return B2C_ERR_TOO_LARGE;
    launch_pdl(index_map_kernel, (unsigned)((total + 255) / 256), 256, 0, st, p, map, g.layout == B2C_LAYOUT_NCHW);
    return check_launch("index_map_kernel");
}

// ---- per-channel sum (bias gradient) ----------------------------------------------------------

#define CS_CHUNKS 64

// NHWC: src is (rows, c). Block (32, 8): x runs over channels, y over rows of one chunk.
template <typename T>
__global__ void channel_sum_nhwc_kernel(const T* __restrict__ src, double* __restrict__ partial, int64_t rows, int c)
{
    pdl_prologue();
    __shared__ double sm[8][33];
    int ch = blockIdx.x * 32 + threadIdx.x;
    int64_t per = (rows + gridDim.y - 1) / gridDim.y;
    int64_t r0 = (int64_t)blockIdx.y * per, r1 = r0 + per < rows ? r0 + per : rows;
    double acc = 0.0;
    if (ch < c)
        for (int64_t r = r0 + threadIdx.y; r < r1; r += 8) acc += (double)src[r * c + ch];
    sm[threadIdx.y][threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.y == 0 && ch < c) {
        double s = 0.0;
        for (int i = 0; i < 8; i++) s += sm[i][threadIdx.x];
        partial[(int64_t)blockIdx.y * c + ch] = s;
    }
}

// NCHW: src is (n, c, hw). One block per (channel, chunk); threads stride over (image, position).
template <typename T>
__global__ void channel_sum_nchw_kernel(const T* __restrict__ src, double* __restrict__ partial, int n, int c, int hw)
{
    pdl_prologue();
    __shared__ double sm[256];
    int ch = blockIdx.x;
    int64_t total = (int64_t)n * hw;
    int64_t per = (total + gridDim.y - 1) / gridDim.y;
    int64_t i0 = (int64_t)blockIdx.y * per, i1 = i0 + per < total ? i0 + per : total;
    double acc = 0.0;
    for (int64_t i = i0 + threadIdx.x; i < i1; i += 256) {
        int64_t img = i / hw, pos = i - img * hw;
        acc += (double)src[(img * c + ch) * hw + pos];
    }
    sm[threadIdx.x] = acc;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) { if (threadIdx.x < s) sm[threadIdx.x] += sm[threadIdx.x + s]; __syncthreads(); }
    if (threadIdx.x == 0) partial[(int64_t)blockIdx.y * c + ch] = sm[0];
}

// A warp per channel: every lane adds its chunks (32 apart) in index order, a shuffle tree adds the lanes.
template <typename T>
__global__ void __launch_bounds__(256) channel_sum_final_kernel(const double* __restrict__ partial, T* __restrict__ dst, int c, int chunks)
{
    pdl_prologue();
    const int ch = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    double s = 0.0;
    if (ch < c) for (int i = lane; i < chunks; i += 32) s += partial[(int64_t)i * c + ch];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (ch < c && lane == 0) dst[ch] = (T)s;
}

// Few rows (a fully connected layer's batch): one launch, block (32 channels, 32 row lanes), a thread adds its rows 32 apart in
// order, the lanes are added in order.
constexpr int CS_FEW_ROWS = 1024;
template <typename T>
__global__ void __launch_bounds__(1024) channel_sum_few_kernel(const T* __restrict__ src, T* __restrict__ dst, int rows, int c)
{
    pdl_prologue();
    __shared__ double sm[32][33];
    const int ch = blockIdx.x * 32 + threadIdx.x;
    double acc = 0.0;
    if (ch < c) {
#pragma unroll 4
        for (int r = threadIdx.y; r < rows; r += 32) acc += (double)src[(int64_t)r * c + ch];
    }
    sm[threadIdx.y][threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.y == 0 && ch < c) {
        double s = 0.0;
#pragma unroll
        for (int i = 0; i < 32; i++) s += sm[i][threadIdx.x];
        dst[ch] = (T)s;
    }
}

// Enough for the float4 fast path to spread over about four CTAs per SM: two doubles per channel and chunk.
size_t channel_sum_workspace_bytes(int n, int c, int hw)
{
    (void)n; (void)hw;
    int gx = c / 256 > 0 ? c / 256 : 1;
    int chunks = (592 + gx - 1) / gx;
    if (chunks < CS_CHUNKS) chunks = CS_CHUNKS;
    return (size_t)chunks * 2 * c * sizeof(double);
}

int channel_sum(int dtype, int layout, int n, int c, int hw, const void* src, void* dst, void* ws, size_t ws_bytes,
                cudaStream_t st)
{
    if (!src || !dst || !ws) return B2C_ERR_NULL_POINTER;
    if (ws_bytes < (size_t)CS_CHUNKS * c * sizeof(double)) return B2C_ERR_WORKSPACE_TOO_SMALL;
    if ((layout == B2C_LAYOUT_NHWC || hw == 1) && (int64_t)n * hw <= CS_FEW_ROWS) {
        if (dtype == B2C_F32) launch_pdl(channel_sum_few_kernel<float>, (c + 31) / 32, dim3(32, 32), 0, st, (const float*)src, (float*)dst, n * hw, c);
        else launch_pdl(channel_sum_few_kernel<double>, (c + 31) / 32, dim3(32, 32), 0, st, (const double*)src, (double*)dst, n * hw, c);
        return check_launch("channel_sum_few_kernel");
    }
    if (dtype == B2C_F32 && layout == B2C_LAYOUT_NHWC) {
        int r = channel_sum_v4(n, c, hw, src, dst, ws, ws_bytes, st);
        if (r != 1) return r;     // 1 = fast path not applicable
    }
    double* partial = (double*)ws;
    int64_t rows = (int64_t)n * hw;
    int chunks = (int)(rows < CS_CHUNKS ? rows : CS_CHUNKS);
    if (chunks < 1) chunks = 1;
    if (layout == B2C_LAYOUT_NHWC) {
        dim3 grid((c + 31) / 32, chunks), block(32, 8);
        if (dtype == B2C_F32) launch_pdl(channel_sum_nhwc_kernel<float>, grid, block, 0, st, (const float*)src, partial, rows, c);
        else launch_pdl(channel_sum_nhwc_kernel<double>, grid, block, 0, st, (const double*)src, partial, rows, c);
    } else {
        if (c > 65535 * 32) return B2C_ERR_TOO_LARGE;
        dim3 grid(c, chunks);
        if (dtype == B2C_F32) launch_pdl(channel_sum_nchw_kernel<float>, grid, 256, 0, st, (const float*)src, partial, n, c, hw);
        else launch_pdl(channel_sum_nchw_kernel<double>, grid, 256, 0, st, (const double*)src, partial, n, c, hw);
    }
    int rc = check_launch("channel_sum");
    if (rc) return rc;
    if (dtype == B2C_F32) launch_pdl(channel_sum_final_kernel<float>, (c + 7) / 8, 256, 0, st, partial, (float*)dst, c, chunks);
    else launch_pdl(channel_sum_final_kernel<double>, (c + 7) / 8, 256, 0, st, partial, (double*)dst, c, chunks);
    return check_launch("channel_sum_final");
}

}  // namespace b2c
