// C ABI of the convolution / FC path: argument checking, engine selection, dispatch.
#include "b2c_common.cuh"
#include <string.h>

namespace b2c {
static thread_local char g_cuda_err[256] = "";
static unsigned long long g_launches = 0;
void count_launch() { __atomic_add_fetch(&g_launches, 1ULL, __ATOMIC_RELAXED); }
void set_cuda_error(cudaError_t e, const char* where) {
    snprintf(g_cuda_err, sizeof(g_cuda_err), "%s: %s", where, cudaGetErrorString(e));
}

// Products summed into one output value (the most over the classes of a strided input gradient).
static int64_t contraction(const Geo& g, int pass) {
    if (pass == B2C_PASS_WGRAD) return g.M;
    if (pass == B2C_PASS_FPROP) return g.K;
    return (int64_t)g.co * ((g.kh + g.vstr - 1) / g.vstr) * ((g.kw + g.hstr - 1) / g.hstr);
}

// Shapes the tensor-core kernels accept but the FMA engine serves better: a weight gradient summed over a handful of pixels
// whose tiles cannot go straight to dw (faster: measured on fully connected layers at batch 32-64), and sums that have to be
// as precise as FMAs (tc_fine_sums) but are so short that only FMAs are: errors against float64 of 0.3, 0.8, 1.0, 1.1 and 1.2e-7
// for 1, 16, 36, 54 and 72 products, against 0.9 to 1.1e-7 of the tensor-core kernels, whatever the length.
static bool fma_is_better(const Geo& g, int pass) {
    if (contraction(g, pass) < 48 && tc_fine_sums(g, pass)) return true;
    const bool one_pixel_images = g.h == 1 && g.w == 1 && g.kh == 1 && g.kw == 1 && g.vpad == 0 && g.hpad == 0;
    return one_pixel_images && g.n <= 128 && pass == B2C_PASS_WGRAD && (g.w_layout != B2C_W_CRSK || g.co % 4);
}

// FMA for everything unless the tensor-core engine takes the shape (AUTO) or is forced.
static int pick_engine(const Geo& g, int pass, int& engine) {
    bool tc = tc_supported(g, pass);
    if (g.engine == B2C_ENGINE_AUTO && tc && fma_is_better(g, pass)) tc = false;
    if (g.engine == B2C_ENGINE_TENSOR) { if (!tc) return B2C_ERR_UNSUPPORTED; engine = B2C_ENGINE_TENSOR; }
    else if (g.engine == B2C_ENGINE_FMA) engine = B2C_ENGINE_FMA;
    else engine = tc ? B2C_ENGINE_TENSOR : B2C_ENGINE_FMA;
    return B2C_OK;
}

// The engine of a call: the shape's, except that channel counts which are no whole blocks on 16-byte pixels also run
// with pointers (x or dx, y or dy) on any alignment, which only the FMA engine takes.
static int call_engine(const Geo& g, int pass, const void* x, const void* y, int& engine) {
    int rc = pick_engine(g, pass, engine);
    if (!rc && engine == B2C_ENGINE_TENSOR && g.engine == B2C_ENGINE_AUTO && !tc_takes_alignment(g, pass, x, y) && !tc_refuses_unaligned(g, pass))
        engine = B2C_ENGINE_FMA;
    return rc;
}
static size_t pass_workspace_bytes(const Geo& g, int pass) {
    int e; if (pick_engine(g, pass, e)) return 0;
    if (e == B2C_ENGINE_FMA) return fma_workspace_bytes(g, pass);
    const size_t t = tc_workspace_bytes(g, pass);
    if (g.engine != B2C_ENGINE_AUTO || tc_refuses_unaligned(g, pass)) return t;
    const size_t f = fma_workspace_bytes(g, pass);
    return t > f ? t : f;
}

// An FC layer is a 1x1 convolution over a (batch, 1, 1, in) NHWC tensor with a (in,1,1,out) filter.
static int fc_geo(int dtype, int engine, int batch, int in_f, int out_f, Geo& g) {
    b2c_conv_desc d{};
    d.layout = B2C_LAYOUT_NHWC; d.dtype = dtype; d.w_layout = B2C_W_CRSK; d.engine = engine;
    d.n = batch; d.h = 1; d.w = 1; d.ci = in_f; d.co = out_f; d.kh = 1; d.kw = 1;
    d.vstr = d.hstr = d.vdil = d.hdil = 1;
    return make_geo(&d, g);
}
}  // namespace b2c

using namespace b2c;

extern "C" const char* b2c_status_string(int status) {
    switch (status) {
        case B2C_OK: return "ok";
        case B2C_ERR_NULL_POINTER: return "null pointer argument";
        case B2C_ERR_BAD_GEOMETRY: return "invalid geometry (non-positive size, empty output, or stride/dilation < 1)";
        case B2C_ERR_BAD_ENUM: return "layout / dtype / weight layout / engine / pass out of range";
        case B2C_ERR_WORKSPACE_TOO_SMALL: return "workspace too small or missing";
        case B2C_ERR_MISALIGNED: return "pointer not aligned as required";
        case B2C_ERR_UNSUPPORTED: return "shape not supported by the requested engine";
        case B2C_ERR_CUDA: return "CUDA launch error";
        case B2C_ERR_TOO_LARGE: return "size exceeds a fixed capacity";
        case B2C_ERR_DEVICE_TIMEOUT: return "a bounded in-kernel wait ran out";
        default: return "unknown status";
    }
}
extern "C" const char* b2c_last_cuda_error(void) { return g_cuda_err; }
extern "C" int b2c_version(void) { return 100; }
extern "C" uint64_t b2c_launch_count(void) { return (uint64_t)__atomic_load_n(&b2c::g_launches, __ATOMIC_RELAXED); }

extern "C" void b2c_note_launches(uint64_t n) { __atomic_add_fetch(&b2c::g_launches, (unsigned long long)n, __ATOMIC_RELAXED); }

extern "C" int b2c_check_device_status(int* detail) {
    int v = 0;
    int rc = tc_read_status(&v);
    if (detail) *detail = v;
    if (rc) return rc;
    return v ? B2C_ERR_DEVICE_TIMEOUT : B2C_OK;
}

extern "C" int b2c_selftest_bounded_wait(int64_t limit_cycles, void* stream) {
    return tc_wait_selftest((long long)limit_cycles, (cudaStream_t)stream);
}

extern "C" int b2c_conv_engine_for(const b2c_conv_desc* desc, int pass) {
    Geo g; int rc = make_geo(desc, g); if (rc) return rc;
    if (pass < 0 || pass > 2) return B2C_ERR_BAD_ENUM;
    int e; rc = pick_engine(g, pass, e); if (rc) return rc;
    return e;
}

extern "C" size_t b2c_conv_workspace_bytes(const b2c_conv_desc* desc, int pass) {
    Geo g; if (make_geo(desc, g)) return 0;
    if (pass < 0 || pass > 2) return 0;
    return pass_workspace_bytes(g, pass);
}

extern "C" int b2c_conv_fprop(const b2c_conv_desc* desc, const void* x, const void* w, const void* bias,
                              const b2c_bn_params* bn, int relu, void* y, void* ws, size_t ws_bytes, void* stream) {
    Geo g; int rc = make_geo(desc, g); if (rc) return rc;
    if (!x || !w || !y) return B2C_ERR_NULL_POINTER;
    if (bn && (!bn->mean || !bn->inv_std || !bn->gamma || !bn->beta)) return B2C_ERR_NULL_POINTER;
    int e; rc = call_engine(g, B2C_PASS_FPROP, x, y, e); if (rc) return rc;
    if (e == B2C_ENGINE_TENSOR) return tc_fprop(g, x, w, bias, bn, relu, y, ws, ws_bytes, (cudaStream_t)stream);
    rc = fma_fprop(g, x, w, bias, bn, relu, y, ws, ws_bytes, (cudaStream_t)stream);
    // a layer that keeps its lowered input has it in the workspace after every forward pass, if the workspace can hold it: one
    // that cannot is refused by the weight gradient, which needs more
    if (rc || !b2c_conv_keeps_lowered_input(desc)) return rc;
    rc = tc_leave_lowered(g, x, ws, ws_bytes, (cudaStream_t)stream);
    return rc == B2C_ERR_WORKSPACE_TOO_SMALL ? B2C_OK : rc;
}

extern "C" size_t b2c_conv_stats_bytes(const b2c_conv_desc* desc) {
    Geo g; if (make_geo(desc, g)) return 0;
    if (g.dtype != B2C_F32) return 0;
    int e; if (pick_engine(g, B2C_PASS_FPROP, e) || e != B2C_ENGINE_TENSOR) return 0;
    return tc_stats_bytes(g);
}

extern "C" int b2c_conv_fprop_stats(const b2c_conv_desc* desc, const void* x, const void* w, const void* bias, void* y,
                                    void* stats, size_t stats_bytes, void* ws, size_t ws_bytes, void* stream) {
    Geo g; int rc = make_geo(desc, g); if (rc) return rc;
    if (!x || !w || !y || !stats) return B2C_ERR_NULL_POINTER;
    if (g.dtype != B2C_F32) return B2C_ERR_UNSUPPORTED;
    int e; rc = call_engine(g, B2C_PASS_FPROP, x, y, e); if (rc) return rc;
    if (e != B2C_ENGINE_TENSOR) return B2C_ERR_UNSUPPORTED;
    return tc_fprop_stats(g, x, w, bias, y, stats, stats_bytes, ws, ws_bytes, (cudaStream_t)stream);
}

extern "C" int b2c_conv_dgrad(const b2c_conv_desc* desc, const void* dy, const void* w, void* dx,
                              void* ws, size_t ws_bytes, void* stream) {
    Geo g; int rc = make_geo(desc, g); if (rc) return rc;
    if (!dy || !w || !dx) return B2C_ERR_NULL_POINTER;
    int e; rc = call_engine(g, B2C_PASS_DGRAD, dx, dy, e); if (rc) return rc;
    if (e == B2C_ENGINE_TENSOR) return tc_dgrad(g, dy, w, dx, ws, ws_bytes, (cudaStream_t)stream);
    return fma_dgrad(g, dy, w, dx, ws, ws_bytes, (cudaStream_t)stream);
}

extern "C" int b2c_conv_keeps_lowered_input(const b2c_conv_desc* desc) {
    Geo g; if (make_geo(desc, g)) return 0;
    int e; if (pick_engine(g, B2C_PASS_WGRAD, e) || e != B2C_ENGINE_TENSOR) return 0;
    if (pick_engine(g, B2C_PASS_FPROP, e) || e != B2C_ENGINE_TENSOR) return 0;
    return tc_keeps_lowered(g) ? 1 : 0;
}

extern "C" int b2c_conv_wgrad_lowered(const b2c_conv_desc* desc, const void* x, const void* dy, void* dw, void* db,
                                      void* ws, size_t ws_bytes, void* stream) {
    Geo g; int rc = make_geo(desc, g); if (rc) return rc;
    if (!x || !dy || !dw) return B2C_ERR_NULL_POINTER;
    if (!b2c_conv_keeps_lowered_input(desc)) return B2C_ERR_UNSUPPORTED;
    int e; rc = call_engine(g, B2C_PASS_WGRAD, x, dy, e); if (rc) return rc;
    if (e != B2C_ENGINE_TENSOR) return B2C_ERR_UNSUPPORTED;
    return tc_wgrad_lowered(g, x, dy, dw, db, ws, ws_bytes, (cudaStream_t)stream);
}

extern "C" int b2c_conv_wgrad(const b2c_conv_desc* desc, const void* x, const void* dy, void* dw, void* db,
                              void* ws, size_t ws_bytes, void* stream) {
    Geo g; int rc = make_geo(desc, g); if (rc) return rc;
    if (!x || !dy || !dw) return B2C_ERR_NULL_POINTER;
    int e; rc = call_engine(g, B2C_PASS_WGRAD, x, dy, e); if (rc) return rc;
    if (e == B2C_ENGINE_TENSOR) return tc_wgrad(g, x, dy, dw, db, ws, ws_bytes, (cudaStream_t)stream);
    return fma_wgrad(g, x, dy, dw, db, ws, ws_bytes, (cudaStream_t)stream);
}

extern "C" int b2c_conv_index_map(const b2c_conv_desc* desc, int64_t* map, void* stream) {
    Geo g; int rc = make_geo(desc, g); if (rc) return rc;
    if (!map) return B2C_ERR_NULL_POINTER;
    return fma_index_map(g, map, (cudaStream_t)stream);
}

extern "C" int b2c_transpose(int dtype, int n, int rows, int cols, const void* src, void* dst, void* stream) {
    if (dtype < 0 || dtype > 1) return B2C_ERR_BAD_ENUM;
    if (n <= 0 || rows <= 0 || cols <= 0) return B2C_ERR_BAD_GEOMETRY;
    if (!src || !dst) return B2C_ERR_NULL_POINTER;
    return transpose_images(dtype, src, dst, n, rows, cols, (cudaStream_t)stream);
}

extern "C" size_t b2c_fc_workspace_bytes(int dtype, int batch, int in_f, int out_f, int engine) {
    Geo g; if (fc_geo(dtype, engine, batch, in_f, out_f, g)) return 0;
    size_t m = 0;
    for (int pass = 0; pass < 3; pass++) {
        size_t b = pass_workspace_bytes(g, pass);
        if (b > m) m = b;
    }
    if (tc_fc_small_batch(dtype, engine, batch, in_f, out_f)) {
        size_t b = tc_fc_small_batch_bytes(batch, in_f, out_f);
        if (b > m) m = b;
    }
    return m;
}

static bool overlap(const void* a, size_t a_floats, const void* b, size_t b_floats) {
    const uintptr_t p = (uintptr_t)a, q = (uintptr_t)b;
    return a && b && p < q + b_floats * 4 && q < p + a_floats * 4;
}

extern "C" int b2c_fc_forward(int dtype, int engine, int batch, int in_f, int out_f, const void* x, const void* w,
                              const void* bias, void* y, void* ws, size_t ws_bytes, void* stream) {
    Geo g; int rc = fc_geo(dtype, engine, batch, in_f, out_f, g); if (rc) return rc;
    if (!x || !w || !y) return B2C_ERR_NULL_POINTER;
    if (engine == B2C_ENGINE_AUTO && fc_tiny(batch, in_f, out_f)) return fc_tiny_forward(dtype, batch, in_f, out_f, x, w, bias, y, (cudaStream_t)stream);
    // The one-launch forms need neither workspace nor alignment; a call with less of either than the other forms ask for is left to them.
    // So is one with an output on an input's memory: there are blocks that read while others store.
    const size_t xs = (size_t)batch * in_f, ys = (size_t)batch * out_f, wts = (size_t)in_f * out_f;
    int e;
    if (fc_mma_takes(dtype, engine, batch, in_f, out_f, false) && !overlap(y, ys, x, xs) && !overlap(y, ys, w, wts) && !overlap(y, ys, bias, out_f) && ws && ws_bytes >= pass_workspace_bytes(g, B2C_PASS_FPROP) &&
        call_engine(g, B2C_PASS_FPROP, x, y, e) == B2C_OK &&
        !(tc_fc_small_batch(dtype, engine, batch, in_f, out_f) &&
          ((((uintptr_t)x | (uintptr_t)w | (uintptr_t)y | (uintptr_t)bias) & 15) || ws_bytes < tc_fc_small_batch_bytes(batch, in_f, out_f))))
        return fc_mma_forward(batch, in_f, out_f, x, w, bias, y, (cudaStream_t)stream);
    if (tc_fc_small_batch(dtype, engine, batch, in_f, out_f))
        return tc_fc_forward_small_batch(batch, in_f, out_f, x, w, bias, y, ws, ws_bytes, (cudaStream_t)stream);
    rc = call_engine(g, B2C_PASS_FPROP, x, y, e); if (rc) return rc;
    if (e == B2C_ENGINE_TENSOR) return tc_fprop(g, x, w, bias, nullptr, 0, y, ws, ws_bytes, (cudaStream_t)stream);
    return fma_fprop(g, x, w, bias, nullptr, 0, y, ws, ws_bytes, (cudaStream_t)stream);
}

extern "C" int b2c_fc_backward(int dtype, int engine, int batch, int in_f, int out_f, const void* x, const void* dy,
                               const void* w, void* dw, void* db, void* dx, void* ws, size_t ws_bytes, void* stream) {
    Geo g; int rc = fc_geo(dtype, engine, batch, in_f, out_f, g); if (rc) return rc;
    if (!dy) return B2C_ERR_NULL_POINTER;
    cudaStream_t st = (cudaStream_t)stream;
    if (engine == B2C_ENGINE_AUTO && fc_tiny(batch, in_f, out_f) && (dw || !db)) {
        if ((dw && !x) || (dx && !w)) return B2C_ERR_NULL_POINTER;
        return fc_tiny_backward(dtype, batch, in_f, out_f, x, dy, w, dw, db, dx, st);
    }
    const size_t xs = (size_t)batch * in_f, ys = (size_t)batch * out_f, wts = (size_t)in_f * out_f;
    auto on_input = [&](const void* out, size_t floats) { return overlap(out, floats, x, xs) || overlap(out, floats, dy, ys) || overlap(out, floats, w, wts); };
    int engine_of;
    if (fc_mma_takes(dtype, engine, batch, in_f, out_f, true) && !on_input(dx, xs) && !on_input(dw, wts) && !on_input(db, out_f) && (dw || (dx && !db)) && (!dw || x) && (!dx || w) && ws &&
        (!dw || ws_bytes >= pass_workspace_bytes(g, B2C_PASS_WGRAD)) && (!dx || ws_bytes >= pass_workspace_bytes(g, B2C_PASS_DGRAD)) &&
        (!dw || call_engine(g, B2C_PASS_WGRAD, x, dy, engine_of) == B2C_OK) && (!dx || call_engine(g, B2C_PASS_DGRAD, dx, dy, engine_of) == B2C_OK) &&
        !(tc_fc_small_batch(dtype, engine, batch, in_f, out_f) &&
          ((((uintptr_t)x | (uintptr_t)dy | (uintptr_t)w | (uintptr_t)dw | (uintptr_t)dx) & 15) || ws_bytes < tc_fc_small_batch_bytes(batch, in_f, out_f))))
        return fc_mma_backward(batch, in_f, out_f, x, dy, w, dw, db, dx, st);
    if (tc_fc_small_batch(dtype, engine, batch, in_f, out_f)) {
        if (dw) {
            if (!x) return B2C_ERR_NULL_POINTER;
            rc = tc_fc_wgrad_small_batch(batch, in_f, out_f, x, dy, dw, db, ws, ws_bytes, st); if (rc) return rc;
        } else if (db) {
            if (!ws || ws_bytes < channel_sum_workspace_bytes(batch, out_f, 1)) return B2C_ERR_WORKSPACE_TOO_SMALL;
            rc = channel_sum(dtype, B2C_LAYOUT_NHWC, batch, out_f, 1, dy, db, ws, ws_bytes, st); if (rc) return rc;
        }
        if (dx) {
            if (!w) return B2C_ERR_NULL_POINTER;
            rc = tc_fc_dgrad_small_batch(batch, in_f, out_f, dy, w, dx, ws, ws_bytes, st);
        }
        return rc;
    }
    if (dw) {
        if (!x) return B2C_ERR_NULL_POINTER;
        int e; rc = call_engine(g, B2C_PASS_WGRAD, x, dy, e); if (rc) return rc;
        rc = e == B2C_ENGINE_TENSOR ? tc_wgrad(g, x, dy, dw, db, ws, ws_bytes, st) : fma_wgrad(g, x, dy, dw, db, ws, ws_bytes, st);
        if (rc) return rc;
    } else if (db) {
        size_t need = channel_sum_workspace_bytes(batch, out_f, 1);
        if (!ws || ws_bytes < need) return B2C_ERR_WORKSPACE_TOO_SMALL;
        rc = channel_sum(dtype, B2C_LAYOUT_NHWC, batch, out_f, 1, dy, db, ws, ws_bytes, st); if (rc) return rc;
    }
    if (dx) {
        if (!w) return B2C_ERR_NULL_POINTER;
        int e; rc = call_engine(g, B2C_PASS_DGRAD, dx, dy, e); if (rc) return rc;
        rc = e == B2C_ENGINE_TENSOR ? tc_dgrad(g, dy, w, dx, ws, ws_bytes, st) : fma_dgrad(g, dy, w, dx, ws, ws_bytes, st);
    }
    return rc;
}
