// Matrix-vector products y = x . W^T over weights in any storage format, with the fusions the decode
// step needs (RMSNorm prologue; residual / SwiGLU epilogues).
//
// Path 0 ("exact", vb_gemv_canon.cu): fp32 activations, weights at their exact fp32 value, fp32 FMA.  It follows the
// reference arithmetic (src/runtime.rs:702-740 with the dequant contract) up to summation order and is the precision
// baseline the tuned paths are checked against.
#include "vb_internal.cuh"
#include "vb_kernels.cuh"

namespace vb {

cudaError_t gemv_fast(const LaunchCfg& lc, const GemvArgs& a, bool* handled);  // vb_gemv_fast.cu

cudaError_t gemv_fast_init();  // vb_gemv_fast.cu

cudaError_t gemv_init() {
    cudaError_t e;
    if ((e = gemv_imma_init()) != cudaSuccess) return e;
    return gemv_fast_init();
}

cudaError_t kernels_init() { return gemv_init(); }

cudaError_t gemv(const LaunchCfg& lc, const GemvArgs& a, int path) {
    if (a.batch == 0 || a.w.rows == 0) return cudaSuccess;
    if (path != 0) {
        bool handled = false;
        cudaError_t e = gemv_mma(lc, a, &handled);
        if (handled || e != cudaSuccess) return e;
        e = gemv_imma(lc, a, &handled);
        if (handled || e != cudaSuccess) return e;
        e = gemv_fast(lc, a, &handled);
        if (handled || e != cudaSuccess) return e;
    }
    return gemv_canon(lc, a);
}

}  // namespace vb

using namespace vb;

extern "C" int32_t vb_op_matmul(float* dst, const float* x, const void* w, const void* scales, int32_t fmt,
                                uint32_t in_dim, uint32_t out_dim, uint32_t batch, void* stream) {
    VB_REQUIRE(dst && x && w, "vb_op_matmul: null pointer");
    VB_REQUIRE(fmt >= VB_FMT_F32 && fmt <= VB_FMT_I8PC, "vb_op_matmul: unknown format %d", fmt);
    VB_REQUIRE(in_dim % 8 == 0 && fmt_shape_ok(fmt, in_dim), "vb_op_matmul: in_dim=%u not valid for format %d", in_dim, fmt);
    VB_REQUIRE(wmat_scale_bytes(fmt, out_dim, in_dim) == 0 || scales, "vb_op_matmul: format %d needs scales", fmt);
    VB_REQUIRE((size_t)in_dim * 4 <= 200 * 1024, "vb_op_matmul: in_dim=%u exceeds 51200, the widest row of a context or an operation", in_dim);
    if (batch == 0 || out_dim == 0) return VB_OK;
    GemvArgs a;
    a.dst = dst; a.x = x;
    a.w.data = w; a.w.scales = scales; a.w.fmt = fmt; a.w.rows = out_dim; a.w.cols = in_dim;
    a.batch = batch;
    LaunchCfg lc; lc.stream = (cudaStream_t)stream;
    VB_CUDA(kernels_init());
    VB_CUDA(gemv(lc, a, 0));
    return VB_OK;
}
