// Matrix-vector products y = x . W^T over weights in their canonical row-major layout, any storage format, fp32
// arithmetic (weights at their exact fp32 value, fp32 activations, fp32 FMA; runtime.rs:702-740 up to summation
// order): the path of fp32 / fp16 / bf16 / q4 group-64 models and the precision baseline of the tuned paths.
//
// What bounds it.  Batches of a few rows stream the weights once, so HBM does, and for models of a few hundred MB the
// chain of launches: what every kernel does between the end of its predecessor and its own first store.
//  * A warp owns four rows of W (two of gate and two of up for SwiGLU) and walks along K, 8 consecutive elements a lane
//    and step: one x value loaded serves four weights, and x (L1-resident after its first touch) needs no staging
//    through shared memory and no barrier.  Several rows of x share the pass over the weights (launch_canon_fmt).
//  * The loads of the next DEPTH steps are in registers or in flight: 128..192 bytes a thread, 64..98 KB an SM at 16
//    warps, what HBM's latency at 44 GB/s an SM asks for.  The first DEPTH steps are requested BEFORE the
//    grid-dependency wait (weights never depend on the kernel before), so at the size of a 135M model the whole
//    matrix is on its way while the predecessor still runs.
//  * RMSNorm is folded in without a pass of its own: W.(x*w)*inv is summed beside sum(x^2), each warp over its K.
//  * KS warps of a block share a row group's K extent where rows alone would leave warps idle.
// The kernel it replaced staged x behind two barriers, loaded one row a warp and started the weights after the wait
// (batch rows re-read them): a token of the 135M fp32 model 0.83 -> 0.57 ms, of the 8B model in q4 group-64 5.05 -> 3.9.
// Alone: fp32 128256 x 4096 292 us (7.2 TB/s), fp16 175 us (6.0), q4 group-64 157 us (1.9: bound by instructions, ~7 a
// weight at IPC 2.3, which is why int4 in tileable shapes goes to the tensor cores).
#include "vb_internal.cuh"
#include "vb_kernels.cuh"

namespace vb {
namespace {

constexpr int GC_R = 4;        // rows of W per warp
constexpr int GC_WARPS = 8;    // per block
constexpr int GC_THREADS = GC_WARPS * 32;
constexpr uint32_t GC_WAVE = 148 * 16;  // warps the chip holds

// words: 32-bit words of 8 consecutive elements; depth: steps requested ahead (depth_rows: where the accumulators of several rows
// of x take the registers)
template <int FMT> struct Canon;
template <> struct Canon<VB_FMT_F32> { static constexpr int words = 8, depth = 1, depth_rows = 1; static constexpr bool group_scale = false; };
template <> struct Canon<VB_FMT_F16> { static constexpr int words = 4, depth = 3, depth_rows = 1; static constexpr bool group_scale = false; };
template <> struct Canon<VB_FMT_BF16> { static constexpr int words = 4, depth = 3, depth_rows = 1; static constexpr bool group_scale = false; };
template <> struct Canon<VB_FMT_I8PC> { static constexpr int words = 2, depth = 4, depth_rows = 2; static constexpr bool group_scale = false; };
template <> struct Canon<VB_FMT_Q4G32> { static constexpr int words = 1, depth = 4, depth_rows = 2; static constexpr bool group_scale = true; };
template <> struct Canon<VB_FMT_Q4G64REF> { static constexpr int words = 1, depth = 4, depth_rows = 2; static constexpr bool group_scale = true; };

struct CanonArgs {
    const void *w, *scales, *w2, *scales2;  // w2: the up matrix of SwiGLU
    uint32_t rows, K;
    const float* x;
    float* dst;
    const void* norm_w; int norm_fmt; float eps;
    const SeqState* state;
    uint32_t batch, dst_stride, dst_offset;
    int epilogue;
    uint32_t ks;  // warps that share a row group's K extent (1, 2, 4, 8)
    unsigned long long* trace;
};

typedef unsigned long long f32x2;  // two floats for the packed FMA of sm_100
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Weights are read once: past L1, which is left to x.
template <int N>
__device__ __forceinline__ void ldg_words(uint32_t (&v)[N], const uint32_t* p) {
    if constexpr (N == 1) asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v[0]) : "l"(p));
    else if constexpr (N == 2) asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "l"(p));
    else {
#pragma unroll
        for (int i = 0; i < N; i += 4)
            asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                         : "=r"(v[i]), "=r"(v[i + 1]), "=r"(v[i + 2]), "=r"(v[i + 3]) : "l"(p + i));
    }
}

// 8 elements of one row as four pairs of floats (q4: the integers, n - 8 for the symmetric format, pair i times 16^i;
// int8: the integers)
template <int FMT>
__device__ __forceinline__ void expand(const uint32_t (&w)[Canon<FMT>::words], f32x2 (&f)[4]) {
    if constexpr (FMT == VB_FMT_F32) {
#pragma unroll
        for (int i = 0; i < 4; ++i) f[i] = pack2(__uint_as_float(w[2 * i]), __uint_as_float(w[2 * i + 1]));
    } else if constexpr (FMT == VB_FMT_F16) {
#pragma unroll
        for (int i = 0; i < 4; ++i) { const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&w[i])); f[i] = pack2(v.x, v.y); }
    } else if constexpr (FMT == VB_FMT_BF16) {
#pragma unroll
        for (int i = 0; i < 4; ++i) f[i] = pack2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xFFFF0000u));
    } else if constexpr (FMT == VB_FMT_I8PC) {
        // an integer below 2^23 in the low bits of 2^23 is that float; the conversion instructions run at 16 a clock and SM
        const uint32_t u[2] = {w[0] ^ 0x80808080u, w[1] ^ 0x80808080u};
        const f32x2 base = pack2(-8388736.0f, -8388736.0f);  // -(2^23 + 128)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t lo = __byte_perm(u[i >> 1], 0x4B000000u, 0x7440 + 2 * (i & 1)), hi = __byte_perm(u[i >> 1], 0x4B000000u, 0x7441 + 2 * (i & 1));
            f[i] = add2(pack2(__uint_as_float(lo), __uint_as_float(hi)), base);
        }
    } else {
        // elements 2i and 2i+1 sit at bits 4i and 16 + 4i: left where they are they read n * 16^i (x carries the 16^-i)
        const uint32_t up = w[0] >> 16;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float b = 8388608.0f + (FMT == VB_FMT_Q4G32 ? 8.0f * (float)(1 << (4 * i)) : 0.0f);
            f[i] = add2(pack2(__uint_as_float(lop3_and_or(w[0], 0xFu << (4 * i), 0x4B000000u)), __uint_as_float(lop3_and_or(up, 0xFu << (4 * i), 0x4B000000u))),
                        pack2(-b, -b));
        }
    }
}

// Sums v[0..V) over the warp; lane l is left with the total of element l >> (5 - log2 V): V - 1 + (5 - log2 V) shuffles.
template <int V>
__device__ __forceinline__ float warp_reduce_scatter(float (&v)[V], uint32_t lane) {
    int o = 16;
#pragma unroll
    for (int n = V; n > 1; n >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < n / 2; ++i) {
            const float send = up ? v[i] : v[i + n / 2], keep = up ? v[i + n / 2] : v[i];
            v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, o);
        }
    }
    float r = v[0];
#pragma unroll
    for (int w = 32 / V; w > 1; w >>= 1) r += __shfl_xor_sync(0xFFFFFFFFu, r, w >> 1);
    return r;
}

// ALIGNED: 16-byte loads; else element by element
template <bool ALIGNED>
__device__ __forceinline__ float4 load_x4(const float* x) {
    if constexpr (ALIGNED) return *reinterpret_cast<const float4*>(x);
    else return make_float4(x[0], x[1], x[2], x[3]);
}
template <bool ALIGNED>
__device__ __forceinline__ void load_norm8(const void* w, int fmt, uint32_t e0, f32x2 (&f)[4]) {
    if constexpr (!ALIGNED) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float v[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const uint32_t at = e0 + 2 * i + e;
                v[e] = fmt == VB_FMT_F16 ? __half2float(((const __half*)w)[at]) : fmt == VB_FMT_BF16 ? __bfloat162float(((const __nv_bfloat16*)w)[at]) : ((const float*)w)[at];
            }
            f[i] = pack2(v[0], v[1]);
        }
    } else if (fmt == VB_FMT_F32) {
        const float4 a = __ldg(reinterpret_cast<const float4*>((const float*)w + e0)), b = __ldg(reinterpret_cast<const float4*>((const float*)w + e0) + 1);
        f[0] = pack2(a.x, a.y); f[1] = pack2(a.z, a.w); f[2] = pack2(b.x, b.y); f[3] = pack2(b.z, b.w);
    } else {
        const uint4 raw = __ldg(reinterpret_cast<const uint4*>((const uint16_t*)w + e0));
        const uint32_t v[4] = {raw.x, raw.y, raw.z, raw.w};
        if (fmt == VB_FMT_F16) expand<VB_FMT_F16>(v, f); else expand<VB_FMT_BF16>(v, f);
    }
}

// grid (blocks of GC_WARPS / ks row groups, passes of NB rows of x), GC_THREADS threads.  ALIGNED: x and the norm weights start on
// 16-byte boundaries (in a context they do; the per-op entry points take any pointer to whole elements)
template <int FMT, int NB, bool ALIGNED>
__global__ void __launch_bounds__(GC_THREADS, 2) k_gemv_canon(const CanonArgs a) {
    constexpr int R = GC_R, W = Canon<FMT>::words, D = NB == 1 ? Canon<FMT>::depth : Canon<FMT>::depth_rows, V = R * NB;
    constexpr bool PAIRS = !Canon<FMT>::group_scale && NB <= 4;  // accumulate even and odd elements apart (packed FMA all the way)
    constexpr bool GS = Canon<FMT>::group_scale;
    __shared__ float part[GC_WARPS][V];
    __shared__ float part_ss[GC_WARPS][NB];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ks = a.ks;
    const uint32_t kq = warp % ks, group = blockIdx.x * (GC_WARPS / ks) + warp / ks;
    const bool swiglu = a.epilogue == EPI_SWIGLU;
    const uint32_t K = a.K, n8 = K / 8;
    // the warp's part of K: `steps` runs of 32 chunks of 8 elements, of which only the last can reach past the row
    const uint32_t all_steps = (n8 + 31) / 32, per = (all_steps + ks - 1) / ks, first = min(kq * per, all_steps), steps = min(per, all_steps - first);
    uint32_t c0 = first * 32 + lane;  // this lane's chunk at the step the pointers below stand at
    trace_mark(a.trace, 0);
    pdl_launch_dependents();

    // rows of this warp: 4 of one matrix, or 2 of gate and the same 2 of up; rows past the end repeat the last one
    const uint32_t row0 = group * (swiglu ? R / 2 : R);
    const uint32_t* wp[R];
    const unsigned char* sp[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int m = swiglu && r >= R / 2;
        uint32_t row = row0 + (swiglu ? r % (R / 2) : r);
        row = row < a.rows ? row : a.rows - 1;
        wp[r] = reinterpret_cast<const uint32_t*>(m ? a.w2 : a.w) + ((size_t)row * n8 + c0) * W;
        if constexpr (GS)
            sp[r] = reinterpret_cast<const unsigned char*>(m ? a.scales2 : a.scales) +
                    (FMT == VB_FMT_Q4G32 ? ((size_t)row * (K / 32) + (c0 >> 2)) * 2 : ((size_t)row * (K / 64) + (c0 >> 3)) * 4);
    }
    uint32_t w[D][R][W], sc[GS ? D : 1][R];
    // step `ahead` of where the pointers stand -> slot d; `last`: lanes past the row read its last chunk (their x is zero)
    auto request = [&](int d, int ahead, bool last) {
        int rel = ahead * 32, rel_s = ahead * (FMT == VB_FMT_Q4G32 ? 8 : 4);
        if (last && c0 + (uint32_t)rel >= n8) {
            rel = (int)(n8 - 1) - (int)c0;
            rel_s = FMT == VB_FMT_Q4G32 ? (int)((n8 - 1) >> 2) - (int)(c0 >> 2) : (int)((n8 - 1) >> 3) - (int)(c0 >> 3);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            ldg_words(w[d][r], wp[r] + rel * W);
            if constexpr (FMT == VB_FMT_Q4G32) sc[d][r] = __ldg(reinterpret_cast<const uint16_t*>(sp[r]) + rel_s);
            if constexpr (FMT == VB_FMT_Q4G64REF) sc[d][r] = __ldg(reinterpret_cast<const uint32_t*>(sp[r]) + rel_s);
        }
    };
#pragma unroll
    for (int d = 0; d < D; ++d)
        if ((uint32_t)d < steps) request(d, d, true);

    pdl_wait();
    trace_mark(a.trace, 1);
    const uint32_t b0 = blockIdx.y * NB;
    const float* xp[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) xp[b] = a.x + (size_t)(b0 + b < a.batch ? b0 + b : b0) * K + (size_t)c0 * 8;
    // the lane that will write (row r, row of x b) of the group, and the value it adds to
    const uint32_t idx = lane / (32 / V), e_r = idx / NB, e_b = idx % NB;
    const uint32_t o = row0 + (swiglu ? e_r % (R / 2) : e_r);
    bool writer = kq == 0 && lane % (32 / V) == 0 && o < a.rows && (!swiglu || e_r < R / 2) && b0 + e_b < a.batch;
    if (writer && a.state) writer = a.state[b0 + e_b].active != 0;
    float* dp = a.dst + (size_t)(b0 + e_b) * a.dst_stride + a.dst_offset + o;
    float resid = 0.0f;
    if (writer && a.epilogue == EPI_RESIDUAL) resid = *dp;

    f32x2 acc2[PAIRS ? R : 1][PAIRS ? NB : 1];
    float acc[PAIRS ? 1 : R][PAIRS ? 1 : NB];
    f32x2 ss2[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        ss2[b] = 0ull;
#pragma unroll
        for (int r = 0; r < R; ++r) { if constexpr (PAIRS) acc2[r][b] = 0ull; else acc[r][b] = 0.0f; }
    }
    uint32_t ahead_left = steps;  // steps from where the pointers stand to the end
    auto consume = [&](int d, bool last) {
        const bool in = !last || c0 + (uint32_t)d * 32 < n8;
        f32x2 f[R][4];
        float scale[R], minimum[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            expand<FMT>(w[d][r], f[r]);
            if constexpr (FMT == VB_FMT_Q4G32) scale[r] = __half2float(__ushort_as_half((unsigned short)sc[d][r]));
            if constexpr (FMT == VB_FMT_Q4G64REF) {
                const float2 sm = __half22float2(*reinterpret_cast<const __half2*>(&sc[d][r]));
                scale[r] = sm.x; minimum[r] = sm.y;
            }
        }
        // the slot's registers are free again
        if (!last) request(d, d + D, false);
        else if ((uint32_t)(d + D) < ahead_left) request(d, d + D, true);
        f32x2 nw[4];
        if (a.norm_w && in) load_norm8<ALIGNED>(a.norm_w, a.norm_fmt, (c0 + d * 32) * 8, nw);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            // (keeps the compiler from holding the x of several steps, or of all eight rows, in registers at once)
            if (b % 2 == 0) asm volatile("" ::: "memory");
            float4 u = make_float4(0.f, 0.f, 0.f, 0.f), v = u;
            if (in) { u = load_x4<ALIGNED>(xp[b] + d * 256); v = load_x4<ALIGNED>(xp[b] + d * 256 + 4); }
            f32x2 x2[4] = {pack2(u.x, u.y), pack2(u.z, u.w), pack2(v.x, v.y), pack2(v.z, v.w)};
            if (a.norm_w && in) {
#pragma unroll
                for (int i = 0; i < 4; ++i) { ss2[b] = fma2(x2[i], x2[i], ss2[b]); x2[i] = mul2(x2[i], nw[i]); }
            }
            float sx = 0.0f;
            if constexpr (FMT == VB_FMT_Q4G64REF) { const float2 t = unpack2(add2(add2(x2[0], x2[1]), add2(x2[2], x2[3]))); sx = t.x + t.y; }
            if constexpr (GS) {
#pragma unroll
                for (int i = 1; i < 4; ++i) { const float p = 1.0f / (float)(1 << (4 * i)); x2[i] = mul2(x2[i], pack2(p, p)); }
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if constexpr (PAIRS) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc2[r][b] = fma2(f[r][i], x2[i], acc2[r][b]);
                } else {
                    const float2 t = unpack2(fma2(f[r][3], x2[3], fma2(f[r][2], x2[2], fma2(f[r][1], x2[1], mul2(f[r][0], x2[0])))));
                    if constexpr (FMT == VB_FMT_Q4G32) acc[r][b] = fmaf(t.x + t.y, scale[r], acc[r][b]);
                    else if constexpr (FMT == VB_FMT_Q4G64REF) acc[r][b] = fmaf(t.x + t.y, scale[r], fmaf(sx, minimum[r], acc[r][b]));
                    else acc[r][b] += t.x + t.y;
                }
            }
        }
    };
    auto advance = [&]() {
        c0 += 32 * D;
#pragma unroll
        for (int r = 0; r < R; ++r) { wp[r] += 32 * D * W; if constexpr (GS) sp[r] += D * 16; }
#pragma unroll
        for (int b = 0; b < NB; ++b) xp[b] += 256 * D;
        ahead_left -= D;
    };
    if constexpr (NB <= 2) {  // (with more rows of x a second copy of the loop body only spills)
        for (; ahead_left > 2 * D; advance()) {  // nothing consumed or requested here reaches the last step
#pragma unroll
            for (int d = 0; d < D; ++d) consume(d, false);
        }
    }
    for (;; advance()) {
#pragma unroll
        for (int d = 0; d < D; ++d)
            if ((uint32_t)d < ahead_left) consume(d, true);
        if (ahead_left <= D) break;
    }

    float v[V];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            if constexpr (!PAIRS) v[r * NB + b] = acc[r][b];
            else { const float2 t = unpack2(acc2[r][b]); v[r * NB + b] = t.x + t.y; }
        }
    float y = warp_reduce_scatter<V>(v, lane);
    float ss = 0.0f;
    if (a.norm_w) {
        float sv[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b) { const float2 t = unpack2(ss2[b]); sv[b] = warp_sum(t.x + t.y); }
#pragma unroll
        for (int b = 0; b < NB; ++b) if ((uint32_t)b == e_b) ss = sv[b];
    }
    if (ks > 1) {
        if (lane % (32 / V) == 0) { part[warp][idx] = y; if (e_r == 0) part_ss[warp][e_b] = ss; }
        __syncthreads();
        if (kq == 0) {
            for (uint32_t i = 1; i < ks; ++i) { y += part[warp + i][idx]; ss += part_ss[warp + i][e_b]; }
        }
    }
    if (kq == 0) {
        if (a.norm_w) y *= 1.0f / sqrtf(ss / (float)K + a.eps);
        if constexpr (FMT == VB_FMT_I8PC) {
            const int m = swiglu && e_r >= R / 2;
            y *= __half2float(__ldg((const __half*)(m ? a.scales2 : a.scales) + (o < a.rows ? o : a.rows - 1)));
        }
        const float up = __shfl_xor_sync(0xFFFFFFFFu, y, 16);  // SwiGLU: the up half of the rows sits 16 lanes away
        if (writer) {
            if (swiglu) *dp = (y / (1.0f + expf(-y))) * up;
            else if (a.epilogue == EPI_RESIDUAL) *dp = resid + y;
            else *dp = y;
        }
    }
    trace_exit(a.trace);
}

template <int FMT, int NB, bool ALIGNED>
cudaError_t launch_canon(const LaunchCfg& lc, const CanonArgs& a) {
    const uint32_t per = a.epilogue == EPI_SWIGLU ? GC_R / 2 : GC_R, groups = (a.rows + per - 1) / per, per_block = GC_WARPS / a.ks;
    return launch(lc, k_gemv_canon<FMT, NB, ALIGNED>, dim3((groups + per_block - 1) / per_block, (a.batch + NB - 1) / NB), dim3(GC_THREADS), 0, a);
}
// Rows of x per pass over the weights.  A matrix whose passes all run at once as one wave of warps gives each the fewest rows, one or
// two: what the pass takes is its own latency, and the weights come from L2 (576 x 576, 3 rows, fp32: 3.1 us in ones, 3.6 in twos, 4.4
// in fours).  Else four rows to a pass: eight share the weights further but
// hold 64 accumulator registers and spill (fp16 28672 x 4096, 16 rows: 252 us in eights, 248 in fours), which only fp32 with its
// eight-byte pairs wins back, where the last pass is more than half full (8 rows 199 / 224 us, 12 rows 363 / 327, 16 rows 370 /
// 429).  One step of the 135M shape, 5 / 9 / 15 / 32 rows, ms: fp32 1.38 / 1.73 / 1.69 / 2.22 with eights throughout, now
// 0.90 / 1.14 / 1.36 / 2.11; q4 group-64 1.23 / 1.66 / 2.46 / 3.93, now 0.79 / 0.98 / 1.18 / 2.05.
template <int FMT>
cudaError_t launch_canon_fmt(const LaunchCfg& lc, const CanonArgs& a, uint32_t warps) {
    if ((((uintptr_t)a.x | (uintptr_t)a.norm_w) & 15) != 0) return launch_canon<FMT, 1, false>(lc, a);
    if (a.batch == 1 || (a.batch > 2 && warps * a.batch <= GC_WAVE)) return launch_canon<FMT, 1, true>(lc, a);
    if (a.batch == 2 || warps * ((a.batch + 1) / 2) <= GC_WAVE) return launch_canon<FMT, 2, true>(lc, a);
    if constexpr (FMT == VB_FMT_F32)
        if ((a.batch - 1) % 8 >= 4 && warps * ((a.batch + 3) / 4) > GC_WAVE) return launch_canon<FMT, 8, true>(lc, a);
    return launch_canon<FMT, 4, true>(lc, a);
}

}  // namespace

cudaError_t gemv_canon(const LaunchCfg& lc, const GemvArgs& g) {
    if (!g.w.data || g.w.cols % 8 != 0) return cudaErrorInvalidValue;  // (a lean context holds no canonical copy)
    CanonArgs a;
    a.w = g.w.data; a.scales = g.w.scales; a.w2 = g.w2.data; a.scales2 = g.w2.scales;
    a.rows = g.w.rows; a.K = g.w.cols; a.x = g.x; a.dst = g.dst;
    a.norm_w = g.norm_w; a.norm_fmt = g.norm_fmt; a.eps = g.eps; a.state = g.state;
    a.batch = g.batch; a.dst_stride = g.dst_stride ? g.dst_stride : g.w.rows; a.dst_offset = g.dst_offset;
    a.epilogue = g.epilogue; a.trace = g.trace;
    // Share K among warps until the row groups make several waves of the warps the chip holds (the last wave is
    // then a small part), as long as every warp keeps four steps; below one wave, down to a single step each.
    const uint32_t per = g.epilogue == EPI_SWIGLU ? GC_R / 2 : GC_R, groups = (a.rows + per - 1) / per, n8 = a.K / 8;
    a.ks = 1;
    while (a.ks < GC_WARPS && ((groups * a.ks < 6 * GC_WAVE && n8 >= 32 * 4 * 2 * a.ks) || (groups * a.ks < GC_WAVE && n8 >= 32 * 2 * a.ks))) a.ks *= 2;
    switch (g.w.fmt) {
    case VB_FMT_F32: return launch_canon_fmt<VB_FMT_F32>(lc, a, groups * a.ks);
    case VB_FMT_F16: return launch_canon_fmt<VB_FMT_F16>(lc, a, groups * a.ks);
    case VB_FMT_BF16: return launch_canon_fmt<VB_FMT_BF16>(lc, a, groups * a.ks);
    case VB_FMT_Q4G32: return launch_canon_fmt<VB_FMT_Q4G32>(lc, a, groups * a.ks);
    case VB_FMT_Q4G64REF: return launch_canon_fmt<VB_FMT_Q4G64REF>(lc, a, groups * a.ks);
    case VB_FMT_I8PC: return launch_canon_fmt<VB_FMT_I8PC>(lc, a, groups * a.ks);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace vb
