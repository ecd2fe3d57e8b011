// Fused elementwise passes of the MLP training step (additive mx_* exports, no counterpart in
// the reference's crate).  Each replaces a chain of single-op calls the reference's autograd
// issues, with the same formulas:
//   mx_bias_gelu       u = z + b ; a = gelu(u)          Linear's bias add (crates/maidenx_nn/src/layers/linear.rs:76-78)
//                                                        + GELU forward (crates/maidenx_cpu/src/ops/unary.rs:268-293)
//   mx_bias_add        u = z + b                         last layer (no activation)
//   mx_gelu_backward   du = dy * gelu'(u)                the 15-op closure at crates/maidenx_tensor/src/ops/unary.rs:324-346
//   mx_mse_loss_grad   loss = mean((p - t)^2), dp = 2 (p - t) / n   crates/maidenx_nn/src/losses/mse.rs:21-29 and its backward
//   mx_sgd_update      w32 -= lr * scale * g ; w16 = round(w32)      crates/maidenx_nn/src/optimizers/sgd.rs:17-26 with an
//                                                        f32 master copy of the 16-bit weights
// All are HBM-bound: 16-byte vector accesses, four vectors in flight per thread, math in f32,
// one rounding per stored value.
#include "fused.cuh"
#include "f32x2.cuh"
#include "abi_common.cuh"
#include "ops.cuh"
#include "matmul_tc.cuh"

namespace mx {

constexpr int kFusedThreads = 256;

template <class T>
__device__ __forceinline__ float ld_scalar_f32(const T* p) {
    if constexpr (is_half_v<T>) return to_f32(*p);
    else return (float)*p;
}
template <class T>
__device__ __forceinline__ T st_from_f32(float v) {
    if constexpr (is_half_v<T>) return from_f32<T>(v);
    else return (T)v;
}
template <class T>
__device__ __forceinline__ float up(T v) {
    if constexpr (is_half_v<T>) return to_f32(v);
    else return (float)v;
}
template <class T>
__device__ __forceinline__ float gelu_fwd(float x) {
    return gelu_f32_fast(x);  // the same function cuda_gelu_<T> evaluates
}

// u = round(z + b), a = round(gelu(u)); `a` may be NULL (bias add only).  The sum is rounded to
// T before the activation, exactly as the two separate ops would.
template <class T>
__global__ void __launch_bounds__(kFusedThreads) bias_gelu_kernel(const T* z, const T* bias, T* u,
                                                                 T* a, uint64_t n) {
    after_previous_kernel();
    constexpr int VEC = 16 / sizeof(T);
    const float b = ld_scalar_f32(bias);
    const uint64_t nvec = n / VEC;
    const uint64_t stride = (uint64_t)gridDim.x * kFusedThreads;
    for (uint64_t v = (uint64_t)blockIdx.x * kFusedThreads + threadIdx.x; v < nvec; v += stride) {
        Vec<T, VEC> zi = *reinterpret_cast<const Vec<T, VEC>*>(z + v * VEC), uo, ao;
#pragma unroll
        for (int j = 0; j < VEC; j++) {
            uo.v[j] = st_from_f32<T>(up(zi.v[j]) + b);
            ao.v[j] = st_from_f32<T>(gelu_fwd<T>(up(uo.v[j])));
        }
        *reinterpret_cast<Vec<T, VEC>*>(u + v * VEC) = uo;
        if (a) *reinterpret_cast<Vec<T, VEC>*>(a + v * VEC) = ao;
    }
    if (blockIdx.x == 0)
        for (uint64_t i = nvec * VEC + threadIdx.x; i < n; i += kFusedThreads) {
            T uu = st_from_f32<T>(up(z[i]) + b);
            u[i] = uu;
            if (a) a[i] = st_from_f32<T>(gelu_fwd<T>(up(uu)));
        }
}

// d/dx of x * sigmoid(2t), t = sqrt(2/pi) (x + 0.044715 x^3) - the tanh form's derivative, 0.5 (1 + tanh t) being sigmoid(2t):
//   sigmoid + x sigmoid (1 - sigmoid) (2t)'
// A dozen instructions and two of the special-function unit, where tanh, its square and the separately rounded products took thirty.  With
// e = exp(-2|t|) and r = 1 / (1 + e) the sigmoid is r or e r and its product with the rest e r^2: no difference of near values on either side.
// Error against 64 bits, of the norm, over [0, 12]: 4.0e-8 (by tanh 1.0e-7); [-12, 0]: 1.05e-7 (4.6e-6); [-6, 6]: 5.7e-8 (5.1e-7); 16-bit results alike.
__device__ __forceinline__ float gelu_grad_f32(float x) {
    const float k1 = -2.302208198f, k2 = -0.102943240f;  // exp(-2t) = 2^(x (k1 + k2 x^2)), as in gelu_f32_fast
    const float c1 = 1.5957691216f, c2 = 0.2140644488f;  // (2t)' = c1 + c2 x^2: 2 sqrt(2/pi), three times 0.044715 of that
    const float x2 = x * x;
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(fabsf(x) * fmaf(k2, x2, k1)));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
    const float er = e * r;
    return fmaf(er * r * x, fmaf(c2, x2, c1), x < 0.0f ? er : r);
}

// Two elements at a time: multiplications and additions in the packed form (each half rounds as the scalar instruction does), which halves what the kernel
// issues.  At the clocks that the products around it leave under the power cap the issue slots, not HBM, bounded it: 16384 x 8192 bf16
// with its sum, behind two products of that size, 222 us by single instructions, 172 so (alone 148 and 131; at 6553 GB/s 123).  f32 elements, half as many a byte, are at HBM's rate as they are.
__device__ __forceinline__ F32x2 gelu_grad_pair(float2 x) {
    const float k1 = -2.302208198f, k2 = -0.102943240f, c1 = 1.5957691216f, c2 = 0.2140644488f;
    const F32x2 xx = pair_of(x), x2 = xx * xx;
    const float2 k = halves(fma2(twice(k2), x2, twice(k1)));
    float2 e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.x) : "f"(fabsf(x.x) * k.x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.y) : "f"(fabsf(x.y) * k.y));
    const F32x2 ep = pair_of(e);
    const float2 d = halves(twice(1.0f) + ep);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(d.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(d.y));
    const F32x2 rp = pair_of(r), er = ep * rp;
    const float2 s = halves(er);
    return fma2(er * rp * xx, fma2(twice(c2), x2, twice(c1)), pair_of(make_float2(x.x < 0.0f ? s.x : r.x, x.y < 0.0f ? s.y : r.y)));
}

// The 32-bit words of a vector of 16-bit elements.
template <class T, int VEC>
__device__ __forceinline__ uint32_t* words(Vec<T, VEC>& v) {
    return reinterpret_cast<uint32_t*>(&v);
}

// The block's sum of v; valid in thread 0.
__device__ __forceinline__ float fused_block_sum(float v) {
    __shared__ float warp_part[kFusedThreads / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    if ((threadIdx.x & 31) == 0) warp_part[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < kFusedThreads / 32; w++) v += warp_part[w];
    return v;
}

// A pass that leaves a sum over everything it writes ends with it: every block leaves its part in `partial`, and the last one to arrive
// folds the parts in block order.  (A launch of its own for that took 2 to 4 us.)  True in every thread of the last block, which then sees all parts.
// `arrived` is a zeroed word, left zeroed.
__device__ __forceinline__ bool fused_last_block(uint32_t* arrived) {
    __shared__ bool last;
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(arrived, 1u) == gridDim.x - 1;
        if (last) *arrived = 0;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// SUM: the sum of du (the bias gradient), which a pass over du used to read it back for.  Two vectors of each operand in flight
// per thread.  Registers for five blocks: the pairs without the bound took 58 and four blocks (2^24 f16 16.2 us, 15.2 so).
template <class T, bool SUM>
__global__ void __launch_bounds__(kFusedThreads, is_half_v<T> || SUM ? 5 : 6) gelu_backward_kernel(const T* dy, const T* u, T* du,
                                                                     uint64_t n, float* partial, uint32_t* arrived, T* grad_sum) {
    after_previous_kernel();
    float acc = 0.0f;
    F32x2 sums = twice(0.0f);
    constexpr int VEC = 16 / sizeof(T), UN = 2;
    const uint64_t nvec = n / VEC;
    const uint64_t stride = (uint64_t)gridDim.x * kFusedThreads;
    for (uint64_t v0 = (uint64_t)blockIdx.x * kFusedThreads + threadIdx.x; v0 < nvec; v0 += UN * stride) {
        Vec<T, VEC> g[UN], x[UN];
#pragma unroll
        for (int i = 0; i < UN; i++)
            if (v0 + i * stride < nvec) {
                g[i] = *reinterpret_cast<const Vec<T, VEC>*>(dy + (v0 + i * stride) * VEC);
                x[i] = *reinterpret_cast<const Vec<T, VEC>*>(u + (v0 + i * stride) * VEC);
            }
#pragma unroll
        for (int i = 0; i < UN; i++)
            if (v0 + i * stride < nvec) {
                Vec<T, VEC> o;
                if constexpr (is_half_v<T>) {
#pragma unroll
                    for (int j = 0; j < VEC / 2; j++) {
                        const float2 r = halves(pair_of(unpack2<T>(words(g[i])[j])) * gelu_grad_pair(unpack2<T>(words(x[i])[j])));
                        words(o)[j] = pack2_rn<T>(r.x, r.y);
                        if (SUM) sums = sums + pair_of(unpack2<T>(words(o)[j]));
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < VEC; j++) {
                        o.v[j] = g[i].v[j] * gelu_grad_f32(x[i].v[j]);
                        if (SUM) acc += o.v[j];
                    }
                }
                *reinterpret_cast<Vec<T, VEC>*>(du + (v0 + i * stride) * VEC) = o;
            }
    }
    acc += halves(sums).x + halves(sums).y;
    if (blockIdx.x == 0)
        for (uint64_t i = nvec * VEC + threadIdx.x; i < n; i += kFusedThreads) {
            du[i] = st_from_f32<T>(up(dy[i]) * gelu_grad_f32(up(u[i])));
            if (SUM) acc += up(du[i]);
        }
    if constexpr (SUM) {
        acc = fused_block_sum(acc);
        if (threadIdx.x == 0) partial[blockIdx.x] = acc;
        if (!fused_last_block(arrived)) return;
        acc = 0.0f;
        for (uint32_t i = threadIdx.x; i < gridDim.x; i += 4 * kFusedThreads) {
            float v[4];
#pragma unroll
            for (uint32_t q = 0; q < 4; q++) v[q] = i + q * kFusedThreads < gridDim.x ? __ldcg(partial + i + q * kFusedThreads) : 0.0f;
#pragma unroll
            for (uint32_t q = 0; q < 4; q++) acc += v[q];
        }
        acc = fused_block_sum(acc);
        if (threadIdx.x == 0) *grad_sum = st_from_f32<T>(acc);
    }
}

// The sum of the blocks' parts in a fixed order; valid in thread 0.
__device__ __forceinline__ float mse_fold(const float* partial, uint32_t count) {
    __shared__ float sm[kFusedThreads];
    float acc = 0.0f;
    for (uint32_t i = threadIdx.x; i < count; i += kFusedThreads) acc += __ldcg(partial + i);
    __syncthreads();  // an earlier fold's result has been read
    sm[threadIdx.x] = acc;
    __syncthreads();
    for (int o = kFusedThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) sm[threadIdx.x] += sm[threadIdx.x + o];
        __syncthreads();
    }
    return sm[0];
}

// The same by half a block, in a tree of its own; valid in the half's first thread.
__device__ __forceinline__ float fused_half_sum(const float* partial, uint32_t count) {
    constexpr uint32_t HALF = kFusedThreads / 2;
    __shared__ float warp_part[kFusedThreads / 32];
    const uint32_t t = threadIdx.x % HALF;
    float acc = 0.0f;
    for (uint32_t i = t; i < count; i += 4 * HALF) {  // four parts in flight: what a trip to L2 takes is the length of this
        float v[4];
#pragma unroll
        for (uint32_t q = 0; q < 4; q++) v[q] = i + q * HALF < count ? __ldcg(partial + i + q * HALF) : 0.0f;
#pragma unroll
        for (uint32_t q = 0; q < 4; q++) acc += v[q];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
    if ((threadIdx.x & 31) == 0) warp_part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (t == 0)
        for (uint32_t w = 1; w < HALF / 32; w++) acc += warp_part[(threadIdx.x >> 5) + w];
    return acc;
}

// grad = 2 (p - t) / n, per-block partial sums of (p - t)^2 into `partial` and, with SUM, of grad behind them; with SUM the last block folds both.
template <class T, bool SUM>
__global__ void __launch_bounds__(kFusedThreads) mse_kernel(const T* p, const T* t, T* grad,
                                                           float* partial, uint64_t n, float two_over_n, float inv_n, float* loss,
                                                           T* grad_sum, uint32_t* arrived) {
    after_previous_kernel();
    constexpr int VEC = 16 / sizeof(T);
    const uint64_t nvec = n / VEC;
    const uint64_t stride = (uint64_t)gridDim.x * kFusedThreads;
    float acc = 0.0f, acc_g = 0.0f;
    for (uint64_t v = (uint64_t)blockIdx.x * kFusedThreads + threadIdx.x; v < nvec; v += stride) {
        Vec<T, VEC> a = *reinterpret_cast<const Vec<T, VEC>*>(p + v * VEC), b = *reinterpret_cast<const Vec<T, VEC>*>(t + v * VEC), o;
#pragma unroll
        for (int j = 0; j < VEC; j++) {
            // the difference is rounded to T first, as the separate sub op would
            float d = up(st_from_f32<T>(up(a.v[j]) - up(b.v[j])));
            acc += d * d;
            o.v[j] = st_from_f32<T>(d * two_over_n);
            if (SUM) acc_g += up(o.v[j]);
        }
        *reinterpret_cast<Vec<T, VEC>*>(grad + v * VEC) = o;
    }
    if (blockIdx.x == 0)
        for (uint64_t i = nvec * VEC + threadIdx.x; i < n; i += kFusedThreads) {
            float d = up(st_from_f32<T>(up(p[i]) - up(t[i])));
            acc += d * d;
            grad[i] = st_from_f32<T>(d * two_over_n);
            if (SUM) acc_g += up(grad[i]);
        }
    __shared__ float warp_part[SUM ? 2 : 1][kFusedThreads / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
        if (SUM) acc_g += __shfl_xor_sync(0xFFFFFFFFu, acc_g, o);
    }
    if ((threadIdx.x & 31) == 0) {
        warp_part[0][threadIdx.x >> 5] = acc;
        if (SUM) warp_part[SUM ? 1 : 0][threadIdx.x >> 5] = acc_g;
    }
    __syncthreads();
    if (threadIdx.x < (SUM ? 64 : 32)) {  // the first warp folds the losses, the second the gradients
        const int which = threadIdx.x >> 5, lane = threadIdx.x & 31;
        float v = lane < kFusedThreads / 32 ? warp_part[which][lane] : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
        if (lane == 0) partial[which * gridDim.x + blockIdx.x] = v;
    }
    if constexpr (SUM) {
        __syncthreads();  // both parts are written: the fence of the thread that counts is behind them
        if (!fused_last_block(arrived)) return;
        // two halves of the block, a sum each
        const uint32_t half = threadIdx.x / (kFusedThreads / 2);
        float v = fused_half_sum(partial + half * gridDim.x, gridDim.x);
        if (threadIdx.x == 0) *loss = v * inv_n;
        if (threadIdx.x == kFusedThreads / 2) *grad_sum = st_from_f32<T>(v);
    }
}
// Without an arrival word (the exported pass, whose caller has none): the loss folded by a launch of one block.
__global__ void __launch_bounds__(kFusedThreads) mse_finish_kernel(const float* partial, int count, float inv_n, float* loss) {
    after_previous_kernel();
    const float l = mse_fold(partial, (uint32_t)count);
    if (threadIdx.x == 0) *loss = l * inv_n;
}

// Bound by HBM.  Two vectors of each operand are loaded before the first store: without restricted pointers, which kernels that wait may not have, the
// compiler leaves the loads of the next step behind the stores of this one (40e6 elements f16 90.9 us, 75.1 so, bf16 80.0, 75.1).
template <class T>
__global__ void __launch_bounds__(kFusedThreads) sgd_kernel(float* w32, const T* g, T* w16, uint64_t n,
                                                           float step, float* b32, const T* gb, T* b16) {
    after_previous_kernel();
    constexpr int VEC = 16 / sizeof(T), UN = 2;  // elements per 16-byte vector of the gradient; w32 moves as VEC floats
    const uint64_t nvec = n / VEC;
    const uint64_t stride = (uint64_t)gridDim.x * kFusedThreads;
    if (b32 && blockIdx.x == 0 && threadIdx.x == 0) {  // the layer's one-element bias
        const float w = *b32 - step * up(*gb);
        *b32 = w;
        *b16 = st_from_f32<T>(w);
    }
    for (uint64_t v0 = (uint64_t)blockIdx.x * kFusedThreads + threadIdx.x; v0 < nvec; v0 += UN * stride) {
        Vec<T, VEC> gi[UN], wo;
        // the master weights are promised 16-byte aligned only: move them as float4 quads, never as one 32-byte access
        float4 w[UN][VEC / 4];
#pragma unroll
        for (int i = 0; i < UN; i++)
            if (v0 + i * stride < nvec) {
                const uint64_t at = (v0 + i * stride) * VEC;
                gi[i] = *reinterpret_cast<const Vec<T, VEC>*>(g + at);
#pragma unroll
                for (int q = 0; q < VEC / 4; q++) w[i][q] = *reinterpret_cast<const float4*>(w32 + at + 4 * q);
            }
#pragma unroll
        for (int i = 0; i < UN; i++)
            if (v0 + i * stride < nvec) {
                const uint64_t at = (v0 + i * stride) * VEC;
#pragma unroll
                for (int q = 0; q < VEC / 4; q++) {
                    float4& x = w[i][q];
                    x.x = x.x - step * up(gi[i].v[4 * q + 0]);
                    x.y = x.y - step * up(gi[i].v[4 * q + 1]);
                    x.z = x.z - step * up(gi[i].v[4 * q + 2]);
                    x.w = x.w - step * up(gi[i].v[4 * q + 3]);
                    wo.v[4 * q + 0] = st_from_f32<T>(x.x);
                    wo.v[4 * q + 1] = st_from_f32<T>(x.y);
                    wo.v[4 * q + 2] = st_from_f32<T>(x.z);
                    wo.v[4 * q + 3] = st_from_f32<T>(x.w);
                    *reinterpret_cast<float4*>(w32 + at + 4 * q) = x;
                }
                *reinterpret_cast<Vec<T, VEC>*>(w16 + at) = wo;
            }
    }
    if (blockIdx.x == 0)
        for (uint64_t i = nvec * VEC + threadIdx.x; i < n; i += kFusedThreads) {
            float w = w32[i] - step * up(g[i]);
            w32[i] = w;
            w16[i] = st_from_f32<T>(w);
        }
}

// Four vectors per thread, up to 16 blocks an SM; small tensors one vector per thread, since four trips to memory one after the other are
// longer than what more blocks cost.
static unsigned fused_grid(uint64_t n, int vec) {
    uint64_t blocks = (n / vec + kFusedThreads * 4 - 1) / (kFusedThreads * 4);
    if (blocks < (uint64_t)sm_count() * 2) blocks = (n / vec + kFusedThreads - 1) / kFusedThreads;
    uint64_t cap = (uint64_t)sm_count() * 16;
    if (blocks > cap) blocks = cap;
    return blocks ? (unsigned)blocks : 1u;
}
static bool aligned16(const void* p) { return ((uintptr_t)p) % 16 == 0; }

template <class T>
void bias_gelu_launch(size_t n, const T* z, const T* bias, T* u, T* a, const char* where) {
    if (!n) return;
    if (!aligned16(z) || !aligned16(u) || (a && !aligned16(a))) {
        set_error(kErrUnsupported, 0, where);
        return;
    }
    launch_kernel(bias_gelu_kernel<T>, fused_grid(n, 16 / sizeof(T)), kFusedThreads, 0, ctx().stream, z, bias, u, a, n);
    check_launch(where);
}
template <class T>
void gelu_backward_launch(size_t n, const T* dy, const T* u, T* du, T* grad_sum, uint32_t* arrived, const char* where) {
    if (!n) return;
    if (!aligned16(dy) || !aligned16(u) || !aligned16(du)) {
        set_error(kErrUnsupported, 0, where);
        return;
    }
    const unsigned blocks = fused_grid(n, 16 / sizeof(T));
    if (!grad_sum) {
        launch_kernel(gelu_backward_kernel<T, false>, blocks, kFusedThreads, 0, ctx().stream, dy, u, du, n, nullptr, nullptr, nullptr);
    } else {
        float* partial = static_cast<float*>(scratch(sizeof(float) * blocks));
        if (!partial) return;
        launch_kernel(gelu_backward_kernel<T, true>, blocks, kFusedThreads, 0, ctx().stream, dy, u, du, n, partial, arrived, grad_sum);
    }
    check_launch(where);
}
template <class T>
void mse_launch(size_t n, const T* p, const T* t, T* grad, float* loss, T* grad_sum, uint32_t* arrived, const char* where) {
    if (!n) return;
    if (!aligned16(p) || !aligned16(t) || !aligned16(grad)) {
        set_error(kErrUnsupported, 0, where);
        return;
    }
    unsigned blocks = fused_grid(n, 16 / sizeof(T));
    float* partial = static_cast<float*>(scratch(sizeof(float) * blocks * (grad_sum ? 2 : 1)));
    if (!partial) return;
    const float two_over_n = 2.0f / (float)n, inv_n = 1.0f / (float)n;
    if (grad_sum) {
        launch_kernel(mse_kernel<T, true>, blocks, kFusedThreads, 0, ctx().stream, p, t, grad, partial, n, two_over_n, inv_n, loss, grad_sum, arrived);
    } else {
        launch_kernel(mse_kernel<T, false>, blocks, kFusedThreads, 0, ctx().stream, p, t, grad, partial, n, two_over_n, inv_n, nullptr, nullptr, nullptr);
        launch_kernel(mse_finish_kernel, 1, kFusedThreads, 0, ctx().stream, partial, (int)blocks, inv_n, loss);
    }
    check_launch(where);
}
template <class T>
void sgd_launch(size_t n, float* w32, const T* g, T* w16, float lr, float grad_scale, const char* where, float* b32 = nullptr, const T* gb = nullptr, T* b16 = nullptr) {
    if (!n) return;
    if (!aligned16(w32) || !aligned16(g) || !aligned16(w16)) {
        set_error(kErrUnsupported, 0, where);
        return;
    }
    launch_kernel(sgd_kernel<T>, fused_grid(n, 16 / sizeof(T)), kFusedThreads, 0, ctx().stream, w32, g, w16, n, lr * grad_scale, b32, gb, b16);
    check_launch(where);
}

template <class T>
void mse_loss_grad_sum(size_t n, const T* pred, const T* target, T* grad, float* loss, T* grad_sum, uint32_t* arrived, const char* where) {
    mse_launch<T>(n, pred, target, grad, loss, grad_sum, arrived, where);
}
template <class T>
void gelu_backward_sum(size_t n, const T* dy, const T* u, T* du, T* grad_sum, uint32_t* arrived, const char* where) {
    gelu_backward_launch<T>(n, dy, u, du, grad_sum, arrived, where);
}
template <class T>
void sgd_update_layer(size_t n, float* w32, const T* grad, T* w16, float* b32, const T* grad_b, T* b16, float lr, float grad_scale, const char* where) {
    sgd_launch<T>(n, w32, grad, w16, lr, grad_scale, where, b32, grad_b, b16);
}
template void mse_loss_grad_sum<bf16>(size_t, const bf16*, const bf16*, bf16*, float*, bf16*, uint32_t*, const char*);
template void mse_loss_grad_sum<f16>(size_t, const f16*, const f16*, f16*, float*, f16*, uint32_t*, const char*);
template void gelu_backward_sum<bf16>(size_t, const bf16*, const bf16*, bf16*, bf16*, uint32_t*, const char*);
template void gelu_backward_sum<f16>(size_t, const f16*, const f16*, f16*, f16*, uint32_t*, const char*);
template void sgd_update_layer<bf16>(size_t, float*, const bf16*, bf16*, float*, const bf16*, bf16*, float, float, const char*);
template void sgd_update_layer<f16>(size_t, float*, const f16*, f16*, float*, const f16*, f16*, float, float, const char*);

}  // namespace mx

#define DEF_FUSED(T)                                                                                                                    \
    void mx_bias_gelu_##T(size_t n, const mx_##T* z, const mx_##T* bias, mx_##T* u, mx_##T* a) {                                        \
        mx::bias_gelu_launch<mx_##T>(n, z, bias, u, a, "mx_bias_gelu_" #T);                                                             \
    }                                                                                                                                   \
    void mx_gelu_backward_##T(size_t n, const mx_##T* dy, const mx_##T* u, mx_##T* du) {                                                \
        mx::gelu_backward_launch<mx_##T>(n, dy, u, du, nullptr, nullptr, "mx_gelu_backward_" #T);                                                \
    }                                                                                                                                   \
    void mx_mse_loss_grad_##T(size_t n, const mx_##T* pred, const mx_##T* target, mx_##T* grad, float* loss) {                          \
        mx::mse_launch<mx_##T>(n, pred, target, grad, loss, nullptr, nullptr, "mx_mse_loss_grad_" #T);                                           \
    }                                                                                                                                   \
    void mx_sgd_update_##T(size_t n, float* w32, const mx_##T* grad, mx_##T* w16, float lr, float grad_scale) {                         \
        mx::sgd_launch<mx_##T>(n, w32, grad, w16, lr, grad_scale, "mx_sgd_update_" #T);                                                 \
    }

// Linear forward in one call: u[rows, out] = x[rows, in] . w[out, in]^T + bias (one element), act = gelu(u) (act may be NULL).
// Large bf16 / f16 layers run the product on the tensor cores with bias and activation in its epilogue; any other
// shape runs cuda_matmul into u followed by the in-place bias / activation pass.  Both give the bits of the three separate
// ops of crates/maidenx_nn/src/layers/linear.rs:60-81 followed by gelu.
#define DEF_LINEAR(T, IS_BF16)                                                                                                          \
    void mx_linear_bias_gelu_##T(size_t rows, size_t in_features, size_t out_features, const mx_##T* x, const mx_##T* w, const mx_##T* bias, \
                                 mx_##T* u, mx_##T* act) {                                                                              \
        if (!rows || !in_features || !out_features) return;                                                                             \
        if (mx::tc_linear_bias_act(IS_BF16, rows, in_features, out_features, x, w, bias, u, act, "mx_linear_bias_gelu_" #T)) return;       \
        const size_t meta[] = {2, 2, 2, rows, out_features, rows, in_features, in_features, out_features, in_features, 1, 1, in_features, 0, 0}; \
        cuda_matmul_##T(rows * out_features, meta, x, w, u);                                                                            \
        mx::bias_gelu_launch<mx_##T>(rows * out_features, u, bias, u, act, "mx_linear_bias_gelu_" #T);                                    \
    }

extern "C" {
DEF_FUSED(bf16)
DEF_FUSED(f16)
DEF_FUSED(f32)
DEF_LINEAR(bf16, true)
DEF_LINEAR(f16, false)
}
