// Conv2d forward and backward composed from the op layer's own entry points, the way the reference's layer
// composes them (crates/maidenx_nn/src/layers/conv.rs:185-307 with the im2col / col2im wrappers at :333-420):
// im2col -> matmul -> (views) -> bias add, and in backward matmul -> col2im for the input gradient, matmul for
// the weight gradient and three sums for the bias gradient.  Every step is a call of a cuda_<op>_<dtype> symbol of
// this library with the metadata the reference's tensor layer would build, but for 16-bit types' input gradient (one product without columns, where that is faster) and
// the first two of their bias sums (one pass with the roundings of both), both in mode 1 alone.
//
// Two compositions are offered (argument `mode`):
//
//   0  "as the reference calls it".  The layer hands the ops a column buffer it declares as [B*oh*ow, C*kh*kw]
//      although im2col writes it as [B][C*kh*kw][oh*ow]; it passes (stride, padding) in the metadata slots where
//      the kernels read (padding, stride); col2im gets num_els = B*C*H*W, so it reads only that many column
//      entries; and the [C*kh*kw, Cout] weight gradient is re-labelled [Cout, C, kh, kw] without a transpose.
//      This mode reproduces those calls literally: it is what an unchanged maidenx_nn would execute on this
//      library, and it is the parity target for the call sequence.  (With stride == padding the slot swap is
//      invisible; the buffer re-labelling is not, so its results are not a convolution.)
//   1  "direct".  The same ops used consistently: the column buffer is read as the [B][K][P] array im2col
//      wrote, so out[b] = W[Cout, K] . cols[b][K, P] is one batched product with the weight shared by every
//      batch (a stride-0 leading dim, which is how Tensor::matmul broadcasts, crates/maidenx_tensor/src/ops/
//      matmul.rs:161-225); grad_cols[b] = W^T . g[b]; col2im reads the whole buffer; grad_W = sum_b g[b] . cols[b]^T.
//      This mode is a convolution and is checked against a direct f64 convolution.
//
// The caller owns every buffer, as everywhere in this ABI: `cols` (B*P*K elements) is written by forward and read
// by backward; `workspace` holds the intermediates (sizes from mx_conv2d_workspace_elems).
#include <algorithm>
#include <atomic>

#include "abi_common.cuh"
#include "matmul_tc.cuh"

namespace mx {

template <class T>
constexpr int half_kind_of() {
    return std::is_same<T, bf16>::value ? 1 : (std::is_same<T, f16>::value ? 2 : 0);
}

namespace {

struct Geometry {
    size_t B, C, H, W, Co, kh, kw, sh, sw, ph, pw, oh, ow, P, K;
};

bool geometry(const MxConv2d* c, Geometry& g) {
    if (!c || !c->batch || !c->in_channels || !c->out_channels || !c->kernel_h || !c->kernel_w || !c->stride_h || !c->stride_w) return false;
    g.B = c->batch;
    g.C = c->in_channels;
    g.H = c->height;
    g.W = c->width;
    g.Co = c->out_channels;
    g.kh = c->kernel_h;
    g.kw = c->kernel_w;
    g.sh = c->stride_h;
    g.sw = c->stride_w;
    g.ph = c->pad_h;
    g.pw = c->pad_w;
    if (g.H + 2 * g.ph < g.kh || g.W + 2 * g.pw < g.kw) return false;
    g.oh = (g.H + 2 * g.ph - g.kh) / g.sh + 1;  // conv.rs:198-199
    g.ow = (g.W + 2 * g.pw - g.kw) / g.sw + 1;
    g.P = g.oh * g.ow;
    g.K = g.C * g.kh * g.kw;
    return true;
}

size_t round16(size_t elems) { return (elems + 15) & ~(size_t)15; }  // keeps every sub-buffer 16-byte aligned for any dtype

// The op entry points of one dtype, with untyped pointers.
struct Ops {
    void (*im2col)(size_t, const size_t*, const void*, void*);
    void (*col2im)(size_t, const size_t*, const void*, void*);
    void (*matmul)(size_t, const size_t*, const void*, const void*, void*);
    void (*add)(size_t, size_t, const size_t*, const void*, const void*, void*);
    void (*add_inplace)(size_t, size_t, const size_t*, void*, const void*);
    void (*sum)(size_t, size_t, size_t, const size_t*, const void*, void*);
    void (*sum_to_shape)(size_t, size_t, const size_t*, const void*, void*);
    void (*contiguous)(size_t, size_t, const size_t*, const void*, void*);
    int half_kind;  // 1 bf16, 2 f16, 0 anything else
    bool is_f32;
};
#define MX_CONV_OPS(T)                                                                                                                  \
    mx::Ops {                                                                                                                           \
        reinterpret_cast<decltype(mx::Ops::im2col)>(cuda_conv2d_im2col_##T), reinterpret_cast<decltype(mx::Ops::col2im)>(cuda_conv2d_col2im_##T), \
            reinterpret_cast<decltype(mx::Ops::matmul)>(cuda_matmul_##T), reinterpret_cast<decltype(mx::Ops::add)>(cuda_add_##T),                 \
            reinterpret_cast<decltype(mx::Ops::add_inplace)>(cuda_add_inplace_##T), reinterpret_cast<decltype(mx::Ops::sum)>(cuda_sum_##T),        \
            reinterpret_cast<decltype(mx::Ops::sum_to_shape)>(cuda_sum_to_shape_##T),                                                     \
            reinterpret_cast<decltype(mx::Ops::contiguous)>(mx_contiguous_##T), mx::half_kind_of<mx_##T>(), std::is_same<mx_##T, float>::value                                  \
    }

// sum over one dim of a dense tensor, metadata as crates/maidenx_tensor/src/ops/reduction.rs:722-733 builds it
void sum_dim(const Ops& ops, const size_t* dims, size_t nd, size_t dim, const void* in, void* out) {
    size_t meta[2 * 8 + 3], strides[8], n = 1;
    for (size_t d = nd; d-- > 0;) {
        strides[d] = n;
        n *= dims[d];
    }
    for (size_t d = 0; d < nd; d++) {
        meta[d] = dims[d];
        meta[nd + d] = strides[d];
    }
    meta[2 * nd] = dims[dim];
    meta[2 * nd + 1] = strides[dim];
    meta[2 * nd + 2] = 0;
    ops.sum(n, nd, 1, meta, in, out);
}

// The first two of the bias gradient's sums, over rows and over their sums, each rounded: out[plane] = round(sum_h round(sum_w in[plane][h][w])).  A warp has a plane, G lanes a row of `nv`
// vectors, four rows in flight.  Bound by the trips of a warp through its plane, one after the other, and by HBM where planes fill the SMs: see plane_sums for where it is taken.
constexpr int kPlaneThreads = 256;
template <class T, int VEC, int G>
__global__ void __launch_bounds__(kPlaneThreads) plane_sums_kernel(const T* in, T* out, size_t planes, uint32_t h, uint32_t w) {
    after_previous_kernel();
    constexpr int Q = 4;
    constexpr uint32_t ROWS = 32 / G;
    const size_t plane = (size_t)blockIdx.x * (kPlaneThreads / 32) + threadIdx.x / 32;
    if (plane >= planes) return;
    const uint32_t lane = threadIdx.x % 32, nv = w / VEC, rounds = (nv + G - 1) / G;
    const T* p = in + plane * h * w;
    float sum = 0.0f;
    for (uint32_t r0 = lane / G; r0 - lane / G < h; r0 += Q * ROWS) {  // the same trips for every lane: the shuffles take the whole warp
        float acc[Q];
#pragma unroll
        for (int q = 0; q < Q; q++) acc[q] = 0.0f;
        for (uint32_t k = 0, v = lane % G; k < rounds; k++, v += G) {
            Vec<T, VEC> x[Q];
#pragma unroll
            for (int q = 0; q < Q; q++)
                if (r0 + q * ROWS < h && v < nv) x[q] = *reinterpret_cast<const Vec<T, VEC>*>(p + (size_t)(r0 + q * ROWS) * w + v * VEC);
#pragma unroll
            for (int q = 0; q < Q; q++)
                if (r0 + q * ROWS < h && v < nv)
#pragma unroll
                    for (int j = 0; j < VEC; j++) acc[q] += to_f32(x[q].v[j]);
        }
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1)
#pragma unroll
            for (int q = 0; q < Q; q++) acc[q] += __shfl_xor_sync(0xFFFFFFFFu, acc[q], o);
#pragma unroll
        for (int q = 0; q < Q; q++)
            if (r0 + q * ROWS < h) sum += to_f32(from_f32<T>(acc[q]));
    }
#pragma unroll
    for (int o = 16; o >= G; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    if (lane == 0) out[plane] = from_f32<T>(sum);
}
// false: the two sums as they are.  One warp a plane pays for small maps, where it saves a launch, until their planes fill the SMs (two sums / a warp each, us, bf16: 512 x 7 x 7 4.4 / 3.7, 840 x 27 x 24
// 5.5 / 4.8, 5720 x 32 x 32 6.5 / 5.5, 4576 x 14 x 14 5.4 / 5.1, 8475 x 10 x 10 5.8 / 6.8, 28556 x 6 x 5 6.1 / 9.2), and for many planes whose rows the first sum reads slower:
// bf16 vectors (16384 x 56 x 56 31.1 / 25.1, 8192 x 80 x 80 40.8 / 30.9, 9456 x 64 x 64 16.6 / 13.1, 9456 x 128 x 128 68.9 / 50.5; 2048 x 160 x 160 38.6 / 41.9, 3200 of them 58.7 / 48.0; f16,
// which it reads faster, 16384 x 56 x 56 21.4 / 24.5, 13024 x 112 x 112 51.6 / 57.9, but 4096 x 48 x 48 8.1 / 7.4; 1150 x 56 x 56 6.1 / 6.1) or elements in a
// warp's two rounds (16384 x 55 x 55 92 / 53, 2048 x 33 x 33 9.9 / 8.4; 16384 x 28 x 28 15.3 / 22.2, 4096 x 109 x 109 29.9 / 54.4).  A few large planes would wait for one
// warp each: 16 x 112 x 112 4.8 / 11.3, 16 x 109 x 109 4.8 / 26.3, 16 x 512 x 512 5.8 / 114.
template <class T>
bool plane_sums(const Geometry& g, const void* grad_out, void* out) {
    const bool vec = g.ow % 8 == 0 && (uintptr_t)grad_out % 16 == 0;
    const size_t planes = g.B * g.Co, nv = vec ? g.ow / 8 : g.ow;
    if (planes > 0x7FFFFFFFull || g.oh > 0x7FFFFFFFull || g.ow > 0x7FFFFFFFull) return false;
    const size_t lanes = vec && nv <= 4 ? 4 : nv <= 8 ? 8 : nv <= 16 ? 16 : 32, trips = (g.oh + 128 / lanes - 1) / (128 / lanes) * ((nv + lanes - 1) / lanes);
    const bool small = trips <= 2 && planes <= (trips > 1 ? 4608 : 8192);
    const bool of_vectors = std::is_same<T, bf16>::value ? g.ow >= 40 && g.ow <= 256 && (trips <= 14 || planes >= 3072) : trips >= 3 && trips <= 4 && g.ow >= 40 && g.ow % 64 != 0 && planes <= 8192;
    const bool many = planes >= 2048 && (vec ? of_vectors : trips <= 32 && g.ow > 32 && g.ow < 64);
    if (!small && !many) return false;
    const auto kernel = vec ? (lanes == 4 ? plane_sums_kernel<T, 8, 4> : lanes == 8 ? plane_sums_kernel<T, 8, 8> : lanes == 16 ? plane_sums_kernel<T, 8, 16> : plane_sums_kernel<T, 8, 32>)
                            : (lanes == 8 ? plane_sums_kernel<T, 1, 8> : lanes == 16 ? plane_sums_kernel<T, 1, 16> : plane_sums_kernel<T, 1, 32>);
    launch_kernel(kernel, (unsigned)((planes + kPlaneThreads / 32 - 1) / (kPlaneThreads / 32)), kPlaneThreads, 0, ctx().stream, static_cast<const T*>(grad_out), static_cast<T*>(out), planes,
                  (uint32_t)g.oh, (uint32_t)g.ow);
    check_launch("mx_conv2d_backward");
    return true;
}

// grad_bias = grad_out.sum(3).sum(2).sum(0) (conv.rs:283-288); tmp holds B*Co*oh + B*Co elements.  The first two as one pass in mode 1 alone: mode 0 is the reference's calls.
void bias_gradient(const Ops& ops, const Geometry& g, size_t es, int mode, const void* grad_out, char* tmp, void* grad_bias) {
    const size_t d4[4] = {g.B, g.Co, g.oh, g.ow}, d3[3] = {g.B, g.Co, g.oh}, d2[2] = {g.B, g.Co};
    char* t1 = tmp;
    char* t2 = tmp + round16(g.B * g.Co * g.oh) * es;
    const bool fused = mode == 1 && (ops.half_kind == 1 ? plane_sums<bf16>(g, grad_out, t2) : ops.half_kind == 2 && plane_sums<f16>(g, grad_out, t2));
    if (!fused) {
        sum_dim(ops, d4, 4, 3, grad_out, t1);
        sum_dim(ops, d3, 3, 2, t1, t2);
    }
    sum_dim(ops, d2, 2, 0, t2, grad_bias);
}

size_t workspace_elems(const Geometry& g, int mode, int backward) {
    const size_t sums = round16(g.B * g.Co * g.oh) + round16(g.B * g.Co);
    if (mode == 0) {
        if (!backward) return round16(g.B * g.P * g.Co);                                 // out_flat
        return round16(g.B * g.P * g.Co) + round16(g.B * g.P * g.K) + sums;              // grad_flat, grad_cols, sums
    }
    if (!backward) return 16;
    return round16(g.B * g.K * g.P) + round16(g.B * g.Co * g.K) + sums;                   // grad_cols, per-batch grad_W, sums
}

void forward(const Ops& ops, size_t es, const MxConv2d* c, int mode, const void* x, const void* w, const void* bias, void* cols, void* workspace,
             void* out) {
    Geometry g;
    if (!geometry(c, g) || !x || !w || !cols || !out || (mode == 0 && !workspace)) {
        set_error(kErrBadMetadata, 0, "mx_conv2d_forward");
        return;
    }
    if (mode == 0 && (g.ph == 0 || g.pw == 0)) {
        // the kernels would read the padding as their stride: a zero stride divides by zero in the reference's CPU backend
        set_error(kErrUnsupported, 0, "mx_conv2d_forward");
        return;
    }
    const size_t ncol = g.B * g.P * g.K;
    if (mode == 0) {
        // conv.rs:345-358: stride in the slots the kernels read as padding, and the other way round
        const size_t cm[12] = {g.B, g.C, g.H, g.W, g.kh, g.kw, g.oh, g.ow, g.sh, g.sw, g.ph, g.pw};
        ops.im2col(ncol, cm, x, cols);
        // cols declared [B*P, K] (conv.rs:334-337) . weight_matrix^T, the transposed view of [Co, K] (conv.rs:214-219)
        const size_t M = g.B * g.P;
        const size_t mm[15] = {2, 2, 2, M, g.Co, M, g.K, g.K, g.Co, g.K, 1, 1, g.K, 0, 0};
        ops.matmul(M * g.Co, mm, cols, w, workspace);
        // reshape [B, oh, ow, Co], transpose(1, 3), transpose(2, 3) (conv.rs:221-222): dims [B, Co, oh, ow] over the flat buffer
        const size_t vs[4] = {g.P * g.Co, 1, g.ow * g.Co, g.Co};
        if (bias) {
            // + bias.reshape([1, Co, 1, 1]) (conv.rs:224-228), broadcast = stride 0
            const size_t am[14] = {g.B, g.Co, g.oh, g.ow, vs[0], vs[1], vs[2], vs[3], 0, 1, 0, 0, 0, 0};
            ops.add(g.B * g.Co * g.P, 4, am, workspace, bias, out);
        } else {
            // the reference returns the strided view itself; here the caller gets its dense copy
            const size_t um[9] = {g.B, g.Co, g.oh, g.ow, vs[0], vs[1], vs[2], vs[3], 0};
            ops.contiguous(g.B * g.Co * g.P, 4, um, workspace, out);
        }
        return;
    }
    const size_t cm[12] = {g.B, g.C, g.H, g.W, g.kh, g.kw, g.oh, g.ow, g.ph, g.pw, g.sh, g.sw};
    ops.im2col(ncol, cm, x, cols);
    // out[B, Co, P] = W[Co, K] (shared by every batch) . cols[B, K, P]
    const size_t mm[20] = {3, 3, 3, g.B, g.Co, g.P, g.B, g.Co, g.K, g.B, g.K, g.P, 0, g.K, 1, g.K * g.P, g.P, 1, 0, 0};
    // 16-bit types: the bias add rides in the product's epilogue (same roundings as the two ops below) when the
    // tensor-core kernel takes the shape
    if (bias && ops.half_kind && tc_batched_row_bias(ops.half_kind == 1, g.B, g.Co, g.K, g.P, w, cols, bias, out, "mx_conv2d_forward")) return;
    ops.matmul(g.B * g.Co * g.P, mm, w, cols, out);
    if (bias) {
        const size_t am[11] = {g.B, g.Co, g.P, g.Co * g.P, g.P, 1, 0, 1, 0, 0, 0};
        ops.add_inplace(g.B * g.Co * g.P, 3, am, out, bias);
    }
}

std::atomic<int> g_implicit{1};  // 0: never, 2: wherever possible (tests, A/B timing)

// Whether the input gradient in one product is faster than by columns: half a tile's rows and a third of the SMs at least, and then by what the product takes (`per`: k-blocks of a 256-wide tile, one
// after the other on an SM, parts of tiles and of waves included) for each million elements of columns that are not written, multiplied and added up.  What columns cost goes by the planes of
// grad_out: whole 128-byte lines the first product and col2im read at their best, vectors off the lines less so, ragged planes several times that.  A kernel of 5 x 5 or 7 x 7 has the
// most columns for each input element; 1 x 1 is one product either way, without columns only where its planes lie off the lines.  Pixels of grad_out (its channels last)
// that are not whole 32-byte sectors cost the kernel half as much again and more (`whole`: 23 x 152 x 32 x 32, 5 x 5 to 208, 216, 224 channels 92, 141, 85 us, by columns 81; 1 x 184 x 112 x 112, 7 x 7
// to 440, 448 channels 198, 103, by columns 171).  The lines stand where 2500 random layers have them.  Columns / in one product, us: 3 x 3 64 x 256 x 56 x 56 -> 256 365 / 205, 24 x 352 x 56 x 56 -> 32
// 639 / 54, 36 x 224 x 14 x 14 -> 112 36 / 21; left: 11 x 88 x 56 x 56 -> 8 25 / 33, 50 x 112 x 28 x 28 -> 488 95 / 123, 3 x 223 x 56 x 56 -> 328 29 / 43; 7 x 7 34 x 208 x 14 x 14 -> 408 116 / 140; 1 x 1 23 x 427
// x 48 x 48 -> 8 31 / 49, but 48 x 344 x 14 x 14 -> 48 28 / 15.
bool implicit_pays(const Geometry& g) {
    const size_t most = 256 / g.W < g.H ? 256 / g.W : g.H, blocks = (g.H + most - 1) / most, rows = (g.H + blocks - 1) / blocks, bn = (rows * g.W + 15) / 16 * 16, sms = (size_t)sm_count();
    const size_t tiles = g.B * ((g.C + 127) / 128) * blocks, taps = g.kh * g.kw, num_kb = taps * ((g.Co + 63) / 64);
    if (g.C < 64 || tiles * 3 < sms) return false;
    const double serial = (double)((tiles + sms - 1) / sms * num_kb) * std::max((128 + bn) / 512.0, 0.4), columns = (double)g.B * g.K * g.P * 1e-6, per = serial / columns;
    const double useful = (double)g.B * g.C * g.H * g.W * taps * g.Co / (128.0 * 256 * 64) / ((double)sms * serial);  // of the multiplications
    const bool lines = g.P % 64 == 0, ragged = g.P % 8 != 0, whole = g.Co % 16 == 0;
    if (taps == 1) return !lines && (columns > 0.96 || tiles <= sms);
    if (taps >= 20 && lines && g.P > 64 && g.H * g.W % 64 == 0) {  // col2im writes whole lines too
        const bool seven = taps >= 40;
        if (g.Co % 64 == 0) return seven ? per <= 3.0 : per <= 1.7 || (per <= 2.7 && useful > 0.4);
        if (whole) return per <= (seven ? 1.8 : 1.4) || (per <= 2.2 && useful > 0.5);
        return per <= (seven ? 1.2 : 0.8);
    }
    if (taps >= 20) return ragged ? per <= (whole ? 6.0 : 4.0) || g.P < 64 : per <= (taps >= 40 ? 3.9 : 2.7);
    if (ragged) return whole ? per <= 2.7 || g.Co <= 280 : per <= 1.95 || g.Co <= 136 || (per <= 2.2 && useful > 0.6);
    if (lines) return columns > 31 ? per <= (whole ? 1.0 : 0.79) : columns > 21 && per <= 0.6 && useful > 1.0 / 12;
    return per <= 1.15 || per <= (columns > 60 ? 2.2 : columns > 30 ? 1.76 : 0.0) || (per <= 4.0 && useful > 0.6);
}

// 16-bit types, strides of 1: the input gradient without its columns, from grad_out with the channels last and the transposed weights, both in the place of the columns.
bool implicit_grad_x(const Ops& ops, const Geometry& g, const void* grad_out, const void* w, char* place, void* grad_x) {
    const int mode = g_implicit.load(std::memory_order_relaxed);
    if (!mode || !ops.half_kind || g.sh != 1 || g.sw != 1 || !conv_grad_input_fits(g.B, g.C, g.H, g.W, g.Co, g.kh, g.kw, g.ph, g.pw)) return false;
    const size_t g_elems = (g.B * g.P * g.Co + 63) / 64 * 64;
    char* base = reinterpret_cast<char*>(((uintptr_t)place + 127) & ~(uintptr_t)127);
    if (g_elems + g.K * g.Co + 64 > g.B * g.K * g.P) return false;
    if (mode == 1 && !implicit_pays(g)) return false;
    char *last = base, *wt = base + g_elems * 2;
    const size_t gm[7] = {g.B, g.P, g.Co, g.Co * g.P, 1, g.P, 0};
    ops.contiguous(g.B * g.P * g.Co, 3, gm, grad_out, last);
    const size_t wm[5] = {g.K, g.Co, 1, g.K, 0};
    ops.contiguous(g.K * g.Co, 2, wm, w, wt);
    return tc_conv_grad_input(ops.half_kind == 1, g.B, g.C, g.H, g.W, g.Co, g.kh, g.kw, g.ph, g.pw, g.oh, g.ow, last, wt, grad_x, "mx_conv2d_backward");
}

void backward(const Ops& ops, size_t es, const MxConv2d* c, int mode, const void* grad_out, const void* w, const void* cols, void* workspace,
              void* grad_x, void* grad_w, void* grad_bias) {
    Geometry g;
    if (!geometry(c, g) || !grad_out || !w || !cols || !workspace) {
        set_error(kErrBadMetadata, 0, "mx_conv2d_backward");
        return;
    }
    if (mode == 0 && (g.ph == 0 || g.pw == 0)) {
        set_error(kErrUnsupported, 0, "mx_conv2d_backward");
        return;
    }
    char* ws = static_cast<char*>(workspace);
    if (mode == 0) {
        char* grad_flat = ws;
        char* grad_cols = grad_flat + round16(g.B * g.P * g.Co) * es;
        char* sums = grad_cols + round16(g.B * g.P * g.K) * es;
        // grad_out.transpose(2, 3).transpose(1, 3) = dims [B, oh, ow, Co] over the dense [B, Co, oh, ow] buffer, then
        // reshape([B*P, Co]), which copies because the view is not contiguous (conv.rs:250-252)
        const size_t um[9] = {g.B, g.oh, g.ow, g.Co, g.Co * g.P, g.ow, 1, g.P, 0};
        ops.contiguous(g.B * g.P * g.Co, 4, um, grad_out, grad_flat);
        const size_t M = g.B * g.P;
        if (grad_x) {
            // grad_cols[B*P, K] = grad_flat[B*P, Co] . weight_matrix[Co, K] (conv.rs:254)
            const size_t mm[15] = {2, 2, 2, M, g.K, M, g.Co, g.Co, g.K, g.Co, 1, g.K, 1, 0, 0};
            ops.matmul(M * g.K, mm, grad_flat, w, grad_cols);
            // col2im with num_els = B*C*H*W and the same slot order as im2col (conv.rs:390-409)
            const size_t cm[12] = {g.B, g.C, g.H, g.W, g.kh, g.kw, g.oh, g.ow, g.sh, g.sw, g.ph, g.pw};
            ops.col2im(g.B * g.C * g.H * g.W, cm, grad_cols, grad_x);
        }
        if (grad_w) {
            // cols.transpose(-1, -2)[K, B*P] . grad_flat[B*P, Co] (conv.rs:277); the [K, Co] result is what the layer
            // then labels [Co, C, kh, kw]
            const size_t mm[15] = {2, 2, 2, g.K, g.Co, g.K, M, M, g.Co, 1, g.K, g.Co, 1, 0, 0};
            ops.matmul(g.K * g.Co, mm, cols, grad_flat, grad_w);
        }
        if (grad_bias) bias_gradient(ops, g, es, mode, grad_out, sums, grad_bias);
        return;
    }
    char* grad_cols = ws;
    char* gw_batch = grad_cols + round16(g.B * g.K * g.P) * es;
    char* sums = gw_batch + round16(g.B * g.Co * g.K) * es;
    if (grad_x && !implicit_grad_x(ops, g, grad_out, w, grad_cols, grad_x)) {
        // grad_cols[B, K, P] = W^T (the transposed view of [Co, K], shared by every batch) . grad_out[B, Co, P]
        const size_t mm[20] = {3, 3, 3, g.B, g.K, g.P, g.B, g.K, g.Co, g.B, g.Co, g.P, 0, 1, g.K, g.Co * g.P, g.P, 1, 0, 0};
        ops.matmul(g.B * g.K * g.P, mm, w, grad_out, grad_cols);
        const size_t cm[12] = {g.B, g.C, g.H, g.W, g.kh, g.kw, g.oh, g.ow, g.ph, g.pw, g.sh, g.sw};
        ops.col2im(g.B * g.K * g.P, cm, grad_cols, grad_x);
    }
    // f32: the sum over the batch is part of the product's reduction where the tensor-core kernel takes it; no per-batch
    // gradient is written and read back (38 MB at 32 x 128 x 14 x 14, 256 channels: product and sum 45 us, now 37).  16-bit types keep the composition's rounding
    // of each batch's gradient.
    if (grad_w && !(ops.is_f32 && tc_batch_sum_f32(g.B, g.Co, g.K, g.P, static_cast<const float*>(grad_out), static_cast<const float*>(cols), static_cast<float*>(grad_w),
                                                   "mx_conv2d_backward"))) {
        // per batch grad_out[b][Co, P] . cols[b]^T (the transposed view of [K, P]), then the sum over the batch
        const size_t mm[20] = {3, 3, 3, g.B, g.Co, g.K, g.B, g.Co, g.P, g.B, g.P, g.K, g.Co * g.P, g.P, 1, g.K * g.P, 1, g.P, 0, 0};
        ops.matmul(g.B * g.Co * g.K, mm, grad_out, cols, gw_batch);
        const size_t d3[3] = {g.B, g.Co, g.K};
        sum_dim(ops, d3, 3, 0, gw_batch, grad_w);
    }
    if (grad_bias && es >= 4) {
        // the bias is broadcast over [B, Co, P]: one fold to [1, Co, 1] (16-bit types keep the roundings of the three sums)
        const size_t fm[10] = {g.B, g.Co, g.P, g.Co * g.P, g.P, 1, 1, g.Co, 1, 0};
        ops.sum_to_shape(g.B * g.Co * g.P, 3, fm, grad_out, grad_bias);
    } else if (grad_bias) {
        bias_gradient(ops, g, es, mode, grad_out, sums, grad_bias);
    }
}

}  // namespace
}  // namespace mx

extern "C" {

size_t mx_conv2d_cols_elems(const MxConv2d* conv) {
    mx::Geometry g;
    return mx::geometry(conv, g) ? g.B * g.P * g.K : 0;
}
size_t mx_conv2d_output_elems(const MxConv2d* conv) {
    mx::Geometry g;
    return mx::geometry(conv, g) ? g.B * g.Co * g.P : 0;
}
size_t mx_conv2d_workspace_elems(const MxConv2d* conv, int mode, int backward) {
    mx::Geometry g;
    return mx::geometry(conv, g) ? mx::workspace_elems(g, mode, backward) : 0;
}

#define DEF_CONV2D(T)                                                                                                                   \
    void mx_conv2d_forward_##T(const MxConv2d* conv, int mode, const mx_##T* x, const mx_##T* weight, const mx_##T* bias, mx_##T* cols, \
                               mx_##T* workspace, mx_##T* out) {                                                                        \
        mx::forward(MX_CONV_OPS(T), sizeof(mx_##T), conv, mode, x, weight, bias, cols, workspace, out);                                 \
    }                                                                                                                                   \
    void mx_conv2d_backward_##T(const MxConv2d* conv, int mode, const mx_##T* grad_out, const mx_##T* weight, const mx_##T* cols,       \
                                mx_##T* workspace, mx_##T* grad_x, mx_##T* grad_weight, mx_##T* grad_bias) {                            \
        mx::backward(MX_CONV_OPS(T), sizeof(mx_##T), conv, mode, grad_out, weight, cols, workspace, grad_x, grad_weight, grad_bias);    \
    }
DEF_CONV2D(bf16)
DEF_CONV2D(f16)
DEF_CONV2D(f32)
DEF_CONV2D(f64)

// 1 (default): a 16-bit layer's input gradient is one product without columns by the rule on its sizes; 0: never; 2: wherever possible
void mx_debug_set_conv_implicit(int mode) { mx::g_implicit.store(mode, std::memory_order_relaxed); }

}  // extern "C"
