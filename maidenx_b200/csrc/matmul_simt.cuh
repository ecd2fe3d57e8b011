// General batched matmul on the CUDA cores: every dtype, every stride pattern, and the
// index quirks of the reference (the parity target is crates/maidenx_cpu/src/ops/matmul.rs).
// The tensor-core paths (matmul_tc.cu, matmul_tc_f32.cu) take the larger products of dense bf16 / f16 /
// f32 operands; these kernels are the rest of those and the only path for f64 and integers.
//
// The same index functions serve forward and both backward products.  The kernels compute
//     out[row * N + col] = sum_{r < K} X[ix(row, r)] * Y[iy(row, r, col)]
// with affine index functions, row = batch * M + mi:
//     ix = batch * xs_b + mi * xs_m + r * xs_r        (term skipped when ix >= x_limit)
//     iy = batch * ys_b + r * ys_r + col * ys_c       (term skipped when iy >= y_limit)
// which covers C = A.B with contiguous or strided operands (matmul.rs:74-113),
// grad_a = g.B^T (:196-219) and grad_b = A^T.g (:231-261), whose loops read A, B and g as
// contiguous whatever their strides, and the bounds checks those loops carry.
//
// Accumulation order is k ascending inside one thread, so results are reproducible and:
// integers are exact (wrapping), f32 / f64 match the reference's element-type accumulation
// bit for bit (no FMA contraction), bf16 / f16 accumulate in f32 and round once.
#pragma once
#include "common.cuh"
#include "ops.cuh"

namespace mx {

struct MmParams {
    uint64_t rows;      // number of output rows (batch * M, or ceil(out_elems / N))
    uint64_t N, K;      // output columns, reduction length
    uint64_t M;         // rows per batch
    uint64_t out_elems; // elements of out that may be written (last row may be short)
    int64_t xs_b, xs_m, xs_r;
    int64_t ys_b, ys_r, ys_c;
    uint64_t x_limit, y_limit;
};

template <class T>
struct MmAcc {
    typedef typename std::conditional<is_half_v<T>, f32,
            typename std::conditional<is_fp_v<T>, T,
            typename std::conditional<sizeof(T) == 8, u64, u32>::type>::type>::type type;
};
template <class T>
__device__ __forceinline__ typename MmAcc<T>::type mm_load(T v) {
    if constexpr (is_half_v<T>) return to_f32(v);
    else return (typename MmAcc<T>::type)v;
}
template <class T>
__device__ __forceinline__ T mm_store(typename MmAcc<T>::type a) {
    if constexpr (is_half_v<T>) return from_f32<T>(a);
    else return (T)a;
}

constexpr int kMmThreads = 256;

// TILE x TILE outputs of one batch per block: 64 (4 x 4 per thread), or 32 (2 x 2) for products whose 64-wide tiles would leave
// most SMs without a block.  Row and batch are resolved once per loaded element, not once per k-step (a 64-bit division each), and
// the next k-step's operands are on their way from memory while the current one is multiplied.  Bound by that latency
// for small products, by the separate multiply and add for large ones.  f32: 64 x 64 x 512 17 us (163 before), 256 x 256 x 128 5.8 (42).
template <class T, int TILE>
__global__ void __launch_bounds__(kMmThreads) matmul_simt_kernel(const T* X, const T* Y, T* out, MmParams P, uint32_t tiles_m, uint64_t first) {
    after_previous_kernel();
    typedef typename MmAcc<T>::type Acc;
    constexpr int kMmK = TILE == 32 ? (sizeof(Acc) == 8 ? 32 : 64) : 16;  // reduction step: the narrow tile is for products with few blocks, which wait for memory once per step
    constexpr int PER = TILE / 16, LOADS = TILE * kMmK / kMmThreads;
    __shared__ Acc xs[2][kMmK][TILE + 1];  // [buffer][r][row]
    __shared__ Acc ys[2][kMmK][TILE + 1];  // [buffer][r][col]
    const uint64_t batch = (first + blockIdx.x) / tiles_m;
    const uint64_t m0 = (first + blockIdx.x) % tiles_m * TILE, col0 = (uint64_t)blockIdx.y * TILE;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;  // 16 x 16 threads; rows ty + 16 i, columns tx + 16 j
    Acc acc[PER][PER];
#pragma unroll
    for (int i = 0; i < PER; i++)
#pragma unroll
        for (int j = 0; j < PER; j++) acc[i][j] = (Acc)0;

    // loader mapping: pick the fast index along the operand's smaller stride
    const bool x_r_fast = (P.xs_r <= P.xs_m) || P.xs_m == 0;
    const bool y_c_fast = (P.ys_c <= P.ys_r) || P.ys_r == 0;
    uint64_t ix[LOADS], iy[LOADS];       // element index at the k-step to be loaded next
    int xr[LOADS], yr[LOADS];            // its r inside the step; -1: a row or column outside the matrix
    int xo[LOADS], yo[LOADS];            // its row or column inside the tile
#pragma unroll
    for (int it = 0; it < LOADS; it++) {
        const int e = threadIdx.x + it * kMmThreads;
        const int r = x_r_fast ? e % kMmK : e / TILE, row = x_r_fast ? e / kMmK : e % TILE;
        const uint64_t mi = m0 + row;
        xo[it] = r * (TILE + 1) + row;
        xr[it] = mi < P.M && batch * P.M + mi < P.rows ? r : -1;
        ix[it] = (uint64_t)((int64_t)batch * P.xs_b + (int64_t)mi * P.xs_m + (int64_t)r * P.xs_r);
        const int yrr = y_c_fast ? e / TILE : e % kMmK, col = y_c_fast ? e % TILE : e / kMmK;
        yo[it] = yrr * (TILE + 1) + col;
        yr[it] = col0 + col < P.N ? yrr : -1;
        iy[it] = (uint64_t)((int64_t)batch * P.ys_b + (int64_t)yrr * P.ys_r + (int64_t)(col0 + col) * P.ys_c);
    }
    Acc xv[LOADS], yv[LOADS];
    auto load = [&](uint64_t k0) {
#pragma unroll
        for (int it = 0; it < LOADS; it++) {
            xv[it] = xr[it] >= 0 && k0 + xr[it] < P.K && ix[it] < P.x_limit ? mm_load<T>(X[ix[it]]) : (Acc)0;
            yv[it] = yr[it] >= 0 && k0 + yr[it] < P.K && iy[it] < P.y_limit ? mm_load<T>(Y[iy[it]]) : (Acc)0;
            ix[it] += (uint64_t)(kMmK * P.xs_r);
            iy[it] += (uint64_t)(kMmK * P.ys_r);
        }
    };
    load(0);
    int buf = 0;
    for (uint64_t k0 = 0; k0 < P.K; k0 += kMmK, buf ^= 1) {
        Acc* xt = &xs[buf][0][0];
        Acc* yt = &ys[buf][0][0];
#pragma unroll
        for (int it = 0; it < LOADS; it++) {
            xt[xo[it]] = xv[it];
            yt[yo[it]] = yv[it];
        }
        __syncthreads();  // one per step: the buffer written next was last read before the previous step's barrier
        if (k0 + kMmK < P.K) load(k0 + kMmK);
#pragma unroll
        for (int kk = 0; kk < kMmK; kk++) {
            Acc xk[PER], yk[PER];
#pragma unroll
            for (int i = 0; i < PER; i++) {
                xk[i] = xs[buf][kk][ty + 16 * i];
                yk[i] = ys[buf][kk][tx + 16 * i];
            }
#pragma unroll
            for (int i = 0; i < PER; i++)
#pragma unroll
                for (int j = 0; j < PER; j++) {
                    if constexpr (is_half_v<T>) acc[i][j] = fmaf(xk[i], yk[j], acc[i][j]);  // product exact in f32
                    else acc[i][j] = acc[i][j] + xk[i] * yk[j];
                }
        }
    }
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const uint64_t mi = m0 + ty + 16 * i, row = batch * P.M + mi;
        if (mi >= P.M || row >= P.rows) continue;
#pragma unroll
        for (int j = 0; j < PER; j++) {
            const uint64_t col = col0 + tx + 16 * j, o = row * P.N + col;
            if (col < P.N && o < P.out_elems) out[o] = mm_store<T>(acc[i][j]);
        }
    }
}

// Many small batches: a tile is 64 output rows whatever batch they belong to.  Rows of the tile's first batch multiply from shared
// memory, the others read their Y element by element, which short reductions of a few rows a batch cost less than a block a
// batch does ([16000] x 1 x 1 x 16 f32: 16 us, 144 with a block each).  Which one: simt_rows_pay.  The order of additions is the same.
template <class T>
__global__ void __launch_bounds__(kMmThreads) matmul_simt_rows_kernel(const T* X, const T* Y, T* out, MmParams P) {
    after_previous_kernel();
    typedef typename MmAcc<T>::type Acc;
    constexpr int TILE = 64, STEP = 16;
    __shared__ Acc xs[STEP][TILE + 1];  // [r][row]
    __shared__ Acc ys[STEP][TILE + 1];  // [r][col]
    const uint64_t row0 = (uint64_t)blockIdx.x * TILE, col0 = (uint64_t)blockIdx.y * TILE;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;  // 16 x 16 threads, 4 x 4 outputs each
    Acc acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = (Acc)0;

    // loader mapping: pick the fast index along the operand's smaller stride
    const bool x_r_fast = (P.xs_r <= P.xs_m) || P.xs_m == 0;
    const bool y_c_fast = (P.ys_c <= P.ys_r) || P.ys_r == 0;

    for (uint64_t k0 = 0; k0 < P.K; k0 += STEP) {
#pragma unroll
        for (int it = 0; it < (TILE * STEP) / kMmThreads; it++) {
            int e = threadIdx.x + it * kMmThreads;
            int lr, lrow;
            if (x_r_fast) {
                lr = e % STEP;
                lrow = e / STEP;
            } else {
                lrow = e % TILE;
                lr = e / TILE;
            }
            uint64_t row = row0 + lrow, r = k0 + lr;
            Acc v = (Acc)0;
            if (row < P.rows && r < P.K) {
                uint64_t batch = row / P.M, mi = row % P.M;
                uint64_t ix = (uint64_t)((int64_t)batch * P.xs_b + (int64_t)mi * P.xs_m + (int64_t)r * P.xs_r);
                if (ix < P.x_limit) v = mm_load<T>(X[ix]);
            }
            xs[lr][lrow] = v;
        }
#pragma unroll
        for (int it = 0; it < (TILE * STEP) / kMmThreads; it++) {
            int e = threadIdx.x + it * kMmThreads;
            int lr, lcol;
            if (y_c_fast) {
                lcol = e % TILE;
                lr = e / TILE;
            } else {
                lr = e % STEP;
                lcol = e / STEP;
            }
            // Y is staged for the batch of the tile's first row; rows of other batches read theirs from memory
            uint64_t col = col0 + lcol, r = k0 + lr;
            Acc v = (Acc)0;
            if (col < P.N && r < P.K) {
                uint64_t batch = row0 / P.M;
                uint64_t iy = (uint64_t)((int64_t)batch * P.ys_b + (int64_t)r * P.ys_r + (int64_t)col * P.ys_c);
                if (iy < P.y_limit) v = mm_load<T>(Y[iy]);
            }
            ys[lr][lcol] = v;
        }
        __syncthreads();
        const uint64_t batch0 = row0 / P.M;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            uint64_t row = row0 + ty * 4 + i;
            if (row >= P.rows) continue;
            uint64_t batch = row / P.M;
            if (batch == batch0) {
#pragma unroll
                for (int kk = 0; kk < STEP; kk++) {
                    Acc xv = xs[kk][ty * 4 + i];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        if constexpr (is_half_v<T>) acc[i][j] = fmaf(xv, ys[kk][tx * 4 + j], acc[i][j]);  // product exact in f32
                        else acc[i][j] = acc[i][j] + xv * ys[kk][tx * 4 + j];
                    }
                }
            } else {
                // this row belongs to a later batch than the staged Y tile: read Y directly
                for (int kk = 0; kk < STEP; kk++) {
                    uint64_t r = k0 + kk;
                    if (r >= P.K) break;
                    Acc xv = xs[kk][ty * 4 + i];
                    for (int j = 0; j < 4; j++) {
                        uint64_t col = col0 + tx * 4 + j;
                        Acc yv = (Acc)0;
                        if (col < P.N) {
                            uint64_t iy = (uint64_t)((int64_t)batch * P.ys_b + (int64_t)r * P.ys_r + (int64_t)col * P.ys_c);
                            if (iy < P.y_limit) yv = mm_load<T>(Y[iy]);
                        }
                        if constexpr (is_half_v<T>) acc[i][j] = fmaf(xv, yv, acc[i][j]);
                        else acc[i][j] = acc[i][j] + xv * yv;
                    }
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        uint64_t row = row0 + ty * 4 + i;
        if (row >= P.rows) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            uint64_t col = col0 + tx * 4 + j;
            uint64_t o = row * P.N + col;
            if (col < P.N && o < P.out_elems) out[o] = mm_store<T>(acc[i][j]);
        }
    }
}

// The two kernels' times from their parts, measured over 300 to 100000 batches, M 1 to 33, N 1 to 128 and K 8 to 300: a block of
// matmul_simt_kernel takes 2.7 ns of the chip and 6.2 more a k-step; 64 shared rows 8 ns and, for every term, 1.6 and 0.5 for each of a
// thread's four columns and 0.04 for further ones, and their chain of loads cannot be shorter than 2 us and 0.7 to 1.5 us a term.  Of 401
// products (f32, f64, i32, bf16) two take the slower kernel by more than a tenth, [4000] x 4 x 20 x 200 f64 440 / 519 us.
inline bool simt_rows_pay(uint64_t rows, uint64_t M, uint64_t N, uint64_t K) {
    if (rows <= M || M >= 64) return false;
    const double own = N < 4 ? (double)N : 4.0, more = N < 64 ? (double)N - own : 60.0, tiles_n = (double)((N + 63) / 64), steps = (double)((K + 15) / 16);
    const double block = (double)((rows + M - 1) / M) * tiles_n * (2.7 + 6.2 * steps);
    const double shared = (double)((rows + 63) / 64) * tiles_n * (8.0 + (double)K * (1.6 + 0.5 * own + 0.04 * more));
    const double chain = 2000.0 + (double)K * (400.0 + 275.0 * own);
    return (shared > chain ? shared : chain) < 0.9 * block;
}

// Few outputs, long reduction (the weight gradient of a narrow Linear layer: [1, batch] . [batch, in] in the reference's
// README example): the tiled kernel would run the whole reduction in one or two blocks.  Here one block owns one output
// element, its threads take k = t, t + 256, ... (each in ascending order) and the partial sums are folded by a fixed
// shuffle tree, so the result is reproducible; integers stay exact (wrapping addition is associative), floats are summed
// in a different order than the element-type loop of the reference and agree with it within the reduction tolerance.
template <class T>
__global__ void __launch_bounds__(kMmThreads) matmul_longk_kernel(const T* X, const T* Y, T* out, MmParams P) {
    after_previous_kernel();
    typedef typename MmAcc<T>::type Acc;
    const uint64_t o = blockIdx.x;
    const uint64_t row = o / P.N, col = o % P.N;
    const uint64_t batch = row / P.M, mi = row % P.M;
    const int64_t x0 = (int64_t)batch * P.xs_b + (int64_t)mi * P.xs_m, y0 = (int64_t)batch * P.ys_b + (int64_t)col * P.ys_c;
    Acc acc = (Acc)0;
    for (uint64_t r = threadIdx.x; r < P.K; r += kMmThreads) {
        const uint64_t ix = (uint64_t)(x0 + (int64_t)r * P.xs_r), iy = (uint64_t)(y0 + (int64_t)r * P.ys_r);
        const Acc xv = ix < P.x_limit ? mm_load<T>(X[ix]) : (Acc)0, yv = iy < P.y_limit ? mm_load<T>(Y[iy]) : (Acc)0;
        if constexpr (is_half_v<T>) acc = fmaf(xv, yv, acc);
        else acc = acc + xv * yv;
    }
    __shared__ Acc part[kMmThreads / 32];
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) acc = acc + __shfl_down_sync(0xFFFFFFFFu, acc, s);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        Acc total = part[0];
#pragma unroll
        for (int w = 1; w < kMmThreads / 32; w++) total = total + part[w];
        if (o < P.out_elems) out[o] = mm_store<T>(total);
    }
}
constexpr uint64_t kLongKMinK = 2048, kLongKMaxOutputs = 1024;

// Host-side description of one matmul call, parsed from the metadata block
// [out_ndim, a_ndim, b_ndim | out_shape | a_shape | b_shape | a_strides | b_strides | a_off, b_off]
// (crates/maidenx_tensor/src/ops/matmul.rs:227-264).
struct MmDesc {
    bool valid;
    size_t out_nd, a_nd, b_nd;
    uint64_t m, n, k_fwd, k_bwd;
    uint64_t g_size;               // product of out_shape (1 when out_ndim == 0)
    bool a_cont, b_cont;
    int64_t a_strides[3];          // batch (a_strides[0]), row (a_strides[nd-2]), col (a_strides[nd-1]); rank 1: col only
    int64_t b_strides[3];
    uint64_t a_off, b_off;
    uint64_t a_elems, b_elems;     // products of the operands' shapes
};
bool mm_parse(const size_t* hm, MmDesc& d);
size_t mm_meta_words(const size_t* head3);

template <class T>
void mm_launch(const MmParams& P, const T* X, const T* Y, T* out, const char* where) {
    if (P.rows == 0 || P.N == 0) return;
    if (P.K >= kLongKMinK && P.out_elems <= kLongKMaxOutputs && P.rows * P.N <= kLongKMaxOutputs) {
        launch_kernel(matmul_longk_kernel<T>, (unsigned)P.out_elems, kMmThreads, 0, ctx().stream, X, Y, out, P);
        check_launch(where);
        return;
    }
    if (P.M && simt_rows_pay(P.rows, P.M, P.N, P.K)) {
        const uint64_t gx = (P.rows + 63) / 64, gy = (P.N + 63) / 64;
        if (gy <= 65535 && gx <= 0x7FFFFFFFull) {
            launch_kernel(matmul_simt_rows_kernel<T>, dim3((unsigned)gx, (unsigned)gy), kMmThreads, 0, ctx().stream, X, Y, out, P);
            check_launch(where);
            return;
        }
    }
    const uint64_t batches = (P.rows + P.M - 1) / P.M;
    auto go = [&](auto kernel, uint64_t tile) {
        const uint64_t tiles_m = ((P.M < P.rows ? P.M : P.rows) + tile - 1) / tile, gx = batches * tiles_m, gy = (P.N + tile - 1) / tile;
        if (gy > 65535) {  // more than 4M output columns
            set_error(kErrUnsupported, 0, where);
            return;
        }
        for (uint64_t first = 0; first < gx; first += 0x7FFFFFFFull) {
            const uint64_t count = gx - first < 0x7FFFFFFFull ? gx - first : 0x7FFFFFFFull;
            launch_kernel(kernel, dim3((unsigned)count, (unsigned)gy), kMmThreads, 0, ctx().stream, X, Y, out, P, (uint32_t)tiles_m, first);
        }
        check_launch(where);
    };
    const uint64_t m = P.M < P.rows ? P.M : P.rows;
    if (batches * ((m + 63) / 64) * ((P.N + 63) / 64) < (uint64_t)sm_count()) go(matmul_simt_kernel<T, 32>, 32);
    else go(matmul_simt_kernel<T, 64>, 64);
}

}  // namespace mx
