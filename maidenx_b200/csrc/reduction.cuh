// Reductions: sum / mean / max / min along dims and sum_to_shape (the broadcast-gradient
// fold of backward).
//
// The reference scatters every input element into out[fold(i)] with one global atomic per
// element (crates/maidenx_cuda/kernels/ops/reduction.cu:18-63) or one mutex acquisition
// (crates/maidenx_cpu/src/ops/reduction.rs:45-58).  Here the host recognises the
// contiguous [outer O, reduced R, inner I] structure and runs one of:
//   rows    (I == 1) each row of R contiguous elements is reduced by a thread, a warp or
//           a block (by length) with 16-byte loads and a warp-shuffle tree; when there are
//           too few rows to fill the GPU each row is split over several blocks;
//   cols    (I > 1) each thread owns a 16-byte strip of columns and walks down R; R is split
//           over blockIdx.y so that a [8192,16384] -> [16384] fold still fills 148 SMs;
// split reductions write per-block partials to scratch and a second launch folds them:
// the classic two-pass grid reduce.  These paths are atomic-free, so their results are
// deterministic, and the output is overwritten (no pre-zero contract).
//   outer   (sum_to_shape of [Q, O, I] to [1, O, 1]: the gradient of a per-channel operand) one of the two above down to
//           wide partials, [O, I] sums over Q or [Q, O] sums over I, and a second launch that folds those; many outputs of
//           few elements each, and partials that no memory is to be had for, take the scatter below.
// Accumulation: bf16/f16 in f32 with one final rounding, f32 in f32, f64 in f64, integers
// wrapping in 32/64 bits (truncation to the element width commutes with wrapping adds).
// Anything else (several reduced dims, non-contiguous input, partial sum_to_shape
// factors) follows the reference's index formulas literally through a scatter kernel with
// wide atomics into scratch.
#pragma once
#include <cfloat>

#include "common.cuh"
#include "ops.cuh"

namespace mx {

enum RedKind { RED_SUM = 0, RED_MEAN = 1, RED_MAX = 2, RED_MIN = 3 };

// ---------------------------------------------------------------------------------
// accumulator traits
// ---------------------------------------------------------------------------------
template <class T, int KIND>
struct RedTraits;

template <class T>
struct SumAcc {
    typedef typename std::conditional<is_half_v<T>, f32,
            typename std::conditional<is_fp_v<T>, T,
            typename std::conditional<sizeof(T) == 8, u64, u32>::type>::type>::type type;
};
template <class T>
struct MaxAcc {
    typedef typename std::conditional<is_half_v<T>, f32,
            typename std::conditional<is_fp_v<T>, T,
            typename std::conditional<sizeof(T) == 8, T,
            typename std::conditional<std::is_signed<T>::value, i32, u32>::type>::type>::type>::type type;
};

template <class T, int KIND>
struct RedTraits {
    static constexpr bool kIsSum = KIND == RED_SUM || KIND == RED_MEAN;
    typedef typename std::conditional<kIsSum, typename SumAcc<T>::type, typename MaxAcc<T>::type>::type Acc;

    __host__ __device__ static Acc init() {
        if constexpr (kIsSum) return (Acc)0;
        else if constexpr (KIND == RED_MAX) {
            // crates/maidenx_cpu/src/ops/reduction.rs:603-614: T::MIN; for 16-bit floats f32::MIN rounds to -inf
            if constexpr (is_half_v<T>) return -INFINITY;
            else if constexpr (std::is_same<T, f32>::value) return -FLT_MAX;
            else if constexpr (std::is_same<T, f64>::value) return -DBL_MAX;
            else return (Acc)std::numeric_limits<T>::min();
        } else {
            if constexpr (is_half_v<T>) return INFINITY;
            else if constexpr (std::is_same<T, f32>::value) return FLT_MAX;
            else if constexpr (std::is_same<T, f64>::value) return DBL_MAX;
            else return (Acc)std::numeric_limits<T>::max();
        }
    }
    __device__ __forceinline__ static Acc load(T v) {
        if constexpr (is_half_v<T>) return to_f32(v);
        else return (Acc)v;  // integers: sign- or zero-extended, then wrapped in Acc
    }
    __device__ __forceinline__ static Acc combine(Acc a, Acc v) {
        // max / min: a NaN never wins (the reference's `if val > *out`), whichever side of a
        // pairwise combine it arrives on.
        if constexpr (kIsSum) return a + v;
        else if constexpr (std::is_same<Acc, f32>::value) {
            // the hardware max / min return the other operand when one is NaN, and the initial
            // value is never NaN, so a NaN can only survive a combine of two NaNs and then loses
            // the next one: the same outcome as the reference's comparison, in one instruction
            if constexpr (KIND == RED_MAX) return fmaxf(a, v);
            else return fminf(a, v);
        } else if constexpr (std::is_same<Acc, f64>::value) {
            if constexpr (KIND == RED_MAX) return fmax(a, v);
            else return fmin(a, v);
        } else if constexpr (KIND == RED_MAX) return v > a ? v : a;
        else return v < a ? v : a;
    }
    // factor: number of reduced elements (mean only)
    __device__ __forceinline__ static T finalize(Acc a, u64 factor) {
        if constexpr (KIND == RED_MEAN) {
            // the reference divides the finished sum by the count converted to the element type
            if constexpr (is_half_v<T>) return from_f32<T>(a / to_f32(from_f32<T>((f32)factor)));
            else return (T)(a / (Acc)(T)factor);
        } else if constexpr (is_half_v<T>) return from_f32<T>(a);
        else return (T)a;
    }
};

// ---------------------------------------------------------------------------------
// block / warp reduce
// ---------------------------------------------------------------------------------
template <class TR>
__device__ __forceinline__ typename TR::Acc warp_reduce(typename TR::Acc v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = TR::combine(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    return v;
}
template <class TR, int THREADS>
__device__ __forceinline__ typename TR::Acc block_reduce(typename TR::Acc v) {
    __shared__ typename TR::Acc warp_part[THREADS / 32];
    v = warp_reduce<TR>(v);
    if ((threadIdx.x & 31) == 0) warp_part[threadIdx.x >> 5] = v;
    __syncthreads();
    v = threadIdx.x < THREADS / 32 ? warp_part[threadIdx.x] : TR::init();
    if (threadIdx.x < 32) v = warp_reduce<TR>(v);
    return v;  // valid in thread 0
}

constexpr int kRedThreads = 256;

// ---------------------------------------------------------------------------------
// rows: in[row * R + r], out[row]
// ---------------------------------------------------------------------------------
// One block per (row, split).  grid = (splits, rows).  VEC > 1 requires R % VEC == 0,
// seg % VEC == 0 and a 16-byte aligned base.
template <class T, int KIND, int VEC, class Src, class SrcTR>
__device__ __forceinline__ typename SrcTR::Acc row_segment(const Src* row, u64 begin, u64 end) {
    typedef typename SrcTR::Acc Acc;
    Acc acc0 = SrcTR::init(), acc1 = SrcTR::init(), acc2 = SrcTR::init(), acc3 = SrcTR::init();
    const u64 step = (u64)kRedThreads * VEC;
    u64 i = begin + (u64)threadIdx.x * VEC;
    // four independent vector loads in flight per thread
    for (; i + 3 * step < end; i += 4 * step) {
        Vec<Src, VEC> a = *reinterpret_cast<const Vec<Src, VEC>*>(row + i);
        Vec<Src, VEC> b = *reinterpret_cast<const Vec<Src, VEC>*>(row + i + step);
        Vec<Src, VEC> c = *reinterpret_cast<const Vec<Src, VEC>*>(row + i + 2 * step);
        Vec<Src, VEC> d = *reinterpret_cast<const Vec<Src, VEC>*>(row + i + 3 * step);
#pragma unroll
        for (int j = 0; j < VEC; j++) {
            acc0 = SrcTR::combine(acc0, SrcTR::load(a.v[j]));
            acc1 = SrcTR::combine(acc1, SrcTR::load(b.v[j]));
            acc2 = SrcTR::combine(acc2, SrcTR::load(c.v[j]));
            acc3 = SrcTR::combine(acc3, SrcTR::load(d.v[j]));
        }
    }
    for (; i < end; i += step) {
        Vec<Src, VEC> a = *reinterpret_cast<const Vec<Src, VEC>*>(row + i);
#pragma unroll
        for (int j = 0; j < VEC; j++) acc0 = SrcTR::combine(acc0, SrcTR::load(a.v[j]));
    }
    return SrcTR::combine(SrcTR::combine(acc0, acc1), SrcTR::combine(acc2, acc3));
}

// Arrival counting for split reductions that fold their partials in the same launch: every block
// publishes its partial (write, __threadfence), then one thread bumps the counter of its output
// group; the block that sees the last ticket re-reads all partials of the group, folds them in
// split order (so the result does not depend on which block came last) and writes the output.
// It also puts the counter back to zero, so the counter array is all-zero between launches.
__device__ __forceinline__ bool last_arrival(u32* counter, u32 expected) {
    __shared__ u32 s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const u32 ticket = atomicAdd(counter, 1u);
        s_last = ticket == expected - 1;
        if (s_last) *counter = 0;
    }
    __syncthreads();
    const bool last = s_last != 0;
    if (last) __threadfence();
    return last;
}
template <class Acc>
__device__ __forceinline__ Acc load_published(const Acc* p) {
    return *reinterpret_cast<const volatile Acc*>(p);  // not through L1: written by other blocks of this launch
}

// The fold of a row's `splits` published parts in split order, eight of them in flight: one thread folds an output while the
// rest of the launch is over, so each trip to L2 counts in full.  One by one (UN = 1) where eight take registers from the main loop: f64 (means of rows 34, 52 with
// eight), and columns (100001 x 16 f32 32.0 us, 37.2; 2047 x 20000 f64 49.7, 54.5) but for vectors of 16-bit floats, whose kernel is held to four blocks an
// SM (bf16 52 registers, 80 without the bound: 130 x 300000 8.8 us, 10.1; with it 2.5 % faster than one by one over 25 shapes, at most 3 % slower).
template <class TR, u32 UN>
__device__ __forceinline__ typename TR::Acc fold_published(const typename TR::Acc* p, u64 stride, u32 splits) {
    typedef typename TR::Acc Acc;
    Acc acc = TR::init();
    for (u32 s = 0; s < splits; s += UN) {
        Acc v[UN];
#pragma unroll
        for (u32 q = 0; q < UN; q++)
            if (s + q < splits) v[q] = load_published(p + (s + q) * stride);
#pragma unroll
        for (u32 q = 0; q < UN; q++)
            if (s + q < splits) acc = TR::combine(acc, v[q]);
    }
    return acc;
}

// counters == nullptr: partials are left for a second launch (reduce_partials_*_kernel).
template <class T, int KIND, int VEC>
__global__ void __launch_bounds__(kRedThreads) reduce_rows_block_kernel(const T* in, T* out, typename RedTraits<T, KIND>::Acc* partial,
                                                                      u64 R, u64 seg, u32 splits, u64 factor, u32* counters, int tree_fold) {
    after_previous_kernel();
    typedef RedTraits<T, KIND> TR;
    typedef typename TR::Acc Acc;
    const u64 row = blockIdx.y;
    const u32 split = blockIdx.x;
    const u64 begin = (u64)split * seg;
    u64 end = begin + seg;
    if (end > R) end = R;
    Acc v = begin < end ? row_segment<T, KIND, VEC, T, TR>(in + row * R, begin, end) : TR::init();
    v = block_reduce<TR, kRedThreads>(v);
    if (threadIdx.x == 0) {
        if (splits == 1) out[row] = TR::finalize(v, factor);
        else partial[row * splits + split] = v;
    }
    if (splits == 1 || !counters) return;
    if (!last_arrival(counters + row, splits)) return;
    const Acc* mine = partial + row * splits;
    if (tree_fold) {  // same shape as reduce_partials_block_kernel
        Acc acc = TR::init();
        for (u32 s2 = threadIdx.x; s2 < splits; s2 += kRedThreads) acc = TR::combine(acc, load_published(mine + s2));
        acc = block_reduce<TR, kRedThreads>(acc);
        if (threadIdx.x == 0) out[row] = TR::finalize(acc, factor);
    } else if (threadIdx.x == 0) {  // same order as reduce_partials_kernel
        out[row] = TR::finalize(fold_published<TR, std::is_same<Acc, f64>::value ? 1 : 8>(mine, 1, splits), factor);
    }
}

// G lanes of a warp per row (up to 32 vectors), G the smallest of 4, 8, 16, 32 that gives every vector of the row a lane: a
// row of 56 bf16 is seven vectors, and a whole warp for it left 25 lanes idle.  Q rows per group with their loads in flight
// together: with one row a block of 256 threads lived for a single load (sums over the last two dims of [64, 256, 56, 56] bf16:
// 124 us with a warp per row, 55 with eight lanes and one row, 32 with eight lanes and four).
template <class T, int KIND, int VEC, int G, int Q>
__global__ void __launch_bounds__(kRedThreads) reduce_rows_short_kernel(const T* in, T* out, u64 rows, u32 R, u64 factor) {
    after_previous_kernel();
    typedef RedTraits<T, KIND> TR;
    constexpr u32 ROWS = kRedThreads / G;  // rows a block has in one step
    const u64 row0 = (u64)blockIdx.x * ROWS * Q + threadIdx.x / G;
    const u32 i = threadIdx.x % G * VEC;
    Vec<T, VEC> v[Q];
    typename TR::Acc acc[Q];
#pragma unroll
    for (int q = 0; q < Q; q++)
        if (i < R && row0 + q * ROWS < rows) v[q] = *reinterpret_cast<const Vec<T, VEC>*>(in + (row0 + q * ROWS) * R + i);
#pragma unroll
    for (int q = 0; q < Q; q++) {
        acc[q] = TR::init();
        if (i < R && row0 + q * ROWS < rows)
#pragma unroll
            for (int j = 0; j < VEC; j++) acc[q] = TR::combine(acc[q], TR::load(v[q].v[j]));
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1)  // the shuffles take the whole warp
#pragma unroll
        for (int q = 0; q < Q; q++) acc[q] = TR::combine(acc[q], __shfl_xor_sync(0xFFFFFFFFu, acc[q], o));
#pragma unroll
    for (int q = 0; q < Q; q++)
        if (threadIdx.x % G == 0 && row0 + q * ROWS < rows) out[row0 + q * ROWS] = TR::finalize(acc[q], factor);
}

// One warp per longer row (R < ~2048): a lane's loads in flight together, four or, of types with 16 elements a vector (whose adds
// bound it), two.  Trips that are whole for every lane, then one with a check per load: checks in every trip cost long rows
// more than they gave (100000 rows of 1023 bf16: 59 us, 46 like this), lanes that leave at different trips the ragged ones.
template <class T, int KIND, int VEC>
__global__ void __launch_bounds__(kRedThreads) reduce_rows_warp_kernel(const T* in, T* out, u64 rows, u32 R, u64 factor) {
    after_previous_kernel();
    typedef RedTraits<T, KIND> TR;
    const u64 row = (u64)blockIdx.x * (kRedThreads / 32) + threadIdx.x / 32;
    if (row >= rows) return;
    constexpr u32 STEP = 32 * VEC, Q = VEC >= 16 ? 2 : 4;
    const T* p = in + row * R;
    typename TR::Acc acc = TR::init();
    u32 i = (threadIdx.x % 32) * VEC;
    for (u32 whole = R / (Q * STEP); whole > 0; whole--, i += Q * STEP) {  // the same trips for every lane
        Vec<T, VEC> v[Q];
#pragma unroll
        for (int q = 0; q < Q; q++) v[q] = *reinterpret_cast<const Vec<T, VEC>*>(p + i + q * STEP);
#pragma unroll
        for (int q = 0; q < Q; q++)
#pragma unroll
            for (int j = 0; j < VEC; j++) acc = TR::combine(acc, TR::load(v[q].v[j]));
    }
    if (R % (Q * STEP)) {
        Vec<T, VEC> v[Q];
#pragma unroll
        for (int q = 0; q < Q; q++)
            if (i + q * STEP < R) v[q] = *reinterpret_cast<const Vec<T, VEC>*>(p + i + q * STEP);
#pragma unroll
        for (int q = 0; q < Q; q++)
            if (i + q * STEP < R)
#pragma unroll
                for (int j = 0; j < VEC; j++) acc = TR::combine(acc, TR::load(v[q].v[j]));
    }
    acc = warp_reduce<TR>(acc);
    if (threadIdx.x % 32 == 0) out[row] = TR::finalize(acc, factor);
}

// Rows that are no whole aligned vectors, by the aligned 16-byte words they lie in: a lane loads a word (which holds at least one element of its row, so
// that nothing outside the tensor's own words is touched) and leaves out the neighbours' elements.  Element by element a row of 197 bf16 takes
// seven loads of two bytes a lane, where one of 16 does (40000 rows of 193 5.5 us, 5.0 so).  G lanes per row with Q rows in flight; which: red_rows_words_launch.
template <class T, int KIND>
struct RowWords {
    typedef RedTraits<T, KIND> TR;
    static constexpr int VEC = 16 / (int)sizeof(T);
    const Vec<T, VEC>* first;
    u32 before, words;  // elements of the first word that belong to the row before; words
    __device__ __forceinline__ RowWords(const T* row, u32 R) {
        const uintptr_t at = reinterpret_cast<uintptr_t>(row), base = at & ~(uintptr_t)15;
        first = reinterpret_cast<const Vec<T, VEC>*>(base);
        before = (u32)(at - base) / (u32)sizeof(T);
        words = (before + R + VEC - 1) / VEC;
    }
    __device__ __forceinline__ typename TR::Acc add(typename TR::Acc acc, const Vec<T, VEC>& v, u32 w, u32 R) const {
        const u32 e0 = w * VEC - before;  // wraps below zero: then not below R
#pragma unroll
        for (int j = 0; j < VEC; j++) acc = TR::combine(acc, e0 + j < R ? TR::load(v.v[j]) : TR::init());
        return acc;
    }
};
template <class T, int KIND, int G, int Q>
__global__ void __launch_bounds__(kRedThreads) reduce_rows_words_kernel(const T* in, T* out, u64 rows, u32 R, u64 factor) {
    after_previous_kernel();
    typedef RedTraits<T, KIND> TR;
    typedef RowWords<T, KIND> RW;
    constexpr u32 ROWS = kRedThreads / G;
    const u64 row0 = (u64)blockIdx.x * ROWS * Q + threadIdx.x / G;
    const u32 lane = threadIdx.x % G;
    Vec<T, RW::VEC> v[Q];
    typename TR::Acc acc[Q];
#pragma unroll
    for (int q = 0; q < Q; q++)
        if (row0 + q * ROWS < rows) {
            const RW w(in + (row0 + q * ROWS) * R, R);
            if (lane < w.words) v[q] = w.first[lane];
        }
#pragma unroll
    for (int q = 0; q < Q; q++) {
        acc[q] = TR::init();
        if (row0 + q * ROWS < rows) {
            const RW w(in + (row0 + q * ROWS) * R, R);
            if (lane < w.words) acc[q] = w.add(acc[q], v[q], lane, R);
        }
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1)  // the shuffles take the whole warp
#pragma unroll
        for (int q = 0; q < Q; q++) acc[q] = TR::combine(acc[q], __shfl_xor_sync(0xFFFFFFFFu, acc[q], o));
#pragma unroll
    for (int q = 0; q < Q; q++)
        if (lane == 0 && row0 + q * ROWS < rows) out[row0 + q * ROWS] = TR::finalize(acc[q], factor);
}

// One thread per row (R < 32, see red_launch).
template <class T, int KIND>
__global__ void __launch_bounds__(kRedThreads) reduce_rows_thread_kernel(const T* in, T* out, u64 rows, u64 R, u64 factor) {
    after_previous_kernel();
    typedef RedTraits<T, KIND> TR;
    const u64 row = (u64)blockIdx.x * kRedThreads + threadIdx.x;
    if (row >= rows) return;
    const T* p = in + row * R;
    typename TR::Acc acc = TR::init();
    for (u64 i = 0; i < R; i++) acc = TR::combine(acc, TR::load(p[i]));
    out[row] = TR::finalize(acc, factor);
}

// Second pass of a split reduction: out[j] = fold of partial[j * S + s] (rows layout) or
// partial[s * count + j] (cols layout).  One thread per output.
template <class T, int KIND>
__global__ void __launch_bounds__(kRedThreads) reduce_partials_kernel(const typename RedTraits<T, KIND>::Acc* partial, T* out, u64 count,
                                                                    u32 S, int cols_layout, u64 factor) {
    after_previous_kernel();
    typedef RedTraits<T, KIND> TR;
    const u64 j = (u64)blockIdx.x * kRedThreads + threadIdx.x;
    if (j >= count) return;
    typename TR::Acc acc = TR::init();
    if (cols_layout) {
        for (u32 s = 0; s < S; s++) acc = TR::combine(acc, partial[(u64)s * count + j]);
    } else {
        for (u32 s = 0; s < S; s++) acc = TR::combine(acc, partial[j * S + s]);
    }
    out[j] = TR::finalize(acc, factor);
}

// Same fold with one block per output, for few outputs with many partials (a full reduction
// split over ~1000 blocks): threads stride over the partials, then a fixed-shape block tree.
template <class T, int KIND>
__global__ void __launch_bounds__(kRedThreads) reduce_partials_block_kernel(const typename RedTraits<T, KIND>::Acc* partial, T* out, u32 S, u64 factor) {
    after_previous_kernel();
    typedef RedTraits<T, KIND> TR;
    const u64 j = blockIdx.x;
    typename TR::Acc acc = TR::init();
    for (u32 s = threadIdx.x; s < S; s += kRedThreads) acc = TR::combine(acc, partial[j * S + s]);
    acc = block_reduce<TR, kRedThreads>(acc);
    if (threadIdx.x == 0) out[j] = TR::finalize(acc, factor);
}

// ---------------------------------------------------------------------------------
// cols: in[(o * R + r) * I + i], out[o * I + i]
// ---------------------------------------------------------------------------------
constexpr int kColLanes = 32;  // threads along the columns
constexpr int kColRows = 8;    // threads along the reduced dim

// The fold of a strip of single columns by the last block, where it has many parts: a column by eight threads, each every eighth part, and then theirs in order, since the trips to L2 are what
// this costs ([17683, 43] bf16, 148 parts, 41.6 us by one thread a column, 7.0 so; [9999, 100] 10.7, 6.0; vectors of f32 [3000, 1000] 7.2, 6.1).  A function of its own and an instantiation of its own
// (TOGETHER): in the kernel that all columns take it cost those without a fold up to 6 %, and vectors' strips, whose main loop it took registers from, up to 30 %.
constexpr u32 kColFoldTogether = 12;
template <class T, int KIND, int VEC>
__device__ __noinline__ void fold_columns(const typename RedTraits<T, KIND>::Acc* parts, T* out, u64 cols, u64 stride, u32 splits, u64 factor, typename RedTraits<T, KIND>::Acc* sm) {
    typedef RedTraits<T, KIND> TR;
    constexpr int LD = kColLanes * VEC, P = kColRows / VEC;  // threads of a column
    const int c = threadIdx.x % LD, y = threadIdx.x / LD;
    typename TR::Acc v = TR::init();
    if ((u64)c < cols && (u32)y < splits) v = fold_published<TR, VEC>(parts + c + (u64)y * stride, P * stride, (splits - y + P - 1) / P);
    sm[y * (LD + 1) + c] = v;
    __syncthreads();
    if (y == 0 && (u64)c < cols) {
#pragma unroll
        for (int q = 1; q < P; q++) v = TR::combine(v, sm[q * (LD + 1) + c]);
        out[c] = TR::finalize(v, factor);
    }
}

// grid = (ceil(I / (32 * VEC)), splits, min(O, 65535)).  VEC > 1 requires I % VEC == 0 and an
// aligned base.
// Vectors of 16-bit floats are held to four blocks an SM (see fold_published), maxima of eight-byte integers to five (they took 54 registers instead of 44 since
// the wait at the top, four blocks: [48950, 873] u64 66 us before, 74, 54 so).  0: the compiler's own choice for all others; 1 would let it take every register (bf16 [130, 300000] 9.0 us, 9.8; minima of f32 [811, 2, 13536] 403, 888).
// The means of f64 with their fold together would take 58 registers and four blocks, 48 without it ([6856, 1784] 11.9 us, 15.9 so).
template <class T, int KIND, bool TOGETHER = false>
constexpr int kColBlocks = is_half_v<T> ? 4 : (KIND >= RED_MAX && std::is_integral<T>::value && sizeof(T) == 8) || (TOGETHER && KIND == RED_MEAN && sizeof(T) == 8) ? 5 : 0;
template <class T, int KIND, int VEC, bool TOGETHER = false>
__global__ void __launch_bounds__(kColLanes* kColRows, VEC > 1 ? kColBlocks<T, KIND, TOGETHER> : 0) reduce_cols_kernel(const T* in, T* out, typename RedTraits<T, KIND>::Acc* partial, u64 O,
                                                                         u64 R, u64 I, u64 seg, u32 splits, u64 factor, u32* counters) {
    after_previous_kernel();
    typedef RedTraits<T, KIND> TR;
    typedef typename TR::Acc Acc;
    __shared__ Acc sm[kColRows][kColLanes * VEC + 1];
    const int lane = threadIdx.x % kColLanes, ty = threadIdx.x / kColLanes;
    const u64 col = ((u64)blockIdx.x * kColLanes + lane) * VEC;
    const u32 split = blockIdx.y;
    const u64 r_begin = (u64)split * seg;
    u64 r_end = r_begin + seg;
    if (r_end > R) r_end = R;
    for (u64 o = blockIdx.z; o < O; o += gridDim.z) {
        Acc acc[VEC];
#pragma unroll
        for (int j = 0; j < VEC; j++) acc[j] = TR::init();
        if (col < I) {
            const T* p = in + o * R * I + col;
            u64 r = r_begin + ty;
            // eight independent 16-byte loads in flight per thread
            for (; r + 7 * kColRows < r_end; r += 8 * kColRows) {
                Vec<T, VEC> x[8];
#pragma unroll
                for (int q = 0; q < 8; q++) x[q] = *reinterpret_cast<const Vec<T, VEC>*>(p + (r + q * kColRows) * I);
#pragma unroll
                for (int j = 0; j < VEC; j++) {
                    Acc s01 = TR::combine(TR::load(x[0].v[j]), TR::load(x[1].v[j]));
                    Acc s23 = TR::combine(TR::load(x[2].v[j]), TR::load(x[3].v[j]));
                    Acc s45 = TR::combine(TR::load(x[4].v[j]), TR::load(x[5].v[j]));
                    Acc s67 = TR::combine(TR::load(x[6].v[j]), TR::load(x[7].v[j]));
                    acc[j] = TR::combine(acc[j], TR::combine(TR::combine(s01, s23), TR::combine(s45, s67)));
                }
            }
            for (; r < r_end; r += kColRows) {
                Vec<T, VEC> a = *reinterpret_cast<const Vec<T, VEC>*>(p + r * I);
#pragma unroll
                for (int j = 0; j < VEC; j++) acc[j] = TR::combine(acc[j], TR::load(a.v[j]));
            }
        }
#pragma unroll
        for (int j = 0; j < VEC; j++) sm[ty][lane * VEC + j] = acc[j];
        __syncthreads();
        // fold the kColRows partial strips; the first kColLanes*VEC threads each own a column
        for (int c = threadIdx.x; c < kColLanes * VEC; c += kColLanes * kColRows) {
            u64 gc = (u64)blockIdx.x * kColLanes * VEC + c;
            if (gc < I) {
                Acc v = sm[0][c];
#pragma unroll
                for (int y = 1; y < kColRows; y++) v = TR::combine(v, sm[y][c]);
                if (splits == 1) out[o * I + gc] = TR::finalize(v, factor);
                else partial[((u64)split * O + o) * I + gc] = v;
            }
        }
        if (splits > 1 && counters) {
            // fold in the same launch: the last block of this (o, column strip) to arrive
            if (last_arrival(counters + o * gridDim.x + blockIdx.x, splits)) {
                if constexpr (TOGETHER) {
                    const u64 c0 = (u64)blockIdx.x * kColLanes * VEC;
                    fold_columns<T, KIND, VEC>(partial + o * I + c0, out + o * I + c0, I - c0, O * I, splits, factor, &sm[0][0]);
                } else {
                    for (int c = threadIdx.x; c < kColLanes * VEC; c += kColLanes * kColRows) {
                        u64 gc = (u64)blockIdx.x * kColLanes * VEC + c;
                        if (gc < I) {
                            const Acc* parts = partial + o * I + gc;
                            Acc v = TR::init();
                            if constexpr (is_half_v<T> && VEC > 1) v = fold_published<TR, 8>(parts, O * I, splits);
                            else
                                for (u32 s2 = 0; s2 < splits; s2++) v = TR::combine(v, load_published(partial + ((u64)s2 * O + o) * I + gc));
                            out[o * I + gc] = TR::finalize(v, factor);
                        }
                    }
                }
            }
        }
        __syncthreads();
    }
}

// The instantiation for a fold of `splits` parts: every entry point that promises another's bits takes it from here.
template <class T, int KIND, int VEC>
auto reduce_cols_choice(bool vec, u64 splits) {
    constexpr int TV = VEC < kColRows ? VEC : 1;  // a wider vector's columns have a thread each
    // what the means of f64 spill for it counts while a thread adds few parts ([11394, 1174], 31 parts, 17.8 us, 19.5 together; 2 x [45888, 146] 26.6, 23.6)
    constexpr u64 FROM = kColFoldTogether * (KIND == RED_MEAN && sizeof(T) == 8 ? 5 : 2);
    if (vec) return TV == VEC && splits >= FROM ? reduce_cols_kernel<T, KIND, TV, true> : reduce_cols_kernel<T, KIND, VEC>;
    return splits >= kColFoldTogether ? reduce_cols_kernel<T, KIND, 1, true> : reduce_cols_kernel<T, KIND, 1>;
}

// Second pass of an "outer" reduction: out[o] = fold of partial[o * so + i * si + j], i < ni, j < nj.  G = 32: a warp per
// output; G = kRedThreads: a block per output.
template <class T, int KIND, int G>
__global__ void __launch_bounds__(kRedThreads) reduce_outer_fold_kernel(const typename RedTraits<T, KIND>::Acc* partial, T* out, u64 count, u64 so, u32 ni,
                                                                      u64 si, u32 nj, FastDiv nj_div, u64 factor) {
    after_previous_kernel();
    typedef RedTraits<T, KIND> TR;
    const u64 o = (u64)blockIdx.x * (kRedThreads / G) + threadIdx.x / G;
    if (G == 32 && o >= count) return;
    const u32 t = threadIdx.x % G, total = ni * nj;
    typename TR::Acc acc = TR::init();
#pragma unroll 4
    for (u32 e = t; e < total; e += G) {
        u32 i, j;
        nj_div.divmod(e, i, j);
        acc = TR::combine(acc, partial[o * so + i * si + j]);
    }
    if constexpr (G == 32) acc = warp_reduce<TR>(acc);
    else acc = block_reduce<TR, kRedThreads>(acc);
    if (t == 0) out[o] = TR::finalize(acc, factor);
}

// ---------------------------------------------------------------------------------
// generic scatter path (literal index formulas, wide atomics into scratch)
// ---------------------------------------------------------------------------------
constexpr int kRedMaxDims = 16;

struct RedGenParams {
    int mode;  // 0 = dim reduction, 1 = sum_to_shape
    u64 n;
    int nd, nr;
    int contiguous;
    u64 dims[kRedMaxDims], strides[kRedMaxDims];
    u64 red_len[kRedMaxDims], red_stride[kRedMaxDims];  // mode 0
    u64 out_dims[kRedMaxDims];                         // mode 1
    u64 off;
};

template <class Acc>
__device__ __forceinline__ void atomic_combine_sum(Acc* p, Acc v) {
    if constexpr (std::is_same<Acc, u64>::value) atomicAdd(reinterpret_cast<unsigned long long*>(p), (unsigned long long)v);
    else atomicAdd(p, v);
}
template <class Acc, bool IS_MAX>
__device__ __forceinline__ void atomic_combine_minmax(Acc* p, Acc v) {
    if constexpr (std::is_same<Acc, f32>::value || std::is_same<Acc, f64>::value) {
        typedef typename std::conditional<sizeof(Acc) == 4, unsigned int, unsigned long long>::type Bits;
        Bits* bp = reinterpret_cast<Bits*>(p);
        Bits old = *bp;
        for (int guard = 0; guard < (1 << 20); guard++) {
            Acc cur;
            memcpy(&cur, &old, sizeof(Acc));
            bool better = IS_MAX ? (v > cur) : (v < cur);
            if (!better) return;
            Bits nb;
            memcpy(&nb, &v, sizeof(Acc));
            Bits prev = atomicCAS(bp, old, nb);
            if (prev == old) return;
            old = prev;
        }
    } else if constexpr (std::is_same<Acc, i64>::value) {
        if (IS_MAX) atomicMax(reinterpret_cast<long long*>(p), (long long)v);
        else atomicMin(reinterpret_cast<long long*>(p), (long long)v);
    } else if constexpr (std::is_same<Acc, u64>::value) {
        if (IS_MAX) atomicMax(reinterpret_cast<unsigned long long*>(p), (unsigned long long)v);
        else atomicMin(reinterpret_cast<unsigned long long*>(p), (unsigned long long)v);
    } else {
        if (IS_MAX) atomicMax(p, v);
        else atomicMin(p, v);
    }
}

template <class T, int KIND>
__global__ void __launch_bounds__(kRedThreads) reduce_fill_kernel(typename RedTraits<T, KIND>::Acc* ws, u64 count) {
    after_previous_kernel();
    for (u64 j = (u64)blockIdx.x * kRedThreads + threadIdx.x; j < count; j += (u64)gridDim.x * kRedThreads) ws[j] = RedTraits<T, KIND>::init();
}
template <class T, int KIND>
__global__ void __launch_bounds__(kRedThreads) reduce_finalize_kernel(const typename RedTraits<T, KIND>::Acc* ws, T* out, u64 count, u64 factor) {
    after_previous_kernel();
    for (u64 j = (u64)blockIdx.x * kRedThreads + threadIdx.x; j < count; j += (u64)gridDim.x * kRedThreads)
        out[j] = RedTraits<T, KIND>::finalize(ws[j], factor);
}

template <class T, int KIND>
__global__ void __launch_bounds__(kRedThreads) reduce_scatter_kernel(const T* in, typename RedTraits<T, KIND>::Acc* ws, RedGenParams P) {
    after_previous_kernel();
    typedef RedTraits<T, KIND> TR;
    for (u64 i = (u64)blockIdx.x * kRedThreads + threadIdx.x; i < P.n; i += (u64)gridDim.x * kRedThreads) {
        u64 src, dst;
        if (P.mode == 0) {
            // crates/maidenx_cpu/src/ops/reduction.rs:45-79
            src = i;
            if (!P.contiguous) {
                u64 rem = i;
                src = 0;
                for (int d = P.nd - 1; d >= 0; d--) {
                    if (P.strides[d] != 0) src += (rem % P.dims[d]) * P.strides[d];
                    rem /= P.dims[d];
                }
            }
            dst = i;
            for (int k = 0; k < P.nr; k++) {
                u64 s = P.red_stride[k], l = P.red_len[k];
                if (s != 0) {
                    u64 pre = dst / s, post = dst % s;
                    dst = (pre / l) * s + post;
                } else {
                    dst /= l;
                }
            }
        } else {
            // crates/maidenx_cpu/src/ops/reduction.rs:127-170
            u64 rem = i, lin = 0, mul = 1;
            src = 0;
            // walk dims from the innermost: coordinate, strided source, row-major index in out_dims
            for (int d = P.nd - 1; d >= 0; d--) {
                u64 c = rem % P.dims[d];
                rem /= P.dims[d];
                src += c * P.strides[d];
                u64 f = P.dims[d] / P.out_dims[d];
                lin += (c / f) * mul;
                mul *= P.out_dims[d];
            }
            dst = lin;
            if (P.contiguous) src = i;
            else src = (src + P.off) % P.n;  // the reference adds the offset a second time and wraps
        }
        typename TR::Acc v = TR::load(in[src]);
        if constexpr (TR::kIsSum) atomic_combine_sum(ws + dst, v);
        else atomic_combine_minmax<typename TR::Acc, KIND == RED_MAX>(ws + dst, v);
    }
}

// ---------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------
enum RedPlanKind { RP_EMPTY = 0, RP_ROWS, RP_COLS, RP_GENERIC, RP_ERROR, RP_OUTER };

struct RedPlan {
    int kind;
    u64 O, R, I;      // rows: O rows of R; cols: [O, R, I]; outer: [R, O, I] -> [O]
    u64 out_count;
    u64 factor;       // elements folded into each output (mean divisor)
    u64 off;
    RedGenParams gen;
};

// How many ways to split each of `groups` independent reductions so that the launch fills the
// GPU's `capacity` resident blocks in ONE wave: a launch of slightly more blocks than fit pays a
// second, nearly empty wave, which on these 50-100 us kernels costs 10-20 %.
inline u64 split_count(u64 groups, u64 capacity) {
    if (groups == 0 || groups >= capacity) return 1;
    u64 s = capacity / groups;
    return s < 1 ? 1 : s;
}
u32* arrival_counters(u64 count);                      // zeroed counters for last_arrival, or nullptr if count is too large

void red_plan_dims(RedPlan& pl, size_t num_els, size_t num_dims, size_t num_red, const size_t* hm);
void red_plan_shape(RedPlan& pl, size_t num_els, size_t num_dims, const size_t* hm);

template <class T, int KIND, int VEC, int G>
void red_rows_short_launch(const T* in, T* out, u64 O, u64 R, u64 factor, cudaStream_t s) {
    constexpr u64 ROWS = kRedThreads / G;
    // four rows per group while that leaves every SM its eight blocks
    if (O >= 4 * ROWS * 8 * (u64)sm_count()) launch_kernel(reduce_rows_short_kernel<T, KIND, VEC, G, 4>, (u32)((O + 4 * ROWS - 1) / (4 * ROWS)), kRedThreads, 0, s, in, out, O, (u32)R, factor);
    else launch_kernel(reduce_rows_short_kernel<T, KIND, VEC, G, 1>, (u32)((O + ROWS - 1) / ROWS), kRedThreads, 0, s, in, out, O, (u32)R, factor);
}
template <class T, int KIND, int VEC>
void red_rows_group_launch(const T* in, T* out, u64 O, u64 R, u64 factor, cudaStream_t s) {
    const u64 lanes = (R + VEC - 1) / VEC;
    if (lanes <= 4) red_rows_short_launch<T, KIND, VEC, 4>(in, out, O, R, factor, s);
    else if (lanes <= 8) red_rows_short_launch<T, KIND, VEC, 8>(in, out, O, R, factor, s);
    else if (lanes <= 16) red_rows_short_launch<T, KIND, VEC, 16>(in, out, O, R, factor, s);
    else if (lanes <= 32) red_rows_short_launch<T, KIND, VEC, 32>(in, out, O, R, factor, s);
    else launch_kernel(reduce_rows_warp_kernel<T, KIND, VEC>, (u32)((O + kRedThreads / 32 - 1) / (kRedThreads / 32)), kRedThreads, 0, s, in, out, O, (u32)R, factor);
}

// Rows of at least 128 bytes that are no whole aligned vectors (see RowWords); false: they are summed element by element.  Leaving out the neighbours costs
// two instructions an element, for one load instead of up to 16, so it pays while a lane has one word.  Elements / words, us (sums; maxima alike):
//   up to 16 words   bf16 65: 600 rows 1.20 / 1.19, 19200 2.63 / 1.90, 300000 22.3 / 14.6; u8 225: 600 1.54 / 1.31, 300000 36.5 / 22.6; f32 57: 9600 1.70 / 1.37
//     four rows a group, f32 57: 600 1.73, 9600 1.83 instead of 1.37, 40000 2.62 instead of 2.71, 300000 10.5 instead of 12.6; 16-bit and bytes no gain at 300000
//   up to 32         bf16 193: 600 1.43 / 1.21, 40000 5.50 / 5.02, 300000 42.0 / 35.4 (four rows a group 5.19, 31.1); f32 97: 9600 1.72 / 1.81, 30000 3.28 / 3.44, four
//                    rows a group 40000 3.99 / 3.83, 300000 31.7 / 26.9; u8 385: 9600 2.40 / 2.52, 40000 6.24 / 7.06, 100000 13.1 / 15.7
//   a warp a row with its words in steps of four a lane was slower than elements over most of what is longer (bf16 263: 40000 5.7 / 9.0; u8 527: 15.1 / 45.7; f32
//   1023: 9600 3.9 / 4.3) and is gone.
template <class T, int KIND>
bool red_rows_words_launch(const T* in, T* out, u64 O, u64 R, u64 factor, cudaStream_t s) {
    constexpr u64 VEC = 16 / sizeof(T);
    const u64 words = (R + 2 * VEC - 2) / VEC;  // at most, wherever a row starts
    auto launch = [&](auto kernel, u64 rows) { launch_kernel(kernel, (u32)((O + rows - 1) / rows), kRedThreads, 0, s, in, out, O, (u32)R, factor); };
    const u64 sms = (u64)sm_count();
    if constexpr (sizeof(T) == 4) {
        const bool many = O >= 256 * sms;
        if (words <= 16 && many) launch(reduce_rows_words_kernel<T, KIND, 16, 4>, 4 * kRedThreads / 16);
        else if (words <= 16) launch(reduce_rows_words_kernel<T, KIND, 16, 1>, kRedThreads / 16);
        else if (words <= 32 && many) launch(reduce_rows_words_kernel<T, KIND, 32, 4>, 4 * kRedThreads / 32);
        else return false;
        return true;
    }
    if constexpr (sizeof(T) < 4) {
        if (words <= 16) {
            launch(reduce_rows_words_kernel<T, KIND, 16, 1>, kRedThreads / 16);
            return true;
        }
    }
    if constexpr (sizeof(T) == 2) {
        if (words <= 32) {
            if (O >= 1024 * sms) launch(reduce_rows_words_kernel<T, KIND, 32, 4>, 4 * kRedThreads / 32);
            else launch(reduce_rows_words_kernel<T, KIND, 32, 1>, kRedThreads / 32);
            return true;
        }
    }
    return false;
}

template <class T, int KIND>
void red_launch(const RedPlan& pl, const T* in, T* out, const char* where) {
    typedef RedTraits<T, KIND> TR;
    typedef typename TR::Acc Acc;
    constexpr int VEC = 16 / sizeof(T);
    cudaStream_t s = ctx().stream;
    const int sms = sm_count();
    if (pl.kind == RP_EMPTY) return;
    if (pl.kind == RP_ERROR) {
        set_error(kErrBadMetadata, 0, where);
        return;
    }
    in += pl.off;
    const bool base_aligned = ((uintptr_t)in) % 16 == 0;
    if (pl.kind == RP_ROWS) {
        const u64 O = pl.O, R = pl.R;
        // Rows below 32 elements: lane groups where a row is two or more aligned vectors (of 8-byte types, whole 64-byte pieces), a thread
        // per row otherwise - its loads of neighbouring rows meet in L1, and a row element by element leaves a group little to do (2000000 rows
        // of 9: f32 10.7 / 43 us in groups, bf16 9.8 / 42; of 16: f32 59 / 22, bf16 31 / 20, u8, one vector, 16.5 / 33; f64 of 12: 35 / 37, of 24: 120 / 75).
        // Few rows are the latency of one thread's chain, which a group shortens (2000 rows of 31: f32 2.7 / 1.6, f64 3.3 / 1.8; 10000 of 20: bf16 1.9 / 2.1, f64 3.0 / 1.9).
        const bool vec_rows = base_aligned && R % VEC == 0;
        if (R < 8 || (R < 32 && O > (sizeof(T) == 8 ? 16384 : 4096) && !(vec_rows && R >= 2 * VEC && (sizeof(T) < 8 || R % 8 == 0)))) {
            u64 blocks = (O + kRedThreads - 1) / kRedThreads;
            launch_kernel(reduce_rows_thread_kernel<T, KIND>, (u32)blocks, kRedThreads, 0, s, in, out, O, R, pl.factor);
        } else if (R < 32 || (R < 2048 && O >= (u64)sms * 4)) {
            if (vec_rows) red_rows_group_launch<T, KIND, VEC>(in, out, O, R, pl.factor, s);
            else if (!(R * sizeof(T) >= 128 && (uintptr_t)in % sizeof(T) == 0 && red_rows_words_launch<T, KIND>(in, out, O, R, pl.factor, s)))
                red_rows_group_launch<T, KIND, 1>(in, out, O, R, pl.factor, s);
        } else {
            // block per (row, split); split long rows when there are too few rows to fill the GPU
            const bool vec = vec_rows;
            const u64 unit = (u64)kRedThreads * VEC * 4;  // one full unrolled trip of a block
            static int occ = 0;  // resident blocks per SM of this instantiation
            if (!occ) occ = resident_blocks((const void*)reduce_rows_block_kernel<T, KIND, VEC>, kRedThreads);
            u64 want = split_count(O, (u64)sms * occ);
            u64 max_splits = (R + unit - 1) / unit;
            u64 splits = want < max_splits ? want : max_splits;
            if (splits < 1) splits = 1;
            u64 seg = (R + splits - 1) / splits;
            seg = (seg + VEC - 1) / VEC * VEC;
            splits = (R + seg - 1) / seg;
            if (O > 65535) {  // grid.y limit: fall back to one warp per row
                red_rows_group_launch<T, KIND, 1>(in, out, O, R, pl.factor, s);
            } else {
                Acc* part = nullptr;
                u32* counters = nullptr;
                if (splits > 1) {
                    part = static_cast<Acc*>(scratch(sizeof(Acc) * O * splits));
                    if (!part) return;
                    counters = arrival_counters(O);  // nullptr: too many groups, fold in a second launch
                }
                const int tree_fold = O <= 64 && splits >= 64;
                dim3 grid((u32)splits, (u32)O);
                if (vec) launch_kernel(reduce_rows_block_kernel<T, KIND, VEC>, grid, kRedThreads, 0, s, in, out, part, R, seg, (u32)splits, pl.factor, counters, tree_fold);
                else launch_kernel(reduce_rows_block_kernel<T, KIND, 1>, grid, kRedThreads, 0, s, in, out, part, R, seg, (u32)splits, pl.factor, counters, tree_fold);
                if (splits > 1 && !counters) {
                    check_launch(where);
                    if (tree_fold) launch_kernel(reduce_partials_block_kernel<T, KIND>, (u32)O, kRedThreads, 0, s, part, out, (u32)splits, pl.factor);
                    else launch_kernel(reduce_partials_kernel<T, KIND>, (u32)((O + kRedThreads - 1) / kRedThreads), kRedThreads, 0, s, part, out, O, (u32)splits, 0, pl.factor);
                }
            }
        }
        check_launch(where);
        return;
    }
    if (pl.kind == RP_COLS) {
        const u64 O = pl.O, R = pl.R, I = pl.I;
        const bool vec = base_aligned && I % VEC == 0;
        const int v = vec ? VEC : 1;
        u64 gx = (I + (u64)kColLanes * v - 1) / ((u64)kColLanes * v);
        u64 gz = O < 65535 ? O : 65535;
        static int occ = 0;
        if (!occ) occ = resident_blocks((const void*)reduce_cols_kernel<T, KIND, VEC>, kColLanes * kColRows);
        u64 want = split_count(gx * gz, (u64)sms * occ);
        u64 max_splits = (R + 63) / 64;  // at least 64 rows per split
        u64 splits = want < max_splits ? want : max_splits;
        if (splits < 1) splits = 1;
        if (splits > 65535) splits = 65535;
        u64 seg = (R + splits - 1) / splits;
        splits = (R + seg - 1) / seg;
        Acc* part = nullptr;
        u32* counters = nullptr;
        if (splits > 1) {
            part = static_cast<Acc*>(scratch(sizeof(Acc) * splits * O * I));
            if (!part) return;
            counters = arrival_counters(O * gx);
        }
        dim3 grid((u32)gx, (u32)splits, (u32)gz);
        launch_kernel(reduce_cols_choice<T, KIND, VEC>(vec, splits), grid, kColLanes * kColRows, 0, s, in, out, part, O, R, I, seg, (u32)splits, pl.factor, counters);
        if (splits > 1 && !counters) {
            check_launch(where);
            u64 count = O * I;
            launch_kernel(reduce_partials_kernel<T, KIND>, (u32)((count + kRedThreads - 1) / kRedThreads), kRedThreads, 0, s, part, out, count, (u32)splits, 1, pl.factor);
        }
        check_launch(where);
        return;
    }
    if (pl.kind == RP_OUTER) {
        const u64 O = pl.O, R = pl.R, I = pl.I;
        const int occ = 8;
        // Long inner runs fold first (one row per (r, o), coalesced, a single value left of each); short ones fold last, so
        // that the first pass walks down R over whole rows of O * I neighbouring elements.  The line: below 1024 elements a
        // block has less than one trip per row; above it the O * I wide partials would be written and read for nothing.
        if (I >= 1024 && R * O <= 65535 && R * 512 <= 0x7FFFFFFFull) {
            const u64 rows = R * O, unit = (u64)kRedThreads * VEC * 4;
            u64 splits = split_count(rows, (u64)sms * occ), max_splits = (I + unit - 1) / unit;
            if (splits > max_splits) splits = max_splits;
            u64 seg = (I + splits - 1) / splits;
            seg = (seg + VEC - 1) / VEC * VEC;
            splits = (I + seg - 1) / seg;
            const u32 pitch = splits < 2 ? 2 : (u32)splits;  // two or more "splits" make the kernel leave its partials
            Acc* part = static_cast<Acc*>(scratch(sizeof(Acc) * rows * pitch));
            if (!part) return;
            dim3 grid((u32)splits, (u32)rows);
            if (base_aligned && I % VEC == 0) launch_kernel(reduce_rows_block_kernel<T, KIND, VEC>, grid, kRedThreads, 0, s, in, out, part, I, seg, pitch, pl.factor, nullptr, 0);
            else launch_kernel(reduce_rows_block_kernel<T, KIND, 1>, grid, kRedThreads, 0, s, in, out, part, I, seg, pitch, pl.factor, nullptr, 0);
            check_launch(where);
            launch_kernel(reduce_outer_fold_kernel<T, KIND, 32>, (u32)((O + 7) / 8), kRedThreads, 0, s, part, out, O, pitch, (u32)R, O * pitch, (u32)splits, FastDiv((u32)splits), pl.factor);
            check_launch(where);
            return;
        }
        // Many outputs of few elements each: the scatter's atomics hardly meet, and the partial results would be as many bytes as the input
        // ([2, 100000, 5] f32 17.8 us, 19.7 in two passes; f64 17.9 / 25.5, [2, 1000000, 25] 679 / 839, [2, 65536, 1024] 2281 / 2014; [3, 50000, 10] f32 24 / 15, f64 24 / 20).
        const bool scatter = O >= 32768 && (R * I <= (sizeof(Acc) < 8 ? 10 : 12) || (sizeof(Acc) == 8 && R <= 2 && I < 512));
        const u64 cols = O * I;
        const bool vec = base_aligned && cols % VEC == 0;
        const int v = vec ? VEC : 1;
        const u64 gx = (cols + (u64)kColLanes * v - 1) / ((u64)kColLanes * v);
        u64 splits = split_count(gx, (u64)sms * occ), max_splits = (R + 63) / 64;
        if (splits > max_splits) splits = max_splits;
        u64 seg = (R + splits - 1) / splits;
        splits = (R + seg - 1) / seg;
        // The partial results grow with the input: what goes beyond the scratch block every thread has is memory of this call alone, and
        // where that is not to be had the scatter serves.
        StreamWorkspace wide;
        Acc* part = nullptr;
        if (!scatter && splits * I <= 0x7FFFFFFFull && gx <= 0x7FFFFFFFull && splits <= 65535) {
            const size_t bytes = sizeof(Acc) * splits * cols;
            if (bytes > kScratchLeast) part = wide.take(bytes) ? static_cast<Acc*>(wide.ptr) : nullptr;
            else if (!(part = static_cast<Acc*>(scratch(bytes)))) return;
        }
        if (part) {
            dim3 grid((u32)gx, (u32)splits, 1);
            const u32 leave = splits < 2 ? 2 : (u32)splits;
            if (vec) launch_kernel(reduce_cols_kernel<T, KIND, VEC>, grid, kColLanes * kColRows, 0, s, in, out, part, 1, R, cols, seg, leave, pl.factor, nullptr);
            else launch_kernel(reduce_cols_kernel<T, KIND, 1>, grid, kColLanes * kColRows, 0, s, in, out, part, 1, R, cols, seg, leave, pl.factor, nullptr);
            check_launch(where);
            const FastDiv div((u32)I);
            if (splits * I <= 2048) launch_kernel(reduce_outer_fold_kernel<T, KIND, 32>, (u32)((O + 7) / 8), kRedThreads, 0, s, part, out, O, I, (u32)splits, cols, (u32)I, div, pl.factor);
            else launch_kernel(reduce_outer_fold_kernel<T, KIND, kRedThreads>, (u32)O, kRedThreads, 0, s, part, out, O, I, (u32)splits, cols, (u32)I, div, pl.factor);
            check_launch(where);
            return;
        }
    }
    // generic scatter
    Acc* ws = static_cast<Acc*>(scratch(sizeof(Acc) * (pl.out_count ? pl.out_count : 1)));
    if (!ws) return;
    u32 fill_blocks = (u32)((pl.out_count + kRedThreads - 1) / kRedThreads);
    if (fill_blocks > (u32)sms * 16) fill_blocks = sms * 16;
    if (fill_blocks == 0) fill_blocks = 1;
    launch_kernel(reduce_fill_kernel<T, KIND>, fill_blocks, kRedThreads, 0, s, ws, pl.out_count);
    u64 sb = (pl.gen.n + kRedThreads - 1) / kRedThreads;
    if (sb > (u64)sms * 16) sb = (u64)sms * 16;
    if (sb) launch_kernel(reduce_scatter_kernel<T, KIND>, (u32)sb, kRedThreads, 0, s, in, ws, pl.gen);
    launch_kernel(reduce_finalize_kernel<T, KIND>, fill_blocks, kRedThreads, 0, s, ws, out, pl.out_count, pl.factor);
    check_launch(where);
}

template <class T, int KIND>
void reduce_entry(size_t n, size_t nd, size_t nr, const size_t* meta, const T* in, T* out, const char* where) {
    const size_t* hm = resolve_metadata(meta, 2 * nd + 2 * nr + 1);
    if (!hm) {
        set_error(kErrBadMetadata, 0, where);
        return;
    }
    RedPlan pl;
    red_plan_dims(pl, n, nd, nr, hm);
    red_launch<T, KIND>(pl, in, out, where);
}
template <class T>
void sum_to_shape_entry(size_t n, size_t nd, const size_t* meta, const T* in, T* out, const char* where) {
    const size_t* hm = resolve_metadata(meta, 3 * nd + 1);
    if (!hm) {
        set_error(kErrBadMetadata, 0, where);
        return;
    }
    RedPlan pl;
    red_plan_shape(pl, n, nd, hm);
    red_launch<T, RED_SUM>(pl, in, out, where);
}

}  // namespace mx
