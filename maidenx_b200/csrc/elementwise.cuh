// Strided elementwise engine shared by the binary, in-place binary, unary and
// unary-with-constant families.
//
// The host reduces the (dims, strides, offsets) metadata of the C ABI to a canonical
// form — size-1 dims dropped, adjacent dims merged wherever every operand allows it —
// and picks one of four kernels:
//   flat     every operand is one contiguous run (or a broadcast scalar): 16-byte
//            vector loads/stores, four vectors in flight per thread;
//   row      every operand has stride 1 or 0 along the innermost dim; outer dims are
//            arbitrary (row-vector / column-vector broadcasts, padded rows): one
//            fast-divmod per 16-byte vector instead of per element;
//   tile     an input is unit-stride along another dim (a transposed view): 64x64
//            tiles staged through shared memory so both the transposed read and the
//            output write are full 128-byte lines;
//   shifted  flat operands whose addresses are not 16-byte aligned (the offset-1 views of the reference's test
//            fixtures): a scalar head brings the output to a 16-byte boundary, then every input vector is
//            assembled from the two aligned 16-byte words it straddles with a funnel shift;
//   dense    a dense output whose inputs fit none of the above (ragged rows, broadcasts along rows that are not
//            vector multiples, permuted views): 16-byte output vectors, contiguous inputs as vectors, the others
//            gathered element by element from one index computation per vector;
//   generic  anything else: per-element fast-divmod gather.
// In-place ops reuse the same kernels with the output aliased to the lhs and the dims
// re-ordered by the lhs strides; an lhs that overlaps itself (stride 0) runs serially
// on one thread, which is the order the CPU backend applies.
#pragma once
#include "common.cuh"
#include "ops.cuh"
#include "tc_ptx.cuh"

namespace mx {

enum EwKind { EW_EMPTY = 0, EW_FLAT, EW_ROW, EW_TILE, EW_GENERIC, EW_SERIAL, EW_ERROR, EW_FLAT_SHIFT };

struct EwPlan {
    int kind;
    int nin;
    uint64_t n;
    int nd;
    uint32_t dim[kMaxDims];
    int64_t st[3][kMaxDims];  // element strides: 0 = out, 1 = a, 2 = b
    int64_t off[3];           // element offsets applied to the base pointers
    int p;                    // tile: the dim along which the transposed inputs are unit-stride
    bool transposed[3];       // tile: operand is read through shared memory
    bool vec;                 // 16-byte vector access is legal for every operand
};

// in_size / out_size: element sizes in bytes; ptrs: base addresses (out, a, b) before offsets.
void ew_make_plan(EwPlan& pl, size_t num_els, size_t num_dims, const size_t* hmeta, int nin, bool inplace, size_t in_size,
                  size_t out_size, const void* out, const void* a, const void* b);

// ---------------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------------
constexpr int kEwThreads = 256;
constexpr int kEwUnroll = 4;

template <class T, int N>
__device__ __forceinline__ Vec<T, N> ld_vec(const T* p) {
    return *reinterpret_cast<const Vec<T, N>*>(p);
}
template <class T, int N>
__device__ __forceinline__ void st_vec(T* p, const Vec<T, N>& v) {
    *reinterpret_cast<Vec<T, N>*>(p) = v;
}
template <class T, int N>
__device__ __forceinline__ Vec<T, N> splat(T x) {
    Vec<T, N> v;
#pragma unroll
    for (int i = 0; i < N; i++) v.v[i] = x;
    return v;
}

template <class F, class T, class O, int NIN, int VEC>
__device__ __forceinline__ Vec<O, VEC> apply_vec(const F& f, const Vec<T, VEC>& a, const Vec<T, VEC>& b) {
    Vec<O, VEC> r;
    if constexpr (F::kNative && VEC % 2 == 0 && NIN == 2) {
        // bf16 / f16 add and sub: the packed hardware instruction rounds exactly as "f32, then round"
        const uint32_t* aw = reinterpret_cast<const uint32_t*>(&a);
        const uint32_t* bw = reinterpret_cast<const uint32_t*>(&b);
        uint32_t* rw = reinterpret_cast<uint32_t*>(&r);
#pragma unroll
        for (int i = 0; i < VEC / 2; i++) rw[i] = f.native(aw[i], bw[i]);
    } else if constexpr (F::kChecked && VEC % 2 == 0) {
        // bf16 / f16 division: approximate quotients, and the few elements the check flags are
        // redone with the exact out-of-line division
        const uint32_t* aw = reinterpret_cast<const uint32_t*>(&a);
        const uint32_t* bw = reinterpret_cast<const uint32_t*>(&b);
        uint32_t* rw = reinterpret_cast<uint32_t*>(&r);
        uint32_t mask = 0;
#pragma unroll
        for (int i = 0; i < VEC / 2; i++) {
            float2 x = unpack2<T>(aw[i]);
            if constexpr (NIN == 2) {
                float2 y = unpack2<T>(bw[i]);
                rw[i] = pack2_rn<T>(f.core_checked(x.x, y.x, mask, 2 * i), f.core_checked(x.y, y.y, mask, 2 * i + 1));
            } else {
                rw[i] = pack2_rn<T>(f.core_checked(x.x, mask, 2 * i), f.core_checked(x.y, mask, 2 * i + 1));
            }
        }
        if (mask) {
#pragma unroll
            for (int i = 0; i < VEC; i++) {
                if ((mask >> i) & 1u) {
                    if constexpr (NIN == 2) r.v[i] = f(a.v[i], b.v[i]);
                    else r.v[i] = f(a.v[i]);
                }
            }
        }
    } else if constexpr (F::kCore && VEC % 2 == 0) {
        // 16-bit floats: unpack / compute in f32 / round two elements at a time
        const uint32_t* aw = reinterpret_cast<const uint32_t*>(&a);
        const uint32_t* bw = reinterpret_cast<const uint32_t*>(&b);
        uint32_t* rw = reinterpret_cast<uint32_t*>(&r);
#pragma unroll
        for (int i = 0; i < VEC / 2; i++) {
            float2 x = unpack2<T>(aw[i]);
            if constexpr (NIN == 2) {
                float2 y = unpack2<T>(bw[i]);
                rw[i] = pack2_rn<T>(f.core(x.x, y.x), f.core(x.y, y.y));
            } else {
                rw[i] = pack2_rn<T>(f.core(x.x), f.core(x.y));
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < VEC; i++) {
            if constexpr (NIN == 2) r.v[i] = f(a.v[i], b.v[i]);
            else r.v[i] = f(a.v[i]);
        }
    }
    return r;
}

// What an incomplete block still does element by element: one, two or three trips.  Vectors give a few threads the work of all and take a second
// path for the rest.  Elements / vectors, us: difference of 100 u8 0.95 / 1.84, bf16 0.94 / 1.33, quotient 1.04 / 2.64, 1.10 / 1.93, f32 1.00 / 1.32; 300 u8 1.20 / 1.84,
// bf16 1.14 / 1.19, quotient 1.39 / 1.78, f32 difference 1.15 / 1.02; 700 u8 1.38 / 1.68, bf16 1.33 / 1.21; square of 1000 u8 1.50 / 1.30, bf16 1.73 / 1.04.
template <int VEC>
constexpr uint64_t kEwTailElements = kEwThreads * (VEC >= 16 ? 3 : VEC == 8 ? 2 : 1);
// `full` blocks of four vectors a thread, all loads in flight together, then blocks of one vector a thread: all of a tensor that would leave an SM one
// block the other way (half of one, with 16 elements a vector), the last, incomplete block of a larger one.  Each is one trip to memory; with its four vectors in a loop an incomplete block was
// the length of the launch (3.4 MB f32 3.3 us, 3.9 so), with all of them in flight it cost the main path registers (product of i16 42, 142 so: 40 MB 21 us, 33).
// One / four vectors a thread, us: difference of 2048 vectors f32 1.3 / 1.5, u8 1.7 / 3.7; 60000 1.5 / 1.9, 2.8 / 3.8; 100000 f32 1.74 / 1.94, bf16 1.73 / 2.04, u8 3.96 /
// 3.77; 150000 1.84 / 1.79, 1.82 / 2.05, 5.1 / 3.8; square root of 8191 f32
// 1.3 / 2.3, 6.4 by elements.
template <int VEC>
inline uint32_t ew_flat_full_blocks(uint64_t n) {
    return n / VEC <= (VEC > 8 ? 2 : 4) * (uint64_t)kEwThreads * sm_count() ? 0 : (uint32_t)(n / ((uint64_t)kEwThreads * VEC * kEwUnroll));
}

// sa / sb: 1 = contiguous, 0 = broadcast scalar
template <class F, class T, class O, int NIN, int VEC>
__global__ void __launch_bounds__(kEwThreads) ew_flat_kernel(F f, const T* a, const T* b, O* out, uint64_t n, int sa, int sb, uint32_t full) {
    after_previous_kernel();
    constexpr uint64_t kChunk = (uint64_t)kEwThreads * VEC * kEwUnroll, kPiece = (uint64_t)kEwThreads * VEC;
    if (blockIdx.x < full) {
        const uint64_t base = (uint64_t)blockIdx.x * kChunk;
        Vec<T, VEC> va[kEwUnroll], vb[kEwUnroll];
#pragma unroll
        for (int u = 0; u < kEwUnroll; u++) {
            uint64_t i = base + ((uint64_t)u * kEwThreads + threadIdx.x) * VEC;
            va[u] = sa ? ld_vec<T, VEC>(a + i) : splat<T, VEC>(a[0]);
            if constexpr (NIN == 2) vb[u] = sb ? ld_vec<T, VEC>(b + i) : splat<T, VEC>(b[0]);
        }
#pragma unroll
        for (int u = 0; u < kEwUnroll; u++) {
            uint64_t i = base + ((uint64_t)u * kEwThreads + threadIdx.x) * VEC;
            st_vec<O, VEC>(out + i, apply_vec<F, T, O, NIN, VEC>(f, va[u], vb[u]));
        }
        return;
    }
    const uint64_t base = full * kChunk + (blockIdx.x - full) * kPiece, end = base + kPiece < n ? base + kPiece : n;
    uint64_t rest = base;
    if (end - base > kEwTailElements<VEC>) {
        const uint64_t i = base + (uint64_t)threadIdx.x * VEC;
        if (i + VEC <= end) {
            const Vec<T, VEC> va = sa ? ld_vec<T, VEC>(a + i) : splat<T, VEC>(a[0]);
            Vec<T, VEC> vb;
            if constexpr (NIN == 2) vb = sb ? ld_vec<T, VEC>(b + i) : splat<T, VEC>(b[0]);
            st_vec<O, VEC>(out + i, apply_vec<F, T, O, NIN, VEC>(f, va, vb));
        }
        rest = end - end % VEC;  // blocks start at whole vectors
    }
    for (uint64_t i = rest + threadIdx.x; i < end; i += kEwThreads) {
        T x = a[sa ? i : 0];
        if constexpr (NIN == 2) out[i] = f(x, b[sb ? i : 0]);
        else out[i] = f(x);
    }
}

// Funnel-shifts the 32 bytes (lo, hi) right by `sh` bytes and returns the low 16.
__device__ __forceinline__ uint4 shift_pair(const uint4& lo, const uint4& hi, uint32_t sh) {
    const uint32_t bits = (sh & 3u) * 8u;
    switch (sh >> 2) {
        case 0:
            return make_uint4(__funnelshift_r(lo.x, lo.y, bits), __funnelshift_r(lo.y, lo.z, bits), __funnelshift_r(lo.z, lo.w, bits),
                              __funnelshift_r(lo.w, hi.x, bits));
        case 1:
            return make_uint4(__funnelshift_r(lo.y, lo.z, bits), __funnelshift_r(lo.z, lo.w, bits), __funnelshift_r(lo.w, hi.x, bits),
                              __funnelshift_r(hi.x, hi.y, bits));
        case 2:
            return make_uint4(__funnelshift_r(lo.z, lo.w, bits), __funnelshift_r(lo.w, hi.x, bits), __funnelshift_r(hi.x, hi.y, bits),
                              __funnelshift_r(hi.y, hi.z, bits));
        default:
            return make_uint4(__funnelshift_r(lo.w, hi.x, bits), __funnelshift_r(hi.x, hi.y, bits), __funnelshift_r(hi.y, hi.z, bits),
                              __funnelshift_r(hi.z, hi.w, bits));
    }
}

// VEC elements starting at an arbitrary element-aligned address: the two aligned 16-byte words the vector straddles,
// shifted together.  `sh` = the address modulo 16 (the same for every vector of a launch).  Both words contain at
// least one byte of the vector, so neither load leaves the allocation.  The second word is the next lane's first
// word, so it comes from L1; handing it over by warp shuffle instead was measured slower (four shuffles per operand
// and vector cost more issue slots than the cached load).
template <class T, int VEC>
__device__ __forceinline__ Vec<T, VEC> ld_vec_shifted(const T* p, uint32_t sh) {
    static_assert(sizeof(T) * VEC == 16, "one 16-byte vector");
    const uintptr_t addr = reinterpret_cast<uintptr_t>(p) - sh;
    const uint4 lo = *reinterpret_cast<const uint4*>(addr);
    if (sh == 0) return *reinterpret_cast<const Vec<T, VEC>*>(&lo);
    const uint4 hi = *reinterpret_cast<const uint4*>(addr + 16);
    const uint4 r = shift_pair(lo, hi, sh);
    return *reinterpret_cast<const Vec<T, VEC>*>(&r);
}

// Flat operands at addresses that are not 16-byte aligned.  Elements [0, head) and [tail_begin, n) are handled one at a
// time by block 0; the body [head, tail_begin) starts where the OUTPUT is aligned for its vector store, and each input
// is read with ld_vec_shifted (sha / shb = its address modulo 16 at the start of the body).  sa / sb: 1 = contiguous,
// 0 = broadcast scalar.
template <class F, class T, class O, int NIN, int VEC>
__global__ void __launch_bounds__(kEwThreads) ew_flat_shift_kernel(F f, const T* a, const T* b, O* out, uint64_t n, uint64_t head, uint64_t body_vecs,
                                                                   int sa, int sb, uint32_t sha, uint32_t shb) {
    after_previous_kernel();
    const uint64_t v0 = (uint64_t)blockIdx.x * kEwThreads * kEwUnroll + threadIdx.x;
    Vec<T, VEC> va[kEwUnroll], vb[kEwUnroll];
#pragma unroll
    for (int u = 0; u < kEwUnroll; u++) {
        const uint64_t v = v0 + (uint64_t)u * kEwThreads;
        if (v < body_vecs) {
            const uint64_t i = head + v * VEC;
            va[u] = sa ? ld_vec_shifted<T, VEC>(a + i, sha) : splat<T, VEC>(a[0]);
            if constexpr (NIN == 2) vb[u] = sb ? ld_vec_shifted<T, VEC>(b + i, shb) : splat<T, VEC>(b[0]);
        }
    }
#pragma unroll
    for (int u = 0; u < kEwUnroll; u++) {
        const uint64_t v = v0 + (uint64_t)u * kEwThreads;
        if (v < body_vecs) st_vec<O, VEC>(out + head + v * VEC, apply_vec<F, T, O, NIN, VEC>(f, va[u], vb[u]));
    }
    if (blockIdx.x == 0) {
        const uint64_t tail_begin = head + body_vecs * VEC;
        const uint64_t edge = head + (n - tail_begin);  // fewer than VEC elements on either side
        for (uint64_t e = threadIdx.x; e < edge; e += kEwThreads) {
            const uint64_t i = e < head ? e : tail_begin + (e - head);
            T x = a[sa ? i : 0];
            if constexpr (NIN == 2) out[i] = f(x, b[sb ? i : 0]);
            else out[i] = f(x);
        }
    }
}

// The same work with the shifted operands staged through shared memory: one thread asks the copy engine of the SM
// (cp.async.bulk, global -> shared, completion on an mbarrier) for the 16-byte-aligned span that covers the block's part
// of each shifted operand - every byte crosses from L2 exactly once, in full lines - and each thread then assembles its
// vectors from two aligned 16-byte shared-memory words.  Used for large operands; the body of the block is kEwThreads *
// kEwUnroll vectors, i.e. 16 KB (+ 16 bytes) of shared memory per shifted operand.  The wait on the barrier is bounded.
constexpr int kEwStageBytes = kEwThreads * kEwUnroll * 16 + 16;

__device__ __forceinline__ bool ew_stage_wait(uint32_t bar, const tc::WaitReport& rep, int code) {
    for (int i = 0; i < (1 << 26); i++) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar)
            : "memory");
        if (ok) return true;
    }
    tc::wait_gave_up(rep, code);  // surfaces as status 5 at the caller's next synchronisation point
    return false;
}

template <class F, class T, class O, int NIN, int VEC>
__global__ void __launch_bounds__(kEwThreads) ew_flat_shift_staged_kernel(F f, const T* a, const T* b, O* out, uint64_t n, uint64_t head,
                                                                          uint64_t body_vecs, int sa, int sb, uint32_t sha, uint32_t shb, int stage_aligned, tc::WaitReport rep) {
    after_previous_kernel();
    extern __shared__ __align__(128) unsigned char ew_stage[];
    __shared__ __align__(8) unsigned long long stage_bar;
    const uint64_t block_v0 = (uint64_t)blockIdx.x * kEwThreads * kEwUnroll;
    const uint64_t left = block_v0 < body_vecs ? body_vecs - block_v0 : 0;
    const uint32_t nv = left < (uint64_t)kEwThreads * kEwUnroll ? (uint32_t)left : (uint32_t)(kEwThreads * kEwUnroll);  // vectors of this block
    // stage_aligned: aligned operands go through shared memory as well (register-heavy functors keep too few loads in flight
    // on their own; the copy engine's queue does not depend on how many threads are resident)
    const bool stage_a = nv && sa && (sha != 0 || stage_aligned), stage_b = nv && NIN == 2 && sb && (shb != 0 || stage_aligned);
    unsigned char* buf_a = ew_stage;
    unsigned char* buf_b = ew_stage + (stage_a ? kEwStageBytes : 0);
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&stage_bar);
    if (stage_a || stage_b) {
        if (threadIdx.x == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            // the aligned words the block's vectors straddle: one extra word only for an operand that is really shifted
            const uint32_t bytes_a = nv * 16 + (sha ? 16 : 0), bytes_b = nv * 16 + (shb ? 16 : 0);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((stage_a ? bytes_a : 0) + (stage_b ? bytes_b : 0)) : "memory");
            if (stage_a) {
                const uintptr_t src = reinterpret_cast<uintptr_t>(a + head + block_v0 * VEC) - sha;
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                 (uint32_t)__cvta_generic_to_shared(buf_a)),
                             "l"(src), "r"(bytes_a), "r"(bar)
                             : "memory");
            }
            if (stage_b) {
                const uintptr_t src = reinterpret_cast<uintptr_t>(b + head + block_v0 * VEC) - shb;
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                 (uint32_t)__cvta_generic_to_shared(buf_b)),
                             "l"(src), "r"(bytes_b), "r"(bar)
                             : "memory");
            }
        }
    }
    // operands that need no staging are read straight from global memory while the copies fly
    Vec<T, VEC> va[kEwUnroll], vb[kEwUnroll];
#pragma unroll
    for (int u = 0; u < kEwUnroll; u++) {
        const uint32_t lv = (uint32_t)u * kEwThreads + threadIdx.x;
        if (lv < nv) {
            const uint64_t i = head + (block_v0 + lv) * VEC;
            if (!stage_a) va[u] = sa ? ld_vec<T, VEC>(a + i) : splat<T, VEC>(a[0]);
            if constexpr (NIN == 2)
                if (!stage_b) vb[u] = sb ? ld_vec<T, VEC>(b + i) : splat<T, VEC>(b[0]);
        }
    }
    bool landed = true;
    if (stage_a || stage_b) {
        __syncthreads();  // the barrier is initialised before anyone polls it
        landed = ew_stage_wait(bar, rep, 21);
    }
    if (landed) {
#pragma unroll
        for (int u = 0; u < kEwUnroll; u++) {
            const uint32_t lv = (uint32_t)u * kEwThreads + threadIdx.x;
            if (lv >= nv) continue;
            if (stage_a) {
                const uint4 lo = *reinterpret_cast<const uint4*>(buf_a + lv * 16);
                uint4 r = lo;
                if (sha) r = shift_pair(lo, *reinterpret_cast<const uint4*>(buf_a + lv * 16 + 16), sha);
                va[u] = *reinterpret_cast<const Vec<T, VEC>*>(&r);
            }
            if constexpr (NIN == 2) {
                if (stage_b) {
                    const uint4 lo = *reinterpret_cast<const uint4*>(buf_b + lv * 16);
                    uint4 r = lo;
                    if (shb) r = shift_pair(lo, *reinterpret_cast<const uint4*>(buf_b + lv * 16 + 16), shb);
                    vb[u] = *reinterpret_cast<const Vec<T, VEC>*>(&r);
                }
            }
            st_vec<O, VEC>(out + head + (block_v0 + lv) * VEC, apply_vec<F, T, O, NIN, VEC>(f, va[u], vb[u]));
        }
    }
    if (blockIdx.x == 0) {
        const uint64_t tail_begin = head + body_vecs * VEC;
        const uint64_t edge = head + (n - tail_begin);
        for (uint64_t e = threadIdx.x; e < edge; e += kEwThreads) {
            const uint64_t i = e < head ? e : tail_begin + (e - head);
            T x = a[sa ? i : 0];
            if constexpr (NIN == 2) out[i] = f(x, b[sb ? i : 0]);
            else out[i] = f(x);
        }
    }
}

struct EwRowParams {
    int nd_outer;
    uint32_t total_vecs;
    uint32_t qv;                    // vectors per row
    uint32_t chunks_per_row;        // long-row mode: blocks per row
    FastDiv qv_div;                 // short-row mode: vectors per row
    FastDiv chunk_div;              // long-row mode: blocks per row
    FastDiv outer_div[kMaxDims];    // outer dims, innermost outer dim last
    int64_t st[3][kMaxDims];        // outer strides per operand
    int sq[3];                      // stride along q per operand (1 or 0)
};

// Long rows (at least one block-load of vectors per row): a block works inside one row, so
// the row's base offsets are computed once per block and each thread only adds its vector
// index — the same instruction stream as the flat kernel.
template <class F, class T, class O, int NIN, int VEC>
__global__ void __launch_bounds__(kEwThreads, 4) ew_row_long_kernel(F f, const T* a, const T* b, O* out, EwRowParams P) {
    after_previous_kernel();
    uint32_t r, chunk;
    P.chunk_div.divmod(blockIdx.x, r, chunk);
    int64_t o_out = 0, o_a = 0, o_b = 0;
    for (int d = P.nd_outer - 1; d >= 0; d--) {  // block-uniform
        uint32_t c;
        P.outer_div[d].divmod(r, r, c);
        o_out += (int64_t)c * P.st[0][d];
        o_a += (int64_t)c * P.st[1][d];
        if constexpr (NIN == 2) o_b += (int64_t)c * P.st[2][d];
    }
    out += o_out;
    a += o_a;
    if constexpr (NIN == 2) b += o_b;
    const uint32_t v0 = chunk * (kEwThreads * kEwUnroll) + threadIdx.x;
    Vec<T, VEC> va[kEwUnroll], vb[kEwUnroll];
    if (P.sq[1]) {
#pragma unroll
        for (int u = 0; u < kEwUnroll; u++)
            if (v0 + u * kEwThreads < P.qv) va[u] = ld_vec<T, VEC>(a + (size_t)(v0 + u * kEwThreads) * VEC);
    } else {
        Vec<T, VEC> s = splat<T, VEC>(a[0]);
#pragma unroll
        for (int u = 0; u < kEwUnroll; u++) va[u] = s;
    }
    if constexpr (NIN == 2) {
        if (P.sq[2]) {
#pragma unroll
            for (int u = 0; u < kEwUnroll; u++)
                if (v0 + u * kEwThreads < P.qv) vb[u] = ld_vec<T, VEC>(b + (size_t)(v0 + u * kEwThreads) * VEC);
        } else {
            Vec<T, VEC> s = splat<T, VEC>(b[0]);
#pragma unroll
            for (int u = 0; u < kEwUnroll; u++) vb[u] = s;
        }
    }
#pragma unroll
    for (int u = 0; u < kEwUnroll; u++) {
        uint32_t v = v0 + u * kEwThreads;
        if (v < P.qv) st_vec<O, VEC>(out + (size_t)v * VEC, apply_vec<F, T, O, NIN, VEC>(f, va[u], vb[u]));
    }
}

// Unary op whose input is one row broadcast over every outer dim (strides [0, ..., 0, 1]):
// f(broadcast(x)) == broadcast(f(x)), so each thread evaluates its vectors once and stores
// them to a slab of output rows — the kernel is a pure store stream.
template <class F, class T, class O, int VEC>
__global__ void __launch_bounds__(kEwThreads) ew_bcast_rows_kernel(F f, const T* a, O* out, uint32_t qv, uint32_t rows, uint32_t rows_per_block) {
    after_previous_kernel();
    const uint32_t v0 = blockIdx.x * (kEwThreads * kEwUnroll) + threadIdx.x;
    const uint32_t r0 = blockIdx.y * rows_per_block;
    const uint32_t r1 = min(rows, r0 + rows_per_block);
    Vec<O, VEC> res[kEwUnroll];
    Vec<T, VEC> dummy;
#pragma unroll
    for (int u = 0; u < kEwUnroll; u++) {
        uint32_t v = v0 + u * kEwThreads;
        if (v < qv) res[u] = apply_vec<F, T, O, 1, VEC>(f, ld_vec<T, VEC>(a + (size_t)v * VEC), dummy);
    }
    for (uint32_t r = r0; r < r1; r++) {
        O* dst = out + (size_t)r * qv * VEC;
#pragma unroll
        for (int u = 0; u < kEwUnroll; u++) {
            uint32_t v = v0 + u * kEwThreads;
            if (v < qv) st_vec<O, VEC>(dst + (size_t)v * VEC, res[u]);
        }
    }
}

// The same store stream issued by the SM's copy engine: the block evaluates its chunk of the row into shared memory once
// and one thread then queues one cp.async.bulk (shared -> global) per output row of the block's slab; no per-element store
// instructions at all.  The chunk is kEwThreads * kEwUnroll output vectors (16 KB when the output type is as wide as the
// input type); rows are VEC * sizeof(O)-byte multiples here, so every copy is 16-byte aligned and sized.
template <class F, class T, class O, int VEC>
__global__ void __launch_bounds__(kEwThreads) ew_bcast_rows_bulk_kernel(F f, const T* a, O* out, uint32_t qv, uint32_t rows, uint32_t rows_per_block) {
    after_previous_kernel();
    extern __shared__ __align__(128) unsigned char ew_stage[];
    const uint32_t chunk_v0 = blockIdx.x * (kEwThreads * kEwUnroll);
    const uint32_t nv = min(qv - chunk_v0, (uint32_t)(kEwThreads * kEwUnroll));
    const uint32_t r0 = blockIdx.y * rows_per_block;
    const uint32_t r1 = min(rows, r0 + rows_per_block);
    Vec<T, VEC> dummy;
#pragma unroll
    for (int u = 0; u < kEwUnroll; u++) {
        const uint32_t lv = u * kEwThreads + threadIdx.x;
        if (lv < nv)
            *reinterpret_cast<Vec<O, VEC>*>(ew_stage + (size_t)lv * VEC * sizeof(O)) =
                apply_vec<F, T, O, 1, VEC>(f, ld_vec<T, VEC>(a + (size_t)(chunk_v0 + lv) * VEC), dummy);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the copy engine reads what the threads just wrote
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t bytes = nv * VEC * (uint32_t)sizeof(O);
        const uint32_t src = (uint32_t)__cvta_generic_to_shared(ew_stage);
        for (uint32_t r = r0; r < r1; r++) {
            O* dst = out + ((size_t)r * qv + chunk_v0) * VEC;
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
        }
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // shared memory stays valid until the copies have read it (and landed)
    }
}

// Short rows: one fast-divmod per vector to find its row.
template <class F, class T, class O, int NIN, int VEC>
__global__ void __launch_bounds__(kEwThreads) ew_row_kernel(F f, const T* a, const T* b, O* out, EwRowParams P) {
    after_previous_kernel();
    const uint32_t base = blockIdx.x * (kEwThreads * kEwUnroll);
#pragma unroll
    for (int u = 0; u < kEwUnroll; u++) {
        uint32_t v = base + u * kEwThreads + threadIdx.x;
        if (v < P.total_vecs) {
            uint32_t r, qv;
            P.qv_div.divmod(v, r, qv);
            int64_t o_out = (int64_t)qv * VEC, o_a = (int64_t)qv * VEC * P.sq[1], o_b = (int64_t)qv * VEC * P.sq[2];
#pragma unroll
            for (int d = kMaxDims - 1; d >= 0; d--) {
                if (d < P.nd_outer) {
                    uint32_t c;
                    P.outer_div[d].divmod(r, r, c);
                    o_out += (int64_t)c * P.st[0][d];
                    o_a += (int64_t)c * P.st[1][d];
                    if constexpr (NIN == 2) o_b += (int64_t)c * P.st[2][d];
                }
            }
            Vec<T, VEC> va = P.sq[1] ? ld_vec<T, VEC>(a + o_a) : splat<T, VEC>(a[o_a]), vb;
            if constexpr (NIN == 2) vb = P.sq[2] ? ld_vec<T, VEC>(b + o_b) : splat<T, VEC>(b[o_b]);
            st_vec<O, VEC>(out + o_out, apply_vec<F, T, O, NIN, VEC>(f, va, vb));
        }
    }
}

struct EwTileParams {
    uint32_t P, Q;                  // extents of the tiled dims
    uint32_t tiles_p, tiles_q;
    FastDiv tiles_q_div, tiles_p_div;
    int nd_batch;
    FastDiv batch_div[kMaxDims];
    int64_t st_batch[3][kMaxDims];
    int64_t st_p[3], st_q[3];
    int transposed[3];              // [1], [2]: input goes through shared memory
    int smem_slot[3];               // [1], [2]: which staging buffer a transposed input uses
};

template <class T>
struct EwTile {
    static constexpr int kTile = sizeof(T) == 8 ? 32 : 64;
    static constexpr int kPitch = kTile * (int)sizeof(T) + (sizeof(T) == 8 ? 8 : 4);  // bytes per staged row
    static constexpr int kBytes = kTile * kPitch;                                     // one staging buffer
};

// A warp covers 8 vectors x 4 rows (VEC > 1) or 32 elements x 1 row (VEC == 1) of the tile:
// 128-byte global segments, and shared-memory word accesses that do not collide.
template <int VPR, int VEC>
__device__ __forceinline__ void ew_tile_coord(int i, int& row, int& vcol) {
    if constexpr (VEC > 1 && VPR >= 8) {
        constexpr int WC = VPR / 8;  // warp-columns per tile row
        int w = i >> 5, lane = i & 31;
        vcol = (w % WC) * 8 + (lane & 7);
        row = (w / WC) * 4 + (lane >> 3);
    } else {
        row = i / VPR;
        vcol = i % VPR;
    }
}

template <class F, class T, class O, int NIN, int VEC>
__global__ void __launch_bounds__(kEwThreads, sizeof(T) == 2 ? 6 : 4) ew_tile_kernel(F f, const T* a, const T* b, O* out, EwTileParams P) {
    after_previous_kernel();
    constexpr int TILE = EwTile<T>::kTile;
    constexpr int PITCH = EwTile<T>::kPitch;
    constexpr int VPR = TILE / VEC;                       // vectors per tile row
    constexpr int ITER = (TILE * VPR + kEwThreads - 1) / kEwThreads;
    extern __shared__ __align__(16) unsigned char ew_smem[];

    uint32_t t = blockIdx.x, tq, tp, bidx;
    P.tiles_q_div.divmod(t, t, tq);
    P.tiles_p_div.divmod(t, bidx, tp);
    int64_t base[3] = {0, 0, 0};
    for (int d = P.nd_batch - 1; d >= 0; d--) {  // block-uniform
        uint32_t c;
        P.batch_div[d].divmod(bidx, bidx, c);
#pragma unroll
        for (int k = 0; k < 3; k++) base[k] += (int64_t)c * P.st_batch[k][d];
    }
    const uint32_t p0 = tp * TILE, q0 = tq * TILE;
#pragma unroll
    for (int k = 0; k < 3; k++) base[k] += (int64_t)p0 * P.st_p[k] + (int64_t)q0 * P.st_q[k];
    const T* in[2] = {a, b};

    // Phase-2 work item: RP consecutive p-rows x one vector along q.  For 2-byte types two rows
    // are handled together, so that one 32-bit shared-memory read (two neighbouring p of one q)
    // feeds both: half the shared-memory instructions of a row-at-a-time walk.
    constexpr int RP = (sizeof(T) == 2 && VEC == 8) ? 2 : 1;
    constexpr int ITER2 = ((TILE / RP) * VPR + kEwThreads - 1) / kEwThreads;
    auto item_coord = [](int i, int& prow, int& qv) {
        if constexpr (RP == 2) {  // a warp covers 8 vectors (128 bytes) x 4 row pairs
            int w = i >> 5, lane = i & 31;
            qv = lane & 7;
            prow = (w * 4 + (lane >> 3)) * 2;
        } else {
            ew_tile_coord<VPR, VEC>(i, prow, qv);
        }
    };

    // All global loads of the tile are issued before the barrier: the direct operands in
    // the phase-2 mapping (rows along p, vectors along q), the transposed operands in the
    // phase-1 mapping (rows along q, vectors along p, their unit-stride dim).
    Vec<T, VEC> direct[NIN][ITER2][RP];
    Vec<T, VEC> staged[NIN][ITER];
#pragma unroll
    for (int x = 0; x < NIN; x++) {
        if (P.transposed[x + 1]) {
            const T* src = in[x] + base[x + 1];
#pragma unroll
            for (int it = 0; it < ITER; it++) {
                int qq, pv;
                ew_tile_coord<VPR, VEC>(threadIdx.x + it * kEwThreads, qq, pv);
                if (qq < TILE && q0 + qq < P.Q && p0 + pv * VEC < P.P) staged[x][it] = ld_vec<T, VEC>(src + (int64_t)qq * P.st_q[x + 1] + pv * VEC);
            }
        } else {
            const T* src = in[x] + base[x + 1];
#pragma unroll
            for (int it = 0; it < ITER2; it++) {
                int pp, qv;
                item_coord(threadIdx.x + it * kEwThreads, pp, qv);
#pragma unroll
                for (int r = 0; r < RP; r++) {
                    if (pp + r < TILE && p0 + pp + r < P.P && q0 + qv * VEC < P.Q) {
                        const T* s = src + (int64_t)(pp + r) * P.st_p[x + 1];
                        direct[x][it][r] = P.st_q[x + 1] ? ld_vec<T, VEC>(s + qv * VEC) : splat<T, VEC>(s[0]);
                    }
                }
            }
        }
    }
    // phase 1: stage the transposed inputs as [q][p]
#pragma unroll
    for (int x = 0; x < NIN; x++) {
        if (!P.transposed[x + 1]) continue;
        unsigned char* buf = ew_smem + P.smem_slot[x + 1] * EwTile<T>::kBytes;
#pragma unroll
        for (int it = 0; it < ITER; it++) {
            int qq, pv;
            ew_tile_coord<VPR, VEC>(threadIdx.x + it * kEwThreads, qq, pv);
            if (qq < TILE && q0 + qq < P.Q && p0 + pv * VEC < P.P) {
                unsigned char* row = buf + qq * PITCH + pv * VEC * (int)sizeof(T);
                if constexpr (VEC * sizeof(T) >= 4 && sizeof(T) < 4) {
                    const uint32_t* w = reinterpret_cast<const uint32_t*>(&staged[x][it]);
#pragma unroll
                    for (int j = 0; j < (int)(VEC * sizeof(T) / 4); j++) reinterpret_cast<uint32_t*>(row)[j] = w[j];
                } else {
#pragma unroll
                    for (int j = 0; j < VEC; j++) reinterpret_cast<T*>(row)[j] = staged[x][it].v[j];
                }
            }
        }
    }
    __syncthreads();

    // phase 2: walk the tile along q (the output's unit-stride dim)
#pragma unroll
    for (int it = 0; it < ITER2; it++) {
        int pp, qv;
        item_coord(threadIdx.x + it * kEwThreads, pp, qv);
        if (pp >= TILE || p0 + pp >= P.P || q0 + qv * VEC >= P.Q) continue;
        Vec<T, VEC> v[2][RP];
#pragma unroll
        for (int x = 0; x < NIN; x++) {
            if (P.transposed[x + 1]) {
                const unsigned char* buf = ew_smem + P.smem_slot[x + 1] * EwTile<T>::kBytes;
                if constexpr (RP == 2) {
                    // word j holds (q = qv*8 + j; p = pp, pp + 1): split the halves into the two rows
                    uint32_t w[VEC];
#pragma unroll
                    for (int j = 0; j < VEC; j++) w[j] = *reinterpret_cast<const uint32_t*>(buf + (qv * VEC + j) * PITCH + pp * 2);
                    uint32_t* r0 = reinterpret_cast<uint32_t*>(&v[x][0]);
                    uint32_t* r1 = reinterpret_cast<uint32_t*>(&v[x][1]);
#pragma unroll
                    for (int j = 0; j < VEC / 2; j++) {
                        r0[j] = __byte_perm(w[2 * j], w[2 * j + 1], 0x5410);
                        r1[j] = __byte_perm(w[2 * j], w[2 * j + 1], 0x7632);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < VEC; j++) v[x][0].v[j] = *reinterpret_cast<const T*>(buf + (qv * VEC + j) * PITCH + pp * (int)sizeof(T));
                }
            } else {
#pragma unroll
                for (int r = 0; r < RP; r++) v[x][r] = direct[x][it][r];
            }
        }
#pragma unroll
        for (int r = 0; r < RP; r++) {
            if (p0 + pp + r < P.P)
                st_vec<O, VEC>(out + base[0] + (int64_t)(pp + r) * P.st_p[0] + qv * VEC, apply_vec<F, T, O, NIN, VEC>(f, v[0][r], v[1][r]));
        }
    }
}

// Tile kernel for 2-byte element types (both in and out), vector-aligned layouts with at most one batch dim.  Every
// operand tile crosses between global and shared memory as ONE tensor copy (a 64 x 64 box, 128-byte swizzle; the inputs
// complete on an mbarrier, the output tile is written back the same way; ragged edges are clipped by the copy engine),
// so no thread spends load/store slots on global memory.  A transposed operand sits in shared memory as [q][p];
// ldmatrix.x4.trans hands each thread the 2 x 4 neighbouring-q pairs of one p-row, i.e. the transposition happens
// inside the instruction, and a direct operand and the output are read/written in that same fragment layout with
// 32-bit accesses.  Under the swizzle the eight 16-byte rows of an 8x8 block, and the 32 words of a fragment access,
// fall in distinct banks.
constexpr int kEwT16 = 64;
constexpr int kEwT16Bytes = kEwT16 * 128;

struct EwTile16Params {
    FastDiv tiles_q_div, tiles_p_div;
    int transposed[3];
    int batched[3];  // 0: the operand's map has one batch entry (broadcast along the batch dim)
};

template <class F, class T, class O, int NIN>
__global__ void __launch_bounds__(kEwThreads) ew_tile16_kernel(F f, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                                                               const __grid_constant__ CUtensorMap map_o, EwTile16Params P, tc::WaitReport rep) {
    after_previous_kernel();
    static_assert(sizeof(T) == 2 && sizeof(O) == 2, "2-byte elements on both sides");
    extern __shared__ unsigned char ew_smem_raw[];
    __shared__ __align__(8) unsigned long long tile_bar;

    uint32_t t = blockIdx.x, tq, tp, bidx;
    P.tiles_q_div.divmod(t, t, tq);
    P.tiles_p_div.divmod(t, bidx, tp);
    const int p0 = (int)tp * kEwT16, q0 = (int)tq * kEwT16;
    const uint32_t smem0 = ((uint32_t)__cvta_generic_to_shared(ew_smem_raw) + 1023u) & ~1023u;  // the swizzle pattern repeats every 1024 bytes
    unsigned char* tiles = ew_smem_raw + (smem0 - (uint32_t)__cvta_generic_to_shared(ew_smem_raw));
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&tile_bar);

    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)NIN * kEwT16Bytes) : "memory");
#pragma unroll
        for (int x = 0; x < NIN; x++) {
            const bool tr = P.transposed[x + 1] != 0;
            tc::tma_load_3d(smem0 + x * kEwT16Bytes, x ? &map_b : &map_a, tr ? p0 : q0, tr ? q0 : p0, P.batched[x + 1] ? (int)bidx : 0, bar);
        }
    }
    __syncthreads();  // the barrier is initialised before anyone polls it
    const bool landed = ew_stage_wait(bar, rep, 22);
    if (landed) {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        unsigned char* obuf = tiles + NIN * kEwT16Bytes;
#pragma unroll
        for (int s = 0; s < 2; s++) {
            const int ws = warp + 8 * s, pb = ws >> 1, qh = ws & 1;  // an 8-row p-block x one 32-wide half of q per warp step
            // fragment word m of this lane: row p = pb*8 + lane/4, 16-byte chunk qh*4 + m (swizzled by the row), word lane%4
            const uint32_t frag_row = (uint32_t)(pb * 8 + (lane >> 2)) * 128u + (uint32_t)(lane & 3) * 4u;
            uint32_t w[2][4] = {};
#pragma unroll
            for (int x = 0; x < NIN; x++) {
                if (P.transposed[x + 1]) {
                    const uint32_t row = (uint32_t)(qh * 32 + lane);
                    const uint32_t addr = smem0 + x * kEwT16Bytes + row * 128u + (((uint32_t)pb ^ (row & 7u)) << 4);
                    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(w[x][0]), "=r"(w[x][1]), "=r"(w[x][2]), "=r"(w[x][3])
                                 : "r"(addr)
                                 : "memory");
                } else {
                    const unsigned char* src = tiles + x * kEwT16Bytes + frag_row;
#pragma unroll
                    for (int m = 0; m < 4; m++) w[x][m] = *reinterpret_cast<const uint32_t*>(src + (((uint32_t)(qh * 4 + m) ^ (uint32_t)(lane >> 2)) << 4));
                }
            }
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const Vec<O, 2> r = apply_vec<F, T, O, NIN, 2>(f, *reinterpret_cast<const Vec<T, 2>*>(&w[0][m]), *reinterpret_cast<const Vec<T, 2>*>(&w[1][m]));
                *reinterpret_cast<uint32_t*>(obuf + frag_row + (((uint32_t)(qh * 4 + m) ^ (uint32_t)(lane >> 2)) << 4)) = *reinterpret_cast<const uint32_t*>(&r);
            }
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the copy engine reads what the threads just wrote
    __syncthreads();
    if (landed && threadIdx.x == 0) {
        tc::tma_store_3d(&map_o, smem0 + NIN * kEwT16Bytes, q0, p0, (int)bidx);
        tc::tma_store_commit();
        tc::tma_store_wait_read<0>();  // shared memory stays valid until the copy has read it
    }
}

struct EwGenParams {
    int nd;
    uint64_t n;
    uint32_t dim[kMaxDims];
    FastDiv div[kMaxDims];
    int64_t st[3][kMaxDims];
};

template <class F, class T, class O, int NIN>
__global__ void __launch_bounds__(kEwThreads) ew_generic_kernel(F f, const T* a, const T* b, O* out, EwGenParams P) {
    after_previous_kernel();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < P.n; i += stride) {
        int64_t o0 = 0, o1 = 0, o2 = 0;
        if (P.n <= 0xFFFFFFFFull) {
            uint32_t r = (uint32_t)i;
            for (int d = P.nd - 1; d >= 0; d--) {
                uint32_t c;
                P.div[d].divmod(r, r, c);
                o0 += (int64_t)c * P.st[0][d];
                o1 += (int64_t)c * P.st[1][d];
                if constexpr (NIN == 2) o2 += (int64_t)c * P.st[2][d];
            }
        } else {
            uint64_t r = i;
            for (int d = P.nd - 1; d >= 0; d--) {
                uint64_t c = r % P.dim[d];
                r /= P.dim[d];
                o0 += (int64_t)c * P.st[0][d];
                o1 += (int64_t)c * P.st[1][d];
                if constexpr (NIN == 2) o2 += (int64_t)c * P.st[2][d];
            }
        }
        if constexpr (NIN == 2) out[o0] = f(a[o1], b[o2]);
        else out[o0] = f(a[o1]);
    }
}

// The same gather for an output that is dense and aligned: a thread produces kEwDenseUnroll vectors of consecutive outputs, each
// from ONE index computation in 32 bits.  An input with the output's own strides is read as a vector when its address
// allows.  Of any other, the elements of a vector come from at most two neighbouring rows (rows of at least VEC elements),
// whose offsets are both known up front, so that all loads are independent; an input that is constant along the rows costs
// two loads per vector.  Shorter rows walk the vector row by row.
// Bound by HBM / L2 where rows are long enough: [8191, 1023] f32 with a per-row operand 12 us (33 on the gather
// kernel; a flat op on the same data 9); [256, 512, 7, 7] bf16 with a per-channel one 9.9 us (33).  These two and a row that repeats have kernels of
// their own below; here stay ops of one input, operands at odd addresses, more than three dims, rows shorter than a vector and vectors of 16 elements.
enum EwDenseKind { EWD_VECTOR = 0, EWD_ELEMENT, EWD_CONST, EWD_STEP };
constexpr int kEwDenseUnroll = 2;
struct EwDenseParams {
    int nd;
    uint32_t n, q;              // elements; extent of the innermost dim
    int kind[3];                // [1], [2]: EwDenseKind of the input
    FastDiv q_div, div[kMaxDims];
    int st[3][kMaxDims];
};
// One vector's place: its first element, how many are inside the tensor and how many of those in its first row.
struct EwDensePlace {
    uint32_t i0;
    int live, left;
};
// o0: offset of the vector's first element, o1: of the place its elements beyond the first row count from
template <class T, int VEC>
__device__ __forceinline__ void ew_dense_load(const T* p, int kind, int sq, const EwDensePlace& w, int o0, int o1, Vec<T, VEC>& v) {
    if (kind == EWD_VECTOR && w.live == VEC) {
        v = ld_vec<T, VEC>(p + w.i0);
    } else if (kind == EWD_CONST) {
        const T x0 = p[o0], x1 = w.left < w.live ? p[o1] : x0;
#pragma unroll
        for (int j = 0; j < VEC; j++) v.v[j] = j < w.left ? x0 : x1;
    } else {
#pragma unroll
        for (int j = 0; j < VEC; j++)
            if (j < w.live) v.v[j] = p[kind == EWD_STEP ? (j < w.left ? o0 : o1) + j * sq : (int)w.i0 + j];
    }
}
template <class F, class T, class O, int NIN, int VEC>
__device__ __forceinline__ void ew_dense_store(const F& f, O* out, const EwDensePlace& w, const Vec<T, VEC>& va, const Vec<T, VEC>& vb) {
    if (w.live == VEC) {
        st_vec<O, VEC>(out + w.i0, apply_vec<F, T, O, NIN, VEC>(f, va, vb));
        return;
    }
#pragma unroll
    for (int j = 0; j < VEC; j++)
        if (j < w.live) {
            if constexpr (NIN == 2) out[w.i0 + j] = f(va.v[j], vb.v[j]);
            else out[w.i0 + j] = f(va.v[j]);
        }
}
template <class F, class T, class O, int NIN, int VEC>
__global__ void __launch_bounds__(kEwThreads) ew_dense_kernel(F f, const T* a, const T* b, O* out, EwDenseParams P) {
    after_previous_kernel();
    auto row_offsets = [&](uint32_t r, int& oa, int& ob) {
        oa = ob = 0;
        for (int d = P.nd - 2; d > 0; d--) {
            uint32_t x;
            P.div[d].divmod(r, r, x);
            oa += (int)x * P.st[1][d];
            if constexpr (NIN == 2) ob += (int)x * P.st[2][d];
        }
        if (P.nd > 1) {
            oa += (int)r * P.st[1][0];
            if constexpr (NIN == 2) ob += (int)r * P.st[2][0];
        }
    };
    const int sa = P.st[1][P.nd - 1], sb = NIN == 2 ? P.st[2][P.nd - 1] : 0;
    EwDensePlace w[kEwDenseUnroll];
    Vec<T, VEC> va[kEwDenseUnroll], vb[kEwDenseUnroll];
#pragma unroll
    for (int u = 0; u < kEwDenseUnroll; u++) {
        const uint64_t first = ((uint64_t)blockIdx.x * kEwDenseUnroll * kEwThreads + u * kEwThreads + threadIdx.x) * VEC;
        w[u].i0 = (uint32_t)first;
        w[u].live = first >= P.n ? 0 : (int)min((uint32_t)VEC, P.n - w[u].i0);
        if (!w[u].live) continue;
        uint32_t row, c;
        P.q_div.divmod(w[u].i0, row, c);
        int oa, ob, oa1 = 0, ob1 = 0;
        row_offsets(row, oa, ob);
        if (P.q >= VEC) {
            w[u].left = (int)min((uint32_t)VEC, P.q - c);
            if (w[u].left < w[u].live) row_offsets(row + 1, oa1, ob1);
            ew_dense_load<T, VEC>(a, P.kind[1], sa, w[u], oa + (int)c * sa, oa1 - w[u].left * sa, va[u]);
            if constexpr (NIN == 2) ew_dense_load<T, VEC>(b, P.kind[2], sb, w[u], ob + (int)c * sb, ob1 - w[u].left * sb, vb[u]);
        } else {
            w[u].left = VEC;
            // the flat inputs as above, the gathered ones (offset c * stride, whatever the stride) row by row
            if (P.kind[1] <= EWD_ELEMENT) ew_dense_load<T, VEC>(a, P.kind[1], 1, w[u], 0, 0, va[u]);
            if constexpr (NIN == 2)
                if (P.kind[2] <= EWD_ELEMENT) ew_dense_load<T, VEC>(b, P.kind[2], 1, w[u], 0, 0, vb[u]);
#pragma unroll
            for (int j = 0; j < VEC; j++) {
                if (j < w[u].live) {
                    if (P.kind[1] > EWD_ELEMENT) va[u].v[j] = a[oa + (int)c * sa];
                    if constexpr (NIN == 2)
                        if (P.kind[2] > EWD_ELEMENT) vb[u].v[j] = b[ob + (int)c * sb];
                    if (++c == P.q && j + 1 < w[u].live) {
                        c = 0;
                        row_offsets(++row, oa, ob);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int u = 0; u < kEwDenseUnroll; u++)
        if (w[u].live) ew_dense_store<F, T, O, NIN, VEC>(f, out, w[u], va[u], vb[u]);
}

// Two inputs, each either the output's own layout (vector loads) or constant along the innermost dim of at most three - a per-row or a per-channel
// operand whose rows are no whole vectors, the commonest call of the kernel above.  What bounds that one there is its instructions (loops over the
// dims, every element's own choice): here the place of a vector costs two divisions by multiplication, the row behind comes from
// the one before it without another, both values a vector can see are loaded whether or not its rows change inside it, and a thread has
// up to two vectors' loads in flight (ew_chan_units).  [256, 512, 7, 7] bf16 with a per-channel operand 4.3 us (8.1 by the kernel above), [8191, 1023] f32 with a per-row
// one 7.8 (10.7).
struct FastDiv31 {  // floor(n / d) for n < 2^31 and d >= 2: with 2^s < d <= 2^(s+1) and m = ceil(2^(32+s) / d), n (m d - 2^(32+s)) < 2^(32+s)
    uint32_t d, m, s;
    void init(uint32_t div) {
        d = div;
        for (s = 0; (2ull << s) < d; s++) {
        }
        m = (uint32_t)(((1ull << (32 + s)) + d - 1) / d);
    }
    __device__ __forceinline__ uint32_t div(uint32_t n) const { return __umulhi(n, m) >> s; }
};
struct EwChanParams {
    uint32_t n, q, channels;    // elements; extent of the innermost dim and of the middle one
    FastDiv31 q_div, channel_div;
    int vector[3];              // [1], [2]: the input has the output's layout
    int s_outer[3], s_channel[3];
    int units;                  // vectors a thread (ew_chan_units)
};
struct EwRepeatParams {
    uint32_t n, q;    // elements; extent of the innermost dim
    FastDiv31 q_div;
    int repeated[3];  // [1], [2]: the input is one row for all rows, else it has the output's layout
    int units;
};
// Two vectors a thread at most, one while that leaves an SM four blocks at most.  Compiled for four the kernels have 46 (f32) to 94 registers (16 bits) instead of 30 to
// 48: fewer blocks an SM, and below 150000 vectors most SMs had none.  Dense kernel / one / two / four, geometric mean and worst over layouts and rows of 92 and 1023,
// of the dense kernel's time: 33000 vectors f32 difference 0.81 0.84 0.93, worst 1.04; bf16 quotient 0.58 0.87 1.44, worst 1.60; i16 comparison 0.60 0.71 1.05, worst
// 1.19; 220000 bf16 quotient 0.84 0.87 1.26; 2400000 f32 difference 0.89 0.85 0.86, bf16 quotient 0.77 0.76 0.84, comparison 0.69 0.62 0.77.  One or two: worst 1.03.
constexpr int kEwChanUnroll = 2;
inline int ew_chan_units(uint64_t vecs) { return vecs <= 4 * (uint64_t)kEwThreads * sm_count() ? 1 : kEwChanUnroll; }
template <class F, class T, class O, int VEC>
__global__ void __launch_bounds__(kEwThreads) ew_chan_kernel(F f, const T* a, const T* b, O* out, EwChanParams P) {
    after_previous_kernel();
    constexpr int U = kEwChanUnroll;
    const uint32_t first = (blockIdx.x * P.units * kEwThreads + threadIdx.x) * VEC;
    Vec<T, VEC> va[U], vb[U];
    T xa[U][2], xb[U][2];
    int left[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        const uint32_t i0 = first + u * kEwThreads * VEC;
        if (u >= P.units || i0 >= P.n) continue;
        const uint32_t row = P.q_div.div(i0), outer = P.channel_div.div(row), channel = row - outer * P.channels;
        left[u] = (int)(P.q - (i0 - row * P.q));  // elements of the vector's first row from i0 on
        const bool wraps = channel + 1 == P.channels, ends = left[u] < VEC && i0 + left[u] < P.n;
        auto load = [&](const T* p, int k, Vec<T, VEC>& v, T(&x)[2]) {
            if (P.vector[k]) {
                if (i0 + VEC <= P.n) v = ld_vec<T, VEC>(p + i0);
                else
#pragma unroll
                    for (int j = 0; j < VEC; j++)
                        if (i0 + j < P.n) v.v[j] = p[i0 + j];
            } else {
                const int o0 = (int)outer * P.s_outer[k] + (int)channel * P.s_channel[k];
                const int o1 = wraps ? (int)(outer + 1) * P.s_outer[k] : o0 + P.s_channel[k];
                x[0] = p[o0];
                x[1] = p[ends ? o1 : o0];
            }
        };
        load(a, 1, va[u], xa[u]);
        load(b, 2, vb[u], xb[u]);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        const uint32_t i0 = first + u * kEwThreads * VEC;
        if (u >= P.units || i0 >= P.n) continue;
        auto spread = [&](int k, Vec<T, VEC>& v, const T(&x)[2]) {
            if (!P.vector[k])
#pragma unroll
                for (int j = 0; j < VEC; j++) v.v[j] = j < left[u] ? x[0] : x[1];
        };
        spread(1, va[u], xa[u]);
        spread(2, vb[u], xb[u]);
        if (i0 + VEC <= P.n) st_vec<O, VEC>(out + i0, apply_vec<F, T, O, 2, VEC>(f, va[u], vb[u]));
        else
#pragma unroll
            for (int j = 0; j < VEC; j++)
                if (i0 + j < P.n) out[i0 + j] = f(va[u].v[j], vb[u].v[j]);
    }
}

// Two inputs of ragged rows, each the output's own layout or the same row for all of them (a bias, a norm's weights): one division by multiplication a
// vector, the repeated row from L1 by elements, up to two vectors a thread.  [8191, 1023] f32 9.5 us (10.8 by the dense kernel), [4099, 1543] bf16 5.9 (7.0).  An
// instantiation of the kernel above for it would have the constants' registers too.
// SHIFTED, for rows of kEwRepeatLong and more: the repeated row's vectors from the two aligned words they lie in instead of by elements, which meet in L1's banks ([4099, 1543] bf16 6.1 us,
// 4.9 so, [2277, 5799] 10.5, 7.8; f32 [8191, 1023] 9.7, 8.9).  In shorter rows the vectors that wrap, which go by elements, are in too many warps ([30000, 197] bf16 5.2,
// 6.1), below two vectors a thread the way to the words is longer than what they save ([3, 100001] bf16 1.7, 2.0), and quotients and saturating sums of 16 bits have
// no registers for it ([5789, 3853] f32 28.1, 31.6; [12489, 523] i16 7.5, 8.4), nor comparisons, whose vectors are longer ([11611, 4195] f32 >= 37.5, 43.6; [16463, 637] f16 8.8, 9.5).
constexpr uint32_t kEwRepeatLong = 512;
template <class F>
struct EwShiftsRepeated : std::true_type {};
template <class T, class O>
struct EwShiftsRepeated<Binary<OpDiv, T, O>> : std::false_type {};
template <class F, class T, class O, int VEC, bool SHIFTED = false>
__global__ void __launch_bounds__(kEwThreads) ew_repeat_kernel(F f, const T* a, const T* b, O* out, EwRepeatParams P) {
    after_previous_kernel();
    constexpr int U = kEwChanUnroll;
    const uint32_t first = (blockIdx.x * P.units * kEwThreads + threadIdx.x) * VEC;
    Vec<T, VEC> va[U], vb[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        const uint32_t i0 = first + u * kEwThreads * VEC;
        if (u >= P.units || i0 >= P.n) continue;
        const uint32_t col = i0 - P.q_div.div(i0) * P.q;
        auto load = [&](const T* p, int repeated, Vec<T, VEC>& v) {
            if (repeated) {
                if (SHIFTED && col + VEC <= P.q) {
                    v = ld_vec_shifted<T, VEC>(p + col, (uint32_t)reinterpret_cast<uintptr_t>(p + col) & 15);
                } else {
#pragma unroll
                    for (int j = 0; j < VEC; j++) v.v[j] = p[col + j < P.q ? col + j : col + j - P.q];
                }
            } else if (i0 + VEC <= P.n) {
                v = ld_vec<T, VEC>(p + i0);
            } else {
#pragma unroll
                for (int j = 0; j < VEC; j++)
                    if (i0 + j < P.n) v.v[j] = p[i0 + j];
            }
        };
        load(a, P.repeated[1], va[u]);
        load(b, P.repeated[2], vb[u]);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        const uint32_t i0 = first + u * kEwThreads * VEC;
        if (u >= P.units) continue;
        if (i0 + VEC <= P.n) {
            st_vec<O, VEC>(out + i0, apply_vec<F, T, O, 2, VEC>(f, va[u], vb[u]));
        } else {
#pragma unroll
            for (int j = 0; j < VEC; j++)
                if (i0 + j < P.n) out[i0 + j] = f(va[u].v[j], vb[u].v[j]);
        }
    }
}

// ---------------------------------------------------------------------------------
// launcher
// ---------------------------------------------------------------------------------
// The dense-output kernel's parameters as those of the kernel of rows and channels; false when they are not of its form.
bool ew_fill_chan_params(const EwDenseParams& D, int vec, EwChanParams& P);
bool ew_fill_repeat_params(const EwDenseParams& D, int vec, EwRepeatParams& P);
// Fills the parameters for the dense-output kernel; false when the output is not dense from `out` on or not vector-aligned, or
// an offset does not fit 31 bits.
bool ew_fill_dense_params(const EwPlan& pl, size_t in_size, size_t out_size, const void* out, const void* a, const void* b, EwDenseParams& P);
void ew_fill_row_params(const EwPlan& pl, int vec, EwRowParams& P);
void ew_fill_tile_params(const EwPlan& pl, int tile, EwTileParams& P, uint32_t& blocks);
void ew_fill_gen_params(const EwPlan& pl, EwGenParams& P);

// Host side of the 2-byte tile kernel: one tensor map per operand (rows along the operand's strided dim, columns along
// its unit-stride dim, the one batch dim as the third coordinate).  Returns false - nothing launched - for layouts the
// maps cannot express (a stride-0 or negative row pitch, two or more batch dims, a pitch the encoder rejects); the
// caller then runs the general tile kernel.
template <class F, class T, class O, int NIN>
bool ew_launch_tile16(const EwPlan& pl, const EwTileParams& TP, uint32_t blocks, const F& f, const T* a, const T* b, O* out, cudaStream_t s) {
    if (TP.nd_batch > 1) return false;
    const uint64_t nb = blocks / ((uint64_t)TP.tiles_p * TP.tiles_q);
    const void* base[3] = {out, a, b};
    CUtensorMap maps[3];
    EwTile16Params P;
    P.tiles_q_div = TP.tiles_q_div;
    P.tiles_p_div = TP.tiles_p_div;
    for (int k = 0; k <= NIN; k++) {
        const bool tr = k != 0 && TP.transposed[k];
        const uint64_t rows = tr ? TP.Q : TP.P, cols = tr ? TP.P : TP.Q;
        const int64_t pitch = tr ? TP.st_q[k] : TP.st_p[k], unit = tr ? TP.st_p[k] : TP.st_q[k];
        const int64_t bs = TP.nd_batch ? TP.st_batch[k][0] : 0;
        if (unit != 1 || pitch <= 0 || bs < 0 || (k == 0 && nb > 1 && bs == 0)) return false;
        P.transposed[k] = tr ? 1 : 0;
        P.batched[k] = (nb > 1 && bs != 0) ? 1 : 0;
        if (!tc::make_map_3d(&maps[k], CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, base[k], rows, cols, nb, (uint64_t)bs, kEwT16, CU_TENSOR_MAP_SWIZZLE_128B, (uint64_t)pitch))
            return false;
    }
    if (NIN == 1) {
        maps[2] = maps[1];
        P.transposed[2] = P.batched[2] = 0;
    }
    launch_kernel(ew_tile16_kernel<F, T, O, NIN>, blocks, kEwThreads, (NIN + 1) * kEwT16Bytes + 1024, s, f, maps[1], maps[2], maps[0], P, tc::next_wait_report());
    return true;
}

template <class F, class T, class O, int NIN>
void ew_launch(const EwPlan& pl, const F& f, const T* a, const T* b, O* out, const char* where) {
    constexpr int VEC = 16 / sizeof(T);
    cudaStream_t s = ctx().stream;
    a += pl.off[1];
    if (NIN == 2) b += pl.off[2];
    out += pl.off[0];
    switch (pl.kind) {
        case EW_EMPTY:
            return;
        case EW_FLAT: {
            uint64_t chunk = (uint64_t)kEwThreads * VEC * kEwUnroll;
            uint64_t blocks = (pl.n + chunk - 1) / chunk;
            if (blocks > 0x7FFFFFFFull) {
                set_error(kErrUnsupported, 0, where);
                return;
            }
            if constexpr (F::kChecked) {
                // 16-bit division (approximate quotient + exact redo): 88 registers per thread leave few loads in flight, so
                // large operands are fed by bulk copies through shared memory instead
                const int sa = (int)pl.st[1][0], sb = NIN == 2 ? (int)pl.st[2][0] : 0;
                const int staged = (sa ? 1 : 0) + (sb ? 1 : 0);
                if (staged && pl.n / VEC >= 4096) {
                    launch_kernel(ew_flat_shift_staged_kernel<F, T, O, NIN, VEC>, (uint32_t)blocks, kEwThreads, (size_t)staged * kEwStageBytes, s, f, a, b, out, pl.n, 0, pl.n / VEC, sa, sb, 0, 0, 1, tc::next_wait_report());
                    break;
                }
            }
            const uint32_t full = ew_flat_full_blocks<VEC>(pl.n);
            const uint64_t piece = (uint64_t)kEwThreads * VEC, pieces = (pl.n - full * chunk + piece - 1) / piece;
            launch_kernel(ew_flat_kernel<F, T, O, NIN, VEC>, full + (uint32_t)pieces, kEwThreads, 0, s, f, a, b, out, pl.n, (int)pl.st[1][0], NIN == 2 ? (int)pl.st[2][0] : 0, full);
            break;
        }
        case EW_FLAT_SHIFT: {
            // head: elements until the output reaches the alignment of its vector store
            const uintptr_t oaddr = reinterpret_cast<uintptr_t>(out);
            const size_t oalign = VEC * sizeof(O);
            uint64_t head = ((oalign - oaddr % oalign) % oalign) / sizeof(O);
            if (head > pl.n) head = pl.n;
            const uint64_t body_vecs = (pl.n - head) / VEC;
            const int sa = (int)pl.st[1][0], sb = NIN == 2 ? (int)pl.st[2][0] : 0;
            const uint32_t sha = sa ? (uint32_t)(reinterpret_cast<uintptr_t>(a + head) % 16) : 0;
            const uint32_t shb = (NIN == 2 && sb) ? (uint32_t)(reinterpret_cast<uintptr_t>(b + head) % 16) : 0;
            uint64_t blocks = (body_vecs + (uint64_t)kEwThreads * kEwUnroll - 1) / ((uint64_t)kEwThreads * kEwUnroll);
            if (blocks == 0) blocks = 1;
            if (blocks > 0x7FFFFFFFull) {
                set_error(kErrUnsupported, 0, where);
                return;
            }
            const int staged = (sa && sha != 0 ? 1 : 0) + (NIN == 2 && sb && shb != 0 ? 1 : 0);
            if (staged && body_vecs >= 4096) {
                // large operands: the shifted ones go through shared memory, one bulk copy per block and operand
                launch_kernel(ew_flat_shift_staged_kernel<F, T, O, NIN, VEC>, (uint32_t)blocks, kEwThreads, (size_t)staged * kEwStageBytes, s, f, a, b, out, pl.n, head, body_vecs, sa, sb, sha, shb, 0, tc::next_wait_report());
                break;
            }
            launch_kernel(ew_flat_shift_kernel<F, T, O, NIN, VEC>, (uint32_t)blocks, kEwThreads, 0, s, f, a, b, out, pl.n, head, body_vecs, sa, sb, sha, shb);
            break;
        }
        case EW_ROW: {
            EwRowParams P;
            ew_fill_row_params(pl, VEC, P);
            uint64_t rows = P.total_vecs / P.qv;
            bool row_bcast = NIN == 1 && P.nd_outer == 1 && P.sq[1] == 1 && P.st[1][0] == 0 && P.st[0][0] == (int64_t)P.qv * VEC && rows >= 8;
            if constexpr (NIN == 1) {
                if (row_bcast) {
                    // enough blocks to fill the GPU, each storing a slab of rows
                    uint32_t want = (uint32_t)sm_count() * 8;
                    uint32_t gy = (want + P.chunks_per_row - 1) / P.chunks_per_row;
                    if (gy > rows) gy = (uint32_t)rows;
                    if (gy > 65535) gy = 65535;
                    uint32_t rpb = (uint32_t)((rows + gy - 1) / gy);
                    gy = (uint32_t)((rows + rpb - 1) / rpb);
                    if ((VEC * sizeof(O)) % 16 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0) {
                        const size_t stage = (size_t)kEwThreads * kEwUnroll * VEC * sizeof(O);
                        launch_kernel(ew_bcast_rows_bulk_kernel<F, T, O, VEC>, dim3(P.chunks_per_row, gy), kEwThreads, stage, s, f, a, out, P.qv, (uint32_t)rows, rpb);
                        break;
                    }
                    launch_kernel(ew_bcast_rows_kernel<F, T, O, VEC>, dim3(P.chunks_per_row, gy), kEwThreads, 0, s, f, a, out, P.qv, (uint32_t)rows, rpb);
                    break;
                }
            }
            if (P.qv >= (uint32_t)kEwThreads && rows * P.chunks_per_row < 0x7FFFFFFFull) {
                launch_kernel(ew_row_long_kernel<F, T, O, NIN, VEC>, (uint32_t)(rows * P.chunks_per_row), kEwThreads, 0, s, f, a, b, out, P);
            } else {
                uint32_t blocks = ceil_div_u32(P.total_vecs, kEwThreads * kEwUnroll);
                launch_kernel(ew_row_kernel<F, T, O, NIN, VEC>, blocks, kEwThreads, 0, s, f, a, b, out, P);
            }
            break;
        }
        case EW_TILE: {
            EwTileParams P;
            uint32_t blocks;
            ew_fill_tile_params(pl, EwTile<T>::kTile, P, blocks);
            int nslots = (P.transposed[1] ? 1 : 0) + (P.transposed[2] ? 1 : 0);
            size_t smem = (size_t)nslots * EwTile<T>::kBytes;
            if constexpr (sizeof(T) == 2 && sizeof(O) == 2) {
                if (pl.vec && ew_launch_tile16<F, T, O, NIN>(pl, P, blocks, f, a, b, out, s)) break;
            }
            if (pl.vec) launch_kernel(ew_tile_kernel<F, T, O, NIN, VEC>, blocks, kEwThreads, smem, s, f, a, b, out, P);
            else launch_kernel(ew_tile_kernel<F, T, O, NIN, 1>, blocks, kEwThreads, smem, s, f, a, b, out, P);
            break;
        }
        case EW_GENERIC:
        case EW_SERIAL: {
            EwDenseParams D;
            if (pl.kind == EW_GENERIC && ew_fill_dense_params(pl, sizeof(T), sizeof(O), out, a, b, D)) {
                const uint64_t vecs = (pl.n + VEC - 1) / VEC;
                if constexpr (NIN == 2 && VEC <= 8) {  // 16 elements a vector would take 145 registers
                    EwChanParams C;
                    EwRepeatParams Q;
                    C.units = Q.units = ew_chan_units(vecs);
                    const uint32_t blocks = (uint32_t)((vecs + kEwThreads * C.units - 1) / (kEwThreads * C.units));
                    if (ew_fill_chan_params(D, VEC, C)) {
                        launch_kernel(ew_chan_kernel<F, T, O, VEC>, blocks, kEwThreads, 0, s, f, a, b, out, C);
                        break;
                    }
                    if (ew_fill_repeat_params(D, VEC, Q)) {
                        constexpr bool kShifts = EwShiftsRepeated<F>::value && std::is_same<T, O>::value && (is_half_v<T> || std::is_same<T, f32>::value);
                        if (kShifts && Q.q >= kEwRepeatLong && Q.units > 1) launch_kernel(ew_repeat_kernel<F, T, O, VEC, kShifts>, blocks, kEwThreads, 0, s, f, a, b, out, Q);
                        else launch_kernel(ew_repeat_kernel<F, T, O, VEC>, blocks, kEwThreads, 0, s, f, a, b, out, Q);
                        break;
                    }
                }
                launch_kernel(ew_dense_kernel<F, T, O, NIN, VEC>, (uint32_t)((vecs + kEwThreads * kEwDenseUnroll - 1) / (kEwThreads * kEwDenseUnroll)), kEwThreads, 0, s, f, a, b, out, D);
                break;
            }
            EwGenParams P;
            ew_fill_gen_params(pl, P);
            if (pl.kind == EW_SERIAL) {
                launch_kernel(ew_generic_kernel<F, T, O, NIN>, 1, 1, 0, s, f, a, b, out, P);
            } else {
                uint64_t blocks = (pl.n + kEwThreads - 1) / kEwThreads;
                uint64_t cap = (uint64_t)sm_count() * 32;
                if (blocks > cap) blocks = cap;
                launch_kernel(ew_generic_kernel<F, T, O, NIN>, (uint32_t)blocks, kEwThreads, 0, s, f, a, b, out, P);
            }
            break;
        }
        default:
            set_error(kErrBadMetadata, 0, where);
            return;
    }
    check_launch(where);
}

// Entry points used by the C-ABI wrappers.  `meta` is the pointer the caller passed
// (device or host memory, or NULL for "contiguous, no offsets").
template <class Op, class T, class O>
void binary_entry(size_t n, size_t nd, const size_t* meta, const T* lhs, const T* rhs, O* out, bool inplace, const char* where) {
    const size_t* hm = meta ? resolve_metadata(meta, 3 * nd + 2) : nullptr;
    if (meta && !hm) return;
    EwPlan pl;
    ew_make_plan(pl, n, nd, hm, 2, inplace, sizeof(T), sizeof(O), out, lhs, rhs);
    ew_launch<Binary<Op, T, O>, T, O, 2>(pl, Binary<Op, T, O>(), lhs, rhs, out, where);
}
template <class Op, class T, class O>
void unary_entry(size_t n, size_t nd, const size_t* meta, const T* in, O* out, const char* where) {
    const size_t* hm = meta ? resolve_metadata(meta, 2 * nd + 1) : nullptr;
    if (meta && !hm) return;
    // The reference accepts input == NULL as "read from the output buffer"; that is
    // only meaningful when input and output have the same element type.
    if (!in) in = reinterpret_cast<const T*>(out);
    EwPlan pl;
    ew_make_plan(pl, n, nd, hm, 1, false, sizeof(T), sizeof(O), out, in, nullptr);
    ew_launch<Unary<Op, T, O>, T, O, 1>(pl, Unary<Op, T, O>(), in, (const T*)nullptr, out, where);
}
template <class Op, class T, class O>
void unary_const_entry(size_t n, size_t nd, const size_t* meta, const T* in, T c, O* out, const char* where) {
    const size_t* hm = meta ? resolve_metadata(meta, 2 * nd + 1) : nullptr;
    if (meta && !hm) return;
    if (!in) in = reinterpret_cast<const T*>(out);
    EwPlan pl;
    ew_make_plan(pl, n, nd, hm, 1, false, sizeof(T), sizeof(O), out, in, nullptr);
    UnaryConst<Op, T, O> f;
    f.c = c;
    ew_launch<UnaryConst<Op, T, O>, T, O, 1>(pl, f, in, (const T*)nullptr, out, where);
}

}  // namespace mx
