// conv2d im2col / col2im for one dtype (MX_T).
// Replaces the symbols declared in crates/maidenx_cuda/src/nn/conv.rs:6-36; semantics follow
// crates/maidenx_cpu/src/nn/conv.rs:13-149.
//   metadata = [B, C, H, W, kh, kw, out_h, out_w, pad_h, pad_w, stride_h, stride_w]
//   col layout [B][C, kh, kw][out_h, out_w]
//
// im2col: a block takes one or a few neighbouring (b, c) image planes.  They are read once into shared memory
// with coalesced loads; the kh*kw shifted copies of a plane (of all of them) are one contiguous run of the column buffer, written
// with 16-byte stores.  DRAM traffic is the algorithmic
// minimum (input once + col once) where the reference re-reads the input kh*kw times.
//
// col2im: gather formulation, one thread per output pixel (strides of 1 and small planes: the column planes of a few
// image planes staged in shared memory) summing the (at most kh*kw) col entries that map to it in the reference's (h_out, w_out) order and in the element type,
// so the result is bit-identical to the CPU backend, deterministic, needs no atomics and
// overwrites the output (the reference's CUDA kernel scatters with atomicAdd into a
// pre-zeroed buffer).  `num_els` bounds the readable part of col: entries at or beyond it
// are skipped, as the CPU backend does (conv.rs:135).
#include "abi_common.cuh"
#include "conv_s1.cuh"
#include "ops.cuh"

#ifndef MX_T
#error "compile with -DMX_T=<dtype suffix> -DMX_TCLASS=<class>"
#endif

namespace mx {

struct ConvParams {
    uint32_t B, C, H, W, KH, KW, OH, OW, PH, PW, SH, SW;
    uint64_t num_els;
    FastDiv ow_div, w_div;
};
// the kernels whose blocks take several planes
struct ConvPlanes : ConvParams {
    uint32_t planes, per_block;  // planes written, planes of one block
    FastDiv ohw_div, hw_div, kk_div, kw_div;
    ConvPlanes(const ConvParams& p, uint64_t n, uint32_t pb) : ConvParams(p), planes((uint32_t)n), per_block(pb) {
        ohw_div.init(OH * OW);
        hw_div.init(H * W);
        kk_div.init(KH * KW);
        kw_div.init(KW);
    }
};

constexpr int kConvThreads = 256;

// `count` consecutive elements into shared memory, as 16-byte vectors where the source allows, all of them in flight; complete behind the caller's barrier.
template <class T>
__device__ __forceinline__ void stage_run(T* dst, const T* src, uint32_t count) {
    constexpr uint32_t VEC = 16 / sizeof(T);
    uint32_t done = 0;
    if ((uintptr_t)src % 16 == 0) {
        done = count / VEC * VEC;
        const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst);
        for (uint32_t i = threadIdx.x * VEC; i < done; i += kConvThreads * VEC)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + i * (uint32_t)sizeof(T)), "l"(src + i) : "memory");
    }
    for (uint32_t i = done + threadIdx.x; i < count; i += kConvThreads) dst[i] = src[i];
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// The block's planes share one flat index over [plane, kh, kw, out_h, out_w], which repeats from group to group of `step` planes, the fewest that make whole vectors: a thread takes VEC
// consecutive columns of a group, finds where they come from once and writes them for all groups of the block.  So small maps (14 x 14: 49 vectors of a
// plane's 441) keep every thread busy and ragged ones (7 x 7) are written as vectors too.  Bound by HBM / L2 writes and by the reads from shared memory (vectors of neighbouring
// lanes meet in its banks): [32, 128, 14, 14] f32, 3 x 3: 7 us, 12 with the places found anew for every plane, 23 with one plane and one kernel offset at a time.
// GROUPS: the block has more than one group; with a single one places kept for later cost what they take ([39, 170, 25, 25] bf16 45.7 us, 48.4).
template <class T, int VEC, bool GROUPS>
__global__ void __launch_bounds__(kConvThreads) im2col_planes_kernel(const T* x, T* col, ConvPlanes P, uint32_t group) {
    after_previous_kernel();
    extern __shared__ __align__(16) unsigned char conv_smem[];
    T* img = reinterpret_cast<T*>(conv_smem);
    const uint32_t bc0 = blockIdx.x * P.per_block, np = min(P.per_block, P.planes - bc0);
    const uint32_t HW = P.H * P.W, OHW = P.OH * P.OW, KK = P.KH * P.KW;
    stage_run(img, x + (uint64_t)bc0 * HW, np * HW);
    __syncthreads();
    const T zero = zero_of<T>();
    const uint64_t base = (uint64_t)bc0 * KK * OHW;
    const uint32_t total = (uint32_t)min((uint64_t)np * KK * OHW, P.num_els - base);
    if constexpr (!GROUPS) {
        for (uint32_t e = threadIdx.x * VEC; e < total; e += kConvThreads * VEC) {
            uint32_t row, o, plane, kk, kh, kw, ho, wo;
            P.ohw_div.divmod(e, row, o);
            P.kk_div.divmod(row, plane, kk);
            P.kw_div.divmod(kk, kh, kw);
            P.ow_div.divmod(o, ho, wo);
            Vec<T, VEC> r;
#pragma unroll
            for (int j = 0; j < VEC; j++) {
                const int hi = (int)(ho * P.SH + kh) - (int)P.PH, wi = (int)(wo * P.SW + kw) - (int)P.PW;
                r.v[j] = (uint32_t)hi < P.H && (uint32_t)wi < P.W && plane < np ? img[plane * HW + hi * P.W + wi] : zero;
                if (++wo == P.OW) {
                    wo = 0;
                    if (++ho == P.OH) {
                        ho = 0;
                        if (++kw == P.KW) {
                            kw = 0;
                            if (++kh == P.KH) {
                                kh = 0;
                                plane++;
                            }
                        }
                    }
                }
            }
            if (e + VEC <= total) {
                *reinterpret_cast<Vec<T, VEC>*>(col + base + e) = r;
            } else {
#pragma unroll
                for (int j = 0; j < VEC; j++)
                    if (e + j < total) col[base + e + j] = r.v[j];
            }
        }
        return;
    }
    const uint32_t period = group * KK * OHW, hop = group * HW;
    for (uint32_t e0 = threadIdx.x * VEC; e0 < min(total, period); e0 += kConvThreads * VEC) {
        uint32_t row, o, plane, kk, kh, kw, ho, wo;
        P.ohw_div.divmod(e0, row, o);
        P.kk_div.divmod(row, plane, kk);
        P.kw_div.divmod(kk, kh, kw);
        P.ow_div.divmod(o, ho, wo);
        int at[VEC];  // the element's place in the group's planes, -1 in the padding
#pragma unroll
        for (int j = 0; j < VEC; j++) {
            const int hi = (int)(ho * P.SH + kh) - (int)P.PH, wi = (int)(wo * P.SW + kw) - (int)P.PW;
            at[j] = (uint32_t)hi < P.H && (uint32_t)wi < P.W ? (int)(plane * HW) + hi * (int)P.W + wi : -1;
            if (++wo == P.OW) {
                wo = 0;
                if (++ho == P.OH) {
                    ho = 0;
                    if (++kw == P.KW) {
                        kw = 0;
                        if (++kh == P.KH) {
                            kh = 0;
                            plane++;
                        }
                    }
                }
            }
        }
        const T* from = img;
#pragma unroll 2
        for (uint32_t e = e0; e < total; e += period, from += hop) {
            Vec<T, VEC> r;  // elements behind the last plane are read from the block's memory all the same, and not written
#pragma unroll
            for (int j = 0; j < VEC; j++) r.v[j] = at[j] < 0 ? zero : from[at[j]];
            if (e + VEC <= total) {
                *reinterpret_cast<Vec<T, VEC>*>(col + base + e) = r;
            } else {
#pragma unroll
                for (int j = 0; j < VEC; j++)
                    if (e + j < total) col[base + e + j] = r.v[j];
            }
        }
    }
}

// One block per plane, one kernel offset at a time.  Large maps keep its threads busy with less arithmetic per element than the flat
// index above takes (see planes_pay).  STAGED: the plane fits shared memory.
template <class T, int VEC, bool STAGED>
__global__ void __launch_bounds__(kConvThreads) im2col_kernel(const T* x, T* col, ConvParams P) {
    after_previous_kernel();
    extern __shared__ __align__(16) unsigned char conv_smem[];
    T* plane = reinterpret_cast<T*>(conv_smem);
    const uint64_t bc = blockIdx.x;  // b * C + c
    const uint32_t HW = P.H * P.W, OHW = P.OH * P.OW, KK = P.KH * P.KW;
    const T* src = x + bc * HW;
    if constexpr (STAGED) {
        for (uint32_t i = threadIdx.x; i < HW; i += kConvThreads) plane[i] = src[i];
        __syncthreads();
    }
    const T* img = STAGED ? plane : src;
    const T zero = zero_of<T>();
    const uint64_t out_base = bc * KK * OHW;
    const uint32_t nvec = (OHW + VEC - 1) / VEC;
    for (uint32_t kk = 0; kk < KK; kk++) {
        const uint32_t kh = kk / P.KW, kw = kk % P.KW;
        T* dst = col + out_base + (uint64_t)kk * OHW;
        const uint64_t dst_lin = out_base + (uint64_t)kk * OHW;
        for (uint32_t v = threadIdx.x; v < nvec; v += kConvThreads) {
            Vec<T, VEC> r;
            uint32_t o0 = v * VEC;
            uint32_t ho, wo;
            P.ow_div.divmod(o0, ho, wo);
#pragma unroll
            for (int j = 0; j < VEC; j++) {
                int hi = (int)(ho * P.SH + kh) - (int)P.PH, wi = (int)(wo * P.SW + kw) - (int)P.PW;
                bool in = hi >= 0 && hi < (int)P.H && wi >= 0 && wi < (int)P.W && o0 + j < OHW;
                r.v[j] = in ? img[hi * P.W + wi] : zero;
                if (++wo == P.OW) {
                    wo = 0;
                    ho++;
                }
            }
            if (VEC > 1 && o0 + VEC <= OHW && dst_lin + o0 + VEC <= P.num_els) {
                *reinterpret_cast<Vec<T, VEC>*>(dst + o0) = r;
            } else {
#pragma unroll
                for (int j = 0; j < VEC; j++)
                    if (o0 + j < OHW && dst_lin + o0 + j < P.num_els) dst[o0 + j] = r.v[j];
            }
        }
    }
}

template <class T>
__device__ __forceinline__ T conv_add(T a, T b) {
    if constexpr (is_half_v<T>) return from_f32<T>(to_f32(a) + to_f32(b));
    else return a + b;
}

// The same sums from shared memory: the KH * KW column planes of the block's image planes arrive in one contiguous run; a
// column entry crosses from L2 once instead of once per term.  Strides of 1: larger ones touch few entries more than once.  K > 0: a K x K kernel, whose terms are so many reads at
// distances known up front, each under a bit of the pixel's row or column; 0: any kernel, by the ranges of its output rows and columns.
// [32, 128, 14, 14] f32, 3 x 3: 8 us, 14 by the ranges, 16 from L2.
template <class T, int K>
__global__ void __launch_bounds__(kConvThreads) col2im_planes_kernel(const T* col, T* out, ConvPlanes P) {
    after_previous_kernel();
    extern __shared__ __align__(16) unsigned char conv_smem[];
    T* cols = reinterpret_cast<T*>(conv_smem);
    const uint32_t bc0 = blockIdx.x * P.per_block, np = min(P.per_block, P.planes - bc0);
    const uint32_t HW = P.H * P.W, OHW = P.OH * P.OW, KK = P.KH * P.KW;
    const uint64_t base = (uint64_t)bc0 * KK * OHW;
    const uint32_t want = np * KK * OHW, have = base >= P.num_els ? 0 : (uint32_t)min((uint64_t)want, P.num_els - base);
    stage_run(cols, col + base, have);
    for (uint32_t i = have + threadIdx.x; i < want; i += kConvThreads) cols[i] = zero_of<T>();  // adding +0 is skipping: the sum is never -0
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < np * HW; i += kConvThreads) {
        uint32_t plane, pix, h, w;
        P.hw_div.divmod(i, plane, pix);
        P.w_div.divmod(pix, h, w);
        const uint32_t hp = h + P.PH, wp = w + P.PW;
        const T* mine = cols + plane * KK * OHW;
        T sum = zero_of<T>();
        if constexpr (K > 0) {
            // output row hp - kh, output column wp - kw; ascending, as conv.rs:121-135 goes through them
            const T* top = mine + hp * P.OW + wp;
            const int kh_step = (int)(K * OHW) - (int)P.OW, kw_step = (int)OHW - 1;
            uint32_t cols_in = 0;
#pragma unroll
            for (int kw = 0; kw < K; kw++) cols_in |= (wp - kw < P.OW ? 1u : 0u) << kw;
#pragma unroll
            for (int kh = K - 1; kh >= 0; kh--) {
                if (hp - kh < P.OH) {
                    T v[K];
#pragma unroll
                    for (int kw = K - 1; kw >= 0; kw--)
                        if (cols_in >> kw & 1) v[kw] = top[kh * kh_step + kw * kw_step];
#pragma unroll
                    for (int kw = K - 1; kw >= 0; kw--)
                        if (cols_in >> kw & 1) sum = conv_add(sum, v[kw]);
                }
            }
        } else {
            // conv.rs:121-125
            const uint32_t hs = hp >= P.KH - 1 ? hp - (P.KH - 1) : 0, ws = wp >= P.KW - 1 ? wp - (P.KW - 1) : 0;
            const uint32_t he = min(hp + 1, P.OH), we = min(wp + 1, P.OW);
            for (uint32_t ho = hs; ho < he; ho++) {
                const uint32_t kh = hp - ho;
                if (kh >= P.KH) continue;
                const T* row = mine + kh * P.KW * OHW + ho * P.OW;
                for (uint32_t wo = ws; wo < we; wo++) {
                    const uint32_t kw = wp - wo;
                    if (kw < P.KW) sum = conv_add(sum, row[kw * OHW + wo]);
                }
            }
        }
        out[(uint64_t)bc0 * HW + i] = sum;
    }
}

template <class T>
__global__ void __launch_bounds__(kConvThreads) col2im_kernel(const T* col, T* out, ConvParams P) {
    after_previous_kernel();
    const uint64_t bc = blockIdx.y;  // b * C + c
    const uint32_t HW = P.H * P.W, OHW = P.OH * P.OW, KK = P.KH * P.KW;
    const uint32_t pix = blockIdx.x * kConvThreads + threadIdx.x;
    if (pix >= HW) return;
    uint32_t h, w;
    P.w_div.divmod(pix, h, w);
    const uint32_t hp = h + P.PH, wp = w + P.PW;
    // conv.rs:121-125
    const uint32_t hs0 = hp >= P.KH - 1 ? hp - (P.KH - 1) : 0, ws0 = wp >= P.KW - 1 ? wp - (P.KW - 1) : 0;
    const uint32_t hs = (hs0 + P.SH - 1) / P.SH, ws = (ws0 + P.SW - 1) / P.SW;
    const uint32_t he = min(hp / P.SH + 1, P.OH), we = min(wp / P.SW + 1, P.OW);
    const uint64_t base = bc * KK * OHW;
    T sum = zero_of<T>();
    for (uint32_t ho = hs; ho < he; ho++) {
        const uint32_t kh = hp - ho * P.SH;
        if (kh >= P.KH) continue;
        for (uint32_t wo = ws; wo < we; wo++) {
            const uint32_t kw = wp - wo * P.SW;
            if (kw >= P.KW) continue;
            uint64_t ci = base + (uint64_t)(kh * P.KW + kw) * OHW + ho * P.OW + wo;
            if (ci < P.num_els) sum = conv_add(sum, col[ci]);
        }
    }
    out[bc * HW + pix] = sum;
}

// The limit is the same in every call, whatever the call needs: with each call setting its own, a thread with small planes
// took back what a thread with large ones had just asked for, and the larger launch was refused.
constexpr int kConvSmemMost = 200 * 1024;
template <class K>
static void allow_shared_memory(K kernel, size_t bytes) {
    if (bytes > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kConvSmemMost);
}

static bool conv_params(const size_t* meta, size_t num_els, ConvParams& P, const char* where) {
    const size_t* m = resolve_metadata(meta, 12);
    if (!m) return false;
    for (int i = 0; i < 12; i++)
        if (m[i] > 0x7FFFFFFFull) {
            set_error(kErrUnsupported, 0, where);
            return false;
        }
    P.B = (uint32_t)m[0];
    P.C = (uint32_t)m[1];
    P.H = (uint32_t)m[2];
    P.W = (uint32_t)m[3];
    P.KH = (uint32_t)m[4];
    P.KW = (uint32_t)m[5];
    P.OH = (uint32_t)m[6];
    P.OW = (uint32_t)m[7];
    P.PH = (uint32_t)m[8];
    P.PW = (uint32_t)m[9];
    P.SH = (uint32_t)m[10];
    P.SW = (uint32_t)m[11];
    P.num_els = num_els;
    if (P.SH == 0 || P.SW == 0) {  // division by zero in the reference's index arithmetic
        set_error(kErrBadMetadata, 0, where);
        return false;
    }
    P.ow_div.init(P.OW);
    P.w_div.init(P.W);
    return true;
}

// Planes of one block of the staged kernels: up to 16 KB of them in shared memory (at least one), so that a block has a few
// vectors or pixels per thread, but not so many that fewer than eight blocks per SM (all its threads) are left;
// a multiple of `step`.  0: not even `step` planes fit `most` bytes.
static uint32_t planes_per_block(uint64_t planes, uint64_t plane_bytes, uint64_t step, uint64_t most) {
    if (step * plane_bytes > most) return 0;
    const uint64_t spread = planes / (8 * (uint64_t)sm_count());
    uint64_t n = spread;
    if (plane_bytes && n > 16 * 1024 / plane_bytes) n = 16 * 1024 / plane_bytes;  // an image of no pixels is all padding
    n = n / step * step;
    return (uint32_t)(n < step ? step : n);
}

// Bytes of planes that a block of the flat im2col takes at most: large planes leave a block or two on an SM, which 16-bit types (half the vectors to make) and maps of
// few outputs gain from all the same ([64, 3, 224, 224] 7 x 7 stride 2 bf16 230 -> 206 us, f32 248 -> 325; [32, 3, 224, 224] 16 x 16 stride 16 f32 98 -> 27).
static uint64_t planes_most(size_t es, uint64_t step, uint64_t ohw) {
    if (step > 1) return 40 * 1024;
    return es == 2 || ohw < kConvThreads ? kConvSmemMost : 48 * 1024;
}

// Planes of a group of the flat im2col, whose places a thread keeps from group to group: a multiple of `step` whose vectors nearly fill the block's
// threads, else the fewest that hold 48 vectors, twice at least in the block's `per_block` planes; else all of these, one group.  Many idle threads cost
// less than places found anew ([30000, 7, 7] f32 3 x 3, 441 vectors: 22.1 -> 10.1 us; [30000, 14, 14] bf16 1 x 1 stride 2, 49: 5.0 -> 4.0), but a few threads
// that write vector after vector cost more (groups of `step` planes, against one group: [30000, 5, 5] bf16 2 x 2, 8 vectors: 5.0 -> 9.2 us; [30000, 7, 7] 1 x 1
// stride 2, 2: 3.8 -> 9.0), and full threads are best ([30000, 7, 7] bf16 5 x 5 stride 2, 50 vectors: 15.2 us in one group, 13.3 in groups of 1, 8.3 of 5).
static uint32_t planes_per_group(uint32_t per_block, uint64_t step, uint64_t chunk, uint64_t vec) {
    const uint64_t vecs = step * chunk / vec;  // of `step` planes
    if (vecs == 0) return per_block;
    uint64_t n = std::max<uint64_t>(1, kConvThreads / vecs);
    if (8 * n * vecs < 7 * kConvThreads || 2 * n * step > per_block) n = vecs < 16 ? per_block : (48 + vecs - 1) / vecs;
    return 2 * n * step <= per_block ? (uint32_t)(n * step) : per_block;
}

// im2col: is the flat form faster than a block per plane and a kernel offset at a time?  It is where a plane's vectors are whole on
// their own (step 1: [16, 64, 30, 30] f32 3 x 3 15.1 -> 11.9 us, [64, 64, 29, 29] bf16 7 x 7 stride 4 113 -> 16.6).  Where `step` planes
// have to share a block to make whole vectors, enough blocks must be left ([4, 64, 27, 27] f32, 64 blocks: 6.3 -> 10.5 us; [16, 64, 21, 21],
// 256: 11.8 -> 9.0), fewer for maps that do not even fill a block's threads ([2, 64, 7, 7], 32 blocks: 4.0 -> 2.5 us).  8-byte
// types have two elements a vector, which large maps do not gain from ([32, 64, 35, 35] f64: 39.8 -> 43.4 us).
static bool planes_pay(size_t es, uint64_t step, uint64_t blocks, uint64_t ohw) {
    if (es == 8 && ohw > 1100) return false;
    return step == 1 || blocks >= 192 || (ohw < kConvThreads && blocks >= 32);
}

template <class T>
void im2col_entry(size_t num_els, const size_t* meta, const T* x, T* col, const char* where) {
    if (!meta || !x || !col) return;  // conv.rs:19-21
    ConvParams P;
    if (!conv_params(meta, num_els, P, where)) return;
    const uint64_t planes = (uint64_t)P.B * P.C;
    const uint64_t chunk = (uint64_t)P.KH * P.KW * P.OH * P.OW;
    if (planes == 0 || chunk == 0 || num_els == 0) return;
    // the reference walks col in chunks of C*kh*kw*oh*ow per batch; planes beyond num_els are never touched
    uint64_t planes_touched = (num_els + chunk - 1) / chunk;
    if (planes_touched > planes) planes_touched = planes;
    if (planes_touched > 0x7FFFFFFFull) {
        set_error(kErrUnsupported, 0, where);
        return;
    }
    constexpr int VEC = 16 / sizeof(T);
    const size_t plane_bytes = (size_t)P.H * P.W * sizeof(T);
    const bool vec = ((uintptr_t)col % 16 == 0) && ((uint64_t)P.OH * P.OW) % VEC == 0;
    cudaStream_t s = ctx().stream;
    const unsigned grid = (unsigned)planes_touched;
    // stride-1 fast path (conv_s1.cuh)
    if (P.SH == 1 && P.SW == 1 && vec && P.OW % VEC == 0 && num_els == planes * chunk && (int)P.KW - 1 <= VEC &&
        (uint64_t)P.OW + P.KW == (uint64_t)P.W + 2 * P.PW + 1 && (uint64_t)P.OH + P.KH == (uint64_t)P.H + 2 * P.PH + 1) {
        ConvS1Params Q;
        Q.H = P.H; Q.W = P.W; Q.KH = P.KH; Q.OH = P.OH; Q.OW = P.OW; Q.PH = P.PH; Q.PW = P.PW;
        Q.owv = P.OW / VEC;
        uint32_t need = (Q.owv + 1) * VEC, wide = (P.W + 2 * P.PW + VEC - 1) / VEC * VEC;
        Q.pitch = need > wide ? need : wide;
        Q.num_els = num_els;
        const size_t smem = (size_t)(P.H + 2 * P.PH) * Q.pitch * sizeof(T);
        auto go = [&](auto kernel) {
            allow_shared_memory(kernel, smem);
            launch_kernel(kernel, grid, kConvS1Threads, smem, s, x, col, Q);
            check_launch(where);
        };
        if (smem <= kConvSmemMost) {
            switch (P.KW) {
                case 1: go(im2col_s1_kernel<T, VEC, 1>); return;
                case 3: if (VEC >= 2) { go(im2col_s1_kernel<T, VEC, 3>); return; } break;
                case 5: if (VEC >= 4) { go(im2col_s1_kernel<T, VEC, 5>); return; } break;
                case 7: if (VEC >= 8) { go(im2col_s1_kernel<T, VEC, 7>); return; } break;
                default: break;
            }
        }
    }
    // a block's columns start on a vector boundary when its planes' chunks add up to whole vectors
    uint64_t step = 1;
    while (step < VEC && (chunk * step) % VEC != 0) step *= 2;
    const uint64_t ohw = (uint64_t)P.OH * P.OW;
    uint32_t pb = (uintptr_t)col % 16 == 0 ? planes_per_block(planes_touched, plane_bytes, step, planes_most(sizeof(T), step, ohw)) : 0;
    // four groups share their places where two blocks an SM are left ([32, 128, 14, 14] bf16, a group of two planes: 10.0 us with one group a block)
    if (pb && pb < 4 * step && 4 * step * plane_bytes <= 16 * 1024 && planes_touched >= 4 * step * 2 * (uint64_t)sm_count()) pb = (uint32_t)(4 * step);
    if (pb && pb * chunk < 0x7FFFFFFFull && planes_pay(sizeof(T), step, (planes_touched + pb - 1) / pb, ohw)) {
        const uint32_t group = planes_per_group(pb, step, chunk, VEC);
        const auto kernel = pb > group ? im2col_planes_kernel<T, VEC, true> : im2col_planes_kernel<T, VEC, false>;
        allow_shared_memory(kernel, pb * plane_bytes);
        launch_kernel(kernel, (unsigned)((planes_touched + pb - 1) / pb), kConvThreads, pb * plane_bytes, s, x, col, ConvPlanes(P, planes_touched, pb), group);
    } else if (plane_bytes <= kConvSmemMost) {
        auto launch = [&](auto kernel) {
            allow_shared_memory(kernel, plane_bytes);
            launch_kernel(kernel, grid, kConvThreads, plane_bytes, s, x, col, P);
        };
        if (vec) launch(im2col_kernel<T, VEC, true>);
        else launch(im2col_kernel<T, 1, true>);
    } else {
        if (vec) launch_kernel(im2col_kernel<T, VEC, false>, grid, kConvThreads, 0, s, x, col, P);
        else launch_kernel(im2col_kernel<T, 1, false>, grid, kConvThreads, 0, s, x, col, P);
    }
    check_launch(where);
}

template <class T>
void col2im_entry(size_t num_els, const size_t* meta, const T* col, T* out, const char* where) {
    if (!meta || !col || !out) return;  // conv.rs:90-92
    ConvParams P;
    if (!conv_params(meta, num_els, P, where)) return;
    const uint64_t planes = (uint64_t)P.B * P.C, HW = (uint64_t)P.H * P.W;
    if (planes == 0 || HW == 0) return;
    if (planes > 65535ull * 65535ull || P.KH == 0 || P.KW == 0) {
        set_error(kErrUnsupported, 0, where);
        return;
    }
    cudaStream_t s = ctx().stream;
    // stride-1 fast path (conv_s1.cuh)
    {
        constexpr int VEC = 16 / sizeof(T);
        const int kw = (int)P.KW, pw = (int)P.PW;
        const bool shape_ok = P.SH == 1 && P.SW == 1 && P.W % VEC == 0 && P.OW % VEC == 0 && num_els % VEC == 0 &&
                              ((uintptr_t)col | (uintptr_t)out) % 16 == 0 && planes <= 65535 && pw < VEC && kw - 1 - pw < VEC && kw - 1 - pw >= 0 &&
                              (uint64_t)P.OW + P.KW == (uint64_t)P.W + 2 * P.PW + 1 && (uint64_t)P.OH + P.KH == (uint64_t)P.H + 2 * P.PH + 1;
        if (shape_ok) {
            ConvS1Params Q;
            Q.H = P.H; Q.W = P.W; Q.KH = P.KH; Q.OH = P.OH; Q.OW = P.OW; Q.PH = P.PH; Q.PW = P.PW;
            Q.pitch = 0;
            Q.owv = P.OW / VEC;
            Q.num_els = num_els;
            const uint32_t items = P.H * (P.W / VEC);
            dim3 grid((items + kConvS1Threads - 1) / kConvS1Threads, (unsigned)planes);
            // every plane readable, 16-byte-multiple planes, at least two blocks' worth of shared memory per SM: staged form
            const uint64_t plane_elems = (uint64_t)P.KH * P.KW * P.OH * P.OW;
            const size_t stage_bytes = (size_t)plane_elems * sizeof(T);
            if (num_els >= planes * plane_elems && stage_bytes % 16 == 0 && stage_bytes <= 112 * 1024 && plane_elems < (1ull << 30)) {
                auto go = [&](auto kernel) {
                    allow_shared_memory(kernel, stage_bytes);
                    launch_kernel(kernel, (unsigned)planes, kConvS1Threads, stage_bytes, s, col, out, Q, tc::next_wait_report());
                    check_launch(where);
                };
                if (kw == 1 && pw == 0) { go(col2im_s1_staged_kernel<T, VEC, 1, 0>); return; }
                if (kw == 3 && pw == 1) { go(col2im_s1_staged_kernel<T, VEC, 3, 1>); return; }
                if (kw == 3 && pw == 0 && VEC > 2) { go(col2im_s1_staged_kernel<T, VEC, 3, 0>); return; }
                if (kw == 5 && pw == 2 && VEC > 2) { go(col2im_s1_staged_kernel<T, VEC, 5, 2>); return; }
                if (kw == 7 && pw == 3 && VEC > 3) { go(col2im_s1_staged_kernel<T, VEC, 7, 3>); return; }
            }
            bool done = true;
            if (kw == 1 && pw == 0) launch_kernel(col2im_s1_kernel<T, VEC, 1, 0>, grid, kConvS1Threads, 0, s, col, out, Q);
            else if (kw == 3 && pw == 1) launch_kernel(col2im_s1_kernel<T, VEC, 3, 1>, grid, kConvS1Threads, 0, s, col, out, Q);
            else if (kw == 3 && pw == 0 && VEC > 2) launch_kernel(col2im_s1_kernel<T, VEC, 3, 0>, grid, kConvS1Threads, 0, s, col, out, Q);
            else if (kw == 5 && pw == 2 && VEC > 2) launch_kernel(col2im_s1_kernel<T, VEC, 5, 2>, grid, kConvS1Threads, 0, s, col, out, Q);
            else if (kw == 7 && pw == 3 && VEC > 3) launch_kernel(col2im_s1_kernel<T, VEC, 7, 3>, grid, kConvS1Threads, 0, s, col, out, Q);
            else done = false;
            if (done) {
                check_launch(where);
                return;
            }
        }
    }
    // Staged planes: strides of 1, column planes of at most 48 KB (four blocks on an SM, so that one loads while others sum: [16, 64, 50, 50]
    // f32, 90 KB: 51 -> 65 us; bf16, 45 KB: 40 -> 38), pixels for half of a block's threads, and where a map has more pixels than a block
    // threads, blocks enough for the whole chip ([32, 64, 35, 35] f32: 48 -> 41 us, [1, 64, 35, 35], 64 blocks: 4.2 -> 8.4), and for 8-byte types
    // one term a pixel ([64, 64, 33, 33] f64: 1 x 1 29.1 -> 23.6 us; [16, 64, 21, 21] 3 x 3 10.2 -> 11.4).
    const uint64_t col_plane = (uint64_t)P.KH * P.KW * P.OH * P.OW;
    const uint32_t pb = P.SH == 1 && P.SW == 1 && planes <= 0x7FFFFFFFull && col_plane && HW < 0x7FFFFFFFull ? planes_per_block(planes, col_plane * sizeof(T), 1, 48 * 1024) : 0;
    if (pb && pb * HW < 0x7FFFFFFFull && pb * HW >= kConvThreads / 2 && (HW <= kConvThreads || ((planes + pb - 1) / pb >= 512 && (sizeof(T) < 8 || P.KH * P.KW == 1)))) {
        // Terms at fixed distances (by the ranges / so, us): 3 x 3, [300, 100, 14, 14] f32 94 / 42, and 5 x 5 in rows of an even length, [300, 100, 14, 14] bf16 181 / 144; odd ones, [300, 100, 13, 13] bf16
        // 190 / 220, and the 49 terms of 7 x 7, [300, 100, 7, 7] bf16 86 / 184, gain nothing from it.  And where at least half of a pixel's terms lie inside the columns' planes; the ranges skip the others (7 x 7
        // without padding [52, 209, 48, 8] bf16 95 / 251).
        const bool inside = P.KH == P.KW && 2 * (uint64_t)P.OH * P.OW >= HW;
        const auto kernel = inside && P.KH == 3 ? col2im_planes_kernel<T, 3> : inside && P.KH == 5 && P.W % 2 == 0 ? col2im_planes_kernel<T, 5> : col2im_planes_kernel<T, 0>;
        launch_kernel(kernel, (unsigned)((planes + pb - 1) / pb), kConvThreads, pb * col_plane * sizeof(T), s, col, out, ConvPlanes(P, planes, pb));
        check_launch(where);
        return;
    }
    // grid.y carries the plane index; fold very large plane counts into several launches
    const unsigned gx = (unsigned)((HW + kConvThreads - 1) / kConvThreads);
    for (uint64_t p0 = 0; p0 < planes; p0 += 65535) {
        uint64_t cnt = planes - p0 < 65535 ? planes - p0 : 65535;
        ConvParams Q = P;
        // shift the views instead of the plane index: col entries of plane p start at p*KK*OHW
        const uint64_t col_shift = p0 * P.KH * P.KW * P.OH * P.OW;
        Q.num_els = num_els > col_shift ? num_els - col_shift : 0;
        launch_kernel(col2im_kernel<T>, dim3(gx, (unsigned)cnt), kConvThreads, 0, s, col + col_shift, out + p0 * HW, Q);
    }
    check_launch(where);
}

}  // namespace mx

#define DEF_CONV_(T)                                                                                          \
    void cuda_conv2d_im2col_##T(size_t n, const size_t* m, const mx_##T* i, mx_##T* o) {                      \
        mx::im2col_entry<mx_##T>(n, m, i, o, "cuda_conv2d_im2col_" #T);                                       \
    }                                                                                                         \
    void cuda_conv2d_col2im_##T(size_t n, const size_t* m, const mx_##T* i, mx_##T* o) {                      \
        mx::col2im_entry<mx_##T>(n, m, i, o, "cuda_conv2d_col2im_" #T);                                       \
    }
#define DEF_CONV(T) DEF_CONV_(T)

extern "C" {
DEF_CONV(MX_T)
}
