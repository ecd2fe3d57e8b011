// Tensor-core path for f32 matmul on sm_100a: tcgen05.mma kind::tf32 with split operands, so the
// product keeps f32-level accuracy although the tensor core multiplies 11-bit significands.
//
// Every f32 operand element x is used as two tf32 values
//     big   = x with the low 13 significand bits dropped (what the tensor core reads from the raw f32 bits),
//     small = x - big   (exact in f32; its own low bits are again dropped by the tensor core),
// and each k-step multiplies
//     a_small * b_big  +  a_big * b_small  +  a_big * b_big
// by three MMAs into one TMEM accumulator, or (long reductions, WIDE) by two: a_big by [b_big | b_small], which lie behind one another, into an
// accumulator of twice the columns, and a_small * b_big into its second half; the halves meet in the epilogue's registers.
// The dropped term a_small * b_small and the truncation of `small` are each below 2^-21 of |a * b|, so a dot
// product agrees with f32 arithmetic to a few 1e-7 relative to sum |a_k * b_k| (the stated f32 matmul tolerance is
// 1e-4).
//
// Two-level accumulation.  The tensor core adds each instruction's products into the f32 accumulator with
// truncation, which pulls a long running sum towards zero by about half an ulp per instruction (measured:
// -6e-6 relative after 147 instructions); over K = 8192 that would eat the whole 1e-4 budget.  So the TMEM
// accumulator only ever holds the sum of a few k-blocks: the epilogue warps drain it after every chunk and keep the
// running total in registers, added with round-to-nearest, while the tensor core fills the other accumulator.  The pull
// towards zero is then bounded by the chunk length whatever K is.  Two lengths: CHUNK_FAST k-blocks (128 values of K, error
// 1e-6 of the result), and one k-block for the ragged products, which the CUDA cores would compute: 2.2e-7 at K = 192, where these
// begin (CUDA cores 2.5e-7; below that K they are the more exact), 3e-7 at K = 4096 (1.1e-6); a drain per k-block no longer hides behind the tensor work (conv products [256 x 1152] . [1152 x 196]: 40 us
// with the long chunk, 58 with the short one).  In a chunk of one the eight products with a small factor come first, so that they are summed while the accumulator is still 2^-11 of the result; longer chunks interleave them.
//
// One persistent CTA per SM, 320 threads in four roles:
//   warp 0      TMA producer: raw f32 A [128 x 32] and B [BN x 32] k-blocks (128-byte swizzle rows of 32 floats)
//               into a ring of stages;
//   warps 6-9   splitter: when a stage has landed, read the raw tiles and write the `small` tiles beside them
//               (element-wise, so the swizzled placement carries over unchanged), then hand the stage to
//   warp 1      the MMA issuer: 4 k-steps x 3 (wide: 2) tcgen05.mma (M128, N up to BN, wide 2 BN, K8) per k-block into one of two TMEM
//               accumulators, switching accumulator every chunk_kb k-blocks; commits the stage back to the
//               producer and each finished chunk to
//   warps 2-5   the epilogue: per chunk tcgen05.ld of the warp's 32 rows x BN columns, added into BN registers per
//               thread; after the tile's last chunk the totals go through a swizzled 4 KB staging tile to TMA stores.
// Operands may be K-major ([MN, K] row-major) or MN-major ([K, MN] row-major, loaded as [32 K-rows x 32 MN] boxes),
// which covers x . W^T, g . W and x^T . g without transposed copies.  Clusters only for the slices of one product; no multicast.
// Infinities and NaNs, for which the split has no form, are found in the totals and their tiles computed again (redo_tile).
// Every mbarrier wait is bounded (see tc_ptx.cuh); on expiry all roles fall through to the common exit.
#include <cuda.h>

#include <atomic>
#include <algorithm>
#include <mutex>
#include <unordered_map>

#include "matmul_tc.cuh"
#include "tc_cluster.cuh"

namespace mx {

using namespace tc;

namespace {

constexpr int BM = 128, BN = 128, BK = 32;     // CTA tile; BK * 4 bytes = one 128-byte swizzle row
constexpr int UMMA_K = 8;                      // tf32: 32 bytes of K per instruction
constexpr int STAGES = 3, MAX_STAGES = 4;      // of 128- and of 64-column tiles
constexpr int A_TILE = BM * BK * 4;            // 16 KB
constexpr int B_TILE = BN * BK * 4;
constexpr int STAGE_BYTES = 2 * (A_TILE + B_TILE);  // [A raw | A small | B raw | B small] of a 128-column tile
constexpr int EPI_WARPS = 4, SPLIT_WARPS = 4;
constexpr int EPI_CHUNK_COLS = 32;             // 32 f32 = 128 bytes per staged row
constexpr int EPI_STAGE_BYTES = 32 * EPI_CHUNK_COLS * 4;  // 4 KB per warp per buffer
constexpr int THREADS = 32 * (2 + EPI_WARPS + SPLIT_WARPS);
constexpr int TMEM_COLS = 4 * BN;              // two f32 accumulators, each [big x big | products with a small factor] (WIDE)
constexpr int GROUP_M = 16;
constexpr int CHUNK_FAST = 4;
constexpr int MN_CHUNK_BYTES = BK * 128;       // one [32 K-rows x 32 MN-elements] box
constexpr int REDO_BITS = 2048;

static_assert(TMEM_COLS == 256 || TMEM_COLS == 512, "TMEM allocations are powers of two");
static_assert(A_TILE % (16 * 32 * SPLIT_WARPS) == 0 && B_TILE / 2 % (16 * 32 * SPLIT_WARPS) == 0, "the splitter moves 16 bytes per thread and step");

struct Smem {
    static constexpr int stages = 0;
    static constexpr int epi = stages + STAGES * STAGE_BYTES;
    static constexpr int bars = epi + EPI_WARPS * 2 * EPI_STAGE_BYTES;
    static constexpr int redo = bars + 256;  // one bit per tile of this CTA (number modulo REDO_BITS), then whether any is set: see redo_tile
    static constexpr int total = redo + REDO_BITS / 8 + 16;
};
constexpr int SMEM_BYTES = Smem::total + 1024;  // slack for the 1024-byte alignment
static_assert(SMEM_BYTES <= 232448, "shared memory per CTA");

__host__ __device__ constexpr uint32_t make_idesc_tf32(bool a_mn_major, bool b_mn_major, int bn) {
    uint32_t d = 0;
    d |= 1u << 4;                               // D format: f32
    d |= 2u << 7;                               // A format: tf32
    d |= 2u << 10;                              // B format: tf32
    d |= (a_mn_major ? 1u : 0u) << 15;
    d |= (b_mn_major ? 1u : 0u) << 16;
    d |= (uint32_t)(bn >> 3) << 17;
    d |= (uint32_t)(BM >> 4) << 24;
    return d;
}

struct Params {
    int tiles_m, tiles_n, num_tiles, num_kb;
    int tiles_per_batch;       // tiles_m * tiles_n; num_tiles = batch * tiles_per_batch
    int a_batched, b_batched;  // 0: the operand is one matrix shared by every batch (third TMA coordinate stays 0)
    int a_mn, b_mn;
    int M, N;
    int chunk_kb;   // k-blocks summed inside TMEM before the registers take over
    int bn;         // columns of an output tile: 64 or 128
    int stages;     // of the ring
    int raw_bytes;  // what TMA delivers per stage: A and bn rows of B
    int split_kb;   // > 0: split-K; batch s of the launch reduces the k-blocks [s * split_kb, (s + 1) * split_kb) of one product
    int kb_per_z;   // > 0: the reduction runs over the operands' batches too: k-block i is block i % kb_per_z of batch i / kb_per_z
    int d_plain;    // != 0: the output's rows (or base) are not 16-byte multiples: the epilogue warps write them to `out` themselves
    // The operands and the output as plain memory, for redo_tile: element (row, k) of batch z at z * bs + row * rs + k * ks.
    const float *a, *b;
    int64_t a_bs, a_rs, a_ks, b_bs, b_rs, b_ks;
    int K, zs;      // zs: batches of the operands (kb_per_z > 0)
    float* out;     // D or the split-K partial results, rows `out_ld` elements apart
    int64_t out_ld;
    // > 0: the K slices of an output tile are the CTAs of one cluster; each leaves its partial result in its own shared memory and adds the
    // rows that fall to it over all of them, in slice order (the sums of the form with a second launch, bit for bit)
    int cluster;
    int vec_out;    // cluster: the rows of `out` may be written by 16-byte vectors
    Gate gate;
};

__device__ __forceinline__ void tile_coords(int tile, const Params& p, int& tm, int& tn, int& tb) {
    tb = tile / p.tiles_per_batch;
    tile -= tb * p.tiles_per_batch;
    const int group_size = GROUP_M * p.tiles_n;
    const int group = tile / group_size;
    const int first_m = group * GROUP_M;
    const int rows = min(GROUP_M, p.tiles_m - first_m);
    const int in_group = tile - group * group_size;
    tm = first_m + in_group % rows;
    tn = in_group / rows;
}

// small = x - (x with its low 13 bits cleared), itself rounded to the 11 significant bits the tensor core will read
// (rounding here instead of letting the hardware truncate keeps the error of the split unbiased); infinities and
// NaNs keep all their weight in `big`.
__device__ __forceinline__ uint32_t small_part(uint32_t bits) {
    const float x = __uint_as_float(bits);
    const float big = __uint_as_float(bits & 0xFFFFE000u);
    const uint32_t s = (__float_as_uint(x - big) + 0x1000u) & 0xFFFFE000u;
    return (bits & 0x7F800000u) == 0x7F800000u ? 0u : s;
}

// Where a CTA of a cluster keeps its partial result: behind what redo_tile stages; a row is 16 bytes longer than 128 floats, so that the threads of a
// warp, a row each, store to different banks.
constexpr int PART_OFF = 64 * 1024, PART_LD = BN + 4;
static_assert(PART_OFF + BM * PART_LD * 4 <= STAGES * STAGE_BYTES && 2 * BK * (BM + 4) * 4 <= PART_OFF, "partial result inside the ring");

// A tile whose result is not finite, again and in f32 arithmetic: the split has no form for infinities (inf times the zero `small` of
// an operand that tf32 holds exactly is NaN) and the tensor core reads a NaN whose payload sits in the low bits as one.  An
// infinity or NaN among the operands always leaves a non-finite sum here, whatever becomes of it, so the epilogue's look at its totals
// finds every such tile at the cost of one FMA per output, and finite operands cost nothing else (products of K = 64: 4 to 7 %; of
// K = 1024 and more: none).  k ascending with separate multiply and add, as on the CUDA cores.  All threads of the block; `stage` is the operand ring, which nothing uses any more.
template <bool INTO_PART>  // into the partial result of a CTA of a cluster
__device__ __forceinline__ void redo_tile(const Params& p, int bn, int tm, int tn, int tb, float* stage) {
    constexpr int LD = BM + 4, T = 16;  // 16 x 16 threads, rows ty + 16 i, columns tx + 16 j
    float *xs = stage, *ys = stage + BK * LD;  // [k][row], [k][column]
    const int tx = threadIdx.x % T, ty = threadIdx.x / T;
    float acc[BM / T][BN / T];
#pragma unroll
    for (int i = 0; i < BM / T; i++)
#pragma unroll
        for (int j = 0; j < BN / T; j++) acc[i][j] = 0.0f;
    for (int kb = 0; kb < p.num_kb; kb++) {
        int block = tb * p.split_kb + kb, za = p.a_batched ? tb : 0, zb = p.b_batched ? tb : 0;
        if (p.kb_per_z) {
            za = zb = block / p.kb_per_z;
            block -= za * p.kb_per_z;
            if (za >= p.zs) break;  // the last slice runs past the last batch
        }
        const int k0 = block * BK;
        if (k0 >= p.K) break;
        for (int e = threadIdx.x; e < BM * BK; e += THREADS) {
            const int k = p.a_mn ? e / BM : e % BK, r = p.a_mn ? e % BM : e / BK;
            xs[k * LD + r] = k0 + k < p.K && tm * BM + r < p.M ? p.a[za * p.a_bs + (tm * BM + r) * p.a_rs + (k0 + k) * p.a_ks] : 0.0f;
        }
        for (int e = threadIdx.x; e < BN * BK; e += THREADS) {
            const int k = p.b_mn ? e / BN : e % BK, c = p.b_mn ? e % BN : e / BK;
            ys[k * LD + c] = c < bn && k0 + k < p.K && tn * bn + c < p.N ? p.b[zb * p.b_bs + (tn * bn + c) * p.b_rs + (k0 + k) * p.b_ks] : 0.0f;
        }
        __syncthreads();
        if (ty < T) {
            for (int k = 0; k < BK; k++) {
                float x[BM / T], y[BN / T];
#pragma unroll
                for (int i = 0; i < BM / T; i++) x[i] = xs[k * LD + ty + T * i];
#pragma unroll
                for (int j = 0; j < BN / T; j++) y[j] = ys[k * LD + tx + T * j];
#pragma unroll
                for (int i = 0; i < BM / T; i++)
#pragma unroll
                    for (int j = 0; j < BN / T; j++) acc[i][j] = acc[i][j] + x[i] * y[j];
            }
        }
        __syncthreads();
    }
    if (ty >= T) return;
#pragma unroll
    for (int i = 0; i < BM / T; i++) {
        const int row = tm * BM + ty + T * i;
#pragma unroll
        for (int j = 0; j < BN / T; j++) {
            const int c = tx + T * j;
            if (row >= p.M || c >= bn || tn * bn + c >= p.N) continue;
            if constexpr (INTO_PART) stage[PART_OFF / 4 + (ty + T * i) * PART_LD + c] = acc[i][j];
            else p.out[((int64_t)tb * p.M + row) * p.out_ld + tn * bn + c] = acc[i][j];
        }
    }
}

// BN_T = 128: the form of 128-column tiles, long chunks and tensor stores, all known to the compiler; 0: everything from the
// parameters.  The difference is the splitter's: with the distance between a raw and its small tile a constant, its loads run
// ahead of its stores (8192 x 4096 x 4096: 164 TFLOP/s, 148 in batches of four).
// FORM: what the slices and the parts of B take is compiled in.  As a parameter the wide form cost the others' epilogue registers (24 bytes spilled, 40 with
// it) and time where a tile is little else: 165 x (8 x 4008 x 8) 75.8 us, 88.9.
enum Form { PLAIN = 0, WIDE = 1, CLUSTERED = 2 };  // WIDE: see kWideLeast; CLUSTERED: Params::cluster
template <int BN_T, int FORM = PLAIN>
__global__ void __launch_bounds__(THREADS, 1)
tc_gemm_f32_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_d,
                   Params p, int* err, int tag) {
    if (p.gate.word) {  // behind a product in pairs: almost always shut
        after_previous_kernel();
        if (p.gate.shut()) return;
    }
    extern __shared__ unsigned char tcf_smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)tcf_smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t smem_base = smem_u32(smem);
    const uint32_t bar_base = smem_base + Smem::bars;
    // barrier slots (8 bytes each): full[MAX_STAGES], split[MAX_STAGES], empty[MAX_STAGES], tmem_full[2], tmem_empty[2]; then the TMEM base word
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto split_bar = [&](int s) { return bar_base + 8u * (MAX_STAGES + s); };
    auto empty_bar = [&](int s) { return bar_base + 8u * (2 * MAX_STAGES + s); };
    auto tfull_bar = [&](int a) { return bar_base + 8u * (3 * MAX_STAGES + a); };
    auto tempty_bar = [&](int a) { return bar_base + 8u * (3 * MAX_STAGES + 2 + a); };
    volatile uint32_t* tmem_base_slot = reinterpret_cast<volatile uint32_t*>(smem + Smem::bars + 8 * (3 * MAX_STAGES + 4));

    const int warp = warp_number(), lane = threadIdx.x & 31;
    const int chunk_kb = BN_T ? CHUNK_FAST : p.chunk_kb;
    const int bn = BN_T ? BN_T : p.bn, stages = BN_T ? STAGES : p.stages, raw_bytes = BN_T ? A_TILE + BN_T * BK * 4 : p.raw_bytes;

    // a CTA of a cluster of slices has one tile and slice: its rank is the batch, and the grid is as long as the tiles
    const int first_tile = FORM == CLUSTERED ? (int)blockIdx.x % p.cluster * p.tiles_per_batch + (int)blockIdx.x / p.cluster : (int)blockIdx.x;

    auto redo = [&] { return reinterpret_cast<uint32_t*>(smem + Smem::redo); };
    if (threadIdx.x <= REDO_BITS / 32) redo()[threadIdx.x] = 0;
    if (threadIdx.x == 0) {
        for (int s = 0; s < MAX_STAGES; s++) {
            mbar_init(full_bar(s), 1);
            mbar_init(split_bar(s), SPLIT_WARPS);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(tfull_bar(a), 1);
            mbar_init(tempty_bar(a), EPI_WARPS);
        }
        fence_barrier_init();
    }
    if (warp == 2 && elect_one()) {
        prefetch_map(&map_a);
        prefetch_map(&map_b);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_base_slot)), TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_base_slot;
    after_previous_kernel();

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (elect_one()) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int tile = first_tile; tile < p.num_tiles && ok; tile += gridDim.x) {
                int tm, tn, tb;
                tile_coords(tile, p, tm, tn, tb);
                int za = p.a_batched ? tb : 0, zb = p.b_batched ? tb : 0;
                for (int kb = 0; kb < p.num_kb; kb++) {
                    if (!mbar_wait(empty_bar(stage), phase ^ 1, err, tag, 1)) {
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(full_bar(stage), raw_bytes);
                    const uint32_t sa = smem_base + Smem::stages + stage * 2 * raw_bytes;
                    const uint32_t sb = sa + 2 * A_TILE;
                    int block = tb * p.split_kb + kb;  // a block past the end of K (or of the batches) is all fill: zeros
                    if (p.kb_per_z) {
                        za = zb = block / p.kb_per_z;
                        block -= za * p.kb_per_z;
                    }
                    const int k = block * BK;
                    if (!p.a_mn) {
                        tma_load_3d(sa, &map_a, k, tm * BM, za, full_bar(stage));
                    } else {
#pragma unroll
                        for (int h = 0; h < BM / 32; h++) tma_load_3d(sa + h * MN_CHUNK_BYTES, &map_a, tm * BM + h * 32, k, za, full_bar(stage));
                    }
                    if (!p.b_mn) {
                        tma_load_3d(sb, &map_b, k, tn * bn, zb, full_bar(stage));
                    } else {
                        for (int h = 0; h < bn / 32; h++) tma_load_3d(sb + h * MN_CHUNK_BYTES, &map_b, tn * bn + h * 32, k, zb, full_bar(stage));
                    }
                    if (++stage == stages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            const uint32_t idesc = make_idesc_tf32(p.a_mn != 0, p.b_mn != 0, bn), idesc_wide = make_idesc_tf32(p.a_mn != 0, p.b_mn != 0, 2 * bn);
            // K-major: 8 floats further along the 128-byte row; MN-major: the next group of eight K-rows
            const uint64_t a_kstep = p.a_mn ? (1024 >> 4) : (32 >> 4), b_kstep = p.b_mn ? (1024 >> 4) : (32 >> 4);
            int stage = 0, acc = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool ok = true;
            for (int tile = first_tile; tile < p.num_tiles && ok; tile += gridDim.x) {
                for (int kb0 = 0; kb0 < p.num_kb && ok; kb0 += chunk_kb) {
                    if (!mbar_wait(tempty_bar(acc), acc_phase ^ 1, err, tag, 2)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t d_tmem = tmem_base + (uint32_t)acc * 2 * BN;
                    const int kb1 = min(kb0 + chunk_kb, p.num_kb);
                    for (int kb = kb0; kb < kb1; kb++) {
                        // the raw tiles (TMA) and the small tiles (splitter) are both operands
                        if (!mbar_wait(full_bar(stage), phase, err, tag, 3) || !mbar_wait(split_bar(stage), phase, err, tag, 6)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t s0 = smem_base + Smem::stages + stage * 2 * raw_bytes;
                        // K-major: rows of 32 floats, groups of eight rows 1024 bytes apart.  MN-major: 32-byte-atom swizzle,
                        // groups of four K-rows 512 bytes apart, 128-byte-wide MN chunks one box (4 KB) apart.
                        const uint64_t a_big = p.a_mn ? smem_desc_sw128_atom32(s0, MN_CHUNK_BYTES, 512) : smem_desc_sw128(s0, 16, 1024);
                        const uint32_t s_b = s0 + 2 * A_TILE, s_bs = s_b + (raw_bytes - A_TILE);
                        const uint64_t b_big = p.b_mn ? smem_desc_sw128_atom32(s_b, MN_CHUNK_BYTES, 512) : smem_desc_sw128(s_b, 16, 1024);
                        const uint64_t a_small = p.a_mn ? smem_desc_sw128_atom32(s0 + A_TILE, MN_CHUNK_BYTES, 512) : smem_desc_sw128(s0 + A_TILE, 16, 1024);
                        const uint64_t b_small = p.b_mn ? smem_desc_sw128_atom32(s_bs, MN_CHUNK_BYTES, 512) : smem_desc_sw128(s_bs, 16, 1024);
                        if constexpr (FORM == WIDE) {  // the small part of B lies behind the raw one: one instruction of twice the columns multiplies a_big by both
#pragma unroll
                            for (int k = 0; k < BK / UMMA_K; k++) {
                                umma_tf32(d_tmem, a_big + a_kstep * k, b_big + b_kstep * k, idesc_wide, (kb != kb0) || (k != 0));
                                umma_tf32(d_tmem + bn, a_small + a_kstep * k, b_big + b_kstep * k, idesc, 1);
                            }
                        } else if (chunk_kb == 1) {
#pragma unroll
                            for (int k = 0; k < BK / UMMA_K; k++) {
                                umma_tf32(d_tmem, a_small + a_kstep * k, b_big + b_kstep * k, idesc, k != 0);
                                umma_tf32(d_tmem, a_big + a_kstep * k, b_small + b_kstep * k, idesc, 1);
                            }
#pragma unroll
                            for (int k = 0; k < BK / UMMA_K; k++) umma_tf32(d_tmem, a_big + a_kstep * k, b_big + b_kstep * k, idesc, 1);
                        } else {
#pragma unroll
                            for (int k = 0; k < BK / UMMA_K; k++) {
                                umma_tf32(d_tmem, a_small + a_kstep * k, b_big + b_kstep * k, idesc, (kb != kb0) || (k != 0));
                                umma_tf32(d_tmem, a_big + a_kstep * k, b_small + b_kstep * k, idesc, 1);
                                umma_tf32(d_tmem, a_big + a_kstep * k, b_big + b_kstep * k, idesc, 1);
                            }
                        }
                        umma_commit(empty_bar(stage));
                        if (++stage == stages) {
                            stage = 0;
                            phase ^= 1;
                        }
                    }
                    if (!ok) break;
                    umma_commit(tfull_bar(acc));  // this chunk's partial sums are complete
                    if (++acc == 2) {
                        acc = 0;
                        acc_phase ^= 1;
                    }
                }
            }
        }
    } else if (warp < 2 + EPI_WARPS) {
        // ------------------------------------------------------------ epilogue (warps 2..5)
        const int quarter = warp & 3;  // TMEM lanes [32 * quarter, 32 * quarter + 32)
        const int ew = warp - 2;
        unsigned char* stage_buf = smem + Smem::epi + ew * 2 * EPI_STAGE_BYTES;
        int acc = 0, buf = 0;
        uint32_t acc_phase = 0;
        bool ok = true;
        for (int tile = first_tile; tile < p.num_tiles && ok; tile += gridDim.x) {
            int tm, tn, tb;
            tile_coords(tile, p, tm, tn, tb);
            float total[BN];  // this thread's row of the tile (registers: every index below is a compile-time constant)
#pragma unroll
            for (int j = 0; j < BN; j++) total[j] = 0.0f;
            for (int kb0 = 0; kb0 < p.num_kb; kb0 += chunk_kb) {
                // the TMEM loads below are warp-collective: leave the loops only as a whole warp
                const bool ready = mbar_wait_relaxed(tfull_bar(acc), acc_phase, err, tag, 4, chunk_kb == 1 ? 20 : 200);
                if (!__all_sync(0xFFFFFFFFu, ready)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)acc * 2 * BN;
#pragma unroll
                for (int c = 0; c < BN / 32; c++) {
                    if (c * 32 >= bn) break;
                    uint32_t v[32];
                    if constexpr (FORM == WIDE) {  // the sum of the small products first
                        tmem_ld_32x32b_x32(t_row + bn + c * 32, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 32; j++) total[c * 32 + j] += __uint_as_float(v[j]);
                    }
                    tmem_ld_32x32b_x32(t_row + c * 32, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; j++) total[c * 32 + j] += __uint_as_float(v[j]);
                }
                // every TMEM read of this accumulator is done: hand it back to the MMA warp
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty_bar(acc));
                if (++acc == 2) {
                    acc = 0;
                    acc_phase ^= 1;
                }
            }
            if (!ok) break;
            float zero = 0.0f;  // NaN from the first total on that is not finite
            if constexpr (FORM == CLUSTERED) {
                float* part = reinterpret_cast<float*>(smem + Smem::stages + PART_OFF) + (quarter * 32 + lane) * PART_LD;  // the ring is done with
#pragma unroll
                for (int j = 0; j < BN; j += 4) {
                    if (j >= bn) break;
                    *reinterpret_cast<float4*>(part + j) = make_float4(total[j], total[j + 1], total[j + 2], total[j + 3]);
                    zero += fmaf(total[j], 0.0f, fmaf(total[j + 1], 0.0f, fmaf(total[j + 2], 0.0f, total[j + 3] * 0.0f)));
                }
                if (__any_sync(0xFFFFFFFFu, zero != 0.0f) && lane == 0) redo()[REDO_BITS / 32] = 1;
                continue;
            }
#pragma unroll
            for (int c = 0; c < BN / EPI_CHUNK_COLS; c++) {
                if (c * EPI_CHUNK_COLS >= bn) break;
                // the staging buffer must have been read by its previous TMA store
                if (lane == 0) tma_store_wait_read<1>();
                __syncwarp();
                unsigned char* dst = stage_buf + buf * EPI_STAGE_BYTES + lane * 128;  // row `lane` of the 32 x 32 tile
#pragma unroll
                for (int j = 0; j < 8; j++)  // eight 16-byte chunks per row, XOR-swizzled by the row index
                    *reinterpret_cast<float4*>(dst + ((j ^ (lane & 7)) << 4)) =
                        make_float4(total[c * 32 + 4 * j], total[c * 32 + 4 * j + 1], total[c * 32 + 4 * j + 2], total[c * 32 + 4 * j + 3]);
                float even = 0.0f, odd = 0.0f;
#pragma unroll
                for (int j = 0; j < 32; j += 2) {
                    even = fmaf(total[c * 32 + j], 0.0f, even);
                    odd = fmaf(total[c * 32 + j + 1], 0.0f, odd);
                }
                zero += even + odd;
                fence_proxy_async_smem();
                __syncwarp();
                const int row0 = tm * BM + quarter * 32, col0 = tn * bn + c * EPI_CHUNK_COLS;
                unsigned char* src = stage_buf + buf * EPI_STAGE_BYTES;
                if (!BN_T && p.d_plain) {
                    float* out = p.out + ((size_t)tb * p.M + row0) * p.N + col0 + lane;
                    for (int r0 = 0; r0 < 32; r0 += 8) {
                        float v[8];
#pragma unroll
                        for (int r = 0; r < 8; r++) v[r] = *reinterpret_cast<const float*>(src + (r0 + r) * 128 + (((lane >> 2) ^ r) << 4) + (lane & 3) * 4);
#pragma unroll
                        for (int r = 0; r < 8; r++)
                            if (row0 + r0 + r < p.M && col0 + lane < p.N) out[(size_t)(r0 + r) * p.N] = v[r];
                    }
                } else if (lane == 0) {
                    tma_store_3d(&map_d, smem_u32(src), col0, row0, tb);
                    tma_store_commit();
                }
                buf ^= 1;
            }
            if (__any_sync(0xFFFFFFFFu, zero != 0.0f) && lane == 0) {
                const int it = (tile - first_tile) / (int)gridDim.x;
                atomicOr(&redo()[it % REDO_BITS / 32], 1u << it % 32);
                redo()[REDO_BITS / 32] = 1;
            }
        }
        if (lane == 0) tma_store_wait_read<0>();  // the staging has been read; the writes themselves belong to the launch, and what follows it waits for them
    } else {
        // ------------------------------------------------------------ splitter (warps 6..9)
        const int t = threadIdx.x - 32 * (2 + EPI_WARPS);
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int tile = first_tile; tile < p.num_tiles && ok; tile += gridDim.x) {
            for (int kb = 0; kb < p.num_kb; kb++) {
                const bool landed = mbar_wait_relaxed(full_bar(stage), phase, err, tag, 5, 40);
                if (!__all_sync(0xFFFFFFFFu, landed)) {
                    ok = false;
                    break;
                }
                uint4* words = reinterpret_cast<uint4*>(smem + Smem::stages + stage * 2 * raw_bytes) + t;  // [A raw | A small | B raw | B small]
                constexpr int A_WORDS = A_TILE / 16, STEP = 32 * SPLIT_WARPS;
                auto split = [](const uint4& q) { return make_uint4(small_part(q.x), small_part(q.y), small_part(q.z), small_part(q.w)); };
                if constexpr (BN_T != 0) {
                    constexpr int B_WORDS = BN_T * BK * 4 / 16;
#pragma unroll 8
                    for (int i = 0; i < A_WORDS; i += STEP) words[i + A_WORDS] = split(words[i]);
#pragma unroll 8
                    for (int i = 0; i < B_WORDS; i += STEP) words[2 * A_WORDS + i + B_WORDS] = split(words[2 * A_WORDS + i]);
                } else {
                    const int b_words = bn * BK * 4 / 16;
                    for (int i0 = 0; i0 < A_WORDS + b_words; i0 += 4 * STEP) {  // loads first: the compiler cannot tell the tiles apart
                        uint4* from = words + (i0 < A_WORDS ? i0 : A_WORDS + i0);
                        const int to = i0 < A_WORDS ? A_WORDS : b_words;
                        uint4 q[4];
#pragma unroll
                        for (int i = 0; i < 4; i++) q[i] = from[i * STEP];
#pragma unroll
                        for (int i = 0; i < 4; i++) from[i * STEP + to] = split(q[i]);
                    }
                }
                fence_proxy_async_smem();  // the tensor core reads these through the async proxy
                __syncwarp();
                if (lane == 0) mbar_arrive(split_bar(stage));
                if (++stage == stages) {
                    stage = 0;
                    phase ^= 1;
                }
            }
        }
    }

    // common exit: TMEM is released by the warp that allocated it, after everyone is done with it
    tc_fence_before();
    __syncthreads();
    if (tc_err_mine(err, tag)) {
        const long long t0 = clock64();
        while (clock64() - t0 < 4000000ll) {
        }
        __syncthreads();
    }
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }

    if constexpr (FORM == CLUSTERED) {
        int tm, tn, tb;
        tile_coords(first_tile, p, tm, tn, tb);
        if (redo()[REDO_BITS / 32]) redo_tile<true>(p, bn, tm, tn, tb, reinterpret_cast<float*>(smem + Smem::stages));
        cluster_sync_all();
        const int r0 = BM * tb / p.cluster, rows = BM * (tb + 1) / p.cluster - r0, vecs = bn / 4;
        for (int e = threadIdx.x; e < rows * vecs; e += THREADS) {
            const int r = r0 + e / vecs, c = e % vecs * 4, row = tm * BM + r, col = tn * bn + c;
            if (row >= p.M || col >= p.N) continue;
            const float4 sum = sum_slices(smem_base + Smem::stages + PART_OFF + (uint32_t)(r * PART_LD + c) * 4, p.cluster);
            float* out = p.out + (int64_t)row * p.out_ld + col;
            if (p.vec_out) {
                *reinterpret_cast<float4*>(out) = sum;
            } else {
                out[0] = sum.x;
                if (col + 1 < p.N) out[1] = sum.y;
                if (col + 2 < p.N) out[2] = sum.z;
                if (col + 3 < p.N) out[3] = sum.w;
            }
        }
        cluster_sync_all();  // the others have read this CTA's part
        return;
    }

    if (!redo()[REDO_BITS / 32]) return;
    // the tile stores have to be made before their places are written again
    if (warp >= 2 && warp < 2 + EPI_WARPS && lane == 0) tma_store_wait_all();
    __syncthreads();
    fence_proxy_async();
    for (int tile = blockIdx.x, it = 0; tile < p.num_tiles; tile += gridDim.x, it++) {
        if (!(redo()[it % REDO_BITS / 32] >> it % 32 & 1)) continue;
        int tm, tn, tb;
        tile_coords(tile, p, tm, tn, tb);
        redo_tile<false>(p, bn, tm, tn, tb, reinterpret_cast<float*>(smem + Smem::stages));
    }
}

bool opt_in_shared_memory() {
    static std::mutex mu;
    static bool done[64] = {false};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    std::lock_guard<std::mutex> lock(mu);
    if (!done[dev]) {
        for (auto kernel : {tc_gemm_f32_kernel<BN>, tc_gemm_f32_kernel<0>, tc_gemm_f32_kernel<BN, WIDE>, tc_gemm_f32_kernel<0, WIDE>, tc_gemm_f32_kernel<BN, CLUSTERED>,
                            tc_gemm_f32_kernel<0, CLUSTERED>})
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess) {
                cudaGetLastError();
                return false;
            }
        done[dev] = true;
    }
    return true;
}

// mn_major: the operand is loaded as [32 K-rows x 32 MN-elements] boxes in the 32-byte-atom form of the 128-byte swizzle
bool make_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t batch, uint64_t batch_stride, uint32_t box_rows,
              bool mn_major = false, uint64_t pitch = 0) {
    return make_map_3d(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, rows, cols, batch, batch_stride, box_rows,
                       mn_major ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B, pitch);
}

// Columns of an output tile: 64 where 128-wide tiles would be half empty (N <= 64) or leave SMs without a tile; a 64-wide
// tile costs three quarters of a 128-wide one (shared-memory traffic of A and B together bounds both).
double tile_cost(int bn, uint64_t tiles_m, uint64_t N, uint64_t batch, int grid) {
    const uint64_t tiles = tiles_m * ((N + bn - 1) / bn) * batch, waves = (tiles + grid - 1) / grid;
    return (double)waves * (128 + bn) / 256.0;
}
int tile_columns(uint64_t tiles_m, uint64_t N, uint64_t batch, int grid) {
    return tile_cost(64, tiles_m, N, batch, grid) < 0.93 * tile_cost(128, tiles_m, N, batch, grid) ? 64 : 128;
}
// what the second launch of a split-K product costs, in k-blocks (about 0.9 us each on one CTA)
constexpr double kSplitFixed32 = 3.0;
// k-blocks from which on big x [big | small] is one instruction of twice the columns: two instructions a k-step instead of three and a third fewer reads of A,
// for twice the accumulator columns to empty every four k-blocks.  32 x (1152 x 196 x 256) 37.3 us, 35.7 so; 4096 x 4096 x 256 59.0, 57.3, x 64 22.6,
// 24.0.  Slices of a split product are short and gain nothing (256 x 512 x 2048 12.9, 13.1).  Error of 32 convolutions [256 x 1152] . [1152 x 196]
// against 64 bits 9.2e-7 (1.0e-6 by three).
constexpr int kWideLeast = 8;
std::atomic<int> g_wide{1};  // 0: never (tests, A/B timing)
// and the sum inside a cluster: more, since the second launch closes up with the first (128 x 300 x 784 10.9 us, 12.2 in a cluster; 512 x 1024 x 1024
// 15.5, 15.9).  A cluster takes products that the other form cuts into few slices or none: 300 x 784 x 8192 68 us, 50 in clusters of seven.
constexpr double kClusterFixed32 = 4.0;
std::atomic<int> g_cluster{1};  // 0: no clusters of slices, 2: wherever they fit (tests, A/B timing)
thread_local int t_last_form[4] = {0, 0, 0, 0};  // of the thread's last launch: slices, CTAs of a cluster (0: none), wide, columns of a tile (tests)

// How a product runs here: in how many slices of K, as CTAs of a cluster or through a second launch, and on which tiles.
struct Choice {
    int grid;
    int slices, cluster;
    int bn_cut, bn_whole;  // columns of a tile where the product is cut along K, where it is not
    double us;             // what it is estimated to take
    uint64_t partial_bytes(uint64_t m, uint64_t n) const { return slices > 1 && !cluster ? (uint64_t)slices * m * ((n + 3) / 4 * 4) * sizeof(float) : 0; }
};
Choice choose(const TcProduct& c) {
    Choice f;
    f.grid = sm_count();
    if (ctx().gemm_sm_limit > 0 && ctx().gemm_sm_limit < f.grid) f.grid = ctx().gemm_sm_limit;
    const uint64_t batch = c.sum_batches ? 1 : c.batch, tiles_m = (c.m + BM - 1) / BM;
    const int num_kb = (int)((c.k + BK - 1) / BK) * (c.sum_batches ? (int)c.batch : 1);
    // few output tiles: cut K into slices that run as the batches of the launch (see tc_ptx.cuh)
    f.bn_cut = c.n <= 64 ? 64 : BN;
    f.bn_whole = tile_columns(tiles_m, c.n, batch, f.grid);
    f.slices = 1;
    f.cluster = 0;
    if (batch == 1) {
        const uint64_t tiles = tiles_m * ((c.n + f.bn_cut - 1) / f.bn_cut);
        const double kb = (128 + f.bn_cut) / 256.0, whole = tile_cost(f.bn_whole, tiles_m, c.n, batch, f.grid) * num_kb;
        if (!c.sum_batches) f.slices = splitk_slices(tiles, c.k, BK, f.grid);
        if (f.slices == 1) f.slices = splitk_short(tiles, (uint64_t)num_kb, f.grid, kb, whole - kSplitFixed32);
        const int form = g_cluster.load(std::memory_order_relaxed);
        double cost = form == 2 ? 1e30 : whole;
        if (form != 2 && f.slices > 1)
            cost = std::min(cost, (double)((tiles * f.slices + f.grid - 1) / f.grid * ((num_kb + f.slices - 1) / f.slices)) * kb + kSplitFixed32 + 0.1 * f.slices);
        if (form)
            f.cluster = cluster_slices(tiles, (uint64_t)num_kb, f.grid, kb, kClusterFixed32, cost,
                                       [](int n) { return resident_clusters(reinterpret_cast<const void*>(tc_gemm_f32_kernel<0, CLUSTERED>), THREADS, SMEM_BYTES, n); });
        if (f.cluster) f.slices = f.cluster;
    }
    // us of a k-block of 64 or 128 columns, of a tile's end, of the launch and of what else is launched, fitted to 1400 products of 1.6e7 to 3e11 multiply-adds (four of five within 11 %)
    const int bn = f.slices > 1 ? f.bn_cut : f.bn_whole, per = (num_kb + f.slices - 1) / f.slices;
    const double waves = (double)((batch * tiles_m * ((c.n + bn - 1) / bn) * f.slices + f.grid - 1) / f.grid), columns = bn / 128.0;
    const bool wide = !c.ragged && f.slices == 1 && num_kb >= kWideLeast;
    const double copies = (c.a_repack ? (double)(c.a_bs ? c.batch : 1) * c.m * c.k : 0.0) + (c.b_repack ? (double)(c.b_bs ? c.batch : 1) * c.n * c.k : 0.0);
    const double kb_us = bn == 64 ? (c.ragged ? 0.79 : 0.76) : c.ragged ? 1.06 : 0.86, end_us = c.d_plain && f.slices == 1 ? 5.9 : wide ? 0.6 : 0.8;
    f.us = waves * (kb_us * per + end_us * columns) + 4.7 + (f.cluster ? 3.3 : f.slices > 1 ? 2.8 : 0.0) + (copies > 0 ? 1.4 + copies * 8 / 8.1e6 : 0.0);
    return f;
}

// D[M,N] = sum_k Aop[m,k] * Bop[n,k]; K-major operand = row-major [MN, K], MN-major = row-major [K, MN].
// Behind a gate (c.gate, `run`) in the same form as alone, slices included: without them 512 x 512 x 8192 took 219 us as pairs with an operand that is not fit, 16 tiles on 16 SMs, 51 so (tf32 alone 38).  The sum of the slices is one launch for this
// product and for the one in pairs, whichever ran.
bool launch(const TcProduct& c, const Choice& f, const PairsRun& run, void* D, const char* where) {
    const bool a_mn = c.a_mn, b_mn = c.b_mn;
    const uint64_t M = c.m, N = c.n, K = c.k;
    uint64_t batch = c.batch;
    if (!opt_in_shared_memory()) return false;
    Params p;
    p.M = (int)M;
    p.N = (int)N;
    p.chunk_kb = c.ragged ? 1 : CHUNK_FAST;
    p.bn = f.bn_cut;
    p.tiles_m = (int)((M + BM - 1) / BM);
    p.tiles_n = (int)((N + p.bn - 1) / p.bn);
    p.num_kb = (int)((K + BK - 1) / BK);
    p.split_kb = 0;
    p.kb_per_z = 0;
    if (c.sum_batches) {
        p.kb_per_z = p.num_kb;
        p.num_kb *= (int)batch;
        batch = 1;
    }
    int grid = f.grid;
    p.gate = c.gate;
    p.cluster = f.cluster;
    int slices = f.slices;
    StreamWorkspace workspace;
    float* partial = run.partial;
    const uint64_t n_pitch = (N + 3) / 4 * 4;
    if (slices > 1 && !p.cluster && !partial) {
        if (workspace.take(f.partial_bytes(M, N), true)) partial = static_cast<float*>(workspace.ptr);
        else slices = 1;
    } else if (slices > 1 && !p.cluster) {
        // A graph captured after this call has no workspace for pairs and runs this kernel, in slices with borrowed partial results: unsplit 512 x 512 x 8192 takes 202 us, 37 so.
        reserve_for_capture(f.partial_bytes(M, N));
    }
    if (slices > 1) {
        p.split_kb = (p.num_kb + slices - 1) / slices;
        p.num_kb = p.split_kb;
        batch = (uint64_t)slices;
    } else {
        p.bn = f.bn_whole;
        p.tiles_n = (int)((N + p.bn - 1) / p.bn);
    }
    p.tiles_per_batch = p.tiles_m * p.tiles_n;
    p.raw_bytes = A_TILE + p.bn * BK * 4;
    p.stages = STAGES * STAGE_BYTES / (2 * p.raw_bytes);
    int tag = 0;
    int* err = next_launch_error_word(&tag);
    if (!err) return false;
    CUtensorMap ma, mb, md;
    const uint64_t a_bs = (uint64_t)c.a_bs, b_bs = (uint64_t)c.b_bs;
    const bool oka = a_mn ? make_map(&ma, c.A, K, M, c.batch, a_bs, BK, true, c.a_pitch) : make_map(&ma, c.A, M, K, c.batch, a_bs, BM, false, c.a_pitch);
    const bool okb = b_mn ? make_map(&mb, c.B, K, N, c.batch, b_bs, BK, true, c.b_pitch) : make_map(&mb, c.B, N, K, c.batch, b_bs, (uint32_t)p.bn, false, c.b_pitch);
    if (!oka || !okb) return false;
    p.d_plain = slices > 1 ? 0 : c.d_plain;
    p.vec_out = N % 4 == 0 && (uintptr_t)D % 16 == 0 ? 1 : 0;
    if (p.d_plain || p.cluster) md = ma;  // not used
    else if (slices > 1 ? !make_map(&md, partial, M, N, batch, M * n_pitch, 32, false, n_pitch) : !make_map(&md, D, M, N, batch, M * N, 32)) return false;
    p.num_tiles = (int)batch * p.tiles_per_batch;
    p.a_batched = (c.batch > 1 && a_bs != 0) ? 1 : 0;
    p.b_batched = (c.batch > 1 && b_bs != 0) ? 1 : 0;
    p.a_mn = a_mn ? 1 : 0;
    p.b_mn = b_mn ? 1 : 0;
    p.a = reinterpret_cast<const float*>(c.A);
    p.b = reinterpret_cast<const float*>(c.B);
    p.a_bs = c.batch > 1 ? c.a_bs : 0;
    p.b_bs = c.batch > 1 ? c.b_bs : 0;
    const int64_t a_ld = (int64_t)(c.a_pitch ? c.a_pitch : a_mn ? M : K), b_ld = (int64_t)(c.b_pitch ? c.b_pitch : b_mn ? N : K);
    p.a_rs = a_mn ? 1 : a_ld;
    p.a_ks = a_mn ? a_ld : 1;
    p.b_rs = b_mn ? 1 : b_ld;
    p.b_ks = b_mn ? b_ld : 1;
    p.K = (int)K;
    p.zs = (int)c.batch;
    p.out = slices > 1 && !p.cluster ? partial : static_cast<float*>(D);
    p.out_ld = (int64_t)(slices > 1 && !p.cluster ? n_pitch : N);
    if (grid > p.num_tiles) grid = p.num_tiles;
    const int form = p.cluster ? CLUSTERED : p.chunk_kb == CHUNK_FAST && slices == 1 && p.num_kb >= kWideLeast && g_wide.load(std::memory_order_relaxed) ? WIDE : PLAIN;
    t_last_form[0] = slices;
    t_last_form[1] = p.cluster;
    t_last_form[2] = form == WIDE;
    t_last_form[3] = p.bn;
    const bool fixed = p.bn == BN && !p.d_plain && p.chunk_kb == CHUNK_FAST;
    const auto kernel = form == CLUSTERED ? (fixed ? tc_gemm_f32_kernel<BN, CLUSTERED> : tc_gemm_f32_kernel<0, CLUSTERED>)
                        : form == WIDE ? (fixed ? tc_gemm_f32_kernel<BN, WIDE> : tc_gemm_f32_kernel<0, WIDE>)
                                       : (fixed ? tc_gemm_f32_kernel<BN> : tc_gemm_f32_kernel<0>);
    launch_clusters(kernel, p.cluster ? p.num_tiles : grid, THREADS, SMEM_BYTES, p.cluster, ma, mb, md, p, err, tag);
    check_launch(where);
    const int to_add = slices > 1 && !p.cluster ? slices : 0, in_pairs = run.slices > 1 ? run.slices : 0;
    if (to_add || in_pairs) splitk_reduce(2, partial, to_add, M, N, n_pitch, D, where, &c.gate, in_pairs);
    return true;
}

}  // namespace

namespace tc {
int resident_clusters(const void* kernel, int threads, size_t shared, int n) {
    static std::mutex mu;
    static std::unordered_map<const void*, int> known[64][CLUSTER_MOST + 1];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    std::lock_guard<std::mutex> lock(mu);
    const auto it = known[dev][n].find(kernel);
    if (it != known[dev][n].end()) return it->second;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(sm_count() / n * n));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = shared;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)n;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int most = 0;
    if (cudaOccupancyMaxActiveClusters(&most, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        most = 0;
    }
    return known[dev][n][kernel] = most;
}
}  // namespace tc

// Pairs of f16 where they are faster, with the kernel above behind them for operands that are not fit; else, and where there is no workspace for pairs, that kernel alone.
// Whatever fails here has launched no less than the product's own kernels would overwrite: the caller computes it another way.
static bool repack_and_launch(TcProduct& c, void* out, const char* where) {
    StreamWorkspace pairs, ws;
    const Choice choice = choose(c);
    PairsRun run;
    tc_launch_f32_pairs(c, choice.us, choice.partial_bytes(c.m, c.n), out, run, pairs, where);
    c.gate = run.gate;
    return repack_operands(4, c, ws, where, run.place, run.room) && launch(c, choice, run, out, where);
}

bool tc_launch_f32(const TcProduct& c, void* out, const char* where) {
    TcProduct mine = c;
    return repack_and_launch(mine, out, where);
}

bool tc_gemm_f32(const MmDesc& d, int which, size_t num_els, size_t nea, size_t neb, const void* x, const void* y, void* out, const char* where) {
    TcProduct c;
    return tc_classify(d, which, 4, num_els, nea, neb, x, y, out, c) && repack_and_launch(c, out, where);
}

}  // namespace mx

// 1 (default): the slices of an f32 product are the CTAs of a cluster where that is the cheapest form; 0: never; 2: wherever they fit
extern "C" void mx_debug_set_gemm_f32_cluster(int on) { mx::g_cluster.store(on < 0 ? 0 : on > 2 ? 2 : on, std::memory_order_relaxed); }
extern "C" void mx_debug_set_gemm_f32_wide(int on) { mx::g_wide.store(on ? 1 : 0, std::memory_order_relaxed); }
extern "C" void mx_debug_gemm_f32_last_form(int* form) {
    for (int i = 0; i < 4; i++) form[i] = mx::t_last_form[i];
}
