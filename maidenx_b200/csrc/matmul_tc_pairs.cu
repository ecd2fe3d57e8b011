// f32 products on the 16-bit tensor cores: every operand element as a pair of f16 values.
//
// The tensor core multiplies f16 at twice the rate of tf32, and a pair of f16 (11 significant bits each, rounded to nearest) holds an f32 to 2^-23: with
//     x * 2^e = h1 + h2 * 2^-12,   h1 = f16(x * 2^e),   h2 = f16((x * 2^e - h1) * 2^12)
// three products h1 g1 + 2^-12 (h1 g2 + h2 g1) replace the three of the tf32 kernel (matmul_tc_f32.cu) in half the tensor time, and because the
// pairs are made once, by a pass before (split_pairs_kernel), no CTA splits what another has split: the tf32 kernel's loop is bound by its splitter warps and the
// shared memory they go through (0.9 us for 128 x 128 x 32, here 0.45 for x 64).  What f16 lacks is range.  Each block of 128 x 128 elements of an operand has its
// own power of two, which puts its largest element into [2^14, 2^15), and the sums are scaled back a block at a time: the accumulator of the tensor core
// only ever holds 128 values of K (as in the tf32 kernel, whose reason - truncating additions - holds here too), and the epilogue warps add it to their totals
// in registers with the scales of the two blocks.
//
// An element far below its block's largest one would lose bits: h2 ends at 2^-24.  Blocks with a nonzero element below 2^-28 of the largest, with a
// largest element outside 2^+-45, or with an infinity or NaN are counted as unfit; then the whole product is computed by the tf32 kernel instead.  Down to 2^-28 h1 is
// a normal f16 and a pair holds 2^-23 of the element; from there on it loses a bit with each power of two, and an element must not be held worse than there
// (elements of one binade by an identity, largest error and rms: tf32 2.4e-7, 7.9e-8 everywhere; pairs 1.2e-7, 4.2e-8 to 2^-27, 6.0e-8 at 2^-28, then 2.4e-7, 1.0e-7 and 4.8e-7, 2.0e-7).
// The host does not wait to know: the split pass leaves the call's tag in a word of the call's workspace, this kernel gives up
// when it finds it there, and the tf32 kernel, launched behind it, gives up when it does not.
//
// tf32 kernel / pairs, all launches, us: 4096^3 745 to 850 / 380, 2048 x 2048 x 1024 62 / 34, 4100 x 1544 x 1000 85 / 48, ragged 4099 x 1543 x 1000 124 / 62, 32 x (1152 x
// 196 x 256) with one A 34.6 / 23.8, [256 x 1152] by 32 x [1152 x 196] 36.0 / 30.6; small products and short reductions stay there (512 x 1024 x 1024 17.5 / 22.5, 128 x (384 x
// 384 x 64) 25.5 / 35). Error against 64 bits (2-norm): K = 1024 normal 4.2e-7 / 2.1e-7, positive 6.6e-7 / 4.6e-7; ragged forms, whose accumulator is emptied every 32
// values of K, 2.4e-7 / 1.5e-7, positive 1.85e-7 / 1.1e-7.  What bounds the loop: tensor pipe 61 % busy (4096 x 4096 x 2048), its stages of 64 KB wait for L2.
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <mutex>

#include "matmul_tc.cuh"
#include "tc_cluster.cuh"

namespace mx {

using namespace tc;

namespace {

constexpr int BM = 128, BN = 128, BK = 64;
constexpr int BLOCK = 128;                          // a scale's block: 128 rows or columns by 128 values of K
constexpr int FIT = 28;                             // powers of two that a block's nonzero elements may lie below its largest
constexpr int STAGES = 3;
constexpr int TILE_BYTES = BM * BK * 2;             // 16 KB: one half of the pairs of an operand's tile
constexpr int STAGE_BYTES = 4 * TILE_BYTES;         // [A h1 | A h2 | B h1 | B h2]
constexpr int MN_CHUNK_BYTES = BK * 128;            // one [64 K-rows x 64 MN] box
constexpr int EPI_WARPS = 8, EPI_STAGE_BYTES = 32 * 32 * 4;
constexpr int THREADS = 32 * (2 + EPI_WARPS);
constexpr int TMEM_COLS = 512;                      // two accumulators of [h1 g1 | the small products]
constexpr int GROUP_M = 16;

struct Smem {
    static constexpr int epi = STAGES * STAGE_BYTES;
    static constexpr int bars = epi + EPI_WARPS * EPI_STAGE_BYTES;
    static constexpr int total = bars + 256;
};
constexpr int SMEM_BYTES = Smem::total + 1024;
static_assert(SMEM_BYTES <= 232448, "shared memory per CTA");

__host__ __device__ constexpr uint32_t make_idesc_f16(bool a_mn_major, bool b_mn_major, int n) {
    return 1u << 4 | (a_mn_major ? 1u : 0u) << 15 | (b_mn_major ? 1u : 0u) << 16 | (uint32_t)(n >> 3) << 17 | (uint32_t)(BM >> 4) << 24;
}

struct Params {
    int M, N;
    int tiles_m, tiles_n, num_tiles, tiles_per_batch;
    int kb_z;          // k-blocks of 64 of one matrix
    int chunks_z;      // its scales along K
    int chunks;        // of an output tile: chunks_z, or those of all matrices (sum), or the run of a slice
    int all_chunks;
    int sliced;        // batch s of the launch reduces the chunks [s * chunks, (s + 1) * chunks) of one product
    int sum;           // chunk c belongs to matrix c / chunks_z of both operands
    int fine;          // the accumulator is emptied after every 32 values of K, else after every chunk
    int a_batched, b_batched, a_zs, b_zs;
    int a_mn, b_mn;
    const float *a_scale, *b_scale;  // [matrix][block of rows or columns][block of K]
    int d_plain;
    float* out;
    const unsigned long long* unfit;
    unsigned long long tag;
};

__device__ __forceinline__ void tile_coords(int tile, const Params& p, int& tm, int& tn, int& tb) {
    tb = tile / p.tiles_per_batch;
    tile -= tb * p.tiles_per_batch;
    const int group_size = GROUP_M * p.tiles_n, group = tile / group_size, first_m = group * GROUP_M, rows = min(GROUP_M, p.tiles_m - first_m), in_group = tile - group * group_size;
    tm = first_m + in_group % rows;
    tn = in_group / rows;
}

// The chunks of an output tile, in the order that all roles go through them: (matrices of A and B, chunk of K, k-blocks of it).
struct Chunk {
    int za, zb, kc, kbs;
};
__device__ __forceinline__ void chunk_range(const Params& p, int tb, int& c0, int& c1) {
    c0 = p.sliced ? tb * p.chunks : 0;
    c1 = min(c0 + p.chunks, p.all_chunks);
}
__device__ __forceinline__ Chunk chunk_at(const Params& p, int tb, int c) {
    Chunk q;
    const int z = p.sum ? c / p.chunks_z : p.sliced ? 0 : tb;
    q.kc = p.sum ? c - z * p.chunks_z : c;
    q.za = p.a_batched ? z : 0;
    q.zb = p.b_batched ? z : 0;
    q.kbs = min(2, p.kb_z - 2 * q.kc);
    return q;
}

__global__ void __launch_bounds__(THREADS, 1)
tc_gemm_pairs_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_d, Params p, int* err, int tag) {
    extern __shared__ unsigned char tcp_smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)tcp_smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t smem_base = smem_u32(smem);
    const uint32_t bar_base = smem_base + Smem::bars;
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
    auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
    auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + 2 + a); };
    volatile uint32_t* tmem_base_slot = reinterpret_cast<volatile uint32_t*>(smem + Smem::bars + 8 * (2 * STAGES + 4));
    const int warp = warp_number(), lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) {
            mbar_init(full_bar(s), 1);
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
    const int num_tiles = *p.unfit == p.tag ? 0 : p.num_tiles;

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (elect_one()) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
                int tm, tn, tb, c0, c1;
                tile_coords(tile, p, tm, tn, tb);
                chunk_range(p, tb, c0, c1);
                for (int c = c0; c < c1 && ok; c++) {
                    const Chunk q = chunk_at(p, tb, c);
                    for (int kb = 0; kb < q.kbs; kb++) {
                        if (!mbar_wait(empty_bar(stage), phase ^ 1, err, tag, 1)) {
                            ok = false;
                            break;
                        }
                        mbar_expect_tx(full_bar(stage), STAGE_BYTES);
                        const uint32_t sa = smem_base + stage * STAGE_BYTES, sb = sa + 2 * TILE_BYTES;
                        const int k = (2 * q.kc + kb) * BK;
#pragma unroll
                        for (int h = 0; h < 2; h++) {  // the halves of the pairs are matrices behind one another
                            if (!p.a_mn) {
                                tma_load_3d(sa + h * TILE_BYTES, &map_a, k, tm * BM, q.za + h * p.a_zs, full_bar(stage));
                            } else {
                                tma_load_3d(sa + h * TILE_BYTES, &map_a, tm * BM, k, q.za + h * p.a_zs, full_bar(stage));
                                tma_load_3d(sa + h * TILE_BYTES + MN_CHUNK_BYTES, &map_a, tm * BM + 64, k, q.za + h * p.a_zs, full_bar(stage));
                            }
                            if (!p.b_mn) {
                                tma_load_3d(sb + h * TILE_BYTES, &map_b, k, tn * BN, q.zb + h * p.b_zs, full_bar(stage));
                            } else {
                                tma_load_3d(sb + h * TILE_BYTES, &map_b, tn * BN, k, q.zb + h * p.b_zs, full_bar(stage));
                                tma_load_3d(sb + h * TILE_BYTES + MN_CHUNK_BYTES, &map_b, tn * BN + 64, k, q.zb + h * p.b_zs, full_bar(stage));
                            }
                        }
                        if (++stage == STAGES) {
                            stage = 0;
                            phase ^= 1;
                        }
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            const uint32_t idesc = make_idesc_f16(p.a_mn != 0, p.b_mn != 0, BN), idesc_wide = make_idesc_f16(p.a_mn != 0, p.b_mn != 0, 2 * BN);
            const uint32_t a_lbo = p.a_mn ? MN_CHUNK_BYTES : 16, b_lbo = p.b_mn ? MN_CHUNK_BYTES : 16;
            const uint64_t a_kstep = p.a_mn ? (2048 >> 4) : (32 >> 4), b_kstep = p.b_mn ? (2048 >> 4) : (32 >> 4);
            int stage = 0, acc = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
                int tm, tn, tb, c0, c1;
                tile_coords(tile, p, tm, tn, tb);
                chunk_range(p, tb, c0, c1);
                for (int c = c0; c < c1 && ok; c++) {
                    const int kbs = chunk_at(p, tb, c).kbs;
                    for (int kb = 0; kb < kbs; kb++) {
                        if (!mbar_wait(full_bar(stage), phase, err, tag, 3)) {
                            ok = false;
                            break;
                        }
                        const uint32_t sa = smem_base + stage * STAGE_BYTES;
                        const uint64_t a1 = smem_desc_sw128(sa, a_lbo, 1024), a2 = smem_desc_sw128(sa + TILE_BYTES, a_lbo, 1024), b = smem_desc_sw128(sa + 2 * TILE_BYTES, b_lbo, 1024);
#pragma unroll
                        for (int k2 = 0; k2 < BK / 32; k2++) {
                            const bool first = k2 == 0 ? p.fine || kb == 0 : p.fine != 0, last = k2 == 0 ? p.fine != 0 : p.fine || kb + 1 == kbs;
                            if (first && !mbar_wait(tempty_bar(acc), acc_phase ^ 1, err, tag, 2)) {
                                ok = false;
                                break;
                            }
                            tc_fence_after();
                            const uint32_t d_tmem = tmem_base + (uint32_t)acc * 2 * BN;
#pragma unroll
                            for (int k = 2 * k2; k < 2 * k2 + 2; k++) {
                                umma_f16(d_tmem, a1 + a_kstep * k, b + b_kstep * k, idesc_wide, !first || k != 2 * k2);  // h1 by [g1 | g2], which lie behind one another
                                umma_f16(d_tmem + BN, a2 + a_kstep * k, b + b_kstep * k, idesc, 1);
                            }
                            if (last) {
                                umma_commit(tfull_bar(acc));
                                if (++acc == 2) {
                                    acc = 0;
                                    acc_phase ^= 1;
                                }
                            }
                        }
                        if (!ok) break;
                        umma_commit(empty_bar(stage));
                        if (++stage == STAGES) {
                            stage = 0;
                            phase ^= 1;
                        }
                    }
                }
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue: two warps for each quarter of the accumulator's lanes, 64 columns each
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        unsigned char* stage_buf = smem + Smem::epi + (warp - 2) * EPI_STAGE_BYTES;
        int acc = 0;
        uint32_t acc_phase = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
            int tm, tn, tb, c0, c1;
            tile_coords(tile, p, tm, tn, tb);
            chunk_range(p, tb, c0, c1);
            float total[2][32];
#pragma unroll
            for (int j = 0; j < 64; j++) total[j / 32][j % 32] = 0.0f;
            float a_next = 0.0f, b_next = 0.0f;  // the next chunk's scales are on their way while this one's sums are added
            auto fetch_scales = [&](int c) {
                if (c >= c1) return;
                const Chunk q = chunk_at(p, tb, c);
                a_next = p.a_scale[((int64_t)q.za * p.tiles_m + tm) * p.chunks_z + q.kc];
                b_next = p.b_scale[((int64_t)q.zb * p.tiles_n + tn) * p.chunks_z + q.kc];
            };
            fetch_scales(c0);
            for (int c = c0; c < c1 && ok; c++) {
                const Chunk q = chunk_at(p, tb, c);
                const float scale = a_next * b_next;  // powers of two within 2^-120 .. 2^62: their product is one too
                fetch_scales(c + 1);
                for (int part = 0; part < (p.fine ? 2 * q.kbs : 1); part++) {
                    const bool ready = mbar_wait_relaxed(tfull_bar(acc), acc_phase, err, tag, 4, p.fine ? 20 : 60);
                    if (!__all_sync(0xFFFFFFFFu, ready)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * 2 * BN + half * 64);
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        uint32_t big[32], small[32];
                        tmem_ld_32x32b_x32(t_row + h * 32, big);
                        tmem_ld_32x32b_x32(t_row + BN + h * 32, small);
                        tmem_ld_wait_for(big);
                        reg_fence(small);
#pragma unroll
                        for (int j = 0; j < 32; j++) total[h][j] = fmaf(fmaf(__uint_as_float(small[j]), 0x1p-12f, __uint_as_float(big[j])), scale, total[h][j]);
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(tempty_bar(acc));
                    if (++acc == 2) {
                        acc = 0;
                        acc_phase ^= 1;
                    }
                }
            }
            if (!ok) break;
            const int row0 = tm * BM + quarter * 32;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int col0 = tn * BN + half * 64 + h * 32;
                if (lane == 0) tma_store_wait_read<0>();
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 8; j++)  // rows of 128 bytes, XOR-swizzled by the row
                    *reinterpret_cast<float4*>(stage_buf + lane * 128 + ((j ^ (lane & 7)) << 4)) = make_float4(total[h][4 * j], total[h][4 * j + 1], total[h][4 * j + 2], total[h][4 * j + 3]);
                if (p.d_plain) {
                    __syncwarp();
                    float* out = p.out + ((size_t)tb * p.M + row0) * p.N + col0 + lane;
                    for (int r0 = 0; r0 < 32; r0 += 8) {
                        float v[8];
#pragma unroll
                        for (int r = 0; r < 8; r++) v[r] = *reinterpret_cast<const float*>(stage_buf + (r0 + r) * 128 + (((lane >> 2) ^ r) << 4) + (lane & 3) * 4);
#pragma unroll
                        for (int r = 0; r < 8; r++)
                            if (row0 + r0 + r < p.M && col0 + lane < p.N) out[(size_t)(r0 + r) * p.N] = v[r];
                    }
                    __syncwarp();
                } else {
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0 && col0 < p.N && row0 < p.M) {
                        tma_store_3d(&map_d, smem_u32(stage_buf), col0, row0, tb);
                        tma_store_commit();
                    }
                }
            }
        }
        if (lane == 0) tma_store_wait_read<0>();
    }

    tc_fence_before();
    __syncthreads();
    if (tc_err_mine(err, tag)) {  // a wait gave up: bulk copies still in flight towards this CTA's shared memory get time to land
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
}

// ---------------------------------------------------------------------------------
// the split pass
// ---------------------------------------------------------------------------------
struct SplitOperand {
    const float* in;   // `zs` matrices of `rows` rows of `cols` elements, `ld` elements apart, `bs` between matrices
    __half* out;       // rows of `pitch` elements; the second halves of the pairs `plane` elements behind the first
    float* scale;
    uint32_t zs, rows, cols, pitch, row_blocks, col_blocks, blocks;
    int64_t ld, bs, plane;
    int k_rows;        // K runs along the rows (MN-major), else along the columns
    int vec;           // rows start at 16-byte boundaries
};
constexpr int SPLIT_THREADS = 512, SPLIT_ROWS = BLOCK / (SPLIT_THREADS / 32);

// One block of 128 x 128 elements: read once into registers, its largest and its smallest nonzero magnitude found, written as pairs.  Bound by HBM or L2:
// four bytes read and four written an element ([256 x 1152] and 32 x [1152 x 196] 12.9 us behind the im2col that writes the latter).
__global__ void __launch_bounds__(SPLIT_THREADS) split_pairs_kernel(SplitOperand a, SplitOperand b, unsigned long long* unfit, unsigned long long tag) {
    __shared__ uint32_t part[2][SPLIT_THREADS / 32];
    after_previous_kernel();
    const SplitOperand& o = blockIdx.x < a.blocks ? a : b;
    const uint32_t id = blockIdx.x < a.blocks ? blockIdx.x : blockIdx.x - a.blocks;
    const uint32_t cb = id % o.col_blocks, rest = id / o.col_blocks, rb = rest % o.row_blocks, z = rest / o.row_blocks;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t col = cb * BLOCK + lane * 4;
    const float* in = o.in + z * o.bs + col;
    float v[SPLIT_ROWS][4];
    uint32_t most = 0, least = 0x7FFFFFFFu;
#pragma unroll
    for (int i = 0; i < SPLIT_ROWS; i++) {
        const uint32_t row = rb * BLOCK + i * (SPLIT_THREADS / 32) + warp;
        const float* src = in + row * o.ld;
        if (o.vec && row < o.rows && col + 4 <= o.cols) {
            const float4 q = *reinterpret_cast<const float4*>(src);
            v[i][0] = q.x, v[i][1] = q.y, v[i][2] = q.z, v[i][3] = q.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++) v[i][j] = row < o.rows && col + j < o.cols ? src[j] : 0.0f;
        }
    }
#pragma unroll
    for (int i = 0; i < SPLIT_ROWS; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t m = __float_as_uint(v[i][j]) & 0x7FFFFFFFu;
            most = max(most, m);
            least = min(least, m - 1);  // zero wraps around to the largest
        }
    most = __reduce_max_sync(0xFFFFFFFFu, most);
    least = __reduce_min_sync(0xFFFFFFFFu, least);
    if (lane == 0) part[0][warp] = most, part[1][warp] = least;
    __syncthreads();
    most = __reduce_max_sync(0xFFFFFFFFu, part[0][lane % (SPLIT_THREADS / 32)]);
    least = __reduce_min_sync(0xFFFFFFFFu, part[1][lane % (SPLIT_THREADS / 32)]);
    const int e = (int)(most >> 23) - 127, low = (int)((least + 1) >> 23) - 127;  // of the largest and of the smallest nonzero element
    const bool zero = most == 0, fit = zero || (e >= -45 && e <= 45 && low >= e - FIT);
    const float up = zero || !fit ? 1.0f : __uint_as_float((uint32_t)(127 + 14 - e) << 23);
    if (threadIdx.x == 0) {
        const uint32_t mb = o.k_rows ? cb : rb, kc = o.k_rows ? rb : cb, mbs = o.k_rows ? o.col_blocks : o.row_blocks, kcs = o.k_rows ? o.row_blocks : o.col_blocks;
        o.scale[((int64_t)z * mbs + mb) * kcs + kc] = zero || !fit ? 1.0f : __uint_as_float((uint32_t)(127 + e - 14) << 23);
        if (!fit) *unfit = tag;
    }
    if (col >= o.cols) return;
#pragma unroll
    for (int i = 0; i < SPLIT_ROWS; i++) {
        const uint32_t row = rb * BLOCK + i * (SPLIT_THREADS / 32) + warp;
        if (row >= o.rows) continue;
        Vec<__half, 4> h1, h2;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float x = v[i][j] * up;
            h1.v[j] = __float2half_rn(x);
            h2.v[j] = __float2half_rn((x - __half2float(h1.v[j])) * 4096.0f);
        }
        __half* dst = o.out + ((int64_t)z * o.rows + row) * o.pitch + col;  // rows are whole lines: a vector that runs past the columns stays inside
        *reinterpret_cast<Vec<__half, 4>*>(dst) = h1;
        *reinterpret_cast<Vec<__half, 4>*>(dst + o.plane) = h2;
    }
}

// ---------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------
bool opt_in_shared_memory() {
    static std::mutex mu;
    static bool done[64] = {false};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    std::lock_guard<std::mutex> lock(mu);
    if (!done[dev]) {
        if (cudaFuncSetAttribute(tc_gemm_pairs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        done[dev] = true;
    }
    return true;
}

std::atomic<int> g_pairs{1};  // 0: never, 2: wherever possible, 3: the same with the accumulator emptied after every 32 values of K (tests, A/B timing)
thread_local int t_last_pairs = 0;
std::atomic<unsigned long long> g_next_tag{1};

// Bytes of a call's workspace: what the pools keep of it between calls.  Beyond it each call maps memory anew, which took longer than pairs gain: [13712 x 4025] by 59
// columns and its gradients 772 us in tf32, 1180 while the copies behind the gate had memory of their own, 716 in the pairs'.
constexpr uint64_t kPairsMost = 512ull << 20;

// From which time in the tf32 kernel on pairs are considered, and by an eighth they have to be faster there, what the estimates are off by.  The two to four launches more, their tensor maps and
// the workspace are 5 us of the calling thread (3.4 to 9.6 us a call, 8.7 to 14.4 as pairs): below this line a pass that is issued from the host waits for them.
// Linear layers op by op, forward and gradients, tf32 / pairs, us: 550 x 192 -> 630 41.9 / 52.2, 596 x 53 -> 3816 62.4 / 75.2, 880 x 43 -> 792 39.2 / 46.9; 162 x (635 x 16 x 88) and its
// gradients 92.7 / 120.
constexpr double kPairsLeastUs = 22.0;

struct Plan {
    uint64_t a_rows, a_cols, b_rows, b_cols, a_zs, b_zs, a_pitch, b_pitch, a_bytes, b_bytes, a_scales, b_scales;
    int tiles_m, tiles_n, kb_z, chunks_z, all_chunks, slices, grid;
    double cost;
};

Plan make_plan(const TcProduct& c) {
    Plan q;
    q.a_rows = c.a_mn ? c.k : c.m, q.a_cols = c.a_mn ? c.m : c.k, q.b_rows = c.b_mn ? c.k : c.n, q.b_cols = c.b_mn ? c.n : c.k;
    q.a_zs = c.a_bs ? c.batch : 1, q.b_zs = c.b_bs ? c.batch : 1;
    q.a_pitch = (q.a_cols + 63) / 64 * 64, q.b_pitch = (q.b_cols + 63) / 64 * 64;
    q.a_bytes = q.a_zs * q.a_rows * q.a_pitch * 4, q.b_bytes = q.b_zs * q.b_rows * q.b_pitch * 4;
    q.tiles_m = (int)((c.m + BM - 1) / BM), q.tiles_n = (int)((c.n + BN - 1) / BN);
    q.kb_z = (int)((c.k + BK - 1) / BK), q.chunks_z = (int)((c.k + BLOCK - 1) / BLOCK);
    q.a_scales = q.a_zs * q.tiles_m * q.chunks_z, q.b_scales = q.b_zs * q.tiles_n * q.chunks_z;
    q.all_chunks = c.sum_batches ? (int)c.batch * q.chunks_z : q.chunks_z;
    q.grid = sm_count();
    if (ctx().gemm_sm_limit > 0 && ctx().gemm_sm_limit < q.grid) q.grid = ctx().gemm_sm_limit;
    const uint64_t tiles = (uint64_t)q.tiles_m * q.tiles_n * (c.sum_batches ? 1 : c.batch);
    const uint64_t blocks = q.a_zs * q.tiles_m * q.chunks_z + q.b_zs * q.tiles_n * q.chunks_z;
    const double most = 0.5 * q.kb_z * (c.sum_batches ? (double)c.batch : 1.0);  // chunks, the last one of a matrix by its k-blocks
    // us of a chunk, of a tile's end, of all launches (the split pass, this kernel, the copies and the kernel behind the gate), of the sum over slices and of the split pass's bytes, fitted as
    // the tf32 kernel's (choose; four of five products within 13 %)
    auto cost = [&](int s) {
        const double waves = (double)((tiles * s + q.grid - 1) / q.grid), per = std::min((double)((q.all_chunks + s - 1) / s), most);
        return waves * (1.32 * per + (c.d_plain && s == 1 ? 3.4 : 1.4)) + 6.8 + (c.a_repack || c.b_repack ? 2.0 : 0.0) + (s > 1 ? 2.0 + (double)s * c.m * c.n * 8 / 1e7 : 0.0) +
               (double)blocks * BLOCK * BLOCK * 8 / 7.4e6;
    };
    q.slices = 1;
    if (c.batch == 1 || c.sum_batches)
        for (int s = 2; s <= std::min(q.all_chunks, 16); s++)
            if (cost(s) < cost(q.slices)) q.slices = s;
    q.slices = (q.all_chunks + (q.all_chunks + q.slices - 1) / q.slices - 1) / ((q.all_chunks + q.slices - 1) / q.slices);
    q.cost = cost(q.slices);
    return q;
}

}  // namespace

// false: nothing was launched and the caller goes on as without this; true: the product has been launched, and `run.gate` says what the caller's own kernel
// has to find in order to run behind it.
bool tc_launch_f32_pairs(const TcProduct& c, double tf32_us, uint64_t partial_bytes, void* D, PairsRun& run, StreamWorkspace& ws, const char* where) {
    t_last_pairs = 0;
    const int mode = g_pairs.load(std::memory_order_relaxed);
    if (!mode) return false;
    if (c.batch > 0x3FFF || c.m > 0x3FFFFFFF || c.n > 0x3FFFFFFF || c.k > 0x3FFFFFFF) return false;
    const Plan q = make_plan(c);
    if (q.a_bytes + q.b_bytes >= kPairsMost || (mode == 1 && (tf32_us < kPairsLeastUs || 1.12 * q.cost > tf32_us))) return false;
    if (q.a_zs * ((q.a_rows + 127) / 128) * ((q.a_cols + 127) / 128) + q.b_zs * ((q.b_rows + 127) / 128) * ((q.b_cols + 127) / 128) > 0x7FFFFFFFull) return false;
    if (!opt_in_shared_memory()) return false;
    auto line = [](uint64_t bytes) { return (bytes + 255) / 256 * 256; };
    const uint64_t n_pitch = (c.n + 3) / 4 * 4, partials = std::max(partial_bytes, q.slices > 1 ? (uint64_t)q.slices * c.m * n_pitch * 4 : 0);
    const uint64_t a_at = 256, b_at = a_at + line(q.a_bytes), sa_at = b_at + line(q.b_bytes), sb_at = sa_at + line(q.a_scales * 4), part_at = sb_at + line(q.b_scales * 4);
    if (part_at + partials > kPairsMost || !ws.take(part_at + partials)) return false;
    char* base = static_cast<char*>(ws.ptr);
    // a tag is never given twice, and what the workspace held before does not look like one
    Gate mine;
    mine.word = reinterpret_cast<unsigned long long*>(base);
    mine.tag = 0x5A17C3E900000000ull ^ g_next_tag.fetch_add(1, std::memory_order_relaxed);
    int tag = 0;
    int* err = next_launch_error_word(&tag);
    if (!err) return false;
    CUtensorMap ma, mb, md;
    const CUtensorMapDataType h = CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    const CUtensorMapSwizzle sw = CU_TENSOR_MAP_SWIZZLE_128B;
    const bool ok = make_map_3d(&ma, h, 2, base + a_at, q.a_rows, q.a_cols, 2 * q.a_zs, q.a_rows * q.a_pitch, c.a_mn ? BK : BM, sw, q.a_pitch) &&
                    make_map_3d(&mb, h, 2, base + b_at, q.b_rows, q.b_cols, 2 * q.b_zs, q.b_rows * q.b_pitch, c.b_mn ? BK : BN, sw, q.b_pitch);
    if (!ok) return false;
    const uint64_t out_batch = q.slices > 1 ? (uint64_t)q.slices : c.sum_batches ? 1 : c.batch;
    const int d_plain = q.slices > 1 ? 0 : (c.n % 4 != 0 || (uintptr_t)D % 16 != 0);
    if (d_plain) md = ma;  // not used
    else if (!make_map_3d(&md, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, q.slices > 1 ? base + part_at : D, c.m, c.n, out_batch, c.m * (q.slices > 1 ? n_pitch : c.n), 32, sw, q.slices > 1 ? n_pitch : 0))
        return false;
    auto operand = [&](const char* in, uint64_t at, uint64_t scale_at, uint64_t zs, uint64_t rows, uint64_t cols, uint64_t pitch, uint64_t ld, int64_t bs, bool k_rows) {
        SplitOperand o;
        o.in = reinterpret_cast<const float*>(in);
        o.out = reinterpret_cast<__half*>(base + at);
        o.scale = reinterpret_cast<float*>(base + scale_at);
        o.zs = (uint32_t)zs, o.rows = (uint32_t)rows, o.cols = (uint32_t)cols, o.pitch = (uint32_t)pitch;
        o.row_blocks = (uint32_t)((rows + BLOCK - 1) / BLOCK), o.col_blocks = (uint32_t)((cols + BLOCK - 1) / BLOCK);
        o.blocks = (uint32_t)(zs * o.row_blocks * o.col_blocks);
        o.ld = (int64_t)ld, o.bs = bs, o.plane = (int64_t)(zs * rows * pitch);
        o.k_rows = k_rows;
        o.vec = (uintptr_t)in % 16 == 0 && ld % 4 == 0 && bs % 4 == 0;
        return o;
    };
    const SplitOperand oa = operand(c.A, a_at, sa_at, q.a_zs, q.a_rows, q.a_cols, q.a_pitch, c.a_pitch ? c.a_pitch : q.a_cols, c.a_bs, c.a_mn);
    const SplitOperand ob = operand(c.B, b_at, sb_at, q.b_zs, q.b_rows, q.b_cols, q.b_pitch, c.b_pitch ? c.b_pitch : q.b_cols, c.b_bs, c.b_mn);
    Params p;
    p.M = (int)c.m, p.N = (int)c.n;
    p.tiles_m = q.tiles_m, p.tiles_n = q.tiles_n, p.tiles_per_batch = q.tiles_m * q.tiles_n;
    p.num_tiles = (int)out_batch * p.tiles_per_batch;
    p.kb_z = q.kb_z, p.chunks_z = q.chunks_z, p.all_chunks = q.all_chunks;
    p.chunks = (q.all_chunks + q.slices - 1) / q.slices;
    p.sliced = q.slices > 1;
    p.sum = c.sum_batches;
    p.fine = mode == 3 || (mode != 2 && c.ragged);
    p.a_batched = q.a_zs > 1, p.b_batched = q.b_zs > 1, p.a_zs = (int)q.a_zs, p.b_zs = (int)q.b_zs;
    p.a_mn = c.a_mn, p.b_mn = c.b_mn;
    p.a_scale = oa.scale, p.b_scale = ob.scale;
    p.d_plain = d_plain;
    p.out = static_cast<float*>(D);
    p.unfit = mine.word, p.tag = mine.tag;
    t_last_pairs = q.slices;
    run.gate = mine;  // only here: a caller whose product was not launched goes on without a gate, for nothing would open it
    run.slices = q.slices;
    run.partial = reinterpret_cast<float*>(base + part_at);
    run.place = base + a_at;
    run.room = sa_at - a_at;
    launch_kernel(split_pairs_kernel, oa.blocks + ob.blocks, SPLIT_THREADS, 0, ctx().stream, oa, ob, reinterpret_cast<unsigned long long*>(base), mine.tag);
    launch_kernel(tc_gemm_pairs_kernel, std::min(q.grid, p.num_tiles), THREADS, SMEM_BYTES, ctx().stream, ma, mb, md, p, err, tag);
    check_launch(where);
    return true;
}

}  // namespace mx

// 1 (default): f32 products as pairs of f16 by the rule on their cost; 0: never; 2: wherever possible; 3: the same, emptying the accumulator after every 32 values of K
extern "C" void mx_debug_set_gemm_f32_pairs(int mode) { mx::g_pairs.store(mode, std::memory_order_relaxed); }
// of the calling thread's last f32 product: 0 not as pairs, else its slices
extern "C" int mx_debug_gemm_f32_last_pairs(void) { return mx::t_last_pairs; }
