// Tensor-core path for bf16 / f16 matmul on sm_100a: tcgen05.mma with the accumulator in
// tensor memory (TMEM), operands staged in shared memory by TMA, epilogue read back with
// tcgen05.ld, converted and written with TMA stores.
//
// One persistent CTA per SM, 192 threads (320 where the warps write the rows themselves or add a bias) in three roles:
//   warp 0      TMA producer: one lane issues cp.async.bulk.tensor loads of the A [128 x 64]
//               and B [64 to 256 x 64] k-blocks into a shared-memory ring (128-byte swizzle) of four
//               stages, up to eight of narrower tiles;
//   warp 1      MMA issuer: one lane issues four tcgen05.mma (M128, N = the tile's columns, K16) per
//               k-block into one of two 256-column TMEM accumulators, commits the stage back to the
//               producer and, after the last k-block (or a run of them, see DRAIN), the accumulator
//               to the epilogue;
//   the others  epilogue: one or two warps own the 32 TMEM lanes that they may address (warp id mod 4),
//               read them 64 columns at a time, round to bf16 / f16, write a swizzled
//               4 KB staging tile and store it with TMA (rows that no tensor map can describe:
//               themselves) while the next tile's MMAs run on the other accumulator.
// No cluster launch: every CTA issues its own (CTA-local) TMA loads; re-use comes from
// L2 through the order in which output tiles are handed out (16 row-tiles per column sweep).
//
// The kernel computes D[M,N] = sum_k A[m,k] * B[n,k]; by default both operands are K-major (row-major
// [M,K] and [N,K]): the reference's forward x . W^T (crates/maidenx_nn/src/layers/linear.rs:74) and
// its grad_a = g . B^T (crates/maidenx_cpu/src/ops/matmul.rs:208-216).  Either operand may instead be
// MN-major (row-major [K,M] / [K,N]): it is then loaded as 64-wide column chunks and described
// to the tensor core with the MN-major descriptor form, which covers grad_b = A^T . g (:244-256)
// and a plain [K,N] B without any transposed copy.
//
// Every mbarrier wait is bounded by a clock64() budget; on expiry the thread records an
// error word, stops issuing work and falls through to the common exit, where TMEM is freed.
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <unordered_map>

#include "f32x2.cuh"
#include "matmul_tc.cuh"
#include "matmul_tc2.cuh"
#include "tc_ptx.cuh"

namespace mx {

using namespace tc;

namespace {

// true: products go to the two-CTA kernel (matmul_tc2.cu); false (default): to the one-CTA kernel below.  On a B200 under
// its power cap the two run at the same rate (the pair form only moves less data through shared memory).
std::atomic<bool> g_two_cta{false};
std::atomic<int> g_group_m{16};  // row-tiles per column sweep of the one-CTA kernel's tile order

constexpr int BM = 128, BN = 256, BK = 64;    // CTA tile; BK * 2 bytes = one 128-byte swizzle row
constexpr int UMMA_K = 16;
constexpr int STAGES = 4;                     // ring stages of full-width tiles; narrower ones get as many as fit the same bytes
constexpr int MAX_STAGES = 8;
constexpr int A_STAGE_BYTES = BM * BK * 2;    // 16 KB
constexpr int B_STAGE_BYTES = BN * BK * 2;    // 32 KB
constexpr int EPI_CHUNK_COLS = 64;            // columns per TMA store (128 bytes of 16-bit)
constexpr int EPI_STAGE_BYTES = 32 * EPI_CHUNK_COLS * 2;  // 4 KB: 32 rows of a chunk; two such buffers per quarter
constexpr int TMEM_COLS = 512;                // two 256-column f32 accumulators
constexpr int GROUP_M = 16;                   // row-tiles per column sweep (L2 re-use)

struct SmemLayout {
    // offsets inside the dynamic shared memory block (base aligned to 1024 bytes)
    static constexpr int ring = 0;  // stage s: A block, then B block (bn rows of 128 bytes), s * stage_bytes further
    static constexpr int epi = ring + STAGES * (A_STAGE_BYTES + B_STAGE_BYTES);
    static constexpr int bars = epi + 4 * 2 * EPI_STAGE_BYTES;
    static constexpr int total = bars + 256;
};
constexpr int TC_SMEM_BYTES = SmemLayout::total + 1024;  // slack for the 1024-byte alignment

// 16-bit products that the CUDA cores would compute (ragged, rank > 3, batched backward, small) with an f32 sum rounded to nearest.  The
// tensor core's additions truncate, which pulls a long sum of one sign towards zero: measured 6e-6 of it in 1024 terms, at most an ulp (2^-23)
// for each instruction's 16.  After runs of these many terms the accumulator is added to f32 totals, so that the pull stays far below the
// rounding to the type (2.2e-4 f16, 1.8e-3 bf16 for positive sums): f16 K = 16385 2.209e-4 on the CUDA cores, 2.237e-4 in one run.
constexpr int kRunMostF16 = 1024, kRunMostBf16 = 4096;

// Split-K of a short reduction: what its second launch and the wider partial results cost, in k-blocks (0.27 us each on one CTA)
constexpr double kSplitFixed16 = 10.0;

constexpr int MN_CHUNK_BYTES = 64 * BK * 2;  // one [64 K-rows x 64 MN] box

// Instruction descriptor of tcgen05.mma kind::f16 with f32 accumulation.
__host__ __device__ constexpr uint32_t make_idesc(bool is_bf16, bool a_mn_major, bool b_mn_major, int bn) {
    uint32_t d = 0;
    d |= 1u << 4;                               // D format: f32
    d |= (is_bf16 ? 1u : 0u) << 7;              // A format: 0 = f16, 1 = bf16
    d |= (is_bf16 ? 1u : 0u) << 10;             // B format
    d |= (a_mn_major ? 1u : 0u) << 15;          // A major: 0 = K, 1 = MN
    d |= (b_mn_major ? 1u : 0u) << 16;          // B major
    d |= (uint32_t)(bn >> 3) << 17;             // N / 8
    d |= (uint32_t)(BM >> 4) << 24;             // M / 16
    return d;
}

struct TcParams {
    int M, N, K;
    int tiles_m, tiles_n, num_tiles, num_kb;
    int tiles_per_batch;   // tiles_m * tiles_n; num_tiles = batch * tiles_per_batch
    int a_batched, b_batched;  // 0: the operand is one matrix shared by every batch (third TMA coordinate stays 0)
    int is_bf16;
    int out_f32;  // split-K partial results: the epilogue stores the f32 accumulators unrounded
    int fuse;     // 0: store the product; 1: u = round(round(product) + bias) through map_d; 2: also act = round(gelu(u)) through map_d2;
                  // 3: as 1 with one bias element per output ROW (bias[row of the batch's matrix]): a convolution's per-channel bias
    const void* bias;  // fuse != 0: one element of the operand type in device memory
    int a_mn, b_mn;  // operand is MN-major in global memory ([K, MN] row-major) instead of K-major ([MN, K])
    int group_m;     // row-tiles per column sweep (L2 re-use of the A panels)
    int bn;          // columns of an output tile: 64, 128, 192 or 256 (tile_columns)
    int stages, stage_bytes;  // of the operand ring
    int split_kb;    // > 0: split-K; batch s of the launch reduces the k-blocks [s * split_kb, (s + 1) * split_kb) of one product
    // The output's rows are not 16-byte multiples (or its base is not aligned), which no tensor map can describe: the epilogue
    // warps copy their staged rows to `d` themselves (store_rows).  0: tensor stores.
    int d_plain;
    void* d;
    int run_kb;      // DRAIN form: k-blocks summed in one accumulator before the epilogue adds them to its own f32 totals
    // Short reductions (num_kb <= STAGES, one batch): `b_keep` CTAs share each column tile, CTA j of them takes the row
    // tiles j, j + b_keep, ...; the B panel of the column tile is loaded once into the B slots of the ring (slot = k-block,
    // the ring is num_kb slots long) and only A streams.  0: the general schedule.
    int b_keep;
    // CONV: the product's B is read out of images, K runs over a kernel's taps and, for each, over the channels of B's images in k-blocks (conv_cb of them); a column tile
    // is conv_rows whole rows of an output image of width conv_w, whose source pixels for tap (i, j) begin at row + conv_y - i, column conv_x - j.
    int conv_cb, conv_kw, conv_rows, conv_w, conv_x, conv_y;
    int poll_ns;  // between the epilogue's looks at a tile's accumulator: 3 to 4 % of the time a tile's reduction takes (training step of 512 x 1024 x 1024 49.5 us at 400, 48.8 so)
};
// CONV: and both operands as plain memory, for conv_redo.  Not among the parameters of the other kernels: a launch that the host does not run ahead of takes 2.02 us where its parameters, rounded up to
// 16 bytes, end 32 behind a multiple of 64, and 2.40 where they end elsewhere (4 maps, these and two words: 668 bytes; with this 700, and three products of 23 x 45 x 496 x 123 19.0 us for 17.8).
struct TcConvParams : TcParams {
    int conv_kh, conv_co, conv_oh, conv_ow;
    const void *conv_g, *conv_wt;
};
static_assert((4 * sizeof(CUtensorMap) + sizeof(TcParams) + sizeof(int*) + sizeof(int) + 15) / 16 * 16 % 64 == 32, "parameters of tc_gemm_kernel");

__device__ __forceinline__ void tile_coords(int tile, const TcParams& p, int& tm, int& tn, int& tb) {
    tb = tile / p.tiles_per_batch;
    tile -= tb * p.tiles_per_batch;
    // sweep GROUP_M row-tiles for each column tile before moving to the next column tile
    const int group_size = p.group_m * p.tiles_n;
    const int group = tile / group_size;
    const int first_m = group * p.group_m;
    const int rows = min(p.group_m, p.tiles_m - first_m);
    const int in_group = tile - group * group_size;
    tm = first_m + in_group % rows;
    tn = in_group / rows;
}

// The it-th tile of this CTA; false when it has none left.  PANELS (short reductions of a batch): the tiles in the order batch, column tile, row
// tile, an equal run of them for each CTA, which loads a B panel once for all row tiles of it.
template <bool PANELS>
__device__ __forceinline__ bool next_tile(int it, const TcParams& p, int& tm, int& tn, int& tb) {
    if constexpr (PANELS) {
        const int tile = (int)((long long)blockIdx.x * p.num_tiles / gridDim.x) + it;
        if (tile >= (int)((long long)(blockIdx.x + 1) * p.num_tiles / gridDim.x)) return false;
        const int panel = tile / p.tiles_m;
        tm = tile - panel * p.tiles_m;
        tb = panel / p.tiles_n;
        tn = panel - tb * p.tiles_n;
        return true;
    }
    if (p.b_keep) {
        tn = (int)blockIdx.x / p.b_keep;
        tm = (int)blockIdx.x % p.b_keep + it * p.b_keep;
        tb = 0;
        return tn < p.tiles_n && tm < p.tiles_m;
    }
    const int tile = (int)blockIdx.x + it * (int)gridDim.x;
    if (tile >= p.num_tiles) return false;
    tile_coords(tile, p, tm, tn, tb);
    return true;
}

__device__ __forceinline__ uint32_t pack2(float lo, float hi, int is_bf16) {
    if (is_bf16) {
        __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<uint32_t*>(&v);
    }
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}

// The epilogue's arithmetic of Linear + bias (+ GELU) on N elements, with the roundings of the separate ops: u = round(round(product) + bias) as 16-byte pieces, and what GELU of u is
// before its rounding.  By pairs, with one branch on the type a chunk: element by element, the type chosen at each, 8192 x 4096 x 512 bf16 took 48.7 us (with GELU, on the same warps, 84.6), 30.1 (58.3) so;
// 512 x 1024 x 1024 7.2 (8.1), 6.8 (7.6); a 1 x 1 convolution 64 x 256 x 55 x 55 -> 64, whose warps write the rows, forward and backward 340 us, 325.  Without arithmetic the one branch gains nothing (128 x (384 x 384 x 64) 10.9 us, 11.4).
template <class T, bool GELU, int N>
__device__ __forceinline__ void bias_gelu(float (&e)[N], float bias, uint4 (&u)[N / 8]) {
#pragma unroll
    for (int j = 0; j < N / 8; j++) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float* x = e + 8 * j + 2 * i;
            float2 f = halves(pair_of(unpack2<T>(pack2_rn<T>(x[0], x[1]))) + twice(bias));
            w[i] = pack2_rn<T>(f.x, f.y);
            if (!GELU) continue;
            f = gelu_f32x2(unpack2<T>(w[i]));
            x[0] = f.x;
            x[1] = f.y;
        }
        u[j] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// The 16 bytes that start 16 - 2 * sh bytes into (lo, hi), sh = 0 .. 7.
__device__ __forceinline__ uint4 vector_before(const uint4& lo, const uint4& hi, uint32_t sh) {
    const uint32_t words = 4 - (sh + 1) / 2, bits = (sh & 1) * 16;
    uint32_t w[9] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w, 0};
#pragma unroll
    for (int s = 4; s; s >>= 1)  // word-wise shift with compile-time indices
#pragma unroll
        for (int i = 0; i + s < 9; i++)
            if (words & s) w[i] = w[i + s];
    return make_uint4(__funnelshift_r(w[0], w[1], bits), __funnelshift_r(w[1], w[2], bits), __funnelshift_r(w[2], w[3], bits), __funnelshift_r(w[3], w[4], bits));
}

// Chunk `c` (64 columns) of 16 rows from r0 on of a quarter's 32 (those below `rows`), written to an output whose rows start anywhere: `tile` is the first element of
// row 0, `ld` the elements between rows, `cols` the tile's columns inside the matrix; `cur` is the staged chunk (XOR-swizzled rows of 128 bytes), `prev` the
// chunk before.  A row that starts sh elements behind a 16-byte boundary is cut at the boundaries: its vector v holds the elements 8 v - sh and following, so that
// every chunk completes exactly eight vectors a row, the first of them with the last sh elements of the chunk before.  Only the
// up to seven elements before a tile's first boundary and after its last are written by themselves.  Stores of one element
// each bound the tiles of short reductions (4096 x 2050 x 512 bf16: 42 us, 24 so with two warps a quarter).
__device__ __forceinline__ void store_rows(uint16_t* tile, size_t ld, int r0, int rows, int cols, int c, const unsigned char* cur, const unsigned char* prev, int lane) {
    if (c * 64 >= cols) return;
    const int r_lane = lane >> 3, j = lane & 7;
    const bool first = c == 0, last = c * 64 + 64 >= cols;
    uint16_t* dst = tile + (r0 + r_lane) * ld;
    uint4 lo[4], hi[4];
    // all loads before the first store: the compiler cannot tell the staging tile from the output
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int r = r0 + 4 * i + r_lane;
        lo[i] = *reinterpret_cast<const uint4*>((j ? cur : prev) + r * 128 + ((((j - 1) & 7) ^ (r & 7)) << 4));
        hi[i] = *reinterpret_cast<const uint4*>(cur + r * 128 + ((j ^ (r & 7)) << 4));
    }
#pragma unroll
    for (int i = 0; i < 4; i++, dst += 4 * ld) {
        const int r = r0 + 4 * i + r_lane;
        const int sh = (int)(reinterpret_cast<uintptr_t>(dst) >> 1) & 7, e0 = c * 64 + j * 8 - sh;
        if (r < rows && e0 >= 0 && e0 + 8 <= cols) *reinterpret_cast<uint4*>(dst + e0) = vector_before(lo[i], hi[i], (uint32_t)sh);
        auto single = [&](int e) {
            const int x = e & 63;
            dst[e] = *reinterpret_cast<const uint16_t*>((e >> 6 == c ? cur : prev) + r * 128 + (((x >> 3) ^ (r & 7)) << 4) + (x & 7) * 2);
        };
        const int head = sh ? 8 - sh : 0;
        if (first && r < rows && j < head && j < cols) single(j);
        if (last) {
            const int e = max(head, ((cols + sh) & ~7) - sh) + j;
            if (r < rows && e < cols) single(e);
        }
    }
}

// What the epilogue does is compiled in: each form keeps its registers and its code to itself, and the plain product's loop is
// not laid out around the others.
// CONV: a pixel outside grad_out arrives as zeros, and zero times a weight that is infinite or NaN is a NaN that the sum over the pixels inside does not have.  The epilogue looks for totals that
// are not finite, and a CTA that saw one goes through its tiles here: a NaN whose taps do not all lie inside is summed anew over those that do, up to the first NaN among them.
// A warp takes a row, eight pixels a lane in flight; bound by the sums' serial chains.  Finite totals cost nothing that shows (64 x 256 x 56 x 56 -> 256, 3 x 3, input gradient 205 us with the look
// and without), one infinite weight 1075, a gradient of NaNs 468.
struct ConvRedo {
    const void *g, *wt;
    void* out;  // of the tile's batch
    int rows, pixels, c0, pix0, n, w, x, y, kh, kw, co, oh, ow;
};
template <class T>
__device__ __noinline__ void conv_redo(const ConvRedo q) {
    const T *const g = static_cast<const T*>(q.g), *const wt = static_cast<const T*>(q.wt);
    const int lane = threadIdx.x & 31;
    auto tap_row = [&](int s) { return (q.pix0 + lane + 32 * s) / q.w + q.y; };  // tap (i, j) of the lane's s-th pixel reads (tap_row - i, tap_col - j)
    auto tap_col = [&](int s) { return (q.pix0 + lane + 32 * s) % q.w + q.x; };
    uint32_t edge = 0;  // the pixels that not all taps of lie inside; a tile has 256 at most
    for (int s = 0; s < 8; s++)
        if (lane + 32 * s < q.pixels && (tap_row(s) >= q.oh || tap_col(s) >= q.ow || tap_row(s) < q.kh - 1 || tap_col(s) < q.kw - 1)) edge |= 1u << s;
    for (int r = threadIdx.x >> 5; r < q.rows; r += blockDim.x >> 5) {
        const int c = q.c0 + r;
        T* const row = static_cast<T*>(q.out) + (size_t)c * q.n + q.pix0 + lane;
        uint32_t wrong = 0;
#pragma unroll
        for (int s = 0; s < 8; s++)
            if (edge >> s & 1 && isnan(to_f32(row[32 * s]))) wrong |= 1u << s;
        for (; wrong; wrong &= wrong - 1) {
            const int s = __ffs(wrong) - 1, y = tap_row(s), x = tap_col(s);
            float sum = 0.0f;
            for (int i = max(0, y - q.oh + 1); i < q.kh && i <= y && !isnan(sum); i++)
                for (int j = max(0, x - q.ow + 1); j < q.kw && j <= x && !isnan(sum); j++) {
                    const T *const a = wt + ((size_t)c * q.kh * q.kw + i * q.kw + j) * q.co, *const b = g + ((size_t)(y - i) * q.ow + (x - j)) * q.co;
                    for (int o = 0; o < q.co && !isnan(sum); o += 8) {  // co is a multiple of 8 and both start on 16-byte boundaries
                        const Vec<T, 8> va = *reinterpret_cast<const Vec<T, 8>*>(a + o), vb = *reinterpret_cast<const Vec<T, 8>*>(b + o);
#pragma unroll
                        for (int k = 0; k < 8; k++) sum = fmaf(to_f32(va.v[k]), to_f32(vb.v[k]), sum);
                    }
                }
            row[32 * s] = from_f32<T>(sum);
        }
    }
}

enum TcMode {
    TC_STORE = 0,  // tensor stores of the rounded product or of f32 split-K partials
    TC_BIAS,       // fuse 1..3, tensor stores
    TC_PLAIN,      // d_plain: rows written by the warps; fuse 0 or 3
};

// BN_T: the tile's columns where they are 256, else 0 (from the parameters).  The ring of full-width tiles is four stages deep and waits
// out a round trip to L2 in them, so the single producer thread's own instructions between a freed stage and its refill count:
// with the geometry from the parameters the products of a 16384 x 8192 layer took 12 % longer at full clock.
// DRAIN (tiles of at most 128 columns): the accumulator is emptied every run_kb k-blocks into totals in registers, added with
// round-to-nearest, so that the pull of the tensor core's truncating additions stays that of one run whatever K is (see kRunMostF16).
// PANELS: TcParams::panels, an instantiation of its own for the same reason (as a branch of the common schedule it cost 4096^3 19 %).
//
// Epilogue warps for each quarter of the accumulator's lanes.  Rows that the warps write themselves take two (4096 x 2050 x 512 bf16: 25 us, 36
// with one), and so do tiles with a bias or an activation: their arithmetic is what a wave of few narrow tiles ends with (training step of two layers 1024 x 2048 x 2048 96.2 us, 94.5 so;
// 256 x 256 x 256 34.9, 33.9) and what full-width tiles of a short reduction wait for (8192 x 4096 x 512 with GELU 58.3 us, 46.9 so; 4096 x 4096 x 1024 39.5, 35.2); products that only leave
// through the copy engine gain nothing from a second one (16384 x 4096 x 256: 55 us, 50 with one; 128 x (384 x 384 x 64) and its gradients 31.1, 29.8).
constexpr int epi_warps(int mode, bool drain) { return mode == TC_PLAIN || (mode == TC_BIAS && !drain) ? 2 : 1; }
constexpr int tc_threads(int w) { return 32 * (2 + 4 * w); }
// CONV (TC_PLAIN): TcConvParams; an instantiation of its own for the producer's sake too.
template <int MODE, int BN_T, bool DRAIN = false, bool PANELS = false, bool CONV = false>
__global__ void __launch_bounds__(tc_threads(epi_warps(MODE, DRAIN)), 1)
tc_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_d,
               const __grid_constant__ CUtensorMap map_d2, std::conditional_t<CONV, TcConvParams, TcParams> p, int* err, int tag) {
    constexpr int W = epi_warps(MODE, DRAIN), CW = EPI_CHUNK_COLS / W;  // columns of a chunk that a warp has
    extern __shared__ unsigned char tc_smem_raw[];
    // 128-byte swizzled TMA tiles and UMMA descriptors want 1024-byte aligned bases
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)tc_smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t smem_base = smem_u32(smem);
    const uint32_t bar_base = smem_base + SmemLayout::bars;
    // barrier slots (8 bytes each): full[MAX_STAGES], empty[MAX_STAGES], tmem_full[2], tmem_empty[2]; then the TMEM base word
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (MAX_STAGES + s); };
    auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * MAX_STAGES + a); };
    auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * MAX_STAGES + 2 + a); };
    volatile uint32_t* tmem_base_slot = reinterpret_cast<volatile uint32_t*>(smem + SmemLayout::bars + 8 * (2 * MAX_STAGES + 4));

    int* const not_finite = reinterpret_cast<int*>(smem + SmemLayout::bars + 8 * (2 * MAX_STAGES + 5));  // CONV: a total of this CTA is not
    const int warp = warp_number(), lane = threadIdx.x & 31;
    const int bn = BN_T ? BN_T : p.bn, stages = BN_T ? STAGES : p.stages, stage_bytes = BN_T ? A_STAGE_BYTES + BN_T * BK * 2 : p.stage_bytes;

    if (threadIdx.x == 0) {
        if (CONV) *not_finite = 0;
        for (int s = 0; s < MAX_STAGES; s++) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(tfull_bar(a), 1);
            mbar_init(tempty_bar(a), 4 * W);
        }
        fence_barrier_init();
    }
    if (warp == 2 && elect_one()) {
        prefetch_map(&map_a);
        prefetch_map(&map_b);
        if (MODE != TC_PLAIN) prefetch_map(&map_d);
    }
    if (warp == 1) {  // the MMA warp owns the TMEM allocation
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
            const int ring = PANELS || p.b_keep ? p.num_kb : stages;
            int tm, tn, tb;
            for (int it = 0; ok && next_tile<PANELS>(it, p, tm, tn, tb); it++) {
                const int za = p.a_batched ? tb : 0, zb = p.b_batched ? tb : 0;
                int k = tb * p.split_kb * BK;              // a k-block past the end of K is all fill: zeros
                const bool load_b = PANELS ? tm == 0 || it == 0 : !p.b_keep || it == 0;  // a kept B panel arrives with its first tile's A blocks
                int cb = 0, ki = 0, kj = 0;  // CONV: k-block of the channels, tap
                for (int kb = 0; kb < p.num_kb; kb++, k += BK) {
                    if (!mbar_wait(empty_bar(stage), phase ^ 1, err, tag, 1)) {
                        ok = false;
                        break;
                    }
                    const uint32_t sa = smem_base + SmemLayout::ring + stage * stage_bytes, sb = sa + A_STAGE_BYTES;
                    if constexpr (CONV) {  // what lies outside an image, or behind the last channel of either operand, arrives as zeros
                        mbar_expect_tx(full_bar(stage), A_STAGE_BYTES + p.conv_rows * p.conv_w * BK * 2);
                        tma_load_3d(sa, &map_a, cb * BK, ki * p.conv_kw + kj, tm * BM, full_bar(stage));
                        tma_load_4d(sb, &map_b, cb * BK, p.conv_x - kj, tn * p.conv_rows + p.conv_y - ki, tb, full_bar(stage));
                        if (++cb == p.conv_cb) {
                            cb = 0;
                            if (++kj == p.conv_kw) {
                                kj = 0;
                                ki++;
                            }
                        }
                        if (++stage == ring) {
                            stage = 0;
                            phase ^= 1;
                        }
                        continue;
                    }
                    mbar_expect_tx(full_bar(stage), A_STAGE_BYTES + (load_b ? bn * BK * 2 : 0));
                    if (!p.a_mn) {
                        tma_load_3d(sa, &map_a, k, tm * BM, za, full_bar(stage));
                    } else {
#pragma unroll
                        for (int h = 0; h < BM / 64; h++) tma_load_3d(sa + h * MN_CHUNK_BYTES, &map_a, tm * BM + h * 64, k, za, full_bar(stage));
                    }
                    if (!load_b) {
                    } else if (!p.b_mn) {
                        tma_load_3d(sb, &map_b, k, tn * bn, zb, full_bar(stage));
                    } else {
#pragma unroll
                        for (int h = 0; h < bn / 64; h++) tma_load_3d(sb + h * MN_CHUNK_BYTES, &map_b, tn * bn + h * 64, k, zb, full_bar(stage));
                    }
                    if (++stage == ring) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            const uint32_t idesc = make_idesc(p.is_bf16 != 0, p.a_mn != 0, p.b_mn != 0, bn);
            // per-operand descriptor geometry: (leading, stride) byte offsets and the K step in 16-byte units
            const uint32_t a_lbo = p.a_mn ? MN_CHUNK_BYTES : 16, b_lbo = p.b_mn ? MN_CHUNK_BYTES : 16;
            const uint64_t a_kstep = p.a_mn ? (2048 >> 4) : (32 >> 4), b_kstep = p.b_mn ? (2048 >> 4) : (32 >> 4);
            int stage = 0, acc = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool ok = true;
            const int ring = PANELS || p.b_keep ? p.num_kb : stages;
            int tm, tn, tb;
            int run = 0;  // first k-block of the accumulator's run (DRAIN: a tile has several)
            for (int it = 0; ok && next_tile<PANELS>(it, p, tm, tn, tb); it += DRAIN && run ? 0 : 1) {
                if (!mbar_wait(tempty_bar(acc), acc_phase ^ 1, err, tag, 2)) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)acc * BN;
                const int run_end = DRAIN ? min(run + p.run_kb, p.num_kb) : p.num_kb;
                for (int kb = run; kb < run_end; kb++) {
                    if (!mbar_wait(full_bar(stage), phase, err, tag, 3)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sa = smem_base + SmemLayout::ring + stage * stage_bytes;
                    const uint64_t da = smem_desc_sw128(sa, a_lbo, 1024), db = smem_desc_sw128(sa + A_STAGE_BYTES, b_lbo, 1024);
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; k++) umma_f16(d_tmem, da + a_kstep * k, db + b_kstep * k, idesc, ((kb - run) | k) != 0);
                    umma_commit(empty_bar(stage));  // the stage may be refilled once these MMAs have read it
                    if (++stage == ring) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (!ok) break;
                umma_commit(tfull_bar(acc));  // accumulator complete
                if (DRAIN) run = run_end < p.num_kb ? run_end : 0;
                if (++acc == 2) {
                    acc = 0;
                    acc_phase ^= 1;
                }
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue (warps 2 to 5 or 9)
        // W warps share a quarter of the accumulator's lanes: each reads, rounds and stages its CW columns of a 64-column chunk, which
        // leaves as one copy.
        const int quarter = warp & 3;  // TMEM lanes [32 * quarter, 32 * quarter + 32)
        const int half = W == 2 ? (warp - 2) >> 2 : 0;
        const bool lead = half == 0 && lane == 0;  // the thread that hands a quarter's chunks to the copy engine
        unsigned char* stage_buf = smem + SmemLayout::epi + quarter * 2 * EPI_STAGE_BYTES;
        auto quarter_sync = [&] {
            if constexpr (W == 2) asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory");
            else __syncwarp();
        };
        int acc = 0, buf = 0;
        uint32_t acc_phase = 0;
        float fused_bias = 0.0f;
        if (MODE == TC_BIAS && p.fuse != 3) fused_bias = p.is_bf16 ? to_f32(*static_cast<const bf16*>(p.bias)) : to_f32(*static_cast<const f16*>(p.bias));
        int tm, tn, tb;
        for (int it = 0; next_tile<PANELS>(it, p, tm, tn, tb); it++) {
            // four or eight warps wait here for most of a tile's reduction: they sleep between polls, so that their polling does not
            // take shared-memory cycles from the TMA writes and the tensor core's operand reads
            if (MODE != TC_STORE && p.fuse == 3) {  // this thread's output row inside the batch's matrix
                const int row = tm * BM + quarter * 32 + lane;
                fused_bias = row < p.M ? (p.is_bf16 ? to_f32(static_cast<const bf16*>(p.bias)[row]) : to_f32(static_cast<const f16*>(p.bias)[row])) : 0.0f;
            }
            // The TMEM loads below take whole warps and the staging all warps of a quarter: these leave the loop together, two by a vote that each
            // of them reaches, its own wait being bounded.
            auto wait_accumulator = [&] {
                const bool ready = mbar_wait_relaxed(tfull_bar(acc), acc_phase, err, tag, 4, (unsigned)p.poll_ns);
                if constexpr (W == 2) {
                    uint32_t both;
                    __syncwarp();
                    asm volatile(
                        "{\n\t.reg .pred p, q;\n\t"
                        "setp.ne.u32 p, %2, 0;\n\t"
                        "barrier.cta.red.and.pred q, %1, 64, p;\n\t"
                        "selp.u32 %0, 1, 0, q;\n\t}"
                        : "=r"(both)
                        : "r"(1 + quarter), "r"((uint32_t)ready)
                        : "memory");
                    if (!both) return false;
                } else if (!__all_sync(0xFFFFFFFFu, ready)) {
                    return false;
                }
                tc_fence_after();
                return true;
            };
            if (!DRAIN && !wait_accumulator()) break;
            const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * BN + half * CW);
            const int rows_here = min(32, p.M - (tm * BM + quarter * 32));  // may be <= 0: this warp's rows lie below the matrix
            // Stages a warp's columns of a chunk (16-byte pieces, XOR-swizzled by the row); the chunk (first output column `col`) then goes to the copy
            // engine, or the warps write its rows themselves.
            auto flush = [&](const CUtensorMap* map, int col, const uint4 (&q)[CW / 8]) {
                if (lead) tma_store_wait_read<1>();  // the buffer's previous chunk has been read
                if (W == 2) __syncwarp();
                quarter_sync();
                unsigned char* src = stage_buf + buf * EPI_STAGE_BYTES;
#pragma unroll
                for (int j = 0; j < CW / 8; j++) *reinterpret_cast<uint4*>(src + lane * 128 + (((half * (CW / 8) + j) ^ (lane & 7)) << 4)) = q[j];
                if (MODE != TC_PLAIN) fence_proxy_async_smem();
                quarter_sync();
                buf ^= 1;
                if constexpr (MODE != TC_PLAIN) {
                    if (lead) {
                        tma_store_3d(map, smem_u32(src), col, tm * BM + quarter * 32, tb);
                        tma_store_commit();
                    }
                } else {
                    const int width = CONV ? p.conv_rows * p.conv_w : bn;  // columns from one tile to the next
                    store_rows(static_cast<uint16_t*>(p.d) + ((size_t)tb * p.M + tm * BM + quarter * 32) * p.N + tn * width, (size_t)p.N, half * 16, rows_here,
                               min(width, p.N - tn * width), (col - tn * bn) / 64, src, stage_buf + buf * EPI_STAGE_BYTES, lane);
                }
            };
            auto pack = [&](const float (&e)[CW], uint4 (&q)[CW / 8]) {
#pragma unroll
                for (int j = 0; j < CW / 8; j++)
                    q[j] = make_uint4(pack2(e[8 * j], e[8 * j + 1], p.is_bf16), pack2(e[8 * j + 2], e[8 * j + 3], p.is_bf16), pack2(e[8 * j + 4], e[8 * j + 5], p.is_bf16),
                                      pack2(e[8 * j + 6], e[8 * j + 7], p.is_bf16));
            };
            auto store_chunk = [&](int c, const uint32_t (&v)[CW / 32][32]) {
                const int col = tn * bn + c * EPI_CHUNK_COLS;
                if constexpr (MODE == TC_STORE) {
                    static_assert(W == 1, "f32 results: a warp stages both halves of a chunk");
                    if (p.out_f32) {
                        // two 32-column f32 chunks (128 bytes per row each), one per staging buffer
#pragma unroll
                        for (int h = 0; h < CW / 32; h++) {
                            if (lane == 0) tma_store_wait_read<1>();
                            __syncwarp();
                            unsigned char* src = stage_buf + buf * EPI_STAGE_BYTES;
#pragma unroll
                            for (int j = 0; j < 8; j++)
                                *reinterpret_cast<uint4*>(src + lane * 128 + ((j ^ (lane & 7)) << 4)) = make_uint4(v[h][4 * j], v[h][4 * j + 1], v[h][4 * j + 2], v[h][4 * j + 3]);
                            fence_proxy_async_smem();
                            __syncwarp();
                            if (lane == 0) {
                                tma_store_3d(&map_d, smem_u32(src), col + h * 32, tm * BM + quarter * 32, tb);
                                tma_store_commit();
                            }
                            buf ^= 1;
                        }
                        return;
                    }
                }
                float e[CW];
                uint4 q[CW / 8];
#pragma unroll
                for (int j = 0; j < CW; j++) e[j] = __uint_as_float(v[j / 32][j % 32]);
                if constexpr (MODE == TC_BIAS) {
                    // Linear + bias (+ GELU) in one pass: bit for bit what cuda_matmul, cuda_add and cuda_gelu give one after the other.
                    const bool gelu = p.fuse == 2;
                    if (p.is_bf16) gelu ? bias_gelu<bf16, true>(e, fused_bias, q) : bias_gelu<bf16, false>(e, fused_bias, q);
                    else gelu ? bias_gelu<f16, true>(e, fused_bias, q) : bias_gelu<f16, false>(e, fused_bias, q);
                    flush(&map_d, col, q);
                    if (gelu) {
                        pack(e, q);
                        flush(&map_d2, col, q);
                    }
                } else {
                    if (MODE == TC_PLAIN && p.fuse) {
                        if (p.is_bf16) bias_gelu<bf16, false>(e, fused_bias, q);
                        else bias_gelu<f16, false>(e, fused_bias, q);
                    } else {
                        pack(e, q);
                    }
                    if constexpr (CONV) {  // columns behind the tile's pixels hold what the ring and the accumulator held before
                        const int mine = p.conv_rows * p.conv_w - c * EPI_CHUNK_COLS - half * CW;
                        F32x2 zero[4] = {twice(0.0f), twice(0.0f), twice(0.0f), twice(0.0f)};  // NaN from the first total on that is not finite
                        if (mine >= CW) {
#pragma unroll
                            for (int j = 0; j < CW; j += 2) zero[j / 2 % 4] = fma2(pair_of(make_float2(e[j], e[j + 1])), twice(0.0f), zero[j / 2 % 4]);
                        } else {
#pragma unroll
                            for (int j = 0; j < CW; j += 2) zero[j / 2 % 4] = fma2(pair_of(make_float2(j < mine ? e[j] : 0.0f, j + 1 < mine ? e[j + 1] : 0.0f)), twice(0.0f), zero[j / 2 % 4]);
                        }
                        const float2 z = halves(zero[0] + zero[1] + (zero[2] + zero[3]));
                        if (z.x + z.y != 0.0f) *not_finite = 1;
                    }
                    flush(&map_d, col, q);
                }
            };
            auto load_chunk = [&](uint32_t at, uint32_t (&v)[CW / 32][32]) {
#pragma unroll
                for (int h = 0; h < CW / 32; h++) tmem_ld_32x32b_x32(at + h * 32, v[h]);
            };
            auto wait_chunk = [&](uint32_t (&v)[CW / 32][32]) {
                tmem_ld_wait_for(v[0]);
                if constexpr (CW > 32) reg_fence(v[CW / 32 - 1]);
            };
            // The TMEM loads of chunk c + 1 are in flight while chunk c is converted and stored.
            const int chunks = CONV ? (bn + EPI_CHUNK_COLS - 1) / EPI_CHUNK_COLS : bn / EPI_CHUNK_COLS;
            auto hand_back = [&] {  // every TMEM read of this accumulator is done: hand it back to the MMA warp
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty_bar(acc));
            };
            if constexpr (DRAIN) {
                uint32_t total[2][CW / 32][32], v[32];  // tiles of at most 128 columns
#pragma unroll
                for (int c = 0; c < 2 * CW; c++) total[c / CW][c % CW / 32][c % 32] = 0;  // 0.0f
                bool ok = true;
                for (int run = 0; run < p.num_kb && ok; run += p.run_kb) {
                    ok = wait_accumulator();
                    if (!ok) break;
                    const uint32_t t_run = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * BN + half * CW);
#pragma unroll
                    for (int c = 0; c < 2; c++) {
                        if (c >= chunks) break;
#pragma unroll
                        for (int h = 0; h < CW / 32; h++) {
                            tmem_ld_32x32b_x32(t_run + c * EPI_CHUNK_COLS + h * 32, v);
                            tmem_ld_wait_for(v);
#pragma unroll
                            for (int j = 0; j < 32; j++) total[c][h][j] = __float_as_uint(__uint_as_float(total[c][h][j]) + __uint_as_float(v[j]));
                        }
                    }
                    hand_back();
                    if (++acc == 2) {
                        acc = 0;
                        acc_phase ^= 1;
                    }
                }
                if (!ok) break;
                store_chunk(0, total[0]);
                if (chunks > 1) store_chunk(1, total[1]);
                continue;
            }
            uint32_t va[CW / 32][32], vb[CW / 32][32];
            load_chunk(t_row, va);
#pragma unroll
            for (int c = 0; c < BN / EPI_CHUNK_COLS; c += 2) {
                if (c >= chunks) break;
                wait_chunk(va);
                if (c + 1 < chunks) load_chunk(t_row + (c + 1) * EPI_CHUNK_COLS, vb);
                else hand_back();
                store_chunk(c, va);
                if (c + 1 >= chunks) break;
                wait_chunk(vb);
                if (c + 2 < chunks) load_chunk(t_row + (c + 2) * EPI_CHUNK_COLS, va);
                else hand_back();
                store_chunk(c + 1, vb);
            }
            if (++acc == 2) {
                acc = 0;
                acc_phase ^= 1;
            }
        }
        // the staging has been read; the writes themselves belong to the launch, and what follows it waits for them
        if (lane == 0) tma_store_wait_read<0>();
    }

    // common exit: TMEM is released by the warp that allocated it, after everyone is done with it
    tc_fence_before();
    __syncthreads();
    if (tc_err_mine(err, tag)) {
        // a wait gave up: give bulk copies still in flight towards this CTA's shared memory time to land
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
    if constexpr (CONV) {
        if (!*not_finite) return;
        int tm, tn, tb;
        for (int it = 0; next_tile<PANELS>(it, p, tm, tn, tb); it++) {
            const int width = p.conv_rows * p.conv_w;
            const uint16_t* g = static_cast<const uint16_t*>(p.conv_g) + (size_t)tb * p.conv_oh * p.conv_ow * p.conv_co;
            const ConvRedo q = {g, p.conv_wt, static_cast<uint16_t*>(p.d) + (size_t)tb * p.M * p.N, min(BM, p.M - tm * BM), min(width, p.N - tn * width), tm * BM, tn * width, p.N, p.conv_w, p.conv_x, p.conv_y,
                                p.conv_kh, p.conv_kw, p.conv_co, p.conv_oh, p.conv_ow};
            if (p.is_bf16) conv_redo<bf16>(q);
            else conv_redo<f16>(q);
        }
    }
}

// ---------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------
// [rows, cols] row-major 16-bit matrix, box = box_rows x 64 columns, 128-byte swizzle
bool make_map(CUtensorMap* map, bool is_bf16, const void* base, uint64_t rows, uint64_t cols, uint64_t batch, uint64_t batch_stride, uint32_t box_rows) {
    return make_map_3d(map, is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, base, rows, cols, batch, batch_stride, box_rows);
}

bool opt_in_shared_memory() {
    static std::mutex mu;
    static bool done[64] = {false};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    std::lock_guard<std::mutex> lock(mu);
    if (!done[dev]) {
        for (auto kernel : {tc_gemm_kernel<TC_STORE, BN>, tc_gemm_kernel<TC_BIAS, BN>, tc_gemm_kernel<TC_STORE, 0>, tc_gemm_kernel<TC_BIAS, 0>, tc_gemm_kernel<TC_PLAIN, 0>, tc_gemm_kernel<TC_STORE, BN, false, true>, tc_gemm_kernel<TC_BIAS, BN, false, true>,
                            tc_gemm_kernel<TC_STORE, 0, true>, tc_gemm_kernel<TC_BIAS, 0, true>, tc_gemm_kernel<TC_PLAIN, 0, true>})
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM_BYTES) != cudaSuccess) {
                cudaGetLastError();
                return false;
            }
        if (cudaFuncSetAttribute(tc_gemm_kernel<TC_PLAIN, 0, false, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM_BYTES) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        done[dev] = true;
    }
    return true;
}

int poll_ns(int num_kb) { return std::max(20, std::min(400, 10 * num_kb)); }

// D[M,N] = sum_k Aop[m,k] * Bop[n,k].  A K-major operand is a dense row-major [MN, K] matrix, an
// MN-major operand a dense row-major [K, MN] matrix; D is dense row-major [M, N].
// fuse: 0 plain product; 1 D = round(round(product) + bias); 2 also D2 = round(gelu(D)) (see the kernel's epilogue)
std::atomic<int> g_keep_b{1};  // 0: the B-panel-resident schedule is never taken (tests, A/B timing)

// CTAs per column tile of the schedule that keeps the B panel of a column tile in shared memory (0 = general schedule).
// Taken when the whole reduction fits the ring (K <= STAGES * BK), there is one batch, and every CTA gets at least four
// row tiles to spread the panel's load over.  With K = 256 a 128 x 256 tile otherwise loads 192 KB to do 2048 cycles
// of tensor work; with the panel resident it loads the 64 KB of A.
int keep_b_ctas(int tiles_m, int tiles_n, int num_kb, int batch, int ctas) {
    if (!g_keep_b.load(std::memory_order_relaxed) || batch != 1 || num_kb > STAGES || tiles_n > ctas) return 0;
    const int per_col = ctas / tiles_n;
    return tiles_m >= 4 * per_col ? per_col : 0;
}

// The same for a batch whose products share A, with five row tiles and more to a panel and enough tiles that the runs' ends do not count.  General schedule /
// panels, bf16, us: A shared 64 x (2304 x 3136 x 256) 316 / 266, 64 x (2304 x 784 x 256) 93 / 80, 300 x (520 x 256 x 256) 36 / 33.  Four row tiles gain nothing (160 x (512 x
// 512 x 256) 32.6 / 33.3), nor does what loads little of B (64 x (1152 x 3136 x 128) 114 / 125, 128 x (1024 x 1024 x 64) 57 / 59), and an A of its own
// for each product is read again for every panel by CTAs that are batches apart (64 x (2304 x 3136 x 256) 285 / 365, 160 x (512 x 512 x 256) 34.6 / 39.5).
bool keep_panels(uint64_t tiles_m, uint64_t tiles_n, int num_kb, uint64_t batch, bool a_shared, int ctas) {
    return g_keep_b.load(std::memory_order_relaxed) && batch > 1 && a_shared && num_kb == STAGES && tiles_m >= 5 && tiles_m * tiles_n * batch >= 8 * (uint64_t)ctas;
}
thread_local int t_last_schedule = 0;  // of the thread's last launch of this kernel: 1 = one B panel kept, 2 = panels of a batch, 0 = general (tests)

// The two-CTA kernel: B is staged in halves of 128 columns, a pair of CTAs owns a 256 x 256 tile.  Its split-K slices are
// sub-matrices behind the third coordinate of the tensor maps.  false: nothing was launched.
bool launch_two_cta(bool is_bf16, const TcProduct& c, void* D, const char* where, int grid) {
    const uint64_t M = c.m, N = c.n;
    uint64_t K = c.k, batch = c.batch, a_bs = (uint64_t)c.a_bs, b_bs = (uint64_t)c.b_bs, a_pitch = 0, b_pitch = 0;
    const int tiles_m = (int)((M + BM - 1) / BM), tiles_n = (int)((N + BN - 1) / BN);
    const int slices = batch == 1 ? splitk_slices((uint64_t)tiles_m * tiles_n, K, BK, grid) : 1;
    float* partial = nullptr;
    if (slices > 1) {
        partial = static_cast<float*>(scratch((size_t)slices * M * N * sizeof(float)));
        if (!partial) return false;
        const uint64_t Ks = K / slices;
        a_pitch = c.a_mn ? M : K;  // rows keep the pitch of the whole matrix
        b_pitch = c.b_mn ? N : K;
        a_bs = c.a_mn ? Ks * M : Ks;  // MN-major: Ks rows further; K-major: Ks columns further
        b_bs = c.b_mn ? Ks * N : Ks;
        K = Ks;
        batch = (uint64_t)slices;
    }
    int tag = 0;
    int* err = next_launch_error_word(&tag);
    if (!err) return false;
    const CUtensorMapDataType t16 = is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    const CUtensorMapSwizzle sw = CU_TENSOR_MAP_SWIZZLE_128B;
    CUtensorMap ma, mb, md;
    const bool oka = c.a_mn ? make_map_3d(&ma, t16, 2, c.A, K, M, batch, a_bs, 64, sw, a_pitch) : make_map_3d(&ma, t16, 2, c.A, M, K, batch, a_bs, tc2::BM, sw, a_pitch);
    const bool okb = c.b_mn ? make_map_3d(&mb, t16, 2, c.B, K, N, batch, b_bs, 64, sw, b_pitch) : make_map_3d(&mb, t16, 2, c.B, N, K, batch, b_bs, tc2::BN_HALF, sw, b_pitch);
    const bool okd = partial ? make_map_3d(&md, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, partial, M, N, batch, M * N, 32) : make_map(&md, is_bf16, D, M, N, batch, M * N, 32);
    if (!oka || !okb || !okd) return false;
    tc2::Params q;
    q.tile_pairs_m = (tiles_m + 1) / 2;
    q.tiles_n = tiles_n;
    q.tiles_per_batch = q.tile_pairs_m * q.tiles_n;
    q.num_tiles = (int)batch * q.tiles_per_batch;
    q.num_kb = (int)((K + BK - 1) / BK);
    q.a_batched = (batch > 1 && a_bs != 0) ? 1 : 0;
    q.b_batched = (batch > 1 && b_bs != 0) ? 1 : 0;
    q.is_bf16 = is_bf16 ? 1 : 0;
    q.out_f32 = partial ? 1 : 0;
    q.a_mn = c.a_mn ? 1 : 0;
    q.b_mn = c.b_mn ? 1 : 0;
    if (!tc2::launch(ma, mb, md, q, grid, err, tag, ctx().stream)) return false;
    check_launch(where);
    if (partial) splitk_reduce(is_bf16 ? 0 : 1, partial, slices, M, N, N, D, where);
    return true;
}

int ring_stages(int bn) { return std::min(MAX_STAGES, STAGES * (A_STAGE_BYTES + B_STAGE_BYTES) / (A_STAGE_BYTES + bn * BK * 2)); }
// k-blocks of tensor-core time (M128 N256 K64: 512 cycles) that one k-block of a bn-wide tile takes: the columns' share; the
// operand reads from shared memory (a k-step of N64 needs 48 cycles for its 6 KB, 32 for its multiplications); or the ring, whose
// stages all wait out one round trip to L2 of about 1.2 us.  The four stages of 192 columns do not: measured, 0.212 us a k-block
// against 0.306 of a 256-wide tile, 0.27 with B MN-major (a copy for each 64 columns); 128 columns 0.200.
double kb_cost(int bn, bool b_mn) {
    if (bn == 192) return b_mn ? 0.87 : 0.70;
    if (bn == 128 && !b_mn) return 0.65;
    return std::max(std::max(bn / 256.0, (128 + bn) / 512.0), 4.4 / ring_stages(bn));
}
// Columns of an output tile.  256 feeds the tensor core best, so narrower tiles are for products that 256-wide tiles serve
// badly: an N that fills its last tile poorly (N = 64 would compute 256 columns, N = 384 512) or too few tiles to reach every
// SM.  The estimate is in k-blocks of a 256-wide tile: a wave's reduction, and its epilogue in proportion to the columns.
// From two waves of 256-wide tiles on only the columns count, and all that narrow tiles load besides: at the power cap a
// part-filled last wave costs nothing (12856 x 2856 x 760 58 us, 65 on tiles of 192).
// bf16 512 x 1024 x 1024 (64 tiles of 64 columns instead of 16): 8.7 us, 10.0 on full-width tiles;
// 4096 x 1536 x 1024 (256 of 192 columns instead of 192) 13.1, 15.4; 2432 x 1008 x 1504 with B MN-major 11.6, 15.3.
double tile_cost(int bn, bool b_mn, uint64_t tiles_m, uint64_t N, uint64_t batch, uint64_t num_kb, int grid) {
    const uint64_t tiles = tiles_m * ((N + bn - 1) / bn) * batch, tiles_256 = tiles_m * ((N + 255) / 256) * batch;
    const double epilogue = 3.0 * bn / 256.0;
    if (tiles_256 > 2 * (uint64_t)grid) return (double)tiles / grid * ((double)num_kb * std::max((128 + bn) / 512.0, 4.4 / ring_stages(bn)) + epilogue);
    return (double)((tiles + grid - 1) / grid) * ((double)num_kb * kb_cost(bn, b_mn) + epilogue);
}
int tile_columns(bool b_mn, uint64_t tiles_m, uint64_t N, uint64_t batch, uint64_t num_kb, int grid) {
    int best = 256;
    for (int bn : {192, 128, 64})
        if (tile_cost(bn, b_mn, tiles_m, N, batch, num_kb, grid) < 0.93 * tile_cost(best, b_mn, tiles_m, N, batch, num_kb, grid)) best = bn;
    return best;
}

bool launch_gemm(bool is_bf16, const TcProduct& c, void* D, const char* where, int fuse = 0, const void* bias = nullptr, void* D2 = nullptr) {
    const void *A = c.A, *B = c.B;
    const bool a_mn = c.a_mn, b_mn = c.b_mn;
    const uint64_t M = c.m, N = c.n;
    const uint64_t K = c.k;
    uint64_t batch = c.batch;
    if (!opt_in_shared_memory()) return false;
    int grid = sm_count();
    if (ctx().gemm_sm_limit > 0 && ctx().gemm_sm_limit < grid) grid = ctx().gemm_sm_limit;
    const CUtensorMapDataType t16 = is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    const CUtensorMapSwizzle sw = CU_TENSOR_MAP_SWIZZLE_128B;
    CUtensorMap ma, mb, md;
    if (g_two_cta.load(std::memory_order_relaxed) && grid >= 2 && !fuse && !c.a_pitch && !c.b_pitch && !c.d_plain)
        if (launch_two_cta(is_bf16, c, D, where, grid)) return true;
    TcParams p;
    p.M = (int)M;
    p.N = (int)N;
    p.K = (int)K;
    p.tiles_m = (int)((M + BM - 1) / BM);
    p.num_kb = (int)((K + BK - 1) / BK);
    p.split_kb = 0;
    p.bn = N < 192 ? (int)((N + 63) / 64 * 64) : BN;
    p.tiles_n = (int)((N + p.bn - 1) / p.bn);
    p.b_keep = keep_b_ctas(p.tiles_m, p.tiles_n, p.num_kb, (int)batch, std::min(grid, (int)std::min<uint64_t>(batch * p.tiles_m * p.tiles_n, 1u << 30)));
    // few output tiles: cut K into slices that run as the batches of this launch
    int slices = 1;
    const int bn_whole = p.b_keep ? p.bn : tile_columns(b_mn, (uint64_t)p.tiles_m, N, batch, (uint64_t)p.num_kb, grid);
    const bool panels = p.bn == BN && bn_whole == BN && !c.d_plain && keep_panels((uint64_t)p.tiles_m, (uint64_t)p.tiles_n, p.num_kb, batch, c.a_bs == 0, grid);
    if (batch == 1 && !fuse && !p.b_keep) {
        slices = splitk_slices((uint64_t)p.tiles_m * p.tiles_n, K, BK, grid);
        if (slices == 1)
            slices = splitk_short((uint64_t)p.tiles_m * p.tiles_n, (uint64_t)p.num_kb, grid, kb_cost(p.bn, b_mn),
                                  tile_cost(bn_whole, b_mn, (uint64_t)p.tiles_m, N, batch, (uint64_t)p.num_kb, grid) - kSplitFixed16);
    }
    StreamWorkspace partial;
    const uint64_t n_pitch = (N + 3) / 4 * 4;
    if (slices > 1 && !partial.take((size_t)slices * M * n_pitch * sizeof(float), true)) slices = 1;
    if (slices > 1) {
        p.split_kb = (p.num_kb + slices - 1) / slices;
        p.num_kb = p.split_kb;
        batch = (uint64_t)slices;
    } else if (!p.b_keep) {
        p.bn = bn_whole;
        p.tiles_n = (int)((N + p.bn - 1) / p.bn);
    }
    p.run_kb = c.nearest ? (is_bf16 ? kRunMostBf16 : kRunMostF16) / BK : 0;
    const bool drain = p.run_kb && p.num_kb > p.run_kb;
    if (drain && p.bn > 128) {
        p.bn = 128;
        p.tiles_n = (int)((N + p.bn - 1) / p.bn);
    }
    p.tiles_per_batch = p.tiles_m * p.tiles_n;
    p.stages = ring_stages(p.bn);
    p.stage_bytes = A_STAGE_BYTES + p.bn * BK * 2;
    int tag = 0;
    int* err = next_launch_error_word(&tag);
    if (!err) return false;
    const uint64_t a_bs = (uint64_t)c.a_bs, b_bs = (uint64_t)c.b_bs;
    const bool oka = a_mn ? make_map_3d(&ma, t16, 2, A, K, M, c.batch, a_bs, 64, sw, c.a_pitch) : make_map_3d(&ma, t16, 2, A, M, K, c.batch, a_bs, BM, sw, c.a_pitch);
    const bool okb = b_mn ? make_map_3d(&mb, t16, 2, B, K, N, c.batch, b_bs, 64, sw, c.b_pitch) : make_map_3d(&mb, t16, 2, B, N, K, c.batch, b_bs, (uint32_t)p.bn, sw, c.b_pitch);
    if (!oka || !okb) return false;
    p.d_plain = slices > 1 ? 0 : c.d_plain;
    p.d = D;
    if (slices > 1) {
        if (!make_map_3d(&md, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, partial.ptr, M, N, batch, M * n_pitch, 32, sw, n_pitch)) return false;
    } else if (p.d_plain) {
        md = ma;  // not used
    } else if (!make_map(&md, is_bf16, D, M, N, batch, M * N, 32)) {
        return false;
    }
    CUtensorMap md2 = md;
    if (fuse == 2 && !make_map(&md2, is_bf16, D2, M, N, batch, M * N, 32)) return false;
    p.fuse = fuse;
    p.bias = bias;
    p.group_m = g_group_m.load(std::memory_order_relaxed);
    p.num_tiles = (int)batch * p.tiles_per_batch;
    p.a_batched = (c.batch > 1 && a_bs != 0) ? 1 : 0;
    p.b_batched = (c.batch > 1 && b_bs != 0) ? 1 : 0;
    p.is_bf16 = is_bf16 ? 1 : 0;
    p.out_f32 = slices > 1 ? 1 : 0;
    p.a_mn = a_mn ? 1 : 0;
    p.b_mn = b_mn ? 1 : 0;
    if (grid > p.num_tiles) grid = p.num_tiles;
    if (p.b_keep) grid = p.b_keep * p.tiles_n;
    p.poll_ns = poll_ns(p.num_kb);
    t_last_schedule = panels ? 2 : p.b_keep ? 1 : 0;
    const bool full = p.bn == BN;
    const auto kernel = panels ? (fuse ? tc_gemm_kernel<TC_BIAS, BN, false, true> : tc_gemm_kernel<TC_STORE, BN, false, true>)
                        : drain ? (p.d_plain ? tc_gemm_kernel<TC_PLAIN, 0, true> : (fuse ? tc_gemm_kernel<TC_BIAS, 0, true> : tc_gemm_kernel<TC_STORE, 0, true>))
                        : p.d_plain ? tc_gemm_kernel<TC_PLAIN, 0>
                                  : (fuse ? (full ? tc_gemm_kernel<TC_BIAS, BN> : tc_gemm_kernel<TC_BIAS, 0>) : (full ? tc_gemm_kernel<TC_STORE, BN> : tc_gemm_kernel<TC_STORE, 0>));
    const int warps = epi_warps(p.d_plain ? TC_PLAIN : fuse ? TC_BIAS : TC_STORE, drain);
    launch_kernel(kernel, grid, tc_threads(warps), TC_SMEM_BYTES, ctx().stream, ma, mb, md, md2, p, err, tag);
    check_launch(where);
    if (slices > 1) splitk_reduce(is_bf16 ? 0 : 1, static_cast<const float*>(partial.ptr), slices, M, N, n_pitch, D, where);
    return true;
}

}  // namespace

// ---------------------------------------------------------------------------------
// shared host helpers (declared in tc_ptx.cuh)
// ---------------------------------------------------------------------------------
namespace tc {

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

bool make_map_2d(CUtensorMap* map, CUtensorMapDataType type, int elem_bytes, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) return false;
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {cols * (uint64_t)elem_bytes};
    cuuint32_t box[2] = {(cuuint32_t)(128 / elem_bytes), box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, type, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

bool make_map_3d(CUtensorMap* map, CUtensorMapDataType type, int elem_bytes, const void* base, uint64_t rows, uint64_t cols, uint64_t batch,
                 uint64_t batch_stride, uint32_t box_rows, CUtensorMapSwizzle swizzle, uint64_t pitch) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) return false;
    if (pitch == 0) pitch = cols;
    const bool bcast = batch_stride == 0 || batch <= 1;
    cuuint64_t dims[3] = {cols, rows, bcast ? 1 : batch};
    cuuint64_t strides[2] = {pitch * (uint64_t)elem_bytes, (bcast ? rows * pitch : batch_stride) * (uint64_t)elem_bytes};
    cuuint32_t box[3] = {(cuuint32_t)(128 / elem_bytes), box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(map, type, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

int splitk_slices(uint64_t tiles, uint64_t K, int block_k, int sms) {
    if (tiles == 0 || tiles * 2 > (uint64_t)sms || K % block_k != 0 || K < 4096) return 1;
    const uint64_t kb = K / block_k;
    // Cost in units of one k-block of tensor-core time per CTA: every wave runs kb / s k-blocks plus about 12 for the
    // pipeline fill and the f32 epilogue of a tile, and the second pass reads s partial tiles per output tile.
    auto cost = [&](uint64_t s) {
        const uint64_t t = tiles * s, waves = (t + sms - 1) / sms;
        return (double)waves * ((double)kb / (double)s + 12.0) + 0.07 * (double)t;
    };
    int best = 1;
    double best_cost = cost(1);
    for (int s = 2; s <= 64; s++) {
        if (kb % s != 0 || K / s < 512) continue;
        const double c = cost((uint64_t)s);
        if (c < best_cost * 0.97) {
            best_cost = c;
            best = s;
        }
    }
    return best;
}

int splitk_short(uint64_t tiles, uint64_t num_kb, int sms, double kb_cost, double below) {
    if (tiles == 0 || tiles * 2 > (uint64_t)sms) return 1;
    int best = 1;
    for (uint64_t s = 2; s * tiles <= (uint64_t)sms && s * 2 <= num_kb && s <= 32; s++) {
        const uint64_t per = (num_kb + s - 1) / s;
        if ((num_kb + per - 1) / per != s) continue;  // the last slices would be empty
        const double cost = (double)per * kb_cost + 0.1 * (double)s;
        if (cost < below) {
            below = cost;
            best = (int)s;
        }
    }
    return best;
}

// `vec` elements per step: 4 when the output's rows are whole vectors (then rows and padded rows coincide), else 1.
template <class T, int VEC>
__global__ void __launch_bounds__(256) splitk_reduce_kernel(const float* partial, int slices, size_t rows, uint32_t cols, uint32_t pitch, FastDiv div,
                                                            T* out, Gate gate, int shut_slices) {
    after_previous_kernel();
    if (gate.shut()) slices = shut_slices;
    if (!slices) return;
    const size_t nvec = rows * cols / VEC, stride = (size_t)gridDim.x * 256, slice = rows * pitch;
    for (size_t v = (size_t)blockIdx.x * 256 + threadIdx.x; v < nvec; v += stride) {
        size_t src = VEC * v;
        if constexpr (VEC == 1) {
            const uint32_t r = div.div((uint32_t)v);
            src = (size_t)r * pitch + ((uint32_t)v - r * cols);
        }
        float acc[VEC];
        *reinterpret_cast<Vec<float, VEC>*>(acc) = *reinterpret_cast<const Vec<float, VEC>*>(partial + src);
        for (int s = 1; s < slices; s++) {
            const Vec<float, VEC> q = *reinterpret_cast<const Vec<float, VEC>*>(partial + (size_t)s * slice + src);
#pragma unroll
            for (int j = 0; j < VEC; j++) acc[j] += q.v[j];
        }
        Vec<T, VEC> o;
#pragma unroll
        for (int j = 0; j < VEC; j++) {
            if constexpr (std::is_same<T, float>::value) o.v[j] = acc[j];
            else o.v[j] = from_f32<T>(acc[j]);
        }
        *reinterpret_cast<Vec<T, VEC>*>(out + VEC * v) = o;
    }
}

template <class T>
static void splitk_reduce_t(const float* partial, int slices, uint64_t rows, uint64_t cols, uint64_t pitch, void* out, const Gate& gate, int shut_slices) {
    const bool vec = cols == pitch && reinterpret_cast<uintptr_t>(out) % (4 * sizeof(T)) == 0;
    size_t blocks = (rows * cols / (vec ? 4 : 1) + 255) / 256;
    const size_t cap = (size_t)sm_count() * 8;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    const FastDiv div((uint32_t)cols);
    if (vec) launch_kernel(splitk_reduce_kernel<T, 4>, (unsigned)blocks, 256, 0, ctx().stream, partial, slices, rows, (uint32_t)cols, (uint32_t)pitch, div, static_cast<T*>(out), gate, shut_slices);
    else launch_kernel(splitk_reduce_kernel<T, 1>, (unsigned)blocks, 256, 0, ctx().stream, partial, slices, rows, (uint32_t)cols, (uint32_t)pitch, div, static_cast<T*>(out), gate, shut_slices);
}

void splitk_reduce(int dtype, const float* partial, int slices, uint64_t rows, uint64_t cols, uint64_t pitch, void* out, const char* where, const Gate* behind, int shut_slices) {
    const Gate gate = behind ? *behind : Gate();
    if (dtype == 0) splitk_reduce_t<bf16>(partial, slices, rows, cols, pitch, out, gate, shut_slices);
    else if (dtype == 1) splitk_reduce_t<f16>(partial, slices, rows, cols, pitch, out, gate, shut_slices);
    else splitk_reduce_t<float>(partial, slices, rows, cols, pitch, out, gate, shut_slices);
    check_launch(where);
}

// Rows of `cols` elements, dense and starting anywhere, copied to rows of `pitch` elements (a multiple of 128 bytes): one
// 16-byte vector of a destination row per thread and step, assembled from the one or two aligned 16-byte words of the
// source it straddles.  The words read all hold at least one element of the vector, so nothing outside the aligned words
// of the source's own elements is touched.  Bound by HBM (or L2): reads and writes the operand once.  Both operands of a product in one launch.
template <class W>
struct RowCopy {
    const W* in;
    W* out;
    uint32_t vecs;  // 0: nothing to copy
    FastDiv per_row;
    uint32_t cols, pitch;
};
constexpr int kCopyUnroll = 4;  // vectors a thread has in flight ([4099, 1543] bf16 4.5 us, 5.6 with one)
template <class W>
__device__ __forceinline__ void repack_vectors(const RowCopy<W>& p, uint32_t v0) {
    constexpr uint32_t VEC = 16 / sizeof(W);
    uint4 lo[kCopyUnroll], hi[kCopyUnroll];
    uint32_t sh[kCopyUnroll];
    W* to[kCopyUnroll];
#pragma unroll
    for (int u = 0; u < kCopyUnroll; u++) {
        const uint32_t v = v0 + u * 256;
        to[u] = nullptr;
        if (v >= p.vecs) continue;
        uint32_t row, c;
        p.per_row.divmod(v, row, c);
        c *= VEC;
        const uint32_t need = min(VEC, p.cols - c) * (uint32_t)sizeof(W);
        const uintptr_t src = reinterpret_cast<uintptr_t>(p.in + (size_t)row * p.cols + c);
        sh[u] = (uint32_t)(src & 15);
        const uint4* words = reinterpret_cast<const uint4*>(src - sh[u]);
        lo[u] = words[0];
        hi[u] = make_uint4(0, 0, 0, 0);
        if (sh[u] + need > 16) hi[u] = words[1];
        to[u] = p.out + (size_t)row * p.pitch + c;
    }
#pragma unroll
    for (int u = 0; u < kCopyUnroll; u++) {
        if (!to[u]) continue;
        uint32_t w[8] = {lo[u].x, lo[u].y, lo[u].z, lo[u].w, hi[u].x, hi[u].y, hi[u].z, hi[u].w};
        uint4 r;
        const uint32_t bits = (sh[u] & 3) * 8;
#pragma unroll
        for (int k = 0; k < 2; k++)  // word-wise shift by sh / 4 in two steps with compile-time indices
#pragma unroll
            for (int i = 0; i < 8; i++)
                if ((sh[u] >> 2) & (2 >> k)) w[i] = i + (2 >> k) < 8 ? w[i + (2 >> k)] : 0;
        r.x = __funnelshift_r(w[0], w[1], bits);
        r.y = __funnelshift_r(w[1], w[2], bits);
        r.z = __funnelshift_r(w[2], w[3], bits);
        r.w = __funnelshift_r(w[3], w[4], bits);
        *reinterpret_cast<uint4*>(to[u]) = r;
    }
}
template <class W>
__global__ void __launch_bounds__(256) repack_rows_kernel(RowCopy<W> a, RowCopy<W> b, Gate gate, uint32_t a_blocks) {
    after_previous_kernel();
    if (gate.shut()) return;
    if (blockIdx.x < a_blocks) repack_vectors(a, blockIdx.x * 256 * kCopyUnroll + threadIdx.x);
    else repack_vectors(b, (blockIdx.x - a_blocks) * 256 * kCopyUnroll + threadIdx.x);
}

// Elements between the rows of a copy.  Whole 128-byte lines, so that a tensor copy's 128-byte box rows read one line each and
// not parts of two (bf16 100000 x 3 x 257: 19 us, 40 with the 257 rows of three elements 16 bytes apart); where rows shorter than a line would
// make that much memory, the 16-byte multiple that a tensor map asks for.
uint64_t copy_pitch(size_t es, uint64_t rows, uint64_t cols) {
    const uint64_t q = (cols * es >= 128 || rows <= kCopyFree / 128 ? 128 : 16) / es;
    return (cols + q - 1) / q * q;
}

// A 16-bit operand whose rows lie 16-byte multiples apart, but no whole 128-byte lines: each row of a tensor copy's box reads parts of two lines.  What that costs a
// product is counted in us a KB of the box's rows inside the matrix and k-block (bf16 4096 x 1536 x 1024 15.0 us; x 1000, 16 bytes off, 24.4, x 1008 18.3, x 992 16.6), on as many
// k-blocks as an SM has of the whole product: with few tiles its slices of K run side by side; a copy in lines costs its bytes, read and written, at 5 TB/s, and 2 us where
// no other operand has to be copied.  In place / by the rule, us: 4104^3 209 / 137, 4112^3 135 / 127, 4128^3 both 126, 4096 x 1536 x 1000 24.6 / 19.9, 16384 x 4088 x
// 520 97 / 79, 8192 x 1000 x 1000 25.0 / 20.4, and both alike 1024 x 1024 x 1000 8.2, 16384 x 200 x 200 10.2.  Left in place, copied: 336 x 8 x 11560 10.0, 13.1; 224 x 32 x 10248 12.3,
// 15.6; 5440 x 6800 x 168 20.2, 22.6 (reductions of fewer than five k-blocks are bound by their output).  The products' sums are the same either way.
std::atomic<int> g_realign{1};  // 0: never, 2: always (tests, A/B timing)
thread_local int t_last_copies = 0;  // operands that the thread's last product copied: 1 A, 2 B (tests)
constexpr uint64_t kRealignMost = 256ull << 20;  // half of what the workspace pools keep between calls: beyond it a call would map memory anew
static double misaligned_us(const TcProduct& c, uint64_t pitch, double box_kb) {
    const uint64_t off = pitch * 2 % 128, num_kb = (c.k + 63) / 64;
    const double us_kb = off == 0 || num_kb < 5 ? 0.0 : off % 32 ? 0.006 : off % 64 ? 0.0025 : 0.00125;
    const double tiles = (double)c.batch * (double)((c.m + 127) / 128) * (double)((c.n + 255) / 256);
    return us_kb * box_kb * (double)num_kb * tiles / sm_count();
}
// Of what an operand's box reads of the matrix, `mn` of at most `most` rows or columns.  MN-major its rows are those of K, and short ones cost what whole ones do, those of 16 bytes twice that, of A where
// they are of 17 to 64 elements less (in place / copied, us: B 32 x (3136 x 8 x 320) 36.6 / 15.3, x 40 x 320 24.8 / 19.9, A 32 x (8 x 3136 x 400) 34.8 / 21.7, 32 x (40 x 12544 x 320) 66.7 / 71.0).
static double box_kb(bool is_a, bool mn_major, uint64_t mn) {
    const double most = is_a ? 16.0 : 32.0, inside = std::min(most, (double)mn / 8.0);
    return !mn_major || (is_a && mn > 16 && mn <= 64) ? inside : mn <= 8 ? 2 * most : most;
}
static double copy_us(uint64_t rows, uint64_t cols) { return (double)rows * (double)cols * 4.0 / 5.0e6; }

template <class W>
static void repack_launch(const RowCopy<W>& a, const RowCopy<W>& b, const Gate& gate) {
    constexpr uint32_t each = 256 * kCopyUnroll;
    const uint32_t a_blocks = (uint32_t)(((uint64_t)a.vecs + each - 1) / each), b_blocks = (uint32_t)(((uint64_t)b.vecs + each - 1) / each);
    launch_kernel(repack_rows_kernel<W>, a_blocks + b_blocks, 256, 0, ctx().stream, a, b, gate, a_blocks);
}

bool repack_operands(size_t es, TcProduct& c, StreamWorkspace& ws, const char* where, char* place, uint64_t room) {
    const uint64_t a_rows = (c.a_mn ? c.k : c.m) * (c.a_bs ? c.batch : 1), a_cols = c.a_mn ? c.m : c.k, a_pitch = copy_pitch(es, a_rows, a_cols);
    const uint64_t b_rows = (c.b_mn ? c.k : c.n) * (c.b_bs ? c.batch : 1), b_cols = c.b_mn ? c.n : c.k, b_pitch = copy_pitch(es, b_rows, b_cols);
    bool a_copy = c.a_repack, b_copy = c.b_repack;
    const bool needed = a_copy || b_copy;
    const int mode = g_realign.load(std::memory_order_relaxed);
    if (es == 2 && mode) {
        const bool a_dense = !c.a_bs || c.a_bs == (int64_t)(c.m * c.k), b_dense = !c.b_bs || c.b_bs == (int64_t)(c.k * c.n);
        const auto fits = [&](uint64_t rows, uint64_t pitch) { return rows * pitch * es <= kRealignMost / 2; };
        const bool a_may = !a_copy && a_dense && a_pitch != a_cols && fits(a_rows, a_pitch), b_may = !b_copy && b_dense && b_pitch != b_cols && fits(b_rows, b_pitch);
        const double a_gain = a_may ? std::max(0.0, misaligned_us(c, a_cols, box_kb(true, c.a_mn, c.m)) - copy_us(a_rows, a_cols)) : 0.0;
        const double b_gain = b_may ? std::max(0.0, misaligned_us(c, b_cols, box_kb(false, c.b_mn, c.n)) - copy_us(b_rows, b_cols)) : 0.0;
        const bool pays = mode == 2 || a_gain + b_gain > (needed ? 0.0 : 2.0);
        a_copy = a_copy || (pays && a_may && (mode == 2 || a_gain > 0.0));
        b_copy = b_copy || (pays && b_may && (mode == 2 || b_gain > 0.0));
    }
    t_last_copies = 0;
    if (!a_copy && !b_copy) return true;
    const uint64_t a_bytes = a_copy ? (a_rows * a_pitch * es + 255) / 256 * 256 : 0, b_bytes = b_copy ? b_rows * b_pitch * es : 0;
    if (a_bytes / 16 + b_bytes / 16 > 0x7FFFFFFFull) return !needed;  // the copy counts vectors in 32 bits
    if (!place || a_bytes + b_bytes > room) {
        if (!ws.take(a_bytes + b_bytes)) return !needed;
        place = static_cast<char*>(ws.ptr);
    }
    char *const a_dst = place, *const b_dst = a_dst + a_bytes;
    auto launch = [&](auto w) {
        typedef decltype(w) W;
        const auto copy = [&](bool yes, const char* in, char* out, uint64_t rows, uint64_t cols, uint64_t pitch) {
            const uint64_t per_row = (cols * es + 15) / 16;  // the padding itself is never read
            return RowCopy<W>{reinterpret_cast<const W*>(in), reinterpret_cast<W*>(out), yes ? (uint32_t)(rows * per_row) : 0u, FastDiv((uint32_t)per_row), (uint32_t)cols, (uint32_t)pitch};
        };
        repack_launch<W>(copy(a_copy, c.A, a_dst, a_rows, a_cols, a_pitch), copy(b_copy, c.B, b_dst, b_rows, b_cols, b_pitch), c.gate);
    };
    if (es == 2) launch(uint16_t());
    else launch(uint32_t());
    t_last_copies = (a_copy ? 1 : 0) + (b_copy ? 2 : 0);
    if (a_copy) {
        c.A = a_dst;
        c.a_pitch = a_pitch;
        if (c.a_bs) c.a_bs = (int64_t)((c.a_mn ? c.k : c.m) * a_pitch);
    }
    if (b_copy) {
        c.B = b_dst;
        c.b_pitch = b_pitch;
        if (c.b_bs) c.b_bs = (int64_t)((c.b_mn ? c.k : c.n) * b_pitch);
    }
    check_launch(where);
    return true;
}

namespace {
struct DeviceState {
    int* err = nullptr;     // device error word
    int seq = 0;            // launches made so far (the tag of a launch is seq & 0x7FFFFF, never 0)
    bool unchecked = false; // a launch was made since the host last read the word
};
thread_local DeviceState t_state[64];

DeviceState* current_state() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    return &t_state[dev];
}
}  // namespace

int* next_launch_error_word(int* tag) {
    DeviceState* s = current_state();
    if (!s) return nullptr;
    if (!s->err) {
        if (cudaMalloc(&s->err, sizeof(int)) != cudaSuccess) {
            cudaGetLastError();
            s->err = nullptr;
            return nullptr;
        }
        cudaMemset(s->err, 0, sizeof(int));
    }
    s->seq = (s->seq + 1) & 0x7FFFFF;
    if (s->seq == 0) s->seq = 1;
    s->unchecked = true;
    *tag = s->seq;
    return s->err;
}

WaitReport next_wait_report() {
    WaitReport w;
    w.tag = 0;
    w.err = next_launch_error_word(&w.tag);
    return w;
}

}  // namespace tc

// Reads the error word of the calling thread's device.  The copy runs on the legacy stream, i.e. after the work the
// thread has queued there; call it after a synchronisation point.  A non-zero word sets the sticky status
// kErrDeviceWait (its detail = the code of the wait that gave up) and is cleared.
static int collect_tc_status(bool only_if_unchecked) {
    tc::DeviceState* s = tc::current_state();
    if (!s || !s->err) return 0;
    if (only_if_unchecked && !s->unchecked) return 0;
    int v = 0;
    if (cudaMemcpy(&v, s->err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    s->unchecked = false;
    if (v != 0) {
        set_error(kErrDeviceWait, v & 0xFF, (v & 0xFF) >= 21 ? "staged elementwise / conv kernel" : "tc_gemm_kernel");
        cudaMemset(s->err, 0, sizeof(int));
    }
    return v & 0xFF;
}

// Called by the ABI's own synchronisation points (cuda_memcpy_d2h, cuda_stream_synchronize): costs one 4-byte
// read-back, and only when a tensor-core launch was made since the last check.
int tc_status_after_sync() { return collect_tc_status(true); }

}  // namespace mx

// Checks the error word of the calling thread's device after a synchronisation point: 0 = fine, else the code of
// the bounded wait that ran out (also recorded as the sticky status kErrDeviceWait).
extern "C" int mx_tc_gemm_status(void) { return mx::collect_tc_status(false); }

// Test hook: writes `value` into the error word the way a kernel of an EARLIER launch would have left it
// (tag 0 is never handed to a launch), so the surfacing of a stale report can be tested without making a wait run out.
extern "C" int mx_debug_tc_gemm_poke_status(int value) {
    int tag = 0;
    int* err = mx::tc::next_launch_error_word(&tag);
    if (!err) return -1;
    const int word = value ? (value & 0xFF) | (0x7FFFFF << 8) : 0;
    return cudaMemcpy(err, &word, sizeof(int), cudaMemcpyHostToDevice) == cudaSuccess ? 0 : -1;
}

namespace mx {

// Sizes the tensor-core kernels can index and are worth a persistent launch for.
// `least`: multiply-adds from which on.
constexpr uint64_t kTcLeast = 1ull << 24;
static bool in_range(uint64_t M, uint64_t N, uint64_t K, uint64_t batch, uint64_t least = kTcLeast) {
    if (M == 0 || N == 0 || K == 0) return false;
    if (M > 0x7FFFFFFFull || N > 0x7FFFFFFFull || K > 0x7FFFFFFFull) return false;
    if (batch > 0x7FFFull) return false;
    if (batch * M * N * K < least) return false;  // small problems are not worth a persistent launch
    return batch * ((M + 127) / 128) * ((N + 63) / 64) <= 0x3FFFFFFFull;
}
// TMA wants 16-byte aligned bases and row pitches: the contiguous extent of every matrix (K for K-major
// operands, MN for MN-major ones, N for D) must be a multiple of 16 / elem_size elements.
static bool eligible(size_t es, uint64_t M, uint64_t N, uint64_t K, uint64_t batch, bool a_mn, bool b_mn, const void* a, const void* b, const void* d,
                     uint64_t least = kTcLeast) {
    const uint64_t q = 16 / es;
    if (!in_range(M, N, K, batch, least)) return false;
    if (N % q != 0) return false;
    if ((a_mn ? M : K) % q != 0 || (b_mn ? N : K) % q != 0) return false;
    if (((uintptr_t)a | (uintptr_t)b | (uintptr_t)d) % 16 != 0) return false;
    if (batch > 1 && (M * N) % q != 0) return false;  // every batch's output starts on a 16-byte boundary
    return true;
}
// f32 products that are not of the plain form (ragged, rank > 3, batched backward) were the CUDA cores' before; they go to the split kernel
// only where that is no less exact.  Error against 64 bits, CUDA cores / split kernel: K = 64 1.5e-7 / 2.2e-7, 128 2.1e-7 / 2.2e-7, 192 2.5e-7
// / 2.2e-7, 1024 5.7e-7 / 2.4e-7 for normal values; K = 128 1.6e-7 / 1.7e-7, 192 2.1e-7 / 1.7e-7 for positive ones.
constexpr uint64_t kSplitLeastK = 192;
// What a product of dense operands needs before the kernels can take it: an operand whose rows (or base) are not
// 16-byte multiples is copied to padded rows first (repack_operands), an output like that is written by the epilogue warps
// without tensor stores.  One pass over the operand against 8 TFLOP/s on the CUDA cores: bf16 4099 x 1543 x 1000, whose
// 1543-wide matrices all need it, takes 20-40 us a product (1804 us on the CUDA cores).
static bool plan_ragged(size_t es, TcProduct& c, const void* d, uint64_t least = kTcLeast) {
    const uint64_t q = 16 / es;
    if (!in_range(c.m, c.n, c.k, c.batch, least) || (es == 4 && c.k < kSplitLeastK)) return false;
    if (((uintptr_t)c.A | (uintptr_t)c.B | (uintptr_t)d) % es != 0) return false;
    const uint64_t a_cols = c.a_mn ? c.m : c.k, b_cols = c.b_mn ? c.n : c.k;
    c.a_repack = a_cols % q != 0 || (uintptr_t)c.A % 16 != 0;
    c.b_repack = b_cols % q != 0 || (uintptr_t)c.B % 16 != 0;
    const uint64_t a_rows = (c.a_mn ? c.k : c.m) * (c.a_bs ? c.batch : 1), b_rows = (c.b_mn ? c.k : c.n) * (c.b_bs ? c.batch : 1);
    const uint64_t a_copy = c.a_repack ? a_rows * tc::copy_pitch(es, a_rows, a_cols) * es : 0, b_copy = c.b_repack ? b_rows * tc::copy_pitch(es, b_rows, b_cols) * es : 0;
    // The copies are workspace that a caller does not see: at most twice the operands where they are large (rows of one to three
    // elements grow up to eightfold), and 8 GB in all.  What is beyond runs on the CUDA cores.
    const uint64_t dense = (c.a_repack ? a_rows * a_cols * es : 0) + (c.b_repack ? b_rows * b_cols * es : 0);
    if (a_copy + b_copy > 2 * dense + 2 * tc::kCopyFree || a_copy + b_copy > (8ull << 30)) return false;
    if (c.batch > 1) {
        // the batches of a copied operand must lie one after the other; an uncopied one's batch stride is a tensor-map stride
        if (c.a_bs != 0 && c.a_bs != (int64_t)(c.m * c.k)) return false;
        if (c.b_bs != 0 && c.b_bs != (int64_t)(c.k * c.n)) return false;
    }
    c.ragged = true;
    c.nearest = es == 2;
    const bool plain = c.n % q != 0 || (uintptr_t)d % 16 != 0;
    c.d_plain = !plain ? 0 : (c.n % 2 == 0 && (uintptr_t)d % 4 == 0 ? 2 : 1);
    return true;
}

// Forward product C[m, n] = sum_k A[m, k] * B[k, n]: can it run on a tensor-core kernel, and with which operand
// majors?  Unbatched, every operand either dense row-major or the transposed view of a dense matrix.
static bool forward_operands(const MmDesc& d, size_t es, size_t num_els, const void* x, const void* y, TcProduct& c) {
    if (d.out_nd < 2 || d.a_nd < 2 || d.b_nd < 2) return false;
    const uint64_t m = d.m, n = d.n, k = d.k_fwd;
    if (m == 0 || n == 0 || k == 0 || num_els % (m * n) != 0) return false;
    const uint64_t batch = num_els / (m * n);
    if (batch > 0x7FFFull) return false;
    c.A = static_cast<const char*>(x) + d.a_off * es;
    c.B = static_cast<const char*>(y) + d.b_off * es;
    bool a_kmajor, a_mnmajor, b_kmajor, b_mnmajor;
    if (d.a_cont && d.b_cont) {
        // the reference's contiguous branch: A is [batch, m, k], B is [batch, k, n], both dense
        a_kmajor = true;
        a_mnmajor = false;
        b_kmajor = false;
        b_mnmajor = true;
        c.a_bs = (int64_t)(m * k);
        c.b_bs = (int64_t)(k * n);
        // ranks other than three: every leading dim folds into the batch, as long as both operands have all of it
        if (batch > 1 && !(d.out_nd == 3 && d.a_nd == 3 && d.b_nd == 3) && (d.a_elems != batch * m * k || d.b_elems != batch * k * n)) return false;
    } else {
        // batched: rank-3 operands only (for higher ranks the reference indexes the batch through strides[0] alone)
        if (batch > 1 && !(d.out_nd == 3 && d.a_nd == 3 && d.b_nd == 3)) return false;
        // strided branch: A[b * as0 + m * as1 + k * as2], B[b * bs0 + k * bs1 + n * bs2]
        a_kmajor = d.a_strides[2] == 1 && d.a_strides[1] == (int64_t)k;
        a_mnmajor = d.a_strides[1] == 1 && d.a_strides[2] == (int64_t)m;  // transposed view of a dense [k, m] matrix
        b_kmajor = d.b_strides[1] == 1 && d.b_strides[2] == (int64_t)k;   // transposed view of a dense [n, k] matrix
        b_mnmajor = d.b_strides[2] == 1 && d.b_strides[1] == (int64_t)n;  // dense [k, n]
        c.a_bs = batch > 1 ? d.a_strides[0] : 0;                          // 0: one matrix broadcast over the batch
        c.b_bs = batch > 1 ? d.b_strides[0] : 0;
    }
    if (!(a_kmajor || a_mnmajor) || !(b_kmajor || b_mnmajor)) return false;
    // batches are whole matrices apart (no overlap tricks)
    if (batch > 1 && (c.a_bs < 0 || c.b_bs < 0 || (c.a_bs != 0 && c.a_bs < (int64_t)(m * k)) || (c.b_bs != 0 && c.b_bs < (int64_t)(k * n)))) return false;
    c.a_mn = !a_kmajor;
    c.b_mn = !b_kmajor;
    c.m = m;
    c.n = n;
    c.k = k;
    c.batch = batch;
    return true;
}

static bool backward_operands(const MmDesc& d, int which, size_t nea, size_t neb, const void* x, const void* y, TcProduct& c) {
    const uint64_t m = d.m, n = d.n, k = d.k_bwd;
    if (d.out_nd < 2 || m == 0 || n == 0 || k == 0 || d.g_size % (m * n) != 0) return false;
    // both gradients have every batch of g (an operand broadcast over the batch has fewer elements): dense batched products
    const uint64_t batch = d.g_size / (m * n);
    if (batch > 0x7FFFull || nea != batch * m * k || neb != batch * k * n) return false;
    c.batch = batch;
    const int64_t g_bs = batch > 1 ? (int64_t)(m * n) : 0, a_bs = batch > 1 ? (int64_t)(m * k) : 0, b_bs = batch > 1 ? (int64_t)(k * n) : 0;
    if (which == 1) {
        c.A = static_cast<const char*>(x);
        c.B = static_cast<const char*>(y);
        c.a_bs = g_bs;
        c.b_bs = b_bs;
        c.a_mn = c.b_mn = false;
        c.m = m;
        c.n = k;
        c.k = n;
    } else {
        c.A = static_cast<const char*>(y);
        c.B = static_cast<const char*>(x);
        c.a_bs = a_bs;
        c.b_bs = g_bs;
        c.a_mn = c.b_mn = true;
        c.m = k;
        c.n = n;
        c.k = m;
    }
    return true;
}

// The batch strides of operands that tensor maps reach in place are multiples of 16 bytes.
static bool aligned_batches(size_t es, const TcProduct& c) {
    const int64_t q = (int64_t)(16 / es);
    return c.batch <= 1 || (c.a_bs % q == 0 && c.b_bs % q == 0);
}

// which = 0: forward (x = A base, y = B base).  1: grad_a[m, k] = sum_n g[m, n] * B[k, n] (x = g, y = B + offset),
// reduction over n, both operands K-major.  2: grad_b[k, n] = sum_m A[m, k] * g[m, n] (x = g, y = A + offset),
// reduction over m, both operands MN-major.  The backward products read g, A and B as dense row-major matrices
// (strides ignored, crates/maidenx_cpu/src/ops/matmul.rs:196-261).
// Few outputs and a long reduction: matmul_longk_kernel (a block per output) is done before 128-row tiles have been cut into runs, copied
// and summed.  16-bit, longk / tensor cores, both operands K-major: 16 x 64 x 4100 7.9 / 12.1 us, x 8192 12.3 / 8.5; 32 x 32 x 2048 5.1 / 7.3; 1 x 64
// x 16384 9.0 / 10.7, x 32768 16.1 / 12.2; an MN-major operand costs longk a line per element: 16 x 64 x 4100 22.9 / 10.3, 1 x 256 x 8192
// 11.2 / 11.2, x 16384 19.9 / 13.1, 100 x 10 x 4100 (A and B) 20.6 / 13.2, and without copies 16 x 64 x 2048 12.5 / 6.9 already.  f32 stays: its fixed
// tree has an error of 5e-8 for values of one sign at any length, the drained tf32 sums 1.9e-7 (normal values 1.9e-7 at K = 20000 to 5.8e-7 at
// 262144, 2.6e-7 to 3.5e-7), although 100 x 10 x 131072 takes 220 us and would take 84.
static bool longk_better(size_t es, const TcProduct& c, bool in_place) {
    const uint64_t outputs = c.batch * c.m * c.n;
    if (c.k < kLongKMinK || outputs > kLongKMaxOutputs) return false;
    if (es != 2) return true;
    const bool b_across = c.b_mn && c.n >= 32;
    const uint64_t many = !b_across && !(c.a_mn && c.m >= 32) ? 8192 : in_place ? kLongKMinK : 4096;
    return !(c.k >= 32768 || (outputs >= 512 && c.k >= many) || (b_across && outputs >= 64 && c.k >= 16384));
}

bool tc_classify(const MmDesc& d, int which, size_t es, size_t num_els, size_t nea, size_t neb, const void* x, const void* y, const void* out,
                     TcProduct& c) {
    if (which == 0 ? !forward_operands(d, es, num_els, x, y, c) : !backward_operands(d, which, nea, neb, x, y, c)) return false;
    // a matrix of one column is the same memory as one of one row, and K-major it needs no copy of its one-element rows
    if (c.m == 1) c.a_mn = false;
    if (c.n == 1) c.b_mn = false;
    c.ragged = d.out_nd > (which == 0 ? 3 : 2);  // aligned, but new to these kernels: batches beyond rank 3, batched backward
    // 16-bit products far below kTcLeast still gain when their reduction is long: the CUDA-core kernel's time is its chain of
    // k-steps (64 x 64 x 512: 22 us, 128 x 10 x 784: 33), the tensor-core kernel's about 4.5 us, 1.6 us more per copied operand.
    // f32 keeps the line: below it results are bit for bit those of the element-type loop.
    const uint64_t least = es == 2 && c.k >= 256 ? 1ull << 18 : kTcLeast;
    if (es == 4 && c.ragged && c.k < kSplitLeastK) return false;
    if (aligned_batches(es, c) && eligible(es, c.m, c.n, c.k, c.batch, c.a_mn, c.b_mn, c.A, c.B, out, least)) {
        const bool plain_form = !c.ragged && c.batch * c.m * c.n * c.k >= kTcLeast;
        c.nearest = es == 2 && !plain_form;
        return plain_form || !longk_better(es, c, true);
    }
    if (longk_better(es, c, false)) return false;
    // the copy reads whole operands: every batch must be there (a size-1 batch dim passes the contiguity test)
    if (which == 0 && c.batch > 1 && d.a_cont && d.b_cont && (d.a_elems != c.batch * c.m * c.k || d.b_elems != c.batch * c.k * c.n)) return false;
    return plan_ragged(es, c, out, least);
}

// x [rows, in] . w[out, in]^T with the bias add (and GELU) in the epilogue; false = shape not taken (the caller runs the ops one by one)
bool tc_linear_bias_act(bool is_bf16, uint64_t rows, uint64_t in_features, uint64_t out_features, const void* x, const void* w, const void* bias,
                        void* u, void* act, const char* where) {
    TcProduct c;
    c.A = static_cast<const char*>(x);
    c.B = static_cast<const char*>(w);
    c.a_mn = c.b_mn = false;
    c.m = rows;
    c.n = out_features;
    c.k = in_features;
    c.batch = 1;
    c.a_bs = c.b_bs = 0;
    if (!bias || !u || !eligible(2, c.m, c.n, c.k, 1, false, false, x, w, u) || (act && (uintptr_t)act % 16 != 0)) return false;
    return launch_gemm(is_bf16, c, u, where, act ? 2 : 1, bias, act);
}

// out[b] = w[rows, k] (shared by every batch) . cols[b][k, n] + bias[rows] broadcast along n, the bias add in the
// product's epilogue with the roundings of the two separate ops; false = shape not taken, nothing launched.
bool tc_batched_row_bias(bool is_bf16, uint64_t batch, uint64_t rows, uint64_t k, uint64_t n, const void* w, const void* cols, const void* bias, void* out,
                         const char* where) {
    TcProduct c;
    c.A = static_cast<const char*>(w);
    c.B = static_cast<const char*>(cols);
    c.a_mn = false;
    c.b_mn = true;  // [k, n] row-major per batch
    c.m = rows;
    c.n = n;
    c.k = k;
    c.batch = batch;
    c.a_bs = 0;
    c.b_bs = (int64_t)(k * n);
    if (!bias || !out || batch == 0 || batch > 0x7FFFull) return false;
    if (!eligible(2, c.m, c.n, c.k, batch, false, true, w, cols, out) && !plan_ragged(2, c, out)) return false;
    StreamWorkspace ws;
    return repack_operands(2, c, ws, where) && launch_gemm(is_bf16, c, out, where, 3, bias, nullptr);
}

// Rows of whole output images in at most 256 columns of a tile, channels that tensor maps can describe, sizes that the kernel indexes in 32 bits.
bool conv_grad_input_fits(uint64_t batch, uint64_t c, uint64_t h, uint64_t w, uint64_t co, uint64_t kh, uint64_t kw, uint64_t ph, uint64_t pw) {
    return batch && c && h && w && co && kh && kw && w <= 256 && co % 8 == 0 && batch <= 0x7FFF && h * w <= 0x3FFFFFFF && c <= 0x3FFFFFFF && kh * kw * ((co + BK - 1) / BK) <= 0xFFFF && ph <= 0x7FFF &&
           pw <= 0x7FFF && batch * ((c + BM - 1) / BM) * h <= 0x3FFFFFFF;
}
// The gradient of a convolution's input, strides of 1: grad_x[b][c] = sum over taps (i, j) and output channels o of w[o][c][i][j] grad_out[b][o] shifted by the tap.  `g` holds
// grad_out with the channels last, `wt` the weights as [c][tap][o]: then every tap is a product whose second operand is a box of neighbouring pixels, zeros outside
// the image, and all of them are one reduction in the f32 accumulator.  No column matrix is written and read, and nothing is rounded on the way.
bool tc_conv_grad_input(bool is_bf16, uint64_t batch, uint64_t c, uint64_t h, uint64_t w, uint64_t co, uint64_t kh, uint64_t kw, uint64_t ph, uint64_t pw, uint64_t oh, uint64_t ow,
                        const void* g, const void* wt, void* grad_x, const char* where) {
    if (!conv_grad_input_fits(batch, c, h, w, co, kh, kw, ph, pw) || ((uintptr_t)g | (uintptr_t)wt) % 16 != 0 || (uintptr_t)grad_x % 2 != 0 || !opt_in_shared_memory()) return false;
    TcConvParams p = {};
    const uint64_t blocks = (h + 256 / w - 1) / (256 / w);
    p.conv_rows = (int)((h + blocks - 1) / blocks);
    p.conv_w = (int)w;
    p.conv_kw = (int)kw;
    p.conv_cb = (int)((co + BK - 1) / BK);
    p.conv_x = (int)pw;
    p.conv_y = (int)ph;
    p.conv_kh = (int)kh;
    p.conv_co = (int)co;
    p.conv_oh = (int)oh;
    p.conv_ow = (int)ow;
    p.conv_g = g;
    p.conv_wt = wt;
    p.M = (int)c;
    p.N = (int)(h * w);
    p.num_kb = (int)(kh * kw) * p.conv_cb;
    p.K = p.num_kb * BK;
    p.bn = (p.conv_rows * p.conv_w + 15) / 16 * 16;
    p.tiles_m = (int)((c + BM - 1) / BM);
    p.tiles_n = (int)((h + p.conv_rows - 1) / p.conv_rows);
    p.tiles_per_batch = p.tiles_m * p.tiles_n;
    p.num_tiles = (int)batch * p.tiles_per_batch;
    p.a_batched = p.b_batched = 1;
    p.is_bf16 = is_bf16 ? 1 : 0;
    p.group_m = g_group_m.load(std::memory_order_relaxed);
    p.stages = ring_stages(p.bn);
    p.stage_bytes = A_STAGE_BYTES + p.bn * BK * 2;
    p.d_plain = 1;
    p.poll_ns = poll_ns(p.num_kb);
    p.d = grad_x;
    int tag = 0;
    int* err = next_launch_error_word(&tag);
    EncodeTiledFn enc = encode_fn();
    if (!err || !enc) return false;
    const CUtensorMapDataType t16 = is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    auto encode = [&](CUtensorMap& map, const void* base, int rank, const cuuint64_t* dims, const cuuint32_t* box) {  // dense
        cuuint64_t strides[3];
        const cuuint32_t ones[4] = {1, 1, 1, 1};
        for (int i = 0; i + 1 < rank; i++) strides[i] = (i ? strides[i - 1] : 2) * dims[i];
        return enc(&map, t16, (cuuint32_t)rank, const_cast<void*>(base), dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    CUtensorMap ma, mb;
    const cuuint64_t a_dims[3] = {co, kh * kw, c}, b_dims[4] = {co, ow, oh, batch};
    const cuuint32_t a_box[3] = {BK, 1, BM}, b_box[4] = {BK, (cuuint32_t)w, (cuuint32_t)p.conv_rows, 1};
    if (!encode(ma, wt, 3, a_dims, a_box) || !encode(mb, g, 4, b_dims, b_box)) return false;
    int grid = sm_count();
    if (ctx().gemm_sm_limit > 0 && ctx().gemm_sm_limit < grid) grid = ctx().gemm_sm_limit;
    if (grid > p.num_tiles) grid = p.num_tiles;
    launch_kernel(tc_gemm_kernel<TC_PLAIN, 0, false, false, true>, grid, tc_threads(epi_warps(TC_PLAIN, false)), TC_SMEM_BYTES, ctx().stream, ma, mb, ma, ma, p, err, tag);
    check_launch(where);
    return true;
}

bool tc_batch_sum_f32(uint64_t batch, uint64_t m, uint64_t n, uint64_t k, const float* a, const float* b, float* out, const char* where) {
    TcProduct c;
    c.A = reinterpret_cast<const char*>(a);
    c.B = reinterpret_cast<const char*>(b);
    c.a_mn = c.b_mn = false;
    c.m = m;
    c.n = n;
    c.k = k;
    c.batch = batch;
    c.a_bs = (int64_t)(m * k);
    c.b_bs = (int64_t)(n * k);
    c.sum_batches = true;
    return batch * k <= 0x7FFFFFFFull && eligible(4, m, n, k, batch, false, false, a, b, out) && tc_launch_f32(c, out, where);
}

bool tc_gemm_bf16_f16(bool is_bf16, const MmDesc& d, int which, size_t num_els, size_t nea, size_t neb, const void* x, const void* y, void* out,
                      const char* where) {
    TcProduct c;
    if (!tc_classify(d, which, 2, num_els, nea, neb, x, y, out, c)) return false;
    StreamWorkspace ws;
    return repack_operands(2, c, ws, where) && launch_gemm(is_bf16, c, out, where);
}

}  // namespace mx

// Host-only view for tests without a GPU: would cuda_matmul[_backward]_<bf16|f16|f32> with this HOST metadata and these base
// addresses run on a tensor-core kernel?  Returns 0 (CUDA-core kernels) or the number of batches, and how the product would be
// launched: operand majors (0 = K-major, 1 = MN-major), extents, and what is prepared for it (include/maidenx_cuda_testing.h).
extern "C" int mx_debug_matmul_plan(size_t elem_size, int which, size_t num_els, size_t nea, size_t neb, const size_t* host_metadata, const void* x, const void* y,
                                    const void* out, int* a_mn_major, int* b_mn_major, size_t* m, size_t* n, size_t* k, int* prepared) {
    mx::MmDesc d;
    if (!host_metadata || !mx::mm_parse(host_metadata, d)) return 0;
    mx::TcProduct c;
    if (!mx::tc_classify(d, which, elem_size, num_els, nea, neb, x, y, out, c)) return 0;
    if (a_mn_major) *a_mn_major = c.a_mn ? 1 : 0;
    if (b_mn_major) *b_mn_major = c.b_mn ? 1 : 0;
    if (m) *m = c.m;
    if (n) *n = c.n;
    if (k) *k = c.k;
    if (prepared) *prepared = (c.a_repack ? 1 : 0) | (c.b_repack ? 2 : 0) | (c.d_plain << 2);
    return (int)c.batch;
}
// 2: bf16 / f16 products run on the two-CTA kernel (pairs of SMs share the B tile); 1: on the one-CTA kernel.
extern "C" void mx_set_gemm_cta_group(int ctas) { mx::g_two_cta.store(ctas == 2, std::memory_order_relaxed); }
extern "C" int mx_debug_gemm_max_resident_pairs(void) { return mx::tc2::max_resident_pairs(); }
extern "C" void mx_debug_set_gemm_group_m(int rows) { mx::g_group_m.store(rows > 0 ? rows : 16, std::memory_order_relaxed); }
// 1 (default): products with a reduction of at most 256 run with the B panel resident in shared memory; 0: general schedule
extern "C" void mx_debug_set_gemm_keep_b(int on) { mx::g_keep_b.store(on ? 1 : 0, std::memory_order_relaxed); }
extern "C" int mx_debug_gemm_last_copies(void) { return mx::tc::t_last_copies; }
extern "C" void mx_debug_set_gemm_realign(int mode) { mx::tc::g_realign.store(mode, std::memory_order_relaxed); }
extern "C" int mx_debug_gemm_keep_b_ctas(int tiles_m, int tiles_n, int num_kb, int batch, int ctas) { return mx::keep_b_ctas(tiles_m, tiles_n, num_kb, batch, ctas); }
extern "C" int mx_debug_gemm_last_schedule(void) { return mx::t_last_schedule; }
extern "C" int mx_debug_splitk_slices(size_t tiles, size_t k, int block_k, int sms) { return mx::tc::splitk_slices(tiles, k, block_k, sms); }
extern "C" int mx_debug_matmul_forward_path(size_t num_els, const size_t* host_metadata, const void* a, const void* b, const void* out, int* a_mn_major,
                                            int* b_mn_major, size_t* m, size_t* n, size_t* k) {
    return mx_debug_matmul_plan(2, 0, num_els, 0, 0, host_metadata, a, b, out, a_mn_major, b_mn_major, m, n, k, nullptr);
}
extern "C" int mx_debug_matmul_forward_path_f32(size_t num_els, const size_t* host_metadata, const void* a, const void* b, const void* out,
                                                int* a_mn_major, int* b_mn_major, size_t* m, size_t* n, size_t* k) {
    return mx_debug_matmul_plan(4, 0, num_els, 0, 0, host_metadata, a, b, out, a_mn_major, b_mn_major, m, n, k, nullptr);
}
