// Interface between the matmul entry points and the tensor-core (tcgen05) kernels.
// Each function returns true when it handled the product; false sends the call to the
// SIMT kernel.  bf16 / f16 run on kind::f16 (matmul_tc.cu), f32 on split-operand kind::tf32
// (matmul_tc_f32.cu); every other dtype has no tensor-core implementation.
#pragma once
#include "matmul_simt.cuh"

namespace mx {

// What a launch looks for before it does anything: it runs when the word holds the tag.  No word: it runs.
struct Gate {
    const unsigned long long* word = nullptr;
    unsigned long long tag = 0;
    __device__ __forceinline__ bool shut() const { return word && *word != tag; }
};

// A product the tensor-core kernels accept: D[m, n] = sum_k Aop[m, k] * Bop[n, k] with dense operands that are
// K-major ([MN, K] row-major) or MN-major ([K, MN] row-major).
struct TcProduct {
    const char* A;
    const char* B;
    bool a_mn, b_mn;
    uint64_t m, n, k;
    uint64_t batch;      // independent products; D is dense [batch, m, n]
    int64_t a_bs, b_bs;  // elements between consecutive batches of each operand; 0 = one matrix shared by all
    uint64_t a_pitch = 0, b_pitch = 0;        // elements between rows of a copied operand (0: dense)
    bool a_repack = false, b_repack = false;  // the operand has to be copied to 16-byte-multiple rows first
    bool ragged = false;                      // not the plain form: rows or bases off 16 bytes, batches beyond rank 3, batched backward
    bool nearest = false;                     // 16-bit: a sum that the CUDA cores would round to nearest (see kRunMostF16)
    bool sum_batches = false;                 // D is one [m, n] matrix, the sum of the batches' products
    Gate gate;                                // f32: the launches for this product run only if it is open
    int d_plain = 0;                          // the output is written without tensor stores: 1 element-wise, 2 in pairs
};
// Every product the kernels compute, with the fields that say what has to be prepared for it: dense and transposed operands, ragged
// rows and unaligned bases (copied operands, plain stores), batches of any rank, batched backward products.
// which: 0 forward, 1 grad_a, 2 grad_b (see matmul_tc.cu); elem_size in bytes.
bool tc_classify(const MmDesc& d, int which, size_t elem_size, size_t num_els, size_t nea, size_t neb, const void* x, const void* y, const void* out,
                 TcProduct& c);

bool tc_gemm_bf16_f16(bool is_bf16, const MmDesc& d, int which, size_t num_els, size_t nea, size_t neb, const void* x, const void* y, void* out,
                      const char* where);
// Linear forward with its bias add and activation folded into the product's epilogue (bf16 / f16): u = x . w^T + bias and,
// when `act` is not NULL, act = gelu(u), each rounded exactly as the separate ops round.  `bias` is one element in device
// memory.  Returns false when the shape does not qualify for the tensor-core kernel; nothing was launched then.
bool tc_linear_bias_act(bool is_bf16, uint64_t rows, uint64_t in_features, uint64_t out_features, const void* x, const void* w, const void* bias,
                        void* u, void* act, const char* where);
// Batched product with a per-row bias in the epilogue (bf16 / f16): out[b] = w[rows, k] . cols[b][k, n] + bias[rows], the
// form of a convolution's forward pass over its column buffer.  false = not taken by the tensor-core kernel, nothing launched.
bool tc_batched_row_bias(bool is_bf16, uint64_t batch, uint64_t rows, uint64_t k, uint64_t n, const void* w, const void* cols, const void* bias, void* out,
                         const char* where);
// out[m, n] = sum_b a[b][m, k] . b[b][n, k]^T over the whole batch in one reduction: the weight gradient of a convolution.
// false = not taken (rows of k or n that are not 16-byte multiples, a small product).
bool tc_batch_sum_f32(uint64_t batch, uint64_t m, uint64_t n, uint64_t k, const float* a, const float* b, float* out, const char* where);
// The gradient of a convolution's input in one product, strides of 1, 16-bit types: g = grad_out as [batch][oh][ow][co], wt = the weights as [c][kh * kw][co].
// false: not taken, nothing launched.
bool conv_grad_input_fits(uint64_t batch, uint64_t c, uint64_t h, uint64_t w, uint64_t co, uint64_t kh, uint64_t kw, uint64_t ph, uint64_t pw);
bool tc_conv_grad_input(bool is_bf16, uint64_t batch, uint64_t c, uint64_t h, uint64_t w, uint64_t co, uint64_t kh, uint64_t kw, uint64_t ph, uint64_t pw, uint64_t oh, uint64_t ow,
                        const void* g, const void* wt, void* grad_x, const char* where);
bool tc_launch_f32(const TcProduct& c, void* out, const char* where);
// The product in pairs of f16 (matmul_tc_pairs.cu), if that is estimated to take less than `tf32_us`.  true: launched, and whoever called runs the product behind
// a gate, which is open when an operand was not fit for pairs and lies in `ws`, and behind that the sum of the slices, of whichever product ran; false: nothing launched.
struct PairsRun {
    Gate gate;
    int slices = 1;            // of the product in pairs: its partial results, [slices][m][n rounded up to 4], are still to be added
    float* partial = nullptr;  // where they are, and where the product behind the gate has its own
    char* place = nullptr;     // the pairs' own memory, for what else runs behind the open gate: nothing reads them there
    uint64_t room = 0;
};
// partial_bytes: what the product behind the gate takes for partial results.
bool tc_launch_f32_pairs(const TcProduct& c, double tf32_us, uint64_t partial_bytes, void* out, PairsRun& run, StreamWorkspace& ws, const char* where);
bool tc_gemm_f32(const MmDesc& d, int which, size_t num_els, size_t nea, size_t neb, const void* x, const void* y, void* out, const char* where);

template <class T>
inline bool tc_dispatch(const MmDesc& d, int which, size_t num_els, size_t nea, size_t neb, const T* x, const T* y, T* out, const char* where) {
    if constexpr (is_half_v<T>) return tc_gemm_bf16_f16(std::is_same<T, bf16>::value, d, which, num_els, nea, neb, x, y, out, where);
    else if constexpr (std::is_same<T, float>::value) return tc_gemm_f32(d, which, num_els, nea, neb, x, y, out, where);
    else return false;
}
template <class T>
inline bool tc_matmul_forward(const MmDesc& d, size_t num_els, const T* a, const T* b, T* c, const char* where) {
    return tc_dispatch<T>(d, 0, num_els, 0, 0, a, b, c, where);
}
template <class T>
inline bool tc_matmul_grad_a(const MmDesc& d, size_t nea, size_t neb, const T* g, const T* b_off, T* ga, const char* where) {
    return tc_dispatch<T>(d, 1, 0, nea, neb, g, b_off, ga, where);
}
template <class T>
inline bool tc_matmul_grad_b(const MmDesc& d, size_t nea, size_t neb, const T* g, const T* a_off, T* gb, const char* where) {
    return tc_dispatch<T>(d, 2, 0, nea, neb, g, a_off, gb, where);
}

}  // namespace mx
