// Embedding backward: scatter-add of the output gradient rows into the table's gradient.
//
//   dW[ids[t], :] += dY[t, :]        for every token t with 0 <= ids[t] < vocab
//
// The usual framework path builds a dense [vocab, hidden] gradient (sort the ids, segment-reduce, write ~vocab x hidden
// elements) and then adds it to the fp32 accumulator in a second pass: for a 128k x 2048 table that is more than 1.5 GB
// of traffic for 16k tokens' worth of information.  Here each token row goes straight into the fp32 accumulator with
// red.global.add (atomics resolve repeated ids), 64 MB for 16k tokens.  Rows whose id falls outside [0, vocab) (other
// vocabulary shards under tensor parallelism, padding) are skipped.
// Reference counterpart: Megatron's VocabParallelEmbedding backward (index_add into main_grad).
#include "common.cuh"

namespace lmoe {

template <typename T>
__global__ void embedding_bwd_kernel(const T* __restrict__ dy, const int64_t* __restrict__ ids, float* __restrict__ dw,
                                     int64_t tokens, int hidden, int64_t vocab, int64_t id_offset) {
    constexpr int VN = Vec<T>::N;
    const int nvec = hidden / VN;
    for (int64_t t = blockIdx.x; t < tokens; t += gridDim.x) {
        const int64_t id = ids[t] - id_offset;
        if (id < 0 || id >= vocab) continue;
        float* row = dw + id * hidden;
        for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
            Vec<T> v;
            v.load(dy + t * hidden + i * VN);
#pragma unroll
            for (int e = 0; e < VN; ++e) atomicAdd(row + i * VN + e, v.get(e));
        }
    }
}

// The dense gradient, where a caller wants one: the table's rows are zeroed once in their own type, a token whose id is its own writes its row,
// and the tokens that share an id meet in fp32 rows, one per first token (`acc` [tokens, hidden]).  An fp32 table and a pass that
// converts it moved 2.5 times the bytes: 4096 tokens, 32000 x 2048: 146 -> 60 us.
__global__ void embedding_owner_kernel(const int64_t* __restrict__ ids, unsigned* __restrict__ first, unsigned* __restrict__ more, int64_t tokens,
                                       int64_t vocab, int64_t id_offset) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= tokens) return;
    const int64_t id = ids[t] - id_offset;
    if (id < 0 || id >= vocab) return;
    atomicMin(first + id, (unsigned)t);
    atomicAdd(more + id, 1u);                            // from 0xffffffff: 0 for one token
}
// FINISH false: single tokens' rows to `out`, the others' into acc.  FINISH true: the first tokens' rows of acc to `out`.
template <typename T, typename O, bool FINISH>
__global__ void embedding_rows_kernel(const T* __restrict__ dy, const int64_t* __restrict__ ids, const unsigned* __restrict__ first,
                                      const unsigned* __restrict__ more, float* __restrict__ acc, O* __restrict__ out, int hidden, int64_t vocab,
                                      int64_t id_offset) {
    const int64_t t = blockIdx.x, id = ids[t] - id_offset;
    if (id < 0 || id >= vocab) return;
    const bool single = more[id] == 0;
    const int64_t owner = first[id];
    if (FINISH && (single || owner != t)) return;
    for (int i = threadIdx.x * 4; i < hidden; i += blockDim.x * 4) {
        const float4 v = FINISH ? load4(acc + t * hidden + i) : load4(dy + t * hidden + i);
        if (FINISH || single) store4(out + id * hidden + i, v);
        else {
            float* a = acc + owner * hidden + i;
            atomicAdd(a, v.x); atomicAdd(a + 1, v.y); atomicAdd(a + 2, v.z); atomicAdd(a + 3, v.w);
        }
    }
}
template <typename T, typename O>
static int dense_grad(const void* dy, const int64_t* ids, void* out, float* acc, unsigned* tables, int64_t tokens, int hidden, int64_t vocab,
                      int64_t id_offset, cudaStream_t st) {
    unsigned *first = tables, *more = tables + vocab;
    int rc = (int)cudaMemsetAsync(out, 0, (size_t)vocab * hidden * sizeof(O), st);
    if (!rc) rc = (int)cudaMemsetAsync(tables, 0xff, (size_t)vocab * 2 * sizeof(unsigned), st);
    if (!rc && tokens > 0) rc = (int)cudaMemsetAsync(acc, 0, (size_t)tokens * hidden * sizeof(float), st);
    if (rc || tokens <= 0) return rc;
    const int threads = hidden >= 1024 ? 256 : (hidden >= 512 ? 128 : 64);
    embedding_owner_kernel<<<(unsigned)((tokens + 255) / 256), 256, 0, st>>>(ids, first, more, tokens, vocab, id_offset);
    embedding_rows_kernel<T, O, false><<<(unsigned)tokens, threads, 0, st>>>((const T*)dy, ids, first, more, acc, (O*)out, hidden, vocab, id_offset);
    embedding_rows_kernel<T, O, true><<<(unsigned)tokens, threads, 0, st>>>((const T*)dy, ids, first, more, acc, (O*)out, hidden, vocab, id_offset);
    return (int)cudaGetLastError();
}

}  // namespace lmoe

using namespace lmoe;

// out [vocab, hidden] (all of it written) from dy [tokens, hidden]; types as in lmoe_embedding_bwd.  Scratch: acc [tokens, hidden] fp32, tables
// [2 vocab] 32-bit.  hidden a multiple of 4, rows 16-byte aligned.
LMOE_API int lmoe_embedding_dense_grad(const void* dy, const int64_t* ids, void* out, float* acc, void* tables, int64_t tokens, int hidden,
                                       int64_t vocab, int64_t id_offset, int dy_dtype, int out_dtype, cudaStream_t st) {
    if (hidden % 4 != 0 || tokens >= 0x7fffffff) return -1;
    unsigned* t = (unsigned*)tables;
    if (dy_dtype == 1) return out_dtype == 1 ? dense_grad<bf16, bf16>(dy, ids, out, acc, t, tokens, hidden, vocab, id_offset, st)
                                             : dense_grad<bf16, float>(dy, ids, out, acc, t, tokens, hidden, vocab, id_offset, st);
    return out_dtype == 1 ? dense_grad<float, bf16>(dy, ids, out, acc, t, tokens, hidden, vocab, id_offset, st)
                          : dense_grad<float, float>(dy, ids, out, acc, t, tokens, hidden, vocab, id_offset, st);
}

// dy [tokens, hidden] (bf16: dtype 1, fp32: dtype 0), ids [tokens] int64, dw [vocab, hidden] fp32 (accumulated into).
LMOE_API int lmoe_embedding_bwd(const void* dy, const int64_t* ids, float* dw, int64_t tokens, int hidden, int64_t vocab,
                                int64_t id_offset, int dtype, cudaStream_t st) {
    if (tokens <= 0) return 0;
    const int vn = dtype == 1 ? 8 : 4;
    if (hidden % vn != 0) return -1;
    const int threads = hidden / vn >= 256 ? 256 : (hidden / vn >= 128 ? 128 : 64);
    const int blocks = (int)(tokens < 148 * 16 ? tokens : 148 * 16);
    if (dtype == 1) embedding_bwd_kernel<bf16><<<blocks, threads, 0, st>>>((const bf16*)dy, ids, dw, tokens, hidden, vocab, id_offset);
    else embedding_bwd_kernel<float><<<blocks, threads, 0, st>>>((const float*)dy, ids, dw, tokens, hidden, vocab, id_offset);
    return (int)cudaGetLastError();
}
