// Front end of the reference harness: COO sort, COO -> CSR offsets and the
// loader's PageRank weights, on the GPU.
//
//   merbit_coo_sort        GRAPH::sort (src/class.cu:143-177): order the COO
//                          triplets by (major, minor); a stable radix sort
//                          of one 64-bit word per triplet that holds major,
//                          minor and the triplet's position, over the bits
//                          that major and minor use, then a gather
//   merbit_coo_to_csr      cusparseXcoo2csr (include/tile.cuh:574): offsets
//                          of a sorted index array
//   merbit_outdegree_values Fun_Values (src/class.cu:2-34): value = 1 /
//                          (number of entries whose row_ind equals this
//                          entry's row_ind)
#include <algorithm>

#include <cub/device/device_radix_sort.cuh>

#include "merbit_internal.cuh"

namespace merbit {
namespace {

int grid_of(long long n) {
    long long g = (n + 255) / 256;
    if (g > 148 * 32) g = 148 * 32;
    return (int)(g > 0 ? g : 1);
}

__global__ void pack_keys(const int* __restrict__ major, const int* __restrict__ minor, int n,
                          int b_minor, unsigned long long* __restrict__ key,
                          int* __restrict__ idx) {
    each_index((unsigned)n, [&](int i) {
        key[i] = ((unsigned long long)(unsigned)major[i] << b_minor) | (unsigned)minor[i];
        idx[i] = i;
    });
}

__global__ void unpack_keys(const unsigned long long* __restrict__ key, int n, int b_minor,
                            int* __restrict__ major, int* __restrict__ minor) {
    const unsigned long long min_mask = (1ull << b_minor) - 1;
    each_index((unsigned)n, [&](int i) {
        major[i] = (int)(key[i] >> b_minor);
        minor[i] = (int)(key[i] & min_mask);
    });
}

// Largest index of each array, as unsigned values.  One atomic per block: one per
// warp, 76,000 on two words, took most of this kernel's time.
__global__ void max_indices(const int* __restrict__ major, const int* __restrict__ minor, int n,
                            unsigned* __restrict__ out) {
    unsigned a = 0u, b = 0u;
    each_index((unsigned)n, [&](int i) {
        a = max(a, (unsigned)major[i]);
        b = max(b, (unsigned)minor[i]);
    });
    __shared__ unsigned top[2];
    if (threadIdx.x < 2) top[threadIdx.x] = 0u;
    __syncthreads();
    a = __reduce_max_sync(0xFFFFFFFFu, a);
    b = __reduce_max_sync(0xFFFFFFFFu, b);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(top, a);
        atomicMax(top + 1, b);
    }
    __syncthreads();
    if (threadIdx.x < 2) atomicMax(out + threadIdx.x, top[threadIdx.x]);
}

// One word per triplet: major, minor (b_minor bits) and position (b_pos bits).
__global__ void pack_words(const int* __restrict__ major, const int* __restrict__ minor, int n,
                           int b_minor, int b_pos, unsigned long long* __restrict__ word) {
    each_index((unsigned)n, [&](int i) {
        word[i] = ((((unsigned long long)(unsigned)major[i] << b_minor) | (unsigned)minor[i]) << b_pos) |
                  (unsigned)i;
    });
}

template <typename V>
__global__ void unpack_words(const unsigned long long* __restrict__ word, int n, int b_minor,
                             int b_pos, int* __restrict__ major, int* __restrict__ minor,
                             const V* __restrict__ src, V* __restrict__ dst) {
    const unsigned long long pos = (1ull << b_pos) - 1, min_mask = (1ull << b_minor) - 1;
    each_index((unsigned)n, [&](int i) {
        const unsigned long long w = word[i];
        major[i] = (int)(w >> (b_minor + b_pos));
        minor[i] = (int)((w >> b_pos) & min_mask);
        if (src) dst[i] = src[w & pos];
    });
}

int bits_of(unsigned long long v) {
    int b = 0;
    while (v >> b) ++b;
    return b;
}

template <typename V>
__global__ void permute_vals(const V* __restrict__ src, const int* __restrict__ perm, int n,
                             V* __restrict__ dst) {
    each_index((unsigned)n, [&](int i) { dst[i] = src[perm[i]]; });
}

// offsets[r] = first position with sorted[pos] >= r, r in [0, nrow].
__global__ void offsets_kernel(const int* __restrict__ sorted, int n, int nrow,
                               int* __restrict__ offsets) {
    each_index((unsigned)n + 1u, [&](int j) {
        const int prev = j == 0 ? -1 : max(min(sorted[j - 1], nrow), -1);
        const int cur = j == n ? nrow : min(sorted[j], nrow);
        for (long long r = (long long)prev + 1; r <= cur; ++r) offsets[r] = j;
    });
}

// cnt[nrow] counts indices outside [0, nrow).
__global__ void count_kernel(const int* __restrict__ idx, int n, int nrow, int* __restrict__ cnt) {
    each_index((unsigned)n, [&](int i) {
        const int r = idx[i];
        atomicAdd(cnt + ((unsigned)r < (unsigned)nrow ? r : nrow), 1);
    });
}

template <typename V>
__global__ void inv_count_kernel(const int* __restrict__ idx, const int* __restrict__ cnt, int n,
                                 int nrow, V* __restrict__ vals) {
    each_index((unsigned)n, [&](int i) {
        const int r = idx[i];
        vals[i] = (V)((unsigned)r < (unsigned)nrow ? 1.0 / (double)cnt[r] : 0.0);
    });
}

}  // namespace
}  // namespace merbit

using namespace merbit;

extern "C" {

int merbit_coo_sort(int32_t nnz, int32_t* d_major, int32_t* d_minor, void* d_vals,
                    merbit_dtype dtype, void* stream) {
    if (nnz < 0) return fail(MERBIT_ERR_INVALID, "coo_sort: negative nnz");
    if (nnz == 0) return MERBIT_OK;
    if (!d_major || !d_minor) return fail(MERBIT_ERR_INVALID, "coo_sort: null pointer");
    cudaStream_t s = (cudaStream_t)stream;
    unsigned long long *k_in = nullptr, *k_out = nullptr;
    int *i_in = nullptr, *i_out = nullptr;
    void* temp = nullptr;
    const size_t vs = dtype_size(dtype);
    auto done = [&](int st) {  // stream-ordered: after the sort's own work on s
        dev_free(k_in, s);
        dev_free(k_out, s);
        dev_free(i_in, s);
        dev_free(i_out, s);
        dev_free(temp, s);
        return st;
    };
#define TRY(call)                                              \
    do {                                                       \
        cudaError_t _e = (call);                               \
        if (_e != cudaSuccess) return done(cuda_fail(_e, #call)); \
    } while (0)
#define TRY_ALLOC(p, bytes)                              \
    do {                                                 \
        int _st = dev_alloc(&(p), (bytes), s);           \
        if (_st != MERBIT_OK) return done(_st);          \
    } while (0)
    // Indices of b1 and b2 bits and positions of b3 fit one word as a rule: then
    // keys alone are sorted, over b1 + b2 bits, between two buffers, and the
    // buffer that is free afterwards takes the values.  4 M triplets of a 250,000
    // node graph: 5 passes over 8 bytes instead of 8 over 12 (0.19 ms instead of
    // 0.42), and 64 MB of work space instead of 144.  That is what the pool keeps
    // mapped when nothing else is alive: the whole call takes 0.38 ms.  From 4.2 M
    // triplets on, or with other blocks alive, part of it is unmapped and mapped again at
    // every call (0.8 ms; 8 M 1.5 ms; 4 M beside a plan and its transpose 1.2 ms).
    TRY_ALLOC(k_in, 8 * (size_t)nnz);
    TRY_ALLOC(k_out, 8 * (size_t)nnz);
    unsigned top[2] = {0u, 0u};
    unsigned* d_top = reinterpret_cast<unsigned*>(k_out);  // not in use yet
    TRY(cudaMemsetAsync(d_top, 0, sizeof(top), s));
    max_indices<<<grid_of(nnz), 256, 0, s>>>(d_major, d_minor, nnz, d_top);
    TRY(cudaMemcpyAsync(top, d_top, sizeof(top), cudaMemcpyDeviceToHost, s));
    TRY(cudaStreamSynchronize(s));
    const int b_pos = bits_of((unsigned)(nnz - 1));
    const int b_minor = std::max(bits_of(top[1]), 1);
    const int b_all = b_pos + b_minor + std::max(bits_of(top[0]), 1);
    if (b_all <= 64) {
        pack_words<<<grid_of(nnz), 256, 0, s>>>(d_major, d_minor, nnz, b_minor, b_pos, k_in);
        cub::DoubleBuffer<unsigned long long> words(k_in, k_out);
        size_t tb = 0;
        TRY(cub::DeviceRadixSort::SortKeys(nullptr, tb, words, nnz, b_pos, b_all, s));
        TRY_ALLOC(temp, tb);
        TRY(cub::DeviceRadixSort::SortKeys(temp, tb, words, nnz, b_pos, b_all, s));
        if (d_vals)
            TRY(cudaMemcpyAsync(words.Alternate(), d_vals, vs * (size_t)nnz,
                                cudaMemcpyDeviceToDevice, s));
#define UNPACK(V)                                                                             \
    unpack_words<V><<<grid_of(nnz), 256, 0, s>>>(                                             \
        words.Current(), nnz, b_minor, b_pos, d_major, d_minor,                               \
        d_vals ? reinterpret_cast<const V*>(words.Alternate()) : nullptr, static_cast<V*>(d_vals))
        if (dtype == MERBIT_F64)
            UNPACK(double);
        else if (dtype == MERBIT_F32)
            UNPACK(float);
        else
            UNPACK(unsigned short);
#undef UNPACK
        TRY(cudaGetLastError());
        TRY(cudaStreamSynchronize(s));
        return done(MERBIT_OK);
    }
    // wider indices (or negative ones, as unsigned): keys and positions apart, sorted
    // over the bits that the indices use: two passes fewer than over 64 bits make up
    // for reading the largest indices back (1 M triplets of 20 million nodes 0.25 ms)
    TRY_ALLOC(i_in, 4 * (size_t)nnz);
    TRY_ALLOC(i_out, 4 * (size_t)nnz);
    pack_keys<<<grid_of(nnz), 256, 0, s>>>(d_major, d_minor, nnz, b_minor, k_in, i_in);
    size_t tb = 0;
    const int b_key = b_all - b_pos;
    TRY(cub::DeviceRadixSort::SortPairs(nullptr, tb, k_in, k_out, i_in, i_out, nnz, 0, b_key, s));
    TRY_ALLOC(temp, tb);
    TRY(cub::DeviceRadixSort::SortPairs(temp, tb, k_in, k_out, i_in, i_out, nnz, 0, b_key, s));
    unpack_keys<<<grid_of(nnz), 256, 0, s>>>(k_out, nnz, b_minor, d_major, d_minor);
    if (d_vals) {
        void* tmpv = k_in;  // free after the sort
        TRY(cudaMemcpyAsync(tmpv, d_vals, vs * (size_t)nnz, cudaMemcpyDeviceToDevice, s));
        if (dtype == MERBIT_F64)
            permute_vals<double><<<grid_of(nnz), 256, 0, s>>>((const double*)tmpv, i_out, nnz,
                                                              (double*)d_vals);
        else if (dtype == MERBIT_F32)
            permute_vals<float><<<grid_of(nnz), 256, 0, s>>>((const float*)tmpv, i_out, nnz,
                                                             (float*)d_vals);
        else
            permute_vals<unsigned short><<<grid_of(nnz), 256, 0, s>>>(
                (const unsigned short*)tmpv, i_out, nnz, (unsigned short*)d_vals);
    }
    TRY(cudaGetLastError());
    TRY(cudaStreamSynchronize(s));
#undef TRY
#undef TRY_ALLOC
    return done(MERBIT_OK);
}

int merbit_coo_to_csr(int32_t nnz, const int32_t* d_sorted_rows, int32_t nrow, int32_t* d_row_ptr,
                      void* stream) {
    if (nnz < 0 || nrow < 0 || !d_row_ptr || (nnz > 0 && !d_sorted_rows))
        return fail(MERBIT_ERR_INVALID, "coo_to_csr: bad arguments");
    offsets_kernel<<<grid_of((long long)nnz + 1), 256, 0, (cudaStream_t)stream>>>(
        d_sorted_rows, nnz, nrow, d_row_ptr);
    MERBIT_CUDA(cudaGetLastError());
    return MERBIT_OK;
}

int merbit_outdegree_values(int32_t nnz, int32_t nrow, const int32_t* d_row_ind, void* d_vals,
                            merbit_dtype dtype, void* stream) {
    if (nnz < 0 || nrow < 0 || (nnz > 0 && (!d_row_ind || !d_vals)))
        return fail(MERBIT_ERR_INVALID, "outdegree_values: bad arguments");
    if (nnz == 0) return MERBIT_OK;
    cudaStream_t s = (cudaStream_t)stream;
    int* cnt = nullptr;
    const size_t cbytes = sizeof(int) * ((size_t)nrow + 1);
    int st = dev_alloc(&cnt, cbytes, s);
    if (st != MERBIT_OK) return st;
    int bad = 0;
    cudaError_t e = cudaMemsetAsync(cnt, 0, cbytes, s);
    if (e == cudaSuccess) {
        count_kernel<<<grid_of(nnz), 256, 0, s>>>(d_row_ind, nnz, nrow, cnt);
        if (dtype == MERBIT_F64)
            inv_count_kernel<double><<<grid_of(nnz), 256, 0, s>>>(d_row_ind, cnt, nnz, nrow,
                                                                  (double*)d_vals);
        else if (dtype == MERBIT_F32)
            inv_count_kernel<float><<<grid_of(nnz), 256, 0, s>>>(d_row_ind, cnt, nnz, nrow,
                                                                 (float*)d_vals);
        else
            inv_count_kernel<__nv_bfloat16><<<grid_of(nnz), 256, 0, s>>>(
                d_row_ind, cnt, nnz, nrow, (__nv_bfloat16*)d_vals);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(&bad, cnt + nrow, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    dev_free(cnt, s);
    if (e != cudaSuccess) return cuda_fail(e, "outdegree_values");
    if (bad) return fail(MERBIT_ERR_MATRIX, "outdegree_values: row index outside [0, nrow)");
    return MERBIT_OK;
}

}  // extern "C"
