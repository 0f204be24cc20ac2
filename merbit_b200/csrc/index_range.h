// Index arithmetic of the kernels at the top of the accepted range (nrow + nnz
// up to INT_MAX - 64), in plain C++ so that it can also be run on the host.
#pragma once

#ifdef __CUDACC__
#define MERBIT_HD __host__ __device__ __forceinline__
#else
#define MERBIT_HD inline
#endif

namespace merbit {

// The SpMM walk counts nonzeros as in the whole matrix, and all lanes of a warp
// take as many steps as the longest of its segments: the counter of a lane group
// that is done runs up to 600 beyond the last nonzero.  It is unsigned, so that
// it stays above every end it is compared with.
// Nonzero c + t of a chunk; past the segment's end one of the tile again.
MERBIT_HD int walk_entry(unsigned c, unsigned t, int last) {
    return c + t < (unsigned)last ? (int)(c + t) : last;
}
// whether nonzero c + t lies in the segment
MERBIT_HD bool walk_in(unsigned c, unsigned t, int end) { return c + t < (unsigned)end; }
// whether no row or segment ends at or before nonzero c + n
MERBIT_HD bool walk_clear(int lim, unsigned c, unsigned n) { return (unsigned)lim > c + n; }

// f(i) for i = first, first + stride, ... below n: unsigned, as the last step
// passes n by up to a grid's threads (1.2 million) and n may be INT_MAX (+ 1)
template <class F>
MERBIT_HD void strided(unsigned first, unsigned stride, unsigned n, F&& f) {
    for (unsigned i = first; i < n; i += stride) f((int)i);
}

// Row groups: whether entry i + ahead of a row or staged run lies before its
// end (unsigned: a lane looks up to 480 entries past the last one)
MERBIT_HD bool before_end(unsigned i, unsigned ahead, int end) { return i + ahead < (unsigned)end; }

}  // namespace merbit
