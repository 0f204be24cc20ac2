// Merge-path SpMM for sm_100a:  Y = alpha * A X + beta * Y  with K
// right-hand sides (row-major X [ncol x ldx], Y [nrow x ldy]), for one
// matrix or a batch of matrices in one persistent launch.
//
// The merge path of each matrix is cut into warp tiles of ITEMS merge
// items, as for the SpMV (spmv_warp.cu): lane 0 stages the tile's row_ptr
// window, col_idx slice and vals slice with cp.async.bulk on an mbarrier.
// Inside the warp, lanes form groups of K/VW lanes (VW = RHS values per
// lane: 1, 2 or 4); each group walks its own segment of ITEMS/G merge items
// (G groups per warp), lane j of a group owning RHS columns
// [j*VW, j*VW + VW).  The x rows of the next CH nonzeros are gathered while
// the current CH are accumulated, so gathers overlap the walk.  A row that
// begins and ends inside a segment is written directly, as vectors where Y
// allows it; the group segmented scan (shuffles with stride K/VW) finishes the
// rows split between groups, and rows split between tiles are finished
// per RHS column as in the SpMV: two-tile rows by an atomicExch
// swap of the partials (the later side writes carry + head), longer rows by
// a fixed-order look-back over the partials their tiles published, queued and
// taken when the warp has no tile left.  No float atomics: results are bitwise
// reproducible.
//
// What bounds it: instructions and the latency of the X-row gathers, not
// bytes.  So the walk has no condition per nonzero: while no group of the warp
// ends a row or its segment within a chunk (one vote), a chunk is loads and
// arithmetic only; row ends take a branch of their own, a row's sum goes to Y
// without passing through double when alpha = 1 and beta = 0, and only the
// slots that a launch uses are emptied for the next one (all of them, they
// were 20 MB of L2 for Zipf-1M at k = 16, whose X of 64 MB then no longer fit).
// Measured on B200 (one launch of a CUDA graph): Zipf-1M FP32 k = 16 347 us, its
// fused backward 525; Zipf-500k FP64 k = 8 147; 32 R-MAT matrices FP32 in one
// launch, k = 4 431 us, k = 32 1,090.
//
// Batches: the tiles of all matrices form one index space; matrix m owns
// tiles [tile_begin_m, tile_begin_m + num_tiles_m).  Warps of the
// persistent cooperative grid take tiles round-robin, so one launch covers
// the whole batch, and the launch can be captured in a CUDA graph and
// replayed (carry slots come in two parities; a launch empties the words that
// it uses in the other one, for the launch that follows).
//
// Fused backward (DV, merbit_spmm_dval): run on the transpose plan of A, the
// walk also forms dL/dval for each nonzero from the G row it has just
// gathered and the current row of X, and stores it through the transpose
// permutation (staged by TMA with the tile's col and vals).
#include <type_traits>

#include "merbit_internal.cuh"

namespace merbit {

namespace {

constexpr size_t a16(size_t b) { return (b + 15) & ~(size_t)15; }

template <int VW>
__device__ __forceinline__ void ld_vec(const float* p, float (&o)[VW]) {
    if (VW == 4) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(p));
        o[0] = t.x;
        o[1] = t.y;
        o[2] = t.z;
        o[3] = t.w;
    } else if (VW == 2) {
        const float2 t = __ldg(reinterpret_cast<const float2*>(p));
        o[0] = t.x;
        o[1] = t.y;
    } else {
        o[0] = __ldg(p);
    }
}
template <int VW>
__device__ __forceinline__ void ld_vec(const double* p, double (&o)[VW]) {
    if (VW >= 2) {
#pragma unroll
        for (int q = 0; q < VW; q += 2) {
            const double2 t = __ldg(reinterpret_cast<const double2*>(p) + q / 2);
            o[q] = t.x;
            o[q + 1] = t.y;
        }
    } else {
        o[0] = __ldg(p);
    }
}

template <typename Y>
__device__ __forceinline__ void st_row(Y* __restrict__ y, size_t off, double v, double alpha,
                                       double beta) {
    double o = alpha * v;
    if (beta != 0.0) o += beta * (double)y[off];
    y[off] = (Y)o;
}

// One lane's VW values of a Y row: a vector store where the address allows it
// (vec), else one store per column.
template <int VW>
__device__ __forceinline__ void st_vec(float* p, const float (&o)[VW], bool vec) {
    if (VW == 4 && vec) {
        __stcs(reinterpret_cast<float4*>(p), make_float4(o[0], o[1 % VW], o[2 % VW], o[3 % VW]));
    } else if (VW == 2 && vec) {
        __stcs(reinterpret_cast<float2*>(p), make_float2(o[0], o[1 % VW]));
    } else {
#pragma unroll
        for (int v = 0; v < VW; ++v) p[v] = o[v];
    }
}
template <int VW>
__device__ __forceinline__ void st_vec(double* p, const double (&o)[VW], bool vec) {
    if (VW >= 2 && vec) {
#pragma unroll
        for (int v = 0; v + 1 < VW; v += 2)
            __stcs(reinterpret_cast<double2*>(p + v), make_double2(o[v], o[(v + 1) % VW]));
    } else {
#pragma unroll
        for (int v = 0; v < VW; ++v) p[v] = o[v];
    }
}

__device__ __forceinline__ unsigned long long dbits(double v) {
    unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return b == kEmpty ? 0x7FF8000000000000ull : b;
}

}  // namespace

// Two floats in one 64-bit register pair, and arithmetic on both (sm_100).
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 f2_pack(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_unpack(f32x2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 f2_add(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 f2_sub(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 f2_fma(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 f2_mul(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// r = a b + c where `on`; r stays where not
__device__ __forceinline__ void f2_fma_if(bool on, f32x2& r, f32x2 a, f32x2 b, f32x2 c) {
    asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %4, 0;\n\t@p fma.rn.f32x2 %0, %1, %2, %3;\n\t}"
        : "+l"(r)
        : "l"(a), "l"(b), "l"(c), "r"((int)on));
}

// One lane's VW values of an X row, as they sit in registers: floats of an
// even width in pairs (as the load delivers them and the packed arithmetic
// takes them, so no moves), else one by one.
template <typename X, int VW>
struct XRow {
    X r[VW];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int v = 0; v < VW; ++v) r[v] = (X)0;
    }
    __device__ __forceinline__ void load(const X* p) { ld_vec<VW>(p, r); }
    __device__ __forceinline__ X operator[](int v) const { return r[v]; }
};
template <int VW>
struct XPairs {
    static_assert(VW == 2 || VW == 4, "pairs");
    f32x2 r[VW / 2];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int h = 0; h < VW / 2; ++h) r[h] = 0ull;
    }
    __device__ __forceinline__ void load(const float* p) {
        if constexpr (VW == 4) {
            const ulonglong2 t = __ldg(reinterpret_cast<const ulonglong2*>(p));
            r[0] = t.x;
            r[1] = t.y;
        } else {
            r[0] = __ldg(reinterpret_cast<const unsigned long long*>(p));
        }
    }
    __device__ __forceinline__ float operator[](int v) const {
        float lo, hi;
        f2_unpack(r[v / 2], lo, hi);
        return (v & 1) ? hi : lo;
    }
};
template <>
struct XRow<float, 2> : XPairs<2> {};
template <>
struct XRow<float, 4> : XPairs<4> {};

// The VW accumulators of one lane.
//   add, set     one product per column: into the sum, or as a row's first
//   add_two      a0 x0 and, with `both`, a1 x1 of the same row
//   add_p        products formed beforehand
//   value        the sum in double; rounded: in the type of Y
//   stash, unstash   to and from this lane's place in a shared-memory area
//                    of 256 * VW bytes
// F64: one double per column.
template <class Acc, int VW, typename P, typename X>
struct AccRow {
    double a[VW];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int v = 0; v < VW; ++v) a[v] = 0.0;
    }
    __device__ __forceinline__ void add(P av, const XRow<X, VW>& x) {
#pragma unroll
        for (int v = 0; v < VW; ++v) a[v] += av * (P)x[v];
    }
    __device__ __forceinline__ void set(P av, const XRow<X, VW>& x) {
#pragma unroll
        for (int v = 0; v < VW; ++v) a[v] = 0.0 + av * (P)x[v];
    }
    __device__ __forceinline__ void add_two(P a0, const XRow<X, VW>& x0, P a1,
                                            const XRow<X, VW>& x1, bool both = true) {
        add(a0, x0);
        if (both) add(a1, x1);
    }
    __device__ __forceinline__ void add_p(const P (&p)[VW]) {
#pragma unroll
        for (int v = 0; v < VW; ++v) a[v] += p[v];
    }
    __device__ __forceinline__ double value(int v) const { return a[v]; }
    __device__ __forceinline__ void rounded(X (&o)[VW]) const {
#pragma unroll
        for (int v = 0; v < VW; ++v) o[v] = (X)a[v];
    }
    __device__ __forceinline__ void stash(unsigned char* p, int lane) const {
        if constexpr (VW == 1) {
            reinterpret_cast<double*>(p)[lane] = a[0];
        } else {
#pragma unroll
            for (int h = 0; h < VW / 2; ++h)
                reinterpret_cast<double2*>(p)[32 * h + lane] = make_double2(a[2 * h], a[2 * h + 1]);
        }
    }
    __device__ __forceinline__ void unstash(const unsigned char* p, int lane) {
        if constexpr (VW == 1) {
            a[0] = reinterpret_cast<const double*>(p)[lane];
        } else {
#pragma unroll
            for (int h = 0; h < VW / 2; ++h) {
                const double2 t = reinterpret_cast<const double2*>(p)[32 * h + lane];
                a[2 * h] = t.x;
                a[2 * h + 1] = t.y;
            }
        }
    }
};

// FP32/BF16, an even number of columns: TwoSum accumulators, two columns per
// packed f32x2 instruction.  The steps are Knuth's, with n = s - t in the
// place of -(t - s): t = s + q, e = (s - (t + n)) + (q + n).  A lone product
// enters with its own rounding error (a x + n instead of q + n); two products
// of one row enter as q = fma(a1, x1, a0 x0), whose two roundings cost at most
// u (2 |a0 x0| + |a1 x1|), u = 2^-24 (half a unit in the last place).
template <int VW>
struct AccRow<AccTwoSum, VW, float, float> {
    static_assert(VW % 2 == 0, "packed TwoSum needs an even width");
    using XR = XRow<float, VW>;
    f32x2 s[VW / 2], c[VW / 2];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int h = 0; h < VW / 2; ++h) s[h] = c[h] = 0ull;  // +0.0f, +0.0f
    }
    // t = s + q; (s, c) take t and its error, `qn` being q + n
    __device__ __forceinline__ void finish(int h, f32x2 t, f32x2 n, f32x2 qn) {
        c[h] = f2_add(c[h], f2_add(f2_sub(s[h], f2_add(t, n)), qn));
        s[h] = t;
    }
    __device__ __forceinline__ void add(float av, const XR& x) {
        const f32x2 a2 = f2_pack(av, av);
#pragma unroll
        for (int h = 0; h < VW / 2; ++h) {
            const f32x2 t = f2_add(s[h], f2_mul(a2, x.r[h]));
            const f32x2 n = f2_sub(s[h], t);
            finish(h, t, n, f2_fma(a2, x.r[h], n));
        }
    }
    __device__ __forceinline__ void set(float av, const XR& x) {
        const f32x2 a2 = f2_pack(av, av);
#pragma unroll
        for (int h = 0; h < VW / 2; ++h) {
            s[h] = f2_mul(a2, x.r[h]);
            c[h] = f2_fma(a2, x.r[h], f2_sub(0ull, s[h]));
        }
    }
    __device__ __forceinline__ void add_two(float a0, const XR& x0, float a1, const XR& x1) {
        const f32x2 b0 = f2_pack(a0, a0), b1 = f2_pack(a1, a1);
#pragma unroll
        for (int h = 0; h < VW / 2; ++h) {
            const f32x2 q = f2_fma(b1, x1.r[h], f2_mul(b0, x0.r[h]));
            const f32x2 t = f2_add(s[h], q);
            const f32x2 n = f2_sub(s[h], t);
            finish(h, t, n, f2_add(q, n));
        }
    }
    // the same when only some lanes of the warp have a second product
    __device__ __forceinline__ void add_two(float a0, const XR& x0, float a1, const XR& x1,
                                            bool both) {
        const f32x2 b0 = f2_pack(a0, a0), b1 = f2_pack(a1, a1);
#pragma unroll
        for (int h = 0; h < VW / 2; ++h) {
            f32x2 q = f2_mul(b0, x0.r[h]);
            f2_fma_if(both, q, b1, x1.r[h], q);
            const f32x2 t = f2_add(s[h], q);
            const f32x2 n = f2_sub(s[h], t);
            f32x2 qn = f2_add(q, n);
            f2_fma_if(!both, qn, b0, x0.r[h], n);
            finish(h, t, n, qn);
        }
    }
    __device__ __forceinline__ void add_p(const float (&p)[VW]) {
#pragma unroll
        for (int h = 0; h < VW / 2; ++h) {
            const f32x2 q = f2_pack(p[2 * h], p[2 * h + 1]);
            const f32x2 t = f2_add(s[h], q);
            const f32x2 n = f2_sub(s[h], t);
            finish(h, t, n, f2_add(q, n));
        }
    }
    __device__ __forceinline__ double value(int v) const {
        float s0, s1, c0, c1;
        f2_unpack(s[v / 2], s0, s1);
        f2_unpack(c[v / 2], c0, c1);
        return (v & 1) ? (double)s1 + (double)c1 : (double)s0 + (double)c0;
    }
    __device__ __forceinline__ void rounded(float (&o)[VW]) const {
#pragma unroll
        for (int h = 0; h < VW / 2; ++h) f2_unpack(f2_add(s[h], c[h]), o[2 * h], o[2 * h + 1]);
    }
    __device__ __forceinline__ void stash(unsigned char* p, int lane) const {
#pragma unroll
        for (int h = 0; h < VW / 2; ++h)
            reinterpret_cast<ulonglong2*>(p)[32 * h + lane] = make_ulonglong2(s[h], c[h]);
    }
    __device__ __forceinline__ void unstash(const unsigned char* p, int lane) {
#pragma unroll
        for (int h = 0; h < VW / 2; ++h) {
            const ulonglong2 t = reinterpret_cast<const ulonglong2*>(p)[32 * h + lane];
            s[h] = t.x;
            c[h] = t.y;
        }
    }
};
// FP32/BF16, one column.
template <>
struct AccRow<AccTwoSum, 1, float, float> {
    using XR = XRow<float, 1>;
    AccTwoSum a;
    __device__ __forceinline__ void zero() { a.zero(); }
    __device__ __forceinline__ void add(float av, const XR& x) { a.add(av * x[0]); }
    __device__ __forceinline__ void set(float av, const XR& x) {
        a.zero();
        add(av, x);
    }
    __device__ __forceinline__ void add_two(float a0, const XR& x0, float a1, const XR& x1,
                                            bool both = true) {
        add(a0, x0);
        if (both) add(a1, x1);
    }
    __device__ __forceinline__ void add_p(const float (&p)[1]) { a.add(p[0]); }
    __device__ __forceinline__ double value(int) const { return a.value(); }
    __device__ __forceinline__ void rounded(float (&o)[1]) const { o[0] = __fadd_rn(a.s, a.c); }
    __device__ __forceinline__ void stash(unsigned char* p, int lane) const {
        reinterpret_cast<float2*>(p)[lane] = make_float2(a.s, a.c);
    }
    __device__ __forceinline__ void unstash(const unsigned char* p, int lane) {
        const float2 t = reinterpret_cast<const float2*>(p)[lane];
        a.s = t.x;
        a.c = t.y;
    }
};

// A row that began two or more tiles before the tile that completes it: its
// carry-in is the sum of the partials of the tiles in between, which other
// warps process at about the same time.  The completing tile leaves its own
// part (the head) in its boundary-swap slot, which such a row does not use,
// and queues the look-back; the warp takes it when the queue is full, else
// after its last tile, so that it does not wait for tiles while it has others
// to process.  (Taken on the spot, the look-backs held up Zipf-1M at k = 16
// for a third of its time.)
struct SpmmLookBack {
    void* y;    // the row of Y
    int head;   // the completing tile (its slots hold the head)
    int first;  // the tile in which the row begins
};
constexpr int kSpmmLookBacks = 8;

// One look-back by one warp: lane l takes column l % K of tiles first + l / K,
// + 32 / K, ...; R loads are in flight before any is summed, so a row of
// hundreds of tiles takes few round trips.  The order of the sums depends only
// on the tiles.
template <int K, typename Y>
__device__ __forceinline__ void spmm_look_back(const SpmmLookBack& e, unsigned long long* slots,
                                               unsigned long long* xch, LaunchState* st,
                                               double alpha, double beta, int cols, int lane) {
    constexpr int TPS = 32 / K;
    constexpr int R = 8;
    const int j = lane % K;
    double sum = 0.0;
    for (int t = e.first + lane / K; t < e.head; t += TPS * R) {
        unsigned long long bits[R];
        load_carries<R>(bits, slots + (size_t)t * K + j, TPS * K, (e.head - t) * K, st);
#pragma unroll
        for (int r = 0; r < R; ++r) sum += __longlong_as_double((long long)bits[r]);
    }
    __syncwarp();
#pragma unroll
    for (int o = K; o < 32; o <<= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    if (lane < cols) {  // cols <= K
        const double head =
            __longlong_as_double((long long)ld_relaxed_u64(xch + (size_t)e.head * K + j));
        st_row(static_cast<Y*>(e.y), j, sum + head, alpha, beta);
    }
}

template <int K, typename Y>
__device__ __forceinline__ void drain_spmm_look_backs(const SpmmLookBack* q, int n,
                                                      const SpmmLaunch& a, unsigned epoch,
                                                      int lane) {
    __syncwarp();
    const size_t par = (size_t)(epoch & 1u) * a.nslots;
    for (int i = 0; i < n; ++i)
        spmm_look_back<K, Y>(q[i], a.slots + par, a.xch + par, a.state, a.alpha, a.beta,
                             a.cols, lane);
    __syncwarp();
}

constexpr bool spmm_staged_products(int k, int vw, int items, bool dv) {
    return k == 2 && vw == 2 && (items == 224 || items == 352) && !dv;
}

// DV: also form dL/dval for each nonzero (SpmmLaunch::dv_*), from the x row
// the walk gathers anyway and the current row of dv_x.
template <int DT, int K, int VW, int ITEMS, bool DV = false>
struct SpmmTile {
    using Pr = Prec<DT>;
    using V = typename Pr::V;
    using X = typename Pr::X;
    using Y = typename Pr::Y;
    using P = typename Pr::P;
    using Acc = typename Pr::Acc;
    static constexpr int LPG = K / VW;      // lanes per group
    static constexpr int G = 32 / LPG;      // groups per warp
    static constexpr int SEG = ITEMS / G;   // merge items per group
    // nonzeros gathered ahead: 8 values per lane; at k = 1 (one lane per
    // group, latency-bound) 4, which measured 12% faster on the 128-matrix
    // R-MAT batch (2.25 -> 1.98 ms; 16 ahead: 2.55 ms).  The chunk size does
    // not change the order of the additions.
    static constexpr int CH = K == 1 ? 4 : 8 / VW;
    // Staged products (one lane per group, tiles of 224 or 352 items, no
    // fused dval): the warp gathers the X rows of all the tile's nonzeros
    // lane-contiguously, every gather in flight at once, and stores the
    // products in shared memory; each lane then walks its segment from
    // there.  The chunked walk instead keeps only CH nonzeros ahead per lane.
    static constexpr bool STAGEP = spmm_staged_products(K, VW, ITEMS, DV);
    static constexpr int NJ = ITEMS / 32;  // staged products per lane
    static constexpr int CAP = ITEMS + 32;
    static constexpr int RPC = ITEMS + 16;  // row_ptr window (any rows per tile, and the
                                            // end of the row that goes on after it)
    static constexpr size_t rp_bytes = a16((size_t)RPC * 4);
    static constexpr size_t col_bytes = a16((size_t)CAP * 4);
    static constexpr size_t val_bytes = a16((size_t)CAP * sizeof(V));
    // DV: the tile's slice of the transpose permutation, staged like col
    static constexpr size_t perm_bytes = DV ? a16((size_t)CAP * 4) : 0;
    static constexpr size_t perm_offset = rp_bytes + col_bytes + val_bytes;
    static constexpr size_t prod_bytes = STAGEP ? a16((size_t)ITEMS * VW * sizeof(P)) : 0;
    static constexpr size_t prod_offset = perm_offset + perm_bytes;
    // each lane's first finished row of its segment, kept until the scan
    static constexpr size_t first_offset = prod_offset + prod_bytes;
    static constexpr size_t first_bytes = (size_t)256 * VW;
    static constexpr size_t bar_offset = first_offset + first_bytes;
    static constexpr size_t bytes = bar_offset + 16;
    static constexpr int GV = 16 / (int)sizeof(V);
    static_assert(LPG >= 1 && LPG <= 32 && 32 % LPG == 0, "K/VW must divide 32");
    static_assert(SEG * G == ITEMS, "ITEMS must be a multiple of the group count");

    static __device__ __forceinline__ void issue(const SpmmDesc& d, int lt, unsigned char* ws,
                                                 uint64_t* bar, int lane,
                                                 const int* perm = nullptr) {
        const int2 c0 = d.coords[lt];
        const int2 c1 = d.coords[lt + 1];
        int* s_rp = reinterpret_cast<int*>(ws);
        int* s_col = reinterpret_cast<int*>(ws + rp_bytes);
        V* s_val = reinterpret_cast<V*>(ws + rp_bytes + col_bytes);
        const V* vals = static_cast<const V*>(d.vals);
        const int nrp = d.nrow + 1;
        const int rp_end = min(c1.y + 2, nrp);  // the trailing row's end too
        // bulk copies need 16-byte aligned global addresses; an array whose
        // base is not 16-byte aligned (a caller's offset view) is staged by
        // plain loads instead (no transaction bytes)
        auto bb = [](const void* src, int s, int e, int n, int g, int esz) -> unsigned {
            if (e <= s || ((uintptr_t)src & 15u) != 0) return 0u;
            const int base = s & ~(g - 1), lim = n & ~(g - 1);
            const int b_end = min((e + g - 1) & ~(g - 1), lim);
            return b_end > base ? (unsigned)(b_end - base) * (unsigned)esz : 0u;
        };
        const unsigned tot = bb(d.row_ptr, c0.y, rp_end, nrp, 4, 4) +
                             bb(d.col, c0.x, c1.x, d.nnz, 4, 4) +
                             bb(vals, c0.x, c1.x, d.nnz, GV, (int)sizeof(V)) +
                             (DV ? bb(perm, c0.x, c1.x, d.nnz, 4, 4) : 0u);
        __syncwarp();
        if (lane == 0) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_arrive_expect_tx(bar, tot);
        }
        const uint64_t pol = l2_evict_first_policy();
        auto stage = [&](auto* dst, const auto* src, int s, int e, int n) {
            using T = typename std::remove_pointer<decltype(dst)>::type;
            constexpr int GG = 16 / (int)sizeof(T);
            if (e <= s) return;
            const int base = s & ~(GG - 1), lim = n & ~(GG - 1);
            if (((uintptr_t)src & 15u) != 0) {  // warp-uniform: plain loads
                for (int i = s + lane; i < e; i += 32) dst[i - base] = src[i];
                return;
            }
            const int b_end = min((e + GG - 1) & ~(GG - 1), lim);
            if (b_end > base && lane == 0)
                bulk_g2s(dst, src + base, (unsigned)(b_end - base) * (unsigned)sizeof(T), bar, pol);
            const int p0 = max(b_end, s);
            if (lane < e - p0) dst[p0 + lane - base] = src[p0 + lane];
        };
        stage(s_rp, d.row_ptr, c0.y, rp_end, nrp);
        stage(s_col, d.col, c0.x, c1.x, d.nnz);
        stage(s_val, vals, c0.x, c1.x, d.nnz);
        if (DV) stage(reinterpret_cast<int*>(ws + perm_offset), perm, c0.x, c1.x, d.nnz);
    }

    static __device__ __forceinline__ void process(const SpmmLaunch& a, const SpmmDesc& d,
                                                   int u, int lt, unsigned epoch,
                                                   unsigned char* ws, int lane,
                                                   SpmmLookBack* lbq, int& nlb) {
        unsigned long long* slots = a.slots;
        unsigned long long* xch = a.xch;
        const int nslots = a.nslots;
        const int* s_rp = reinterpret_cast<const int*>(ws);
        const int* s_col = reinterpret_cast<const int*>(ws + rp_bytes);
        const V* s_val = reinterpret_cast<const V*>(ws + rp_bytes + col_bytes);
        const int2 c0 = d.coords[lt];
        const int2 c1 = d.coords[lt + 1];
        const int prev_x = lt > 0 ? d.coords[lt - 1].x : 0;
        const int x0 = c0.x, y0 = c0.y, x1 = c1.x, y1 = c1.y;
        const int nz = x1 - x0, nr = y1 - y0, L = nz + nr;
        const int rpo = y0 - (y0 & ~3);
        const int g = lane / LPG;        // group
        const int jl = lane % LPG;       // lane within group
        const int j0 = jl * VW;          // first RHS column of this lane
        // With fewer columns than K the lanes beyond them run along on the
        // first lane's X (no further sectors) and store nothing.
        const bool active = j0 < a.cols;
        // this lane's columns of X, and the distance of its rows in bytes (32
        // bits with vector loads: one wide multiply-add per address)
        using Step = typename std::conditional<(VW > 1), unsigned, unsigned long long>::type;
        const char* __restrict__ xl =
            reinterpret_cast<const char*>(static_cast<const X*>(d.x) + (active ? j0 : 0));
        const Step xstep = (Step)((unsigned long long)d.ldx * sizeof(X));
        char* __restrict__ yl = reinterpret_cast<char*>(static_cast<Y*>(d.y) + j0);
        const Step ystep = (Step)((unsigned long long)d.ldy * sizeof(Y));
        auto y_row = [&](int r) {  // row r of the matrix
            return reinterpret_cast<Y*>(yl + (unsigned long long)(unsigned)r * ystep);
        };
        const int nrow = d.nrow;
        const double alpha = a.alpha, beta = a.beta;
        // plain product: a row's sum is rounded to Y as it is
        const bool plain = alpha == 1.0 && beta == 0.0;
        // Y rows of this lane start on its vector width
        const bool vecy = VW > 1 && (((uintptr_t)yl | ystep) &
                                     (VW * sizeof(Y) < 16 ? VW * sizeof(Y) - 1 : 15)) == 0;
        // row r of Y from its sum in double
        auto finish_row = [&](int r, const double (&v)[VW]) {
            if (!active) return;
            Y* yr = y_row(r);
            if (plain) {
                Y o[VW];
#pragma unroll
                for (int q = 0; q < VW; ++q) o[q] = (Y)v[q];
                st_vec<VW>(yr, o, vecy);
            } else {
#pragma unroll
                for (int q = 0; q < VW; ++q) st_row(yr, q, v[q], alpha, beta);
            }
        };

        // ---- this group's segment of the tile's merge path; it ends where
        // the next group's starts.  Nonzeros are counted as in the whole
        // matrix: rp_t[r] is the end of the tile's row r - 1, col_t[e] and
        // val_t[e] belong to nonzero e.
        const int* rp_t = s_rp + rpo;
        const int* col_t = s_col - (x0 & ~3);
        const V* val_t = s_val - (x0 & ~(GV - 1));
        int lx, ly;
        {
            const int ds = min(g * SEG, L);
            int lo = max(ds - nz, 0), hi = min(ds, nr);
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (rp_t[mid + 1] - x0 <= ds - mid - 1)
                    lo = mid + 1;
                else
                    hi = mid;
            }
            ly = lo;
            lx = x0 + ds - lo;
        }
        int lx_end = x1, ly_end = nr;
        if (G > 1) {
            const int tx = __shfl_down_sync(0xFFFFFFFFu, lx, LPG);
            const int ty = __shfl_down_sync(0xFFFFFFFFu, ly, LPG);
            if (g < G - 1) {
                lx_end = tx;
                ly_end = ty;
            }
        }

        AccRow<Acc, VW, P, X> acc;
        acc.zero();
        unsigned char* s_first = ws + first_offset;
        const bool any_end = ly < ly_end;  // a row ends in this segment
        // The row open where the segment starts (`open`: it began before, in an
        // earlier group or tile) is kept for the scan when it ends here; the
        // rows that begin and end in the segment go to Y.  Rows without
        // nonzeros are written after the walk.
        const int first_row = ly;
        bool open = any_end && rp_t[ly] < lx;
        const bool had_open = open;
        // end of the current row (INT_MAX past the segment's last row), kept in
        // a register so the walk reads row_ptr once per row, not per nonzero;
        // lim: the nonzero at which the current row or the segment ends
        int next_end, lim;
        auto next_row = [&](int e) {  // the first row from ly on that ends beyond e
            for (;;) {
                next_end = ly < ly_end ? rp_t[ly + 1] : INT_MAX;
                if (next_end > e) break;
                ++ly;
            }
            lim = min(next_end, lx_end);
        };
        if (open && rp_t[ly + 1] == lx) {  // its nonzeros all came before
            acc.stash(s_first, lane);
            open = false;
            ++ly;
        }
        next_row(lx);

        // fused dval: this lane's VW values of dv_x's current row, loaded when
        // the segment has a nonzero of it.  (Loading the row after it ahead, or
        // one shuffle tree for two nonzeros, was no faster: Zipf-1M FP32 at k = 16
        // took 542 and 539 us against 537.  The scattered dval writes bind this
        // form: their 97 MB and G's 64 MB do not fit L2 together.)
        const int* perm_t = reinterpret_cast<const int*>(ws + perm_offset) - (x0 & ~3);
        XRow<X, VW> xrow;
        auto dv_row = [&](int e) {  // ly is the current row, e the next nonzero
            if (e < lx_end)
                xrow.load(static_cast<const X*>(a.dv_x) + (size_t)(y0 + ly) * a.dv_ldx + j0);
        };
        if (DV) {
            xrow.zero();
            dv_row(lx);
        }
        const unsigned gmask = LPG == 32 ? 0xFFFFFFFFu : (((1u << LPG) - 1u) << (g * LPG));
        // dval of nonzero e: in the x type, VW fused multiply-adds per lane, then
        // a tree over the group's lanes (error within (VW + log2 LPG) roundings
        // of sum |g x|)
        X* __restrict__ dvo = static_cast<X*>(a.dv_out);
        auto dv_one = [&](int e, const XRow<X, VW>& xr) {
            X dd = (X)0;
#pragma unroll
            for (int v = 0; v < VW; ++v) dd = fma(xr[v], xrow[v], dd);
#pragma unroll
            for (int o = LPG / 2; o > 0; o >>= 1) dd += __shfl_xor_sync(gmask, dd, o);
            if (jl == 0) dvo[perm_t[e]] = dd;
        };

        // the current row ends at nonzero e
        auto end_row = [&](int e) {
            if (open) {
                acc.stash(s_first, lane);
                open = false;
            } else if (plain) {
                Y o[VW];
                acc.rounded(o);
                if (active) st_vec<VW>(y_row(y0 + ly), o, vecy);
            } else if (active) {
                Y* yr = y_row(y0 + ly);
#pragma unroll
                for (int v = 0; v < VW; ++v) st_row(yr, v, acc.value(v), alpha, beta);
            }
            acc.zero();
            ++ly;
            next_row(e);
            if (DV) dv_row(e);
        };

        // ---- walk: chunks of CH nonzeros, the next chunk's x rows in flight
        // (two named buffers, so both stay in registers)
        XRow<X, VW> xa[CH], xb[CH];
        V va[CH], vb[CH];
        // (past the segment's end a nonzero of the tile is read again: loads
        // without conditions; used only when the tile has nonzeros)
        const int e_last = max(lx_end - 1, x0);
        auto load_chunk = [&](unsigned c, XRow<X, VW> (&xr)[CH], V (&vv)[CH]) {
#pragma unroll
            for (int t = 0; t < CH; ++t) {
                const int e = walk_entry(c, t, e_last);
                const unsigned colv = (unsigned)col_t[e];
                vv[t] = val_t[e];
                xr[t].load(reinterpret_cast<const X*>(xl + (unsigned long long)colv * xstep));
            }
        };
        // nonzeros c .. c + CH - 1 (those below lx_end); every row that ends at
        // or before c is finished, so c belongs to row ly.  Called by all
        // lanes of the warp.
        auto consume = [&](unsigned at, const XRow<X, VW> (&xr)[CH], const V (&vv)[CH]) {
            const int c = (int)at;  // used below lx_end only
            if (__all_sync(0xFFFFFFFFu, walk_clear(lim, at, CH))) {  // no row or segment ends here
                if constexpr (CH == 2) {
                    // F32/BF16: one compensated addition of the fused pair
                    acc.add_two(to_p(vv[0]), xr[0], to_p(vv[1]), xr[1]);
                    if (DV) {
                        dv_one(c, xr[0]);
                        dv_one(c + 1, xr[1]);
                    }
                } else {
#pragma unroll
                    for (int t = 0; t < CH; ++t) {
                        acc.add(to_p(vv[t]), xr[t]);
                        if (DV) dv_one(c + t, xr[t]);
                    }
                }
                return;
            }
            if constexpr (CH == 2) {
                const bool both = walk_clear(lim, at, 1);
                if (walk_in(at, 0, lx_end)) {
                    acc.add_two(to_p(vv[0]), xr[0], to_p(vv[1]), xr[1], both);
                    if (DV) {
                        dv_one(c, xr[0]);
                        if (both) dv_one(c + 1, xr[1]);
                    }
                    if (next_end == c + 1) {
                        end_row(c + 1);
                        if (c + 1 < lx_end) {
                            acc.set(to_p(vv[1]), xr[1]);
                            if (DV) dv_one(c + 1, xr[1]);
                        }
                    }
                    if (next_end == c + 2) end_row(c + 2);
                }
            } else {
#pragma unroll
                for (int t = 0; t < CH; ++t) {
                    if (walk_in(at, t, lx_end)) {
                        acc.add(to_p(vv[t]), xr[t]);
                        if (DV) dv_one(c + t, xr[t]);
                        if (next_end == c + t + 1) end_row(c + t + 1);
                    }
                }
            }
            __syncwarp();
        };
        if constexpr (STAGEP) {
            // products of the tile's nonzero i at s_prod[i * VW]
            P* s_prod = reinterpret_cast<P*>(ws + prod_offset);
            {
                int cidx[NJ];
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    const int i = lane + 32 * j;
                    cidx[j] = i < nz ? col_t[x0 + i] : 0;
                }
                XRow<X, VW> xr[NJ];
#pragma unroll
                for (int j = 0; j < NJ; ++j)
                    if (lane + 32 * j < nz)
                        xr[j].load(reinterpret_cast<const X*>(
                            xl + (unsigned long long)(unsigned)cidx[j] * xstep));
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    const int i = lane + 32 * j;
                    if (i < nz) {
                        const P av = to_p(val_t[x0 + i]);
#pragma unroll
                        for (int v = 0; v < VW; ++v) s_prod[(size_t)i * VW + v] = av * (P)xr[j][v];
                    }
                }
            }
            __syncwarp();
            for (int e = lx; e < lx_end; ++e) {
                P pv[VW];
#pragma unroll
                for (int v = 0; v < VW; ++v) pv[v] = s_prod[(size_t)(e - x0) * VW + v];
                acc.add_p(pv);
                if (next_end == e + 1) end_row(e + 1);
            }
        } else {
            // as many steps for every lane: the longest segment's
            const int steps = __reduce_max_sync(0xFFFFFFFFu, (lx_end - lx + 2 * CH - 1) / (2 * CH));
            // The last step loads no chunk beyond it where segments are short, a few
            // steps each (k = 1: 5% less time); on longer ones the branch costs more
            // than the load, and FP64 kernels would pass the registers they are bound to.
            constexpr bool kLastLoad = K >= 16 || (DT == MERBIT_F64 && (!DV || K >= 8));
            unsigned c = (unsigned)lx;
            if (steps > 0) load_chunk(c, xa, va);
            for (int i = 1; i <= steps; ++i) {
                load_chunk(c + CH, xb, vb);
                consume(c, xa, va);
                if (kLastLoad || i < steps) load_chunk(c + 2 * CH, xa, va);  // warp-uniform
                consume(c + CH, xb, vb);
                c += 2 * CH;
            }
        }

        // ---- rows without nonzeros, G at a time
        for (int r0 = 0; r0 < nr; r0 += 32) {
            const int rl = r0 + lane;
            const unsigned m =
                __ballot_sync(0xFFFFFFFFu, rl < nr && rp_t[min(rl, nr - 1) + 1] == rp_t[min(rl, nr - 1)]);
            if (m == 0u) continue;
            for (int i = g; i < 32; i += G) {
                if ((m >> i) & 1u) {
                    double zero[VW];
#pragma unroll
                    for (int v = 0; v < VW; ++v) zero[v] = 0.0;
                    finish_row(y0 + r0 + i, zero);
                }
            }
        }

        // ---- group segmented scan, per RHS column (stride LPG lanes)
        int f = any_end;
        double sv[VW];
#pragma unroll
        for (int v = 0; v < VW; ++v) sv[v] = acc.value(v);
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
            double t[VW];
#pragma unroll
            for (int v = 0; v < VW; ++v) t[v] = __shfl_up_sync(0xFFFFFFFFu, sv[v], o * LPG);
            const int tf = __shfl_up_sync(0xFFFFFFFFu, f, o * LPG);
            if (g >= o) {
                if (!f) {
#pragma unroll
                    for (int v = 0; v < VW; ++v) sv[v] = t[v] + sv[v];
                }
                f |= tf;
            }
        }
        double ev[VW];
#pragma unroll
        for (int v = 0; v < VW; ++v) {
            ev[v] = G > 1 ? __shfl_up_sync(0xFFFFFFFFu, sv[v], LPG) : 0.0;
            if (g == 0) ev[v] = 0.0;
        }
        const int rs = s_rp[rpo];
        const bool need_lb = nr > 0 && rs < x0;
        const bool holds_first = had_open && first_row == 0 && need_lb;
        AccRow<Acc, VW, P, X> first;
        first.zero();
        if (had_open) first.unstash(s_first, lane);
        double rv[VW];
#pragma unroll
        for (int v = 0; v < VW; ++v) rv[v] = ev[v] + first.value(v);
        if (had_open && !holds_first) finish_row(y0 + first_row, rv);

        // ---- the tile's trailing partial (last group).  Row y1 ends in tile
        // lt_end: if it began in this tile and ends in the next, the two swap
        // their partials; if it spans more tiles, the partial is published for
        // the look-back of the tile it ends in.  The words that this launch
        // uses are emptied in the other parity, for the next launch: which
        // they are depends on the matrix and the tile size alone.
        const size_t par = (size_t)(epoch & 1u) * nslots;
        const size_t other = (size_t)((epoch + 1u) & 1u) * nslots;
        if (g == G - 1 && y1 < nrow && lt + 1 < d.num_tiles) {
            const bool began_here = rp_t[nr] >= x0 && rp_t[nr] < x1;
            const int lt_end = (int)((unsigned)(rp_t[nr + 1] + y1) / (unsigned)ITEMS);
            if (began_here && lt_end == lt + 1) {
                const size_t w = (size_t)(u + 1) * K + j0;
#pragma unroll
                for (int v = 0; v < VW; ++v) {
                    st_relaxed_u64(xch + other + w + v, kEmpty);
                    const unsigned long long o = atomicExch(xch + par + w + v, dbits(sv[v]));
                    if (o != kEmpty && active)
                        st_row(y_row(y1), v,
                               sv[v] + __longlong_as_double((long long)o), alpha, beta);
                }
            } else if (rp_t[nr] < x1) {  // (a row that starts at x1 has nothing here)
                const size_t w = (size_t)u * K + j0;
#pragma unroll
                for (int v = 0; v < VW; ++v) {
                    st_relaxed_u64(slots + other + w + v, kEmpty);
                    st_relaxed_u64(slots + par + w + v, dbits(sv[v]));
                }
            }
        }

        // ---- row y0 when it began in an earlier tile
        if (need_lb) {
            if (prev_x <= rs) {
                if (holds_first) {
#pragma unroll
                    for (int v = 0; v < VW; ++v) {
                        const unsigned long long o =
                            atomicExch(xch + par + (size_t)u * K + j0 + v, dbits(rv[v]));
                        if (o != kEmpty && active)
                            st_row(y_row(y0), v,
                                   __longlong_as_double((long long)o) + rv[v], alpha, beta);
                    }
                }
            } else {
                if (nlb == kSpmmLookBacks) {  // warp-uniform
                    drain_spmm_look_backs<K, Y>(lbq, nlb, a, epoch, lane);
                    nlb = 0;
                }
                if (holds_first) {
#pragma unroll
                    for (int v = 0; v < VW; ++v)
                        st_relaxed_u64(xch + par + (size_t)u * K + j0 + v, dbits(rv[v]));
                }
                if (lane == 0) {
                    SpmmLookBack e;
                    e.y = y_row(y0);
                    e.head = u;
                    // the row's first nonzero is item rs + y0 of the merge path
                    e.first = d.tile_begin + (int)((unsigned)(rs + y0) / (unsigned)ITEMS);
                    lbq[nlb] = e;
                }
                ++nlb;
            }
        }
        __syncwarp();
    }
};

// The stage of a warp when a launch takes tiles of ITEMS or ITEMS2 items
// (ITEMS2 = 0: ITEMS only): large enough for either, one mbarrier after both.
template <int DT, int K, int VW, int ITEMS, int ITEMS2, bool DV>
struct SpmmStage {
    using T1 = SpmmTile<DT, K, VW, ITEMS, DV>;
    using T2 = SpmmTile<DT, K, VW, ITEMS2 ? ITEMS2 : ITEMS, DV>;
    static constexpr size_t bar_offset =
        T1::bar_offset > T2::bar_offset ? T1::bar_offset : T2::bar_offset;
    static constexpr size_t bytes = bar_offset + 16;
};

// ITEMS2 != 0: a batch whose matrices take tiles of either size; descriptor
// field `ipt` holds the tile items of its matrix (0 or ITEMS: ITEMS).
//
// Resident CTAs of 4 warps per SM that the registers must allow: 5 (96
// registers).  On Zipf-1M FP32 at k = 16 the forward ran 427, 351 and 373 us
// at 4, 5 and 6, and without a bound (80 registers, spills) 367.  FP64 with the
// fused dval, with two tile sizes or with 8 scalar gathers ahead would spill
// at 5; FP32 with staged products takes 6 (80 registers; an 80 x 70 x 60
// 27-point stencil at k = 2: 80, 71, 68 and 76 us at 4, 5, 6 and 7).
//
// One column, one lane per group, is the most latency-bound: FP32 takes 6, with the
// fused dval 7 (72 registers), FP64 5 (us at 5, 6, 7 and 8: Zipf-1M FP32 product in
// 480-item tiles 145, 144, 145, 204 and random rows of 0 to 40 29, 24, 27, 42; backward in
// 256-item tiles Zipf-1M 270, 250, 251, 238, the stencil 83, 76, 72, 68, R-MAT-300k 84, 84,
// 87, 88; FP64 backward at 4, 5, 6 R-MAT-300k 99, 94, 100, Zipf-300k 96, 89, 89).  The
// FP32 backward of two columns takes 7 as well (at 5, 6 and 7 the stencil 95, 94, 88,
// the random rows 50, 46, 43, R-MAT-40k 22, 25, 20, Zipf-1M 285, 275, 287, R-MAT-300k 93,
// 97, 102).
constexpr int spmm_ctas(int dt, int k, int vw, int items, int items2, bool dv) {
    if (k == 1) return dt == MERBIT_F64 ? 5 : dv ? 7 : 6;
    if (k == 2 && vw == 2 && dv && dt != MERBIT_F64) return 7;
    if (dt == MERBIT_F64) return dv || items2 != 0 || vw == 1 ? 4 : 5;
    return spmm_staged_products(k, vw, items, dv) ? 6 : 5;
}

template <int DT, int K, int VW, int ITEMS, int ITEMS2, int WARPS, bool DV>
__global__ void __launch_bounds__(WARPS * 32, spmm_ctas(DT, K, VW, ITEMS, ITEMS2, DV))
    spmm_kernel(const SpmmLaunch a) {
    using St = SpmmStage<DT, K, VW, ITEMS, ITEMS2, DV>;
    using T = typename St::T1;
    using T2 = typename St::T2;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ unsigned s_epoch;
    __shared__ SpmmLookBack s_lbq[WARPS][kSpmmLookBacks];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_epoch = *(volatile unsigned*)&a.state->epoch;
    unsigned char* ws = smem + (size_t)warp * St::bytes;
    uint64_t* bar = reinterpret_cast<uint64_t*>(ws + St::bar_offset);
    if (lane == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    const unsigned epoch = s_epoch;
    const int nw = (int)gridDim.x * WARPS;
    unsigned phase = 0;
    int nlb = 0;  // queued look-backs of this warp
    int m = 0;  // matrix of the current tile (tiles are visited in increasing order)
    for (int u = (int)blockIdx.x * WARPS + warp; u < a.total_tiles; u += nw) {
        const SpmmDesc* dp;
        if (a.ndesc == 0) {
            dp = &a.single;
        } else {
            while (m + 1 < a.ndesc && a.descs[m + 1].tile_begin <= u) ++m;
            dp = a.descs + m;
        }
        const SpmmDesc& d = *dp;
        const int lt = u - d.tile_begin;
        const bool second = ITEMS2 != 0 && d.ipt == ITEMS2;  // warp-uniform
        if (second)
            T2::issue(d, lt, ws, bar, lane, a.dv_perm);
        else
            T::issue(d, lt, ws, bar, lane, a.dv_perm);
        const bool ok = __all_sync(0xFFFFFFFFu, mbar_wait_bounded(bar, phase, a.state));
        phase ^= 1u;
        __syncwarp();
        if (ok) {
            if (second)
                T2::process(a, d, u, lt, epoch, ws, lane, s_lbq[warp], nlb);
            else
                T::process(a, d, u, lt, epoch, ws, lane, s_lbq[warp], nlb);
        } else {  // nothing published: leave no word of an earlier launch behind
            const size_t other = (size_t)((epoch + 1u) & 1u) * a.nslots;
            if (lane < K) {
                st_relaxed_u64(a.slots + other + (size_t)u * K + lane, kEmpty);
                if (u + 1 < a.total_tiles)
                    st_relaxed_u64(a.xch + other + (size_t)(u + 1) * K + lane, kEmpty);
            }
        }
    }
    drain_spmm_look_backs<K, typename T::Y>(s_lbq[warp], nlb, a, epoch, lane);
    __syncthreads();
    if (threadIdx.x == 0) finish_launch(a.state, epoch);
}

namespace {

template <int DT, int K, int VW, int ITEMS, int WARPS, bool DV, int ITEMS2 = 0>
int launch_spmm_cfg(const SpmmLaunch& a, cudaStream_t s) {
    constexpr size_t smem = SpmmStage<DT, K, VW, ITEMS, ITEMS2, DV>::bytes * WARPS;
    static int grid_cap[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 64) return fail(MERBIT_ERR_UNSUPPORTED, "spmm: device ordinal >= 64");
    auto kern = spmm_kernel<DT, K, VW, ITEMS, ITEMS2, WARPS, DV>;
    // per-device cache; threads that race here compute the same value
    int cap = __atomic_load_n(&grid_cap[dev], __ATOMIC_ACQUIRE);
    if (cap == 0) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(spmm)");
        int per_sm = 0, sms = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, WARPS * 32, smem);
        if (e != cudaSuccess) return cuda_fail(e, "occupancy(spmm)");
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cap = per_sm > 0 && sms > 0 ? per_sm * sms : 1;
        __atomic_store_n(&grid_cap[dev], cap, __ATOMIC_RELEASE);
    }
    const long long need = ((long long)a.total_tiles + WARPS - 1) / WARPS;
    const int grid = (int)(need < cap ? need : cap);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(WARPS * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, a);
    if (e == cudaSuccess) e = cudaGetLastError();
    return e == cudaSuccess ? (int)MERBIT_OK : cuda_fail(e, "spmm_kernel launch");
}

// Configurations: (K, VW, ITEMS).  WARPS = 4.
template <int DT>
int launch_spmm_dt(int k, int vw, int items, int items2, const SpmmLaunch& a, cudaStream_t s) {
    constexpr bool kDv = DT != MERBIT_BF16;  // fused dval: F64 and F32 plans
    if (a.dv_out && !kDv) return fail(MERBIT_ERR_UNSUPPORTED, "spmm: fused dval needs F64 or F32 values");
    if (items2) {
        // batches whose matrices take either of two tile sizes (vector width 4)
        if (a.dv_out) return fail(MERBIT_ERR_UNSUPPORTED, "spmm: tile pairs take no fused dval");
#define MERBIT_SPMM_PAIR(KK, I1, I2) \
        if (k == KK && vw == 4 && items == I1 && items2 == I2) \
            return launch_spmm_cfg<DT, KK, 4, I1, 4, false, I2>(a, s);
        MERBIT_SPMM_PAIR(4, 256, 512)
        MERBIT_SPMM_PAIR(4, 288, 480)
        MERBIT_SPMM_PAIR(8, 256, 512)
        MERBIT_SPMM_PAIR(8, 272, 496)
        MERBIT_SPMM_PAIR(16, 256, 512)
        MERBIT_SPMM_PAIR(16, 264, 504)
        MERBIT_SPMM_PAIR(32, 256, 512)
        MERBIT_SPMM_PAIR(32, 260, 508)
#undef MERBIT_SPMM_PAIR
        return fail(MERBIT_ERR_INVALID, "spmm: no such tile pair");
    }
#define MERBIT_SPMM_CASE(KK, VV, II)                                                  \
    if (k == KK && vw == VV && items == II)                                           \
        return a.dv_out ? launch_spmm_cfg<DT, KK, VV, II, 4, kDv>(a, s)                \
                        : launch_spmm_cfg<DT, KK, VV, II, 4, false>(a, s);
    MERBIT_SPMM_CASE(1, 1, 256)
    MERBIT_SPMM_CASE(2, 1, 256)
    MERBIT_SPMM_CASE(2, 2, 256)
    MERBIT_SPMM_CASE(4, 1, 256)
    MERBIT_SPMM_CASE(4, 2, 256)
    MERBIT_SPMM_CASE(4, 4, 256)
    MERBIT_SPMM_CASE(8, 1, 256)
    MERBIT_SPMM_CASE(8, 2, 256)
    MERBIT_SPMM_CASE(8, 4, 256)
    MERBIT_SPMM_CASE(16, 1, 256)
    MERBIT_SPMM_CASE(16, 2, 256)
    MERBIT_SPMM_CASE(16, 4, 256)
    MERBIT_SPMM_CASE(32, 1, 256)
    MERBIT_SPMM_CASE(32, 2, 256)
    MERBIT_SPMM_CASE(32, 4, 256)
    MERBIT_SPMM_CASE(1, 1, 512)
    MERBIT_SPMM_CASE(4, 4, 512)
    MERBIT_SPMM_CASE(8, 4, 512)
    MERBIT_SPMM_CASE(16, 4, 512)
    MERBIT_SPMM_CASE(32, 4, 512)
    // odd segments per lane group (tile = groups x odd length): the groups'
    // shared-memory reads start in different banks
    MERBIT_SPMM_CASE(1, 1, 288)
    MERBIT_SPMM_CASE(1, 1, 480)
    MERBIT_SPMM_CASE(4, 4, 288)
    MERBIT_SPMM_CASE(4, 4, 480)
    MERBIT_SPMM_CASE(8, 4, 272)
    MERBIT_SPMM_CASE(8, 4, 496)
    MERBIT_SPMM_CASE(16, 4, 264)
    MERBIT_SPMM_CASE(16, 4, 504)
    MERBIT_SPMM_CASE(32, 4, 260)
    MERBIT_SPMM_CASE(32, 4, 508)
    // k = 2, one lane per group with staged products (SpmmTile::STAGEP):
    // 2.12 ms against 2.84 for the 128-matrix R-MAT batch; at k = 4 the
    // product slice and registers cost more warps than it saves (3.12 ms
    // against 2.39), so k = 4 has no such tile
    MERBIT_SPMM_CASE(2, 2, 224)
    MERBIT_SPMM_CASE(2, 2, 352)
    // odd segments at vector width 2, single matrices
    MERBIT_SPMM_CASE(4, 2, 496)
    MERBIT_SPMM_CASE(8, 2, 504)
    MERBIT_SPMM_CASE(16, 2, 508)
    MERBIT_SPMM_CASE(32, 2, 510)
    // the same tiles at width 1: for operands that allow no more, while a capturing
    // stream leaves the slots of these tiles only
    MERBIT_SPMM_CASE(2, 1, 224)
    MERBIT_SPMM_CASE(2, 1, 352)
    MERBIT_SPMM_CASE(4, 1, 496)
    MERBIT_SPMM_CASE(8, 1, 504)
    MERBIT_SPMM_CASE(16, 1, 508)
    MERBIT_SPMM_CASE(32, 1, 510)
#undef MERBIT_SPMM_CASE
    return fail(MERBIT_ERR_INVALID, "spmm: no such configuration");
}

}  // namespace

bool spmm_config_exists(int k, int vw, int items) {
    if (items == 256) return (k == 1 && vw == 1) || (k >= 2 && k <= 32 && (k & (k - 1)) == 0 && vw <= 4 && vw <= k && (vw & (vw - 1)) == 0 && !(k == 2 && vw == 4));
    if (items == 512) return (k == 1 && vw == 1) || (k >= 4 && k <= 32 && (k & (k - 1)) == 0 && vw == 4);
    if (items == 224 || items == 352) return k == 2 && vw == 2;
    if (k == 1) return vw == 1 && (items == 288 || items == 480);
    if (vw != 4) return false;
    switch (k) {
    case 4: return items == 288 || items == 480;
    case 8: return items == 272 || items == 496;
    case 16: return items == 264 || items == 504;
    case 32: return items == 260 || items == 508;
    }
    return false;
}

int spmm_resident_warps(int dtype, int k, int vw, int items, bool dv, int sms) {
    return 4 * spmm_ctas(dtype, k, vw, items, 0, dv) * sms;
}

bool spmm_single_exists(int k, int vw, int items) {
    if (k == 2 && vw == 1 && (items == 224 || items == 352)) return true;
    return spmm_config_exists(k, vw, items) || (k >= 4 && vw <= 2 && items == spmm_odd_tile2(k));
}

int spmm_tile_candidates(int k, int* out) {
    int n = 0;
    out[n++] = 256;
    out[n++] = 512;
    static const int odd[6][2] = {{288, 480}, {0, 0}, {288, 480}, {272, 496}, {264, 504}, {260, 508}};
    const int row = k == 1 ? 0 : k == 4 ? 2 : k == 8 ? 3 : k == 16 ? 4 : k == 32 ? 5 : 1;
    for (int j = 0; j < 2; ++j)
        if (odd[row][j]) out[n++] = odd[row][j];
    if (k == 2) {  // staged products
        out[n++] = 224;
        out[n++] = 352;
    }
    return n;
}

int spmm_odd_tile(int k) {
    switch (k) {
    case 4: return 480;
    case 8: return 496;
    case 16: return 504;
    case 32: return 508;
    }
    return 0;
}

int spmm_small_tile(int k) {
    switch (k) {
    case 4: return 288;
    case 8: return 272;
    case 16: return 264;
    case 32: return 260;
    }
    return 0;
}

int spmm_odd_tile2(int k) {
    switch (k) {
    case 4: return 496;
    case 8: return 504;
    case 16: return 508;
    case 32: return 510;
    }
    return 0;
}

bool spmm_pair_exists(int k, int vw, int items, int items2) {
    if (vw != 4 || !(k == 4 || k == 8 || k == 16 || k == 32)) return false;
    if (items == 256 && items2 == 512) return true;
    return items2 == spmm_odd_tile(k) && items == spmm_small_tile(k);
}

int spmm_launch(int dtype, int k, int vw, int items, const SpmmLaunch& a, cudaStream_t s,
                int items2) {
    if (a.total_tiles <= 0) return MERBIT_OK;
    switch (dtype) {
    case MERBIT_F64: return launch_spmm_dt<MERBIT_F64>(k, vw, items, items2, a, s);
    case MERBIT_F32: return launch_spmm_dt<MERBIT_F32>(k, vw, items, items2, a, s);
    case MERBIT_BF16: return launch_spmm_dt<MERBIT_BF16>(k, vw, items, items2, a, s);
    }
    return fail(MERBIT_ERR_INVALID, "spmm: bad dtype");
}

}  // namespace merbit
