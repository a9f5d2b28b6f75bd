// Warp-level bodies of the SDDMM and SpMM kernels, shared by the local
// kernels (local_ops.cu) and the fused compute+communication kernels
// (fused_impl.cuh).  Where dense rows come from and where results go is a
// template policy:
//
//   SDDMM   A rows:  RowsByStride (one local block) here, RowsByPeerRef (rows
//                    that stay in their owners' memory, local or peer) in the
//                    fused kernel, which has a loop of its own (sddmm_units)
//           output:  StoreLocal | the fused kernel's slice-routing store
//   SpMM    emit:    EmitLocal (Y = beta*Y + acc) | the fused kernel's
//                    owned-or-push emit; one loop for both families
//
// Layout of the math: a dense row is cut into vectors of NB bytes (16, 8 or 4:
// the widest that the width and the alignment of the operands allow); a group
// of G lanes holds R vectors per lane, and the 32/G groups of a warp work on
// different nonzeros.  Column indices and values are taken four at a time.
//
// Reference loops: src/core_ops.cpp:5-35.
#pragma once
#include "sp3_cuda.cuh"

#include <atomic>
#include <cstdlib>
#include <type_traits>

namespace sp3 {

template <int G> __device__ __forceinline__ unsigned group_mask(int slot) {
    return G == 32 ? 0xffffffffu : (((1u << G) - 1u) << (slot * G));
}

// ---- a lane's vector of a dense row ------------------------------------------
// fp32 vectors of 8 and 16 bytes keep their values as pairs in 64-bit registers and use the packed
// multiply-add of sm_100 (`fma.rn.f32x2`: two fp32 products per instruction, each rounded like `fmaf`).
using u64 = unsigned long long;
__device__ __forceinline__ u64 pack2(float a, float b) { u64 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ float2 unpack2(u64 v) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v)); return r; }
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) { u64 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ u64 add2(u64 a, u64 b) { u64 d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ u64 mul2(u64 a, u64 b) { u64 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }

template <typename T, int NB> struct Row;
template <> struct Row<float, 16> { using E = u64; static constexpr int N = 2; E x[2]; };
template <> struct Row<float, 8> { using E = u64; static constexpr int N = 1; E x[1]; };
template <> struct Row<float, 4> { using E = float; static constexpr int N = 1; E x[1]; };
template <> struct Row<double, 16> { using E = double; static constexpr int N = 2; E x[2]; };
template <> struct Row<double, 8> { using E = double; static constexpr int N = 1; E x[1]; };

// Dense rows, values, index lists and work items are read by ordinary loads, never through the read-only path
// (`ld.global.nc`, `__ldg`, or a `const __restrict__` kernel parameter, from which the compiler infers it): that path is
// defined only for memory that nobody writes while the kernel runs.  A kernel launched early runs while the kernel before
// it writes what may be its values, rows or lists (see after_previous_kernel), and in the fused kernels other warps of
// the launch write the pulled rows.  Ordinary loads are ordered behind the wait, or the acquire, that says the data is
// there.  (Lists through the read-only path took the same time: 192 products of 10 to 600 thousand nonzeros within 0.2 %.)
template <typename T, int NB> __device__ __forceinline__ void row_load(Row<T, NB>& v, const char* p) {
    using E = typename Row<T, NB>::E;
    if constexpr (NB == 16 && sizeof(T) == 4) {
        const ulonglong2* q = reinterpret_cast<const ulonglong2*>(p);
        const ulonglong2 t = *q;
        v.x[0] = t.x; v.x[1] = t.y;
    } else if constexpr (NB == 16) {
        const double2* q = reinterpret_cast<const double2*>(p);
        const double2 t = *q;
        v.x[0] = t.x; v.x[1] = t.y;
    } else {
        const E* q = reinterpret_cast<const E*>(p);
        v.x[0] = *q;
    }
}
template <typename T, int NB> __device__ __forceinline__ void row_store(char* p, const Row<T, NB>& v) {
    using E = typename Row<T, NB>::E;
    if constexpr (NB == 16 && sizeof(T) == 4) *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v.x[0], v.x[1]);
    else if constexpr (NB == 16) *reinterpret_cast<double2*>(p) = make_double2(v.x[0], v.x[1]);
    else *reinterpret_cast<E*>(p) = v.x[0];
}
// past the L1: rows that other warps of the same launch wrote
template <typename T, int NB> __device__ __forceinline__ void row_load_cg(Row<T, NB>& v, const char* p) {
    using E = typename Row<T, NB>::E;
#pragma unroll
    for (int h = 0; h < Row<T, NB>::N; ++h) v.x[h] = __ldcg(reinterpret_cast<const E*>(p) + h);
}
template <typename T, int NB> __device__ __forceinline__ void row_zero(Row<T, NB>& v) {
#pragma unroll
    for (int h = 0; h < Row<T, NB>::N; ++h) v.x[h] = 0;
}
// elementwise sums and products of the register elements (a pair of fp32 values or one value)
__device__ __forceinline__ u64 e_fma(u64 a, u64 b, u64 c) { return fma2(a, b, c); }
__device__ __forceinline__ float e_fma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double e_fma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ u64 e_add(u64 a, u64 b) { return add2(a, b); }
__device__ __forceinline__ float e_add(float a, float b) { return a + b; }
__device__ __forceinline__ double e_add(double a, double b) { return a + b; }
template <typename E, typename T> __device__ __forceinline__ E e_splat(T s) {
    if constexpr (sizeof(E) == 8 && sizeof(T) == 4) return pack2(s, s);
    else return s;
}
template <typename T, int NB> __device__ __forceinline__ void row_fma(Row<T, NB>& acc, T s, const Row<T, NB>& x) {
    using E = typename Row<T, NB>::E;
    const E w = e_splat<E>(s);
#pragma unroll
    for (int h = 0; h < Row<T, NB>::N; ++h) acc.x[h] = e_fma(w, x.x[h], acc.x[h]);
}
template <typename T, int NB> __device__ __forceinline__ void row_add(Row<T, NB>& acc, const Row<T, NB>& x) {
#pragma unroll
    for (int h = 0; h < Row<T, NB>::N; ++h) acc.x[h] = e_add(acc.x[h], x.x[h]);
}
// this lane's part of a dot product over R vectors; vectors q with on[q] false do not count
template <bool ALL, typename T, int NB, int R>
__device__ __forceinline__ T row_dot(const Row<T, NB> (&a)[R], const Row<T, NB> (&b)[R], const bool (&on)[R]) {
    using E = typename Row<T, NB>::E;
    E s = 0;
#pragma unroll
    for (int q = 0; q < R; ++q)
        if (ALL || (q < R - 1 && R < 8) || on[q])   // (pick_shape: only the last vector of a lane can be past the row, but for R = 8)
#pragma unroll
            for (int h = 0; h < Row<T, NB>::N; ++h) s = e_fma(a[q].x[h], b[q].x[h], s);
    if constexpr (sizeof(E) == 8 && sizeof(T) == 4) {
        const float2 f = unpack2(s);
        return f.x + f.y;
    } else {
        return s;
    }
}

// Four consecutive values base[i .. i+3] of a list, i a multiple of 4 counted from a 16-byte boundary when `aligned`;
// positions at or past `end` repeat the last value before it.
template <typename I> struct __align__(16) Quad { I v[4]; };
__device__ __forceinline__ Quad<int> quad_load_vec(const int* p) {
    const int4 t = *reinterpret_cast<const int4*>(p);
    return {{t.x, t.y, t.z, t.w}};
}
__device__ __forceinline__ Quad<float> quad_load_vec(const float* p) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    return {{t.x, t.y, t.z, t.w}};
}
__device__ __forceinline__ Quad<double> quad_load_vec(const double* p) {
    const double2 a = *reinterpret_cast<const double2*>(p), b = *(reinterpret_cast<const double2*>(p) + 1);
    return {{a.x, a.y, b.x, b.y}};
}
template <typename I> __device__ __forceinline__ Quad<I> quad_load(const I* base, int i, int end, bool aligned) {
    if (aligned && i + 4 <= end) return quad_load_vec(base + i);
    Quad<I> q;
#pragma unroll
    for (int j = 0; j < 4; ++j) q.v[j] = base[i + j < end ? i + j : end - 1];
    return q;
}

// First in a kernel that is launched early (see launch_early): the next kernel of the stream may start, and the one
// before has written what it writes.  No memory is read ahead of the wait, index lists and work items included: callers
// hand over any tensors, and what the kernel before writes is visible behind the wait only, whether that kernel signals
// early or just ends.
__device__ __forceinline__ void after_previous_kernel() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __threadfence();
}

// ---- row access policies ---------------------------------------------------
// `resolve` turns a 31-bit *reference* to a row into its address (pure arithmetic); references are what a loop compares
// to detect a row change.  In one local block they are the row indices.  Rows at their owners have a table of them, which
// `ref` reads, by every lane for its own nonzeros when a window of indices is read, so that the lookup is off the
// critical path.
struct RowsByStride {
    const char* base;
    unsigned ld_bytes;
    __device__ __forceinline__ const char* resolve(int r) const { return base + (u64)(unsigned)r * ld_bytes; }
};
// The same for lists sorted by chunk of columns: what is read once per chunk (A rows, indices) leaves the L2 first, so
// that the chunk's rows of B stay there (without that 48 % of the sectors hit with chunks of 96 MB; Erdos-Renyi 1 M rows,
// 32 a row, k = 128: 1945 us without, 1782 with; uniform 500 thousand rows, 20 a row: 503 and 463).
struct RowsPassing : RowsByStride {};
template <typename R> struct passes_by { static constexpr bool value = false; };
template <> struct passes_by<RowsPassing> { static constexpr bool value = true; };
__device__ __forceinline__ u64 evict_first_policy() {
    u64 p;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
template <typename T> __device__ __forceinline__ void row_load_passing(Row<T, 16>& v, const char* p, u64 policy) {
    u64 a, b;
    asm volatile("ld.global.L2::cache_hint.v2.u64 {%0, %1}, [%2], %3;" : "=l"(a), "=l"(b) : "l"(p), "l"(policy));
    if constexpr (sizeof(T) == 4) { v.x[0] = a; v.x[1] = b; }
    else { v.x[0] = __longlong_as_double((long long)a); v.x[1] = __longlong_as_double((long long)b); }
}
// Rows that live in the owners' heaps: reference = owner rank (6 bits) and row
// number inside the owner's block (25 bits); `bases` (shared memory) holds the
// block address of every rank as mapped into this process.
constexpr int PEER_REF_SHIFT = 25;
struct RowsByPeerRef {
    const int* table;                  // [local rows] references; null: every row is in this rank's own block
    const unsigned long long* bases;   // [ranks] block base addresses
    unsigned row_bytes;
    int self_bits;                     // this rank << PEER_REF_SHIFT (used when table is null)
    __device__ __forceinline__ int ref(int row) const { return table ? __ldg(table + row) : (self_bits | row); }
    __device__ __forceinline__ const char* resolve(int r) const {
        return reinterpret_cast<const char*>(bases[r >> PEER_REF_SHIFT] +
                                             (u64)(unsigned)(r & ((1 << PEER_REF_SHIFT) - 1)) * row_bytes);
    }
};

// Where values go: `put4(i, n, dots)` stores min(n, 4) values from nonzero i on (i a multiple of 4), dot products times
// values.  Quads are written as vectors where the places of all quads are 16-byte aligned (`vectors`).  `scale(i)` is the
// value of nonzero i, `put(i, v)` stores one that is scaled.
template <typename T> __device__ __forceinline__ void quad_store(T* p, const Quad<T>& q, int n, bool vectors) {
    if (vectors && n >= 4) {
        using V = typename Vec<T>::type;
#pragma unroll
        for (int j = 0; j < 4; j += Vec<T>::N) *reinterpret_cast<V*>(p + j) = *reinterpret_cast<const V*>(q.v + j);
        return;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (j < n) p[j] = q.v[j];
}
template <typename T> struct StoreLocal {
    T* out;
    const T* sval;    // null: no scaling
    bool vectors;
    __device__ __forceinline__ Quad<T> scaled(long long i, int n, const T* dots) const {
        Quad<T> q = quad_load(dots, 0, 4, true);
        if (sval) {
            const Quad<T> s = quad_load(sval + i, 0, n, vectors);
#pragma unroll
            for (int j = 0; j < 4; ++j) q.v[j] *= s.v[j];
        }
        return q;
    }
    __device__ __forceinline__ void put4(long long i, int n, const T* dots) const {
        quad_store(out + i, scaled(i, n, dots), n, vectors);
    }
    __device__ __forceinline__ T scale(long long i) const { return sval ? sval[i] : (T)1; }
    __device__ __forceinline__ void put(long long i, T v) const { out[i] = v; }
};
template <typename T> struct StoreTwice : StoreLocal<T> {
    T* also;          // a second place for the values (a form of its own: the choice in the kernel cost 1 %)
    __device__ __forceinline__ void put4(long long i, int n, const T* dots) const {
        const Quad<T> q = this->scaled(i, n, dots);
        quad_store(this->out + i, q, n, this->vectors);
        quad_store(also + i, q, n, this->vectors);
    }
    __device__ __forceinline__ void put(long long i, T v) const { this->out[i] = v; also[i] = v; }
};
template <typename T> struct StoreScattered : StoreLocal<T> {
    const int* orig;  // result position of nonzero i
    __device__ __forceinline__ void put4(long long i, int n, const T* dots) const {
        const Quad<T> q = this->scaled(i, n, dots);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j < n) this->out[orig[i + j]] = q.v[j];
    }
    __device__ __forceinline__ void put(long long i, T v) const { this->out[orig[i]] = v; }
};

// Sums four values per lane over a group of G lanes (4 <= G) with a halving butterfly: log2(G) + 1 shuffles
// instead of 4 log2(G).  On return lane gl holds the total of value number gl / (G / 4).
template <typename T, int G> __device__ __forceinline__ T group_sum4(T (&v)[4], int gl) {
    {
        constexpr int m = G / 2;
        const bool up = (gl & m) != 0;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const T send = up ? v[t] : v[t + 2], keep = up ? v[t + 2] : v[t];
            v[t] = keep + __shfl_xor_sync(0xffffffffu, send, m);
        }
    }
    {
        constexpr int m = G / 4;
        const bool up = (gl & m) != 0;
        const T send = up ? v[0] : v[1], keep = up ? v[1] : v[0];
        v[0] = keep + __shfl_xor_sync(0xffffffffu, send, m);
    }
#pragma unroll
    for (int m = G / 8; m > 0; m >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], m);
    return v[0];
}

// ---------------------------------------------------------------------------
// SDDMM over windows first, first + step, ... < end of `wn` consecutive nonzeros each (wn a multiple of 4, at
// most 128), one warp per window.  The indices of a window lie in shared memory, copied there asynchronously while the
// window before it is computed; the groups of G lanes take its quads of nonzeros in turn: four
// dense B rows in flight, four dot products reduced together, the A row kept in registers until the row changes (the
// list is sorted by row).
//
// Bound by the row gathers out of the L2 and by what a warp does while it has none in flight.  So the rows of the next
// quad (and the A row it ends in, if that is another one) are requested as soon as the products of this one are summed
// per lane, and travel while the lanes are added up and the results stored; and the lanes per row are few, so that an
// instruction of the reduction serves 32 / G nonzeros.
// ---------------------------------------------------------------------------
constexpr int WINDOW_MAX = 128;
template <typename T> struct WindowLists {   // shared memory of a warp
    int4 cols[2][WINDOW_MAX / 4], rows[2][WINDOW_MAX / 4];
    T dots[WINDOW_MAX];
};

// Nonzeros per window: 128, less when that would leave warps without work.
__host__ __device__ inline int window_nnz(long long nnz, long long nwarps, int groups_per_warp) {
    const int quantum = 4 * groups_per_warp;
    const long long share = (nnz + nwarps - 1) / nwarps;
    const long long w = (share + quantum - 1) / quantum * quantum;
    return (int)(w < quantum ? quantum : (w > WINDOW_MAX ? WINDOW_MAX : w));
}

// The same, and equal rounds where the warps take up to four windows each: with windows of 128 the last round may find work
// for a fifth of them (Zipf rows, 357 thousand nonzeros, fp64, k = 32: 2790 windows on 2368 warps 14.3 us, as two rounds
// of 80 nonzeros 11.2; k = 128, fp32 23.5 and 18.7).  Four rounds and more are level or lose to the longer windows (R-MAT
// scale 17, k = 192, seven rounds: 113 us with windows of 120, 104 with 128).
inline int balanced_window_nnz(long long nnz, long long nwarps, int groups_per_warp) {
    const long long rounds = (nnz - 1) / (nwarps * WINDOW_MAX) + 1;
    return window_nnz(nnz, rounds <= 4 ? rounds * nwarps : nwarps, groups_per_warp);
}

template <bool PASSING> __device__ __forceinline__ void copy_quad_async(int4* dst, const int* src, u64 policy) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (PASSING) asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "l"(policy) : "memory");
    else asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// A quad that ends in one row or has two or more, as the list of a window marks it: the row it ends in, negative where it
// is not all of that row (a list sorted by row class by class may also leave and re-enter a row).
__device__ __forceinline__ int quad_tag(const int4& r) {
    return r.x == r.w && r.y == r.w && r.z == r.w ? r.w : r.w | (1 << 31);
}
// Products of the rows in `b` with row `cur` in `a` and the row the quad ends in, in `a2` unless that is `cur` and the
// whole quad with it; afterwards the latter is `cur`.  `second(h)` brings the rows of the second half where only half a
// quad is in flight, `rows()` the quad's row indices, `fetch_a(row)` a row to `a`.
template <typename T, int NB, int R, int U, bool EXACT, typename Rows, typename Second, typename FetchA>
__device__ __forceinline__ void quad_products(T (&d)[4], Row<T, NB> (&a)[R], Row<T, NB> (&a2)[R], Row<T, NB> (&b)[U][R],
                                              const bool (&on)[R], int& cur, int next, Rows&& rows, Second&& second,
                                              FetchA&& fetch_a) {
    constexpr unsigned FULL = 0xffffffffu;
    if (__all_sync(FULL, next >= 0)) {      // every group: four nonzeros of one row
        if (next != cur) {
            cur = next;
#pragma unroll
            for (int q = 0; q < R; ++q) a[q] = a2[q];
        }
#pragma unroll
        for (int h = 0; h < 4; h += U) {
            second(h);
#pragma unroll
            for (int u = 0; u < U; ++u) d[h + u] = row_dot<EXACT>(a, b[u], on);
        }
    } else {
        // where a row ends in a quad, both of its rows are here as a rule: both products, and the one that counts
        const int4 rq = rows();
        const int r[4] = {rq.x, rq.y, rq.z, rq.w};
        const bool here = (r[0] == cur || r[0] == r[3]) && (r[1] == cur || r[1] == r[3]) && (r[2] == cur || r[2] == r[3]);
        const bool both = __all_sync(FULL, here);
#pragma unroll
        for (int h = 0; h < 4; h += U) {
            second(h);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (!both && r[h + u] != cur && r[h + u] != r[3]) {
                    cur = r[h + u];
                    fetch_a(cur);
                }
                const T d1 = row_dot<EXACT>(a, b[u], on), d2 = row_dot<EXACT>(a2, b[u], on);
                d[h + u] = r[h + u] == r[3] ? d2 : d1;
            }
        }
        cur = r[3];
#pragma unroll
        for (int q = 0; q < R; ++q) a[q] = a2[q];
    }
}

template <typename T, int NB, int G, int R, int U, bool EXACT, typename ARows, typename Store>
__device__ __forceinline__ void sddmm_windows(long long first, long long step, long long end, int wn, long long nnz,
                                              const int* rowidx, const int* colidx,
                                              const ARows& arows, const char* B, unsigned ldb_bytes,
                                              int nvec, bool aligned, const Store& store, WindowLists<T>& lists, int lane) {
    static_assert(G >= 4, "a group reduces four values");
    static_assert(std::is_base_of<RowsByStride, ARows>::value, "row indices are used as they are");
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int SLOTS = 32 / G;
    const int slot = lane / G, gl = lane % G;
    unsigned off[R];
    bool on[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {   // lanes past the row's last vector read it too and do not count
        const int v = gl + q * G;
        on[q] = EXACT || v < nvec;
        off[q] = (unsigned)(on[q] ? v : nvec - 1) * NB;
    }
    constexpr bool PASSING = passes_by<ARows>::value;
    const u64 policy = PASSING ? evict_first_policy() : 0;
    auto length = [&](long long w) { return (int)(nnz - w * wn < wn ? nnz - w * wn : (long long)wn); };
    // copies the indices of window w to buffer k, a quad per lane (behind the last quad: that quad again)
    auto stage = [&](long long w, int k) {
        const int n = length(w), i = 4 * lane < n ? 4 * lane : (n - 1) & ~3;
        const int *c = colidx + w * wn, *r = rowidx + w * wn;
        if (aligned && i + 4 <= n) {
            copy_quad_async<PASSING>(&lists.cols[k][lane], c + i, policy);
            copy_quad_async<PASSING>(&lists.rows[k][lane], r + i, policy);
        } else {
            const Quad<int> cq = quad_load(c, i, n, false), rq = quad_load(r, i, n, false);
            lists.cols[k][lane] = make_int4(cq.v[0], cq.v[1], cq.v[2], cq.v[3]);
            lists.rows[k][lane] = make_int4(rq.v[0], rq.v[1], rq.v[2], rq.v[3]);
        }
    };
    auto fetch = [&](Row<T, NB> (&a)[R], const char* p) {
#pragma unroll
        for (int q = 0; q < R; ++q) row_load(a[q], p + (off[q] - off[0]));
    };
    auto fetch_a = [&](Row<T, NB> (&a)[R], const char* p) {
        if constexpr (PASSING) {
#pragma unroll
            for (int q = 0; q < R; ++q) row_load_passing<T>(a[q], p + (off[q] - off[0]), policy);
        } else {
            fetch(a, p);
        }
    };
    if (first >= end) return;
    B += off[0];
    const bool writer = gl % (G / 4) == 0;      // (lane gl ends up with value gl / (G / 4) of its group's quad)
    long long w = first;
    int k = 1, tag = 0;
    int src = 0, quads = 0;                     // quad of this group, quads of the window (rounded up for all groups)
    auto enter = [&]() {                        // window w, whose indices are on their way to the other buffer
        asm volatile("cp.async.wait_all;" ::: "memory");
        k ^= 1;
        tag = quad_tag(lists.rows[k][lane]);
        __syncwarp();
        if (w + step < end) stage(w + step, k ^ 1);
        src = slot;
        quads = (((length(w) + 3) >> 2) + SLOTS - 1) / SLOTS * SLOTS;
    };
    int cur = -1, next = -1;                    // row in `a`; tag of the quad in flight
    Row<T, NB> a[R], a2[R], b[U][R];
#pragma unroll
    for (int q = 0; q < R; ++q) { row_zero(a[q]); row_zero(a2[q]); }
    auto request = [&]() {                      // the rows of B of quad src, the row of A it ends in if that is another one
        const int4 c = lists.cols[k][src];
        const int cs[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
        for (int u = 0; u < U; ++u) fetch(b[u], B + (u64)(unsigned)cs[u] * ldb_bytes);
        next = __shfl_sync(FULL, tag, src);
        if (__any_sync(FULL, next != cur)) fetch_a(a2, arows.resolve(next & 0x7fffffff) + off[0]);
    };
    stage(first, 0);
    enter();
    request();
    for (bool more = true; more;) {
        auto second = [&](int h) {              // the rows of the second half, where only half a quad is in flight
            if (h > 0) {
                const int4 c = lists.cols[k][src];
                const int cs[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
                for (int u = 0; u < U; ++u) fetch(b[u], B + (u64)(unsigned)cs[(h + u) & 3] * ldb_bytes);
            }
        };
        T d[4];
        quad_products<T, NB, R, U, EXACT>(d, a, a2, b, on, cur, next, [&] { return lists.rows[k][src]; }, second,
                                          [&](int row) { fetch_a(a, arows.resolve(row) + off[0]); });
        // the next quad travels while this one is reduced and stored (behind the last one: that one again)
        T* const place = lists.dots + 4 * src + gl / (G / 4);
        const bool last = src + SLOTS >= quads;
        if (!last) {
            src += SLOTS;
        } else {
            w += step;
            more = w < end;
            if (more) enter();
        }
        request();
        const T total = group_sum4<T, G>(d, gl);
        if (writer) *place = total;
        if (last) {                             // the values of the window, four per lane
            __syncwarp();
            const long long at = (w - step) * wn;
            const int j = 4 * lane, n = (int)(nnz - at < wn ? nnz - at : (long long)wn);
            if (j < n) store.put4(at + j, n - j, lists.dots + j);
            __syncwarp();
        }
    }
}

// ---------------------------------------------------------------------------
// The same for matrices with no more windows than warps: window w, one per warp.  Nothing but the trips to memory one after
// the other counts there, and there are three: the lists, the rows with the values, the store.  So the lists come by
// ordinary loads and pass through shared memory without a second buffer, the values travel with the rows, every value is
// stored when it is there, and nothing is requested behind the last quad.  5 to 400 thousand nonzeros, k = 16 to 256,
// back to back: 27 % less time than sddmm_windows (10 thousand of 4 a row, k = 64: 2.5 against 3.7 us; 200 thousand of 6 a
// row, k = 32: 3.9 against 5.5).  Two windows per warp and more are faster there (600 thousand nonzeros of 6 a row, k = 50:
// 17.4 us, 18.8 with this).
//
// A group takes every SLOTS-th quad where rows are long, so that all groups are in the same row, and its share in one piece
// where a quarter of the quads or more end a row (rows of 6: 5.2 against 4.7 us).
// ---------------------------------------------------------------------------
template <typename T, int NB, int G, int R, int U, bool EXACT, typename Store>
__device__ __forceinline__ void sddmm_window(long long w, int wn, long long nnz, const int* rowidx, const int* colidx,
                                             const RowsByStride& arows, const char* B, unsigned ldb_bytes, int nvec,
                                             bool aligned, const Store& store, int4 (&cols)[WINDOW_MAX / 4],
                                             int4 (&rows)[WINDOW_MAX / 4], int lane) {
    static_assert(G >= 4, "a group reduces four values");
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int SLOTS = 32 / G;
    const int slot = lane / G, gl = lane % G;
    const long long w0 = w * wn;
    if (w0 >= nnz) return;
    const int n = (int)(nnz - w0 < wn ? nnz - w0 : (long long)wn);
    unsigned off[R];
    bool on[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {   // lanes past the row's last vector read it too and do not count
        const int v = gl + q * G;
        on[q] = EXACT || v < nvec;
        off[q] = (unsigned)(on[q] ? v : nvec - 1) * NB;
    }
    B += off[0];
    auto fetch = [&](Row<T, NB> (&a)[R], const char* p) {
#pragma unroll
        for (int q = 0; q < R; ++q) row_load(a[q], p + (off[q] - off[0]));
    };
    int tag;
    {
        const int i = 4 * lane < n ? 4 * lane : (n - 1) & ~3;   // (behind the last quad: that quad again)
        const Quad<int> c = quad_load(colidx + w0, i, n, aligned), r = quad_load(rowidx + w0, i, n, aligned);
        cols[lane] = make_int4(c.v[0], c.v[1], c.v[2], c.v[3]);
        rows[lane] = make_int4(r.v[0], r.v[1], r.v[2], r.v[3]);
        tag = quad_tag(rows[lane]);
        __syncwarp();
    }
    const int quads = (n + 3) >> 2, each = (quads + SLOTS - 1) / SLOTS;
    const bool apart = 4 * __popc(__ballot_sync(FULL, tag < 0 && lane < quads)) >= quads;
    int src = apart ? slot * each : slot;       // quad of this group
    const int inc = apart ? 1 : SLOTS;
    const int mine = gl / (G / 4);              // which of the four results ends up in this lane
    const bool writer = gl % (G / 4) == 0;
    int cur = -1, next = -1;                    // row in `a`; tag of the quad in flight
    T s_next = 1;
    Row<T, NB> a[R], a2[R], b[U][R];
#pragma unroll
    for (int q = 0; q < R; ++q) { row_zero(a[q]); row_zero(a2[q]); }
    auto fetch_b = [&](int h) {                 // the rows of nonzeros h .. h + U - 1 of quad src
        const int4 c = cols[src];
        const int cs[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
        for (int u = 0; u < U; ++u) fetch(b[u], B + (u64)(unsigned)cs[(h + u) & 3] * ldb_bytes);
    };
    auto request = [&]() {                      // as in sddmm_windows, and the value that this lane will scale
        fetch_b(0);
        next = __shfl_sync(FULL, tag, src);
        if (__any_sync(FULL, next != cur)) fetch(a2, arows.resolve(next & 0x7fffffff) + off[0]);
        const int pos = 4 * src + mine;
        s_next = store.scale(w0 + (pos < n ? pos : n - 1));
    };
    request();
    for (int left = each - 1; left >= 0; --left) {
        const int pos = 4 * src + mine;
        const T s = s_next;
        T d[4];
        quad_products<T, NB, R, U, EXACT>(d, a, a2, b, on, cur, next, [&] { return rows[src]; },
                                          [&](int h) { if (h > 0) fetch_b(h); },
                                          [&](int row) { fetch(a, arows.resolve(row) + off[0]); });
        if (left > 0) {
            src += inc;
            request();
        }
        const T total = group_sum4<T, G>(d, gl);
        if (writer && pos < n) store.put(w0 + pos, total * s);
    }
}

// ---------------------------------------------------------------------------
// SpMM
// ---------------------------------------------------------------------------
constexpr int SPMM_PIECE_SHIFT = 20;   // at most 2^20 split rows, 2^11 pieces per row
constexpr int SPMM_ITEM_ROWS = 32;     // most rows of a rows item: a lane holds the end of one row

struct SpmmLong {
    const int* first_piece;  // [nlong] first carry slot of each long row
    const int* npieces;      // [nlong]
    int* counters;           // [nlong] zero at launch; reset by the finishing warp
    void* carry;             // [total pieces, ldc] scratch
    long long ldc;           // elements per carry row
    int* ticket;             // optional work counters {next item, blocks done}, zero between launches: items are
                             // then handed out dynamically
};

// Previous values of a block of result rows on their way into the L2 (each row end waits for its own, one by one).
__device__ __forceinline__ void prefetch_rows(const char* p, long long bytes, int lane) {
    for (long long o = lane * 128; o < bytes; o += 32 * 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + o));
}

template <typename T, int NB> struct EmitLocal {
    char* Y;
    long long ldy_bytes;
    T beta;
    __device__ __forceinline__ void expect(int row, int n, int nvec, int lane) const {
        if (beta != (T)0) prefetch_rows(Y + row * ldy_bytes, (n - 1) * ldy_bytes + nvec * NB, lane);
    }
    // writes vector v of row `row`
    __device__ __forceinline__ void operator()(int row, int v, Row<T, NB> acc) const {
        char* y = Y + row * ldy_bytes + (long long)v * NB;
        if (beta != (T)0) {
            Row<T, NB> old;
            row_load(old, y);
            row_fma(acc, beta, old);
        }
        row_store(y, acc);
    }
};

// Rows of k values without padding, written value by value (X rows are padded, result rows are not).
template <typename T> struct EmitPacked {
    T* Y;
    long long ldy;
    int k;
    T beta;
    __device__ __forceinline__ void expect(int row, int n, int, int lane) const {
        if (beta != (T)0) prefetch_rows(reinterpret_cast<const char*>(Y + row * ldy), ((n - 1) * ldy + k) * (long long)sizeof(T), lane);
    }
    __device__ __forceinline__ void operator()(int row, int v, const Row<T, 16>& acc) const {
        constexpr int N = 16 / (int)sizeof(T);
        if (v * N >= k) return;   // X may be wider by whole vectors: nothing of this one belongs to the row
        T x[N];
        if constexpr (sizeof(T) == 4) {
            const float2 a = unpack2(acc.x[0]), b = unpack2(acc.x[1]);
            x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
        } else {
            x[0] = acc.x[0]; x[1] = acc.x[1];
        }
        T* y = Y + row * ldy + v * N;
        if (beta != (T)0) {
            T old[N];
#pragma unroll
            for (int j = 0; j < N; ++j) old[j] = y[v * N + j < k ? j : 0];
#pragma unroll
            for (int j = 0; j < N; ++j) x[j] += beta * old[j];
        }
#pragma unroll
        for (int j = 0; j < N; ++j)
            if (v * N + j < k) y[j] = x[j];
    }
};

// Shared memory of a warp that works on items: the rows of the item that hold nonzeros, as (end, row number), behind
// them a sentinel, and from the back the numbers of the empty rows; and for every lane the part of a row that began in
// an earlier group (see below).
template <int R, int N, typename E, bool HEADS> struct ItemScratch {
    int2 rows[SPMM_ITEM_ROWS + 2];
    int4 item;
    E heads[HEADS ? R * N * 32 : 1];
};
template <typename T, int NB, int G, int R>
using ItemSmem = ItemScratch<R, Row<T, NB>::N, typename Row<T, NB>::E, (32 / G > 1)>;

// One item, one warp (see build_spmm_items in ops/cuda_ops.py):
//   rows item   (first row, end row, first nonzero, -1 - nonzeros): at most SPMM_ITEM_ROWS whole rows; a first
//               nonzero that 32 bits do not hold is -1 and read from the row pointer
//   piece item  (row, first nonzero, end nonzero, long-row slot | piece number << SPMM_PIECE_SHIFT)
//
// The nonzeros of an item are dealt to the lane groups in equal shares of whole quads, wherever the rows end: a
// group emits the rows that lie inside its share, and the sums of rows that go on in the next group travel along
// the groups by shuffle, in order, at the end.  (Dealing whole rows to the groups left most lanes idle behind the
// longest one: R-MAT scale 20, k = 32, 0.44 ms against 0.26 ms.)  Indices and values come as quads that all lanes of
// a group read, requested one quad ahead; U x R dense vectors are in flight per lane.  No atomics on values: bitwise
// reproducible.
//
// Bound by the latency of the row gathers: a warp that adds up, or ends a row, has none in flight, and a quad waits for
// the slowest of its rows.  So what lies between two quads is kept short -- one comparison tells whether a quad ends a
// row, the rows that hold nonzeros are listed once per item, empty rows are written apart from them -- and what is not
// needed in every quad (where rows end, the part of a group's first row) stays in shared memory, so that the loop spills
// little or nothing within the registers of 32 (one vector per row and lane), 24 or 16 warps per SM.
template <typename T, int NB, int G, int R, int U, bool EXACT, typename Emit>
__device__ __forceinline__ void spmm_warp_item(const int4 item, const long long* rowptr, long long nnz,
                                               const int* colidx, const T* val,
                                               const char* X, unsigned ldx_bytes, int nvec, bool aligned,
                                               const Emit& emit, const SpmmLong& lg, ItemSmem<T, NB, G, R>& sm, int lane) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int SLOTS = 32 / G;            // G need not divide 32: the lanes of slot SLOTS have no share
    constexpr int N = Row<T, NB>::N;
    constexpr int NO_END = 0x7fffffff;
    const int slot = lane / G, gl = lane % G;
    unsigned off[R];
    bool on[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {   // lanes past the row's last vector read it too and emit nothing
        const int v = gl + q * G;
        on[q] = EXACT || (q < R - 1 && R < 8) || v < nvec;   // (see row_dot)
        off[q] = (unsigned)(on[q] ? v : nvec - 1) * NB;
    }
    X += off[0];
    auto clear = [&](Row<T, NB> (&v)[R]) {
#pragma unroll
        for (int q = 0; q < R; ++q) row_zero(v[q]);
    };
    auto flush = [&](int row, const Row<T, NB> (&v)[R]) {
#pragma unroll
        for (int q = 0; q < R; ++q)
            if ((q < R - 1 && R < 8) || on[q]) emit(row, gl + q * G, v[q]);
    };
    const bool is_piece = item.w >= 0, is_rows = !is_piece && item.y - item.x > 1;   // else: one whole row
    const int nr = item.y - item.x;
    const long long p0 = is_piece ? item.y : (item.z >= 0 ? item.z : rowptr[item.x]);
    const int n = is_piece ? item.z - item.y : -1 - item.w;
    // positions count from the 16-byte boundary at or before the first nonzero
    const int lead = (int)(p0 & 3), stop = lead + n;
    const int share = ((stop + 4 * SLOTS - 1) / (4 * SLOTS)) * 4;
    const int begin = slot < SLOTS ? slot * share : stop, end = begin + share < stop ? begin + share : stop;
    const int* cp = colidx + (p0 - lead);
    const T* vp = val + (p0 - lead);
    const int avail = (int)(nnz - (p0 - lead) < NO_END ? nnz - (p0 - lead) : NO_END);
    int row_end_lane = stop;                 // lane l: end of row l of the item
    if (is_rows && lane < nr) row_end_lane = lead + (int)(rowptr[item.x + lane + 1] - p0);
    Row<T, NB> acc[R];
    clear(acc);
    int r = 0;                               // row (of those that hold nonzeros) this group is in
    bool open = false;                       // it began in an earlier group
    if (is_rows) {
        int row_begin_lane = __shfl_up_sync(FULL, row_end_lane, 1);
        if (lane == 0) row_begin_lane = lead;
        const bool mine = lane < nr, full = mine && row_end_lane > row_begin_lane;
        const unsigned filled = __ballot_sync(FULL, full), below = (1u << lane) - 1;
        const int n_full = __popc(filled), n_empty = nr - n_full;
        if (full) sm.rows[__popc(filled & below)] = make_int2(row_end_lane, item.x + lane);
        else if (mine) sm.rows[SPMM_ITEM_ROWS + 1 - __popc(~filled & below)].y = item.x + lane;
        if (lane == 0) sm.rows[n_full].x = NO_END;
#pragma unroll
        for (int g = 1; g < SLOTS; ++g) {
            const unsigned done = __ballot_sync(FULL, full && row_end_lane <= g * share);
            if (slot == g) r = __popc(done);
        }
        __syncwarp();
        for (int e = slot; e < n_empty; e += SLOTS)   // (slot SLOTS: every row is written by a group before it)
            if (slot < SLOTS) flush(sm.rows[SPMM_ITEM_ROWS + 1 - e].y, acc);
        open = slot > 0 && begin < end && (r == 0 ? lead : sm.rows[r - 1].x) < begin;
    } else {
        if (lane == 0) {
            sm.rows[0].x = NO_END;
            sm.item = item;
        }
        __syncwarp();
    }
    bool in_head = open;
    // quads that end at or before `plain` lie inside the item and end no row
    int plain = 0;
    auto look = [&]() {
        const int row_end = sm.rows[r].x;
        plain = row_end <= end ? row_end - 1 : end;
    };
    if (begin >= lead) look();
    auto close = [&]() {                     // the current row ends here
        if (SLOTS > 1 && in_head) {
#pragma unroll
            for (int q = 0; q < R; ++q)
#pragma unroll
                for (int h = 0; h < N; ++h) sm.heads[(q * N + h) * 32 + lane] = acc[q].x[h];
            in_head = false;
        } else {
            flush(sm.rows[r].y, acc);
        }
        clear(acc);
        ++r;
    };
    // VEC: every quad of the item lies inside the lists, and is a vector of them
    auto walk = [&](auto vec) {
        constexpr bool VEC = decltype(vec)::value;
        auto columns = [&](int i) {
            if constexpr (VEC) return quad_load_vec(cp + i);
            else return quad_load(cp, i, avail, false);
        };
        const int tail = (end - 1) & ~3;     // last quad of this group
        Quad<int> c4 = columns(begin);
        for (int i = begin; i < end; i += 4) {
            Quad<T> v4;
            const bool fast = i + 4 <= plain;
#pragma unroll
            for (int h = 0; h < 4; h += U) {
                Row<T, NB> x[U][R];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    // Positions outside the item are read too (their columns are those of the neighbouring items) and
                    // left out below: with the loads under a condition the kernel took 0.71 ms instead of 0.65 ms
                    // (R-MAT scale 20, k = 128).
                    const char* row = X + (u64)(unsigned)c4.v[h + u] * ldx_bytes;
#pragma unroll
                    for (int q = 0; q < R; ++q) row_load(x[u][q], row + (off[q] - off[0]));
                }
                // the values, and the indices of the next quad, are requested behind the rows of this one: loads come
                // back in order, and the lists may have to come from device memory (requested ahead of the rows: 0.84
                // ms instead of 0.66 ms at R-MAT scale 20, k = 128)
                if (h == 0) {
                    if constexpr (VEC) v4 = quad_load_vec(vp + i);
                    else v4 = quad_load(vp, i, avail, false);
                }
                if (h + U == 4) c4 = columns(i < tail ? i + 4 : tail);
                if (fast) {
#pragma unroll
                    for (int u = 0; u < U; ++u)
#pragma unroll
                        for (int q = 0; q < R; ++q) row_fma(acc[q], v4.v[h + u], x[u][q]);
                } else {
                    int row_end = sm.rows[r].x;
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int p = i + h + u;
                        if (p >= lead && p < end) {
#pragma unroll
                            for (int q = 0; q < R; ++q) row_fma(acc[q], v4.v[h + u], x[u][q]);
                            if (p + 1 == row_end) {
                                close();
                                row_end = sm.rows[r].x;
                            }
                        }
                    }
                    if (h + U == 4) look();
                }
            }
        }
    };
    if (begin < end) {
        if (aligned && ((stop + 3) & ~3) <= avail) walk(std::true_type{});
        else walk(std::false_type{});
    }
    if (is_rows) {
        // A row that goes on: its sum so far (acc) moves to the next group.  in_head still set: the whole share
        // lies inside one row that began earlier and goes on.
        if (SLOTS > 1 && __any_sync(FULL, open)) {
            Row<T, NB> carry[R];
            clear(carry);
#pragma unroll
            for (int g = 1; g < SLOTS; ++g)
#pragma unroll
                for (int q = 0; q < R; ++q)
#pragma unroll
                    for (int h = 0; h < N; ++h) {
                        const auto sum = in_head ? e_add(carry[q].x[h], acc[q].x[h]) : acc[q].x[h];
                        const auto up = __shfl_up_sync(FULL, sum, G);
                        if (slot == g) carry[q].x[h] = up;
                    }
            if (open && !in_head) {
#pragma unroll
                for (int q = 0; q < R; ++q)
#pragma unroll
                    for (int h = 0; h < N; ++h) carry[q].x[h] = e_add(carry[q].x[h], sm.heads[(q * N + h) * 32 + lane]);
                int h = 0;           // the row in which this share begins
                while (sm.rows[h].x <= begin) ++h;
                flush(sm.rows[h].y, carry);
            }
        }
        __syncwarp();
        return;
    }
    __syncwarp();
    // one row: add up the groups; a piece of a long row leaves the sum in the carry, and the last piece to arrive adds
    // the carries in order
    auto add_groups = [&]() {                // slot 0 gets the sum of all slots
        if constexpr ((G & (G - 1)) == 0) {
#pragma unroll
            for (int m = G; m < 32; m <<= 1)
#pragma unroll
                for (int q = 0; q < R; ++q)
#pragma unroll
                    for (int h = 0; h < Row<T, NB>::N; ++h)
                        acc[q].x[h] = e_add(acc[q].x[h], __shfl_xor_sync(FULL, acc[q].x[h], m));
        } else {
#pragma unroll
            for (int q = 0; q < R; ++q)
#pragma unroll
                for (int h = 0; h < Row<T, NB>::N; ++h) {
                    auto sum = acc[q].x[h];
#pragma unroll
                    for (int g = 1; g < SLOTS; ++g) sum = e_add(sum, __shfl_sync(FULL, acc[q].x[h], gl + g * G));
                    acc[q].x[h] = sum;
                }
        }
    };
    add_groups();
    const int row = sm.item.x, code = sm.item.w;
    if (code < 0) {
        if (slot == 0) flush(row, acc);
        __syncwarp();
        return;
    }
    const int lr = code & ((1 << SPMM_PIECE_SHIFT) - 1);
    const int first_piece = lg.first_piece[lr], np = lg.npieces[lr];
    char* carry = static_cast<char*>(lg.carry);
    const long long ldc_bytes = lg.ldc * (long long)sizeof(T);
    if (slot == 0)
#pragma unroll
        for (int q = 0; q < R; ++q)
            if (on[q]) row_store(carry + (first_piece + (code >> SPMM_PIECE_SHIFT)) * ldc_bytes + (gl + q * G) * NB, acc[q]);
    __threadfence();
    __syncwarp();
    int old = 0;
    if (lane == 0) old = atomicAdd(lg.counters + lr, 1);
    old = from_lane0(old);
    if (old != np - 1) return;
    __threadfence();
    // group g adds every SLOTS-th carry, then the groups are added up (more loads in flight here would take registers
    // from the loop above: the kernel is compiled for a fixed number of warps)
    clear(acc);
    carry += first_piece * ldc_bytes + off[0];
#pragma unroll 4
    for (int j = slot < SLOTS ? slot : np; j < np; j += SLOTS) {
        Row<T, NB> x[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            row_load_cg(x[q], carry + j * ldc_bytes + (off[q] - off[0]));
            row_add(acc[q], x[q]);
        }
    }
    add_groups();
    if (slot == 0) flush(row, acc);
    if (lane == 0) lg.counters[lr] = 0;
}

// Dense vectors a lane has in flight (U nonzeros x R vectors of NB bytes) and blocks of 256 threads an SM should hold: about
// half of the registers belong to loads in flight; more would halve the warps, fewer leave the memory idle.  More blocks
// than these spill registers in the inner loops.  What counts in the SpMM is the bytes of a lane: three or four vectors of 4
// bytes take the registers of one of 16, and in the blocks that three or four wide ones leave they have a quarter of the
// bytes in flight (SpMM, R-MAT scale 14, items fitted to the warps of each: k = 75 22.5 us in two blocks, 13.3 in four;
// k = 101 24.2 and 14.8; scale 16 5 % less).  In the SDDMM that pays for rows of 16 lanes and more (8-byte vectors, k = 90, 126, 178 7 to 11 %; rows of 8 lanes
// level, 15 % either way) and for five vectors and more.
__host__ __device__ constexpr int spmm_unroll(int R, int NB = 16) { return R * NB <= 64 ? 4 : 1; }
__host__ __device__ constexpr int sddmm_unroll(int R, bool f32, int NB = 16) {
    return R <= (f32 ? 4 : 3) || (NB < 16 && R * NB <= 48) ? 4 : 2;
}
__host__ __device__ constexpr int sddmm_min_blocks(int R, bool f32, int NB = 16, int G = 32) {
    if (NB < 16 && R > 2 && R <= 4 && G >= 16 && f32) return R * NB <= 16 ? 4 : 3;
    return R == 1 ? 4 : (R == 2 && f32 ? 3 : (R <= 4 || R * NB <= 48 ? 2 : 1));
}
__host__ __device__ constexpr int spmm_min_blocks(int R, int NB = 16) { return R * NB <= 16 ? 4 : (R * NB <= 32 ? 3 : 2); }

// All items of an SpMM, by block `block` of `nblocks` blocks of 256 threads that do so (every one of them calls it).
template <typename T, int NB, int G, int R, bool EXACT, typename Emit>
__device__ __forceinline__ void spmm_items(unsigned block, unsigned nblocks, int nitems, const int4* items, int nrows,
                                           const long long* rowptr, const int* colidx, const T* val, const char* X,
                                           unsigned ldx_bytes, int nvec, bool aligned, const Emit& emit, const SpmmLong& lg,
                                           ItemSmem<T, NB, G, R>& sm) {
    const int lane = threadIdx.x & 31;
    const int warp0 = (int)(((long long)block * blockDim.x + threadIdx.x) >> 5);
    const int nwarps = (int)(((long long)nblocks * blockDim.x) >> 5);
    const long long nnz = rowptr[nrows];
    auto run = [&](int it) {
        const int4 item = items[it];
        // (items of fewer rows wait for the previous values less often than the requests cost: Erdos-Renyi, 24 nonzeros
        // a row, fp64, k = 64, 457 us with them, 448 without; R-MAT scale 20, k = 32, beta 0.5, 280 against 313)
        if (item.w < 0 && item.y - item.x >= 8) emit.expect(item.x, item.y - item.x, nvec, lane);
        spmm_warp_item<T, NB, G, R, spmm_unroll(R, NB), EXACT>(item, rowptr, nnz, colidx, val, X, ldx_bytes, nvec,
                                                                 aligned, emit, lg, sm, lane);
    };
    if (lg.ticket && nitems > nwarps) {
        // dynamic hand-out: items differ too much in cost (cached or not, hub or not) for a fixed assignment to balance
        // (a ticket drawn while the item before it runs binds work to a busy warp: R-MAT scale 17, k = 33, 51 us
        // instead of 48)
        for (int it = warp0; it < nitems;) {
            run(it);
            if (lane == 0) it = nwarps + atomicAdd(lg.ticket, 1);
            it = __shfl_sync(0xffffffffu, it, 0);
        }
        // the last block to finish leaves the counters at zero for the next launch (no memset per launch)
        __syncthreads();
        if (threadIdx.x == 0 && atomicAdd(lg.ticket + 1, 1) == (int)nblocks - 1) {
            lg.ticket[0] = 0;
            lg.ticket[1] = 0;
        }
        return;
    }
    for (int it = warp0; it < nitems; it += nwarps) run(it);
}

// Work items per ticket of a dynamically scheduled kernel: about 1/32 of a warp's share, at most max_per.
__device__ __forceinline__ int per_ticket(long long n_work, int nwarps, int max_per) {
    const long long p = n_work / ((long long)nwarps * 32);
    return p < 1 ? 1 : (p > max_per ? max_per : (int)p);
}

// ---- launch helpers ----------------------------------------------------------
inline int env_int(const char* name, int dflt) {
    const char* e = getenv(name);
    return e ? atoi(e) : dflt;
}

// Launch that may begin while the previous kernel of the stream drains (programmatic dependent launch): the kernel
// has to call `after_previous_kernel` before it touches memory, and to read what an earlier kernel of this library may
// have written by ordinary loads (see row_load): it is resident while that kernel still writes.
template <typename... P, typename... A>
inline int launch_early(void (*kernel)(P...), unsigned blocks, size_t smem, cudaStream_t st, const A&... args) {
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

constexpr int MAX_DEVICES = 64;

// Blocks of `threads` threads of a persistent launch of `kernel`: all that fit at once, at most `needed` (0: no
// limit), none if not even one does.  `cache` belongs to this kernel and keeps the answer for the dynamic shared memory
// asked for last: the occupancy query costs more than a launch.  Without the attribute a launch has 48 KB, static and
// dynamic shared memory together; it is raised to what a block can have, the same value whoever sets it.
struct ResidentCache { std::atomic<unsigned long long> last[MAX_DEVICES] = {}; };   // smem << 32 | blocks
template <typename K>
unsigned resident_blocks(K kernel, ResidentCache& cache, long long needed, int threads = 256, size_t smem = 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 1;
    unsigned long long v = dev < MAX_DEVICES ? cache.last[dev].load(std::memory_order_relaxed) : 0;
    if (v == 0 || v >> 32 != smem) {
        int sms = 0, per_sm = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (smem > 0) {
            int most = 0;
            cudaFuncAttributes own = {};
            cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
            if (cudaFuncGetAttributes(&own, kernel) != cudaSuccess ||
                cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)own.sharedSizeBytes) != cudaSuccess)
                return 0;
        }
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm < 1 || sms < 1) return 0;
        v = (unsigned long long)smem << 32 | (unsigned)(sms * per_sm);
        if (dev < MAX_DEVICES) cache.last[dev].store(v, std::memory_order_relaxed);
    }
    const long long b = (long long)(v & 0xffffffffu);
    return (unsigned)(needed > 0 && needed < b ? needed : b);
}

// Lanes per row (G) and vectors per lane (R) for a row of `nvec` vectors, at most 256.
//   SDDMM  few lanes with several vectors each: every step of the reduction then serves 32 / G nonzeros (R-MAT scale
//          20, fp32: k = 64 278 us as 8 x 2, 394 as 16 x 1; k = 128 490 us as 8 x 4, 568 as 16 x 2, 707 as 32 x 1).  9 to
//          12 vectors go as 4 x 3 (R-MAT scale 17, k = 40: 39 us, 47 as 8 x 2, where a third of the lanes idles); 13 to
//          16 do not fit 4 x 4 as well (k = 64, scale 20: 0.375 ms).
//   SpMM   several vectors per lane from 11 vectors on: what all lanes of a group read and compute for a nonzero (its
//          index, its value, its address) then serves that many more bytes.  R-MAT scale 20: k = 64 331 us as 8 x 2, 350
//          as 16 x 1; k = 128 569 as 16 x 2, 571 as 8 x 4, 606 as 32 x 1; scale 17: 43 against 48 us, 72 (8 x 4), 76
//          (16 x 2) and 88.  25 to 32 vectors go as 8 x 4 where X comes out of the L2 (`cached`), and as 16 x 2, which
//          keeps half as many warps more, where it does not (scale 22: 2640 against 2692 us).  49 to 64: 16 x 4 (Zipf
//          rows, k = 256: 885 us, 909 as 32 x 2).  17 to 24 go as 8 x 3 (k = 96, scale 17: 67 us, 100 as 32 x 1), 33 to
//          48 as 16 x 3 (k = 192: 110 us, 140 as 32 x 2), and groups of 5, 6 and 10 lanes share a warp one group more than
//          8 or 16 do (k = 40: 41 us as 10 x 1, 51 as 16 x 1; k = 20: 32 against 35 us; groups of 2 and 3 gained nothing
//          over 4).
//
// 129 to 192 vectors narrower than 16 bytes (`narrow`) go as 32 x 5 and 32 x 6; wider rows take eight per lane, where up to
// three read the last vector again.
inline void pick_shape(int nvec, int* G, int* R, bool spmm, bool cached = false, bool narrow = false) {
    int g = 4;
    const int top = spmm ? 32 : (nvec <= 32 ? 8 : (nvec <= 64 ? 16 : 32));
    while (g < top && g < nvec) g <<= 1;
    if (spmm) {
        if (nvec == 5 || nvec == 6) g = nvec;
        if (nvec == 9 || nvec == 10) g = 10;
        if (nvec > 10 && nvec <= 24) g = 8;
        if (nvec > 24 && nvec <= 32) g = cached ? 8 : 16;
        if (nvec > 32 && nvec <= 64) g = 16;
    } else if (nvec > 8 && nvec <= 12) {
        g = 4;
    }
    int r = (nvec + g - 1) / g;
    r = r <= (narrow ? 6 : 4) ? r : 8;
    *G = g;
    *R = r;
}
// Dense operands of at most this many bytes are expected to stay in the L2 (126 MB, part of it held twice, once per
// die, and shared with the results and the sparse matrix).
constexpr long long CACHED_BYTES = 64ll << 20;

#define SP3_SDDMM_SHAPES(MACRO)                                                                           \
    switch (G * 16 + R) {                                                                                 \
        case 4 * 16 + 1: MACRO(4, 1); break;   case 8 * 16 + 1: MACRO(8, 1); break;                       \
        case 4 * 16 + 3: MACRO(4, 3); break;                                                              \
        case 8 * 16 + 2: MACRO(8, 2); break;   case 8 * 16 + 3: MACRO(8, 3); break;                       \
        case 8 * 16 + 4: MACRO(8, 4); break;   case 16 * 16 + 3: MACRO(16, 3); break;                     \
        case 16 * 16 + 4: MACRO(16, 4); break; case 32 * 16 + 3: MACRO(32, 3); break;                     \
        case 32 * 16 + 4: MACRO(32, 4); break; default: MACRO(32, 8); break;                              \
    }
#define SP3_SPMM_SHAPES(MACRO)                                                                            \
    switch (G * 16 + R) {                                                                                 \
        case 4 * 16 + 1: MACRO(4, 1); break;   case 8 * 16 + 1: MACRO(8, 1); break;                       \
        case 5 * 16 + 1: MACRO(5, 1); break;   case 6 * 16 + 1: MACRO(6, 1); break;                       \
        case 10 * 16 + 1: MACRO(10, 1); break; case 8 * 16 + 2: MACRO(8, 2); break;                       \
        case 16 * 16 + 1: MACRO(16, 1); break; case 32 * 16 + 1: MACRO(32, 1); break;                     \
        case 8 * 16 + 3: MACRO(8, 3); break;   case 16 * 16 + 2: MACRO(16, 2); break;                     \
        case 8 * 16 + 4: MACRO(8, 4); break;   case 16 * 16 + 3: MACRO(16, 3); break;                     \
        case 16 * 16 + 4: MACRO(16, 4); break; case 32 * 16 + 3: MACRO(32, 3); break;                     \
        case 32 * 16 + 4: MACRO(32, 4); break; default: MACRO(32, 8); break;                              \
    }
}  // namespace sp3
