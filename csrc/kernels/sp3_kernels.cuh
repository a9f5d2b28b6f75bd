// Warp-level bodies of the SDDMM and SpMM kernels, shared by the local
// kernels (local_ops.cu) and the fused compute+communication kernels
// (fused_impl.cuh).  Where dense rows come from and where results go is a
// template policy, so both families run the same inner loops:
//
//   SDDMM   A rows:  RowsByStride (one local block) | RowsByPeerRef (rows that
//                    stay in their owners' memory, local or peer)
//           output:  StoreLocal | the fused kernel's slice-routing store
//   SpMM    emit:    EmitLocal (Y = beta*Y + acc) | the fused kernel's
//                    owned-or-push emit
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

// Dense rows and values are read by ordinary loads, never through the read-only path (`ld.global.nc`, `__ldg`, or a
// `const __restrict__` kernel parameter, from which the compiler infers it): that path is defined only for memory that
// nobody writes while the kernel runs.  A kernel launched early runs while the kernel before it writes what may be its
// values or rows (see after_previous_kernel), and in the fused kernels other warps of the launch write the pulled rows.
// Ordinary loads are ordered behind the wait, or the acquire, that says the data is there.  Index arrays and work items
// are fixed when an operator is built and keep the read-only path.
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
        if (ALL || (q < R - 1 && R <= 4) || on[q])   // (pick_shape: only the last vector of a lane can be past the row)
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
// positions at or past `end` repeat the last value before it.  Lists of int are index lists (read-only path).
template <typename I> struct Quad { I v[4]; };
__device__ __forceinline__ Quad<int> quad_load_vec(const int* p) {
    const int4 t = __ldg(reinterpret_cast<const int4*>(p));
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
__device__ __forceinline__ int list_load(const int* p) { return __ldg(p); }
template <typename T> __device__ __forceinline__ T list_load(const T* p) { return *p; }
template <typename I> __device__ __forceinline__ Quad<I> quad_load(const I* base, int i, int end, bool aligned) {
    if (aligned && i + 4 <= end) return quad_load_vec(base + i);
    Quad<I> q;
#pragma unroll
    for (int j = 0; j < 4; ++j) q.v[j] = list_load(base + (i + j < end ? i + j : end - 1));
    return q;
}

// ---- row access policies ---------------------------------------------------
// A policy turns the local row index of a nonzero into a 31-bit *reference*
// (`ref`, evaluated by every lane for its own nonzeros when a window of indices
// is read, so a table lookup is off the critical path) and a reference into
// the address of the dense row (`resolve`, pure arithmetic).  The reference is
// what the lane group passes round by shuffle and compares to detect a row
// change.
struct RowsByStride {
    const char* base;
    unsigned ld_bytes;
    __device__ __forceinline__ int ref(int row) const { return row; }
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
__device__ __forceinline__ Quad<int> quad_load_passing(const int* base, int i, int end, bool aligned, u64 policy) {
    if (!aligned || i + 4 > end) return quad_load(base, i, end, false);
    Quad<int> q;
    asm volatile("ld.global.nc.L2::cache_hint.v4.s32 {%0, %1, %2, %3}, [%4], %5;"
        : "=r"(q.v[0]), "=r"(q.v[1]), "=r"(q.v[2]), "=r"(q.v[3]) : "l"(base + i), "l"(policy));
    return q;
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

// Where values go: `scale(i)` is read together with the dense rows, `put(i, v)` stores dot * scale.
template <typename T> struct StoreLocal {
    T* out;
    const T* sval;    // null: no scaling
    __device__ __forceinline__ T scale(long long i) const { return sval ? sval[i] : (T)1; }
    __device__ __forceinline__ void put(long long i, T v) const { out[i] = v; }
};
template <typename T> struct StoreTwice : StoreLocal<T> {
    T* also;          // a second place for the values (a form of its own: the choice in the kernel cost 1 %)
    __device__ __forceinline__ void put(long long i, T v) const { this->out[i] = v; also[i] = v; }
};
template <typename T> struct StoreScattered {
    T* out;
    const T* sval;
    const int* orig;  // result position of nonzero i
    __device__ __forceinline__ T scale(long long i) const { return sval ? sval[i] : (T)1; }
    __device__ __forceinline__ void put(long long i, T v) const { out[__ldg(orig + i)] = v; }
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
// most 128), one warp per window.  Lane l holds the indices of nonzeros 4l .. 4l+3 (one 16-byte load per array,
// requested a whole window ahead); every group of G lanes works through an equal share of these quads: four
// column indices by shuffle, four dense B rows in flight, four dot products reduced together, the A row kept in
// registers until the row changes (the list is sorted by row).
//
// Bound by the row gathers out of L2 and by the issue of what surrounds them, so the split keeps the lanes per
// row few (each shuffle then serves 32/G nonzeros) and fetches the A row of a quad's last nonzero together with
// its B rows.
// ---------------------------------------------------------------------------
constexpr int WINDOW_MAX = 128;

// Nonzeros per window: 128, less when that would leave warps without work.
__host__ __device__ inline int window_nnz(long long nnz, long long nwarps, int groups_per_warp) {
    const int quantum = 4 * groups_per_warp;
    const long long share = (nnz + nwarps - 1) / nwarps;
    const long long w = (share + quantum - 1) / quantum * quantum;
    return (int)(w < quantum ? quantum : (w > WINDOW_MAX ? WINDOW_MAX : w));
}

template <typename T, int NB, int G, int R, int U, bool EXACT, typename ARows, typename Store>
__device__ __forceinline__ void sddmm_windows(long long first, long long step, long long end, int wn, long long nnz,
                                              const int* __restrict__ rowidx, const int* __restrict__ colidx,
                                              const ARows& arows, const char* B, unsigned ldb_bytes,
                                              int nvec, bool aligned, const Store& store, int lane) {
    static_assert(G >= 4, "a group reduces four values");
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
    auto load = [&](long long w, Quad<int>& c, Quad<int>& r) {
        const int n = length(w), i = 4 * lane < n ? 4 * lane : (n - 1) & ~3;
        if constexpr (PASSING) {
            c = quad_load_passing(colidx + w * wn, i, n, aligned, policy);
            r = quad_load_passing(rowidx + w * wn, i, n, aligned, policy);
        } else {
            c = quad_load(colidx + w * wn, i, n, aligned);
            r = quad_load(rowidx + w * wn, i, n, aligned);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) r.v[j] = arows.ref(r.v[j]);
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
    const int mine = gl / (G / 4);              // which of the four results ends up in this lane
    const bool writer = gl % (G / 4) == 0;
    Quad<int> c4, r4;
    load(first, c4, r4);
    int cur = -1;
    Row<T, NB> a[R];
#pragma unroll
    for (int q = 0; q < R; ++q) row_zero(a[q]);
    for (long long w = first; w < end; w += step) {
        Quad<int> cn = c4, rn = r4;
        if (w + step < end) load(w + step, cn, rn);
        const int n = length(w);
        const long long w0 = w * wn;
        const int nq = (((n + 3) >> 2) + SLOTS - 1) / SLOTS;   // quads per group
        // lanes whose quad is not all one row (a list sorted by row class by class may leave and re-enter a row)
        const unsigned mixed = __ballot_sync(FULL, r4.v[0] != r4.v[3] || r4.v[1] != r4.v[3] || r4.v[2] != r4.v[3]);
        for (int i = 0; i < nq; ++i) {
            const int src = slot * nq + i;                     // lane that holds this group's quad
            int c[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) c[u] = __shfl_sync(FULL, c4.v[u], src);
            const int last = __shfl_sync(FULL, r4.v[3], src);
            Row<T, NB> b[U][R];
#pragma unroll
            for (int u = 0; u < U; ++u) fetch(b[u], B + (u64)(unsigned)c[u] * ldb_bytes);
            const int pos = 4 * src + mine;
            const bool st = writer && pos < n;
            const T s = store.scale(w0 + (pos < n ? pos : n - 1));
            T d[4];
            if (__all_sync(FULL, last == cur && !(mixed >> src & 1))) {
#pragma unroll
                for (int h = 0; h < 4; h += U) {
                    if (h > 0)
#pragma unroll
                        for (int u = 0; u < U; ++u) fetch(b[u], B + (u64)(unsigned)c[h + u] * ldb_bytes);
#pragma unroll
                    for (int u = 0; u < U; ++u) d[h + u] = row_dot<EXACT>(a, b[u], on);
                }
            } else {
                int r[4];
#pragma unroll
                for (int u = 0; u < 3; ++u) r[u] = __shfl_sync(FULL, r4.v[u], src);
                r[3] = last;
                Row<T, NB> a2[R];
                const bool staged = last != cur;
                fetch_a(a2, arows.resolve(last) + off[0]);   // (unconditional: a load under a condition costs more)
#pragma unroll
                for (int h = 0; h < 4; h += U) {
                    if (h > 0)
#pragma unroll
                        for (int u = 0; u < U; ++u) fetch(b[u], B + (u64)(unsigned)c[h + u] * ldb_bytes);
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        if (r[h + u] != cur) {
                            cur = r[h + u];
                            if (staged && cur == last) {
#pragma unroll
                                for (int q = 0; q < R; ++q) a[q] = a2[q];
                            } else {
                                fetch_a(a, arows.resolve(cur) + off[0]);
                            }
                        }
                        d[h + u] = row_dot<EXACT>(a, b[u], on);
                    }
                }
            }
            const T total = group_sum4<T, G>(d, gl);
            if (st) store.put(w0 + pos, total * s);
        }
        c4 = cn;
        r4 = rn;
    }
}

// ---------------------------------------------------------------------------
// SpMM
// ---------------------------------------------------------------------------
constexpr int SPMM_PIECE_SHIFT = 20;   // at most 2^20 split rows, 2^11 pieces per row
constexpr int SPMM_ITEM_ROWS = 32;     // most rows of a rows item: a lane holds the end of one row
constexpr int SPMM_ENDS = SPMM_ITEM_ROWS + 1;   // ints of shared memory per warp for the row ends

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

// One item, one warp (see build_spmm_items in ops/cuda_ops.py):
//   rows item   (first row, end row, first nonzero, -1 - nonzeros): at most SPMM_ITEM_ROWS whole rows; a first
//               nonzero that 32 bits do not hold is -1 and read from the row pointer
//   piece item  (row, first nonzero, end nonzero, long-row slot | piece number << SPMM_PIECE_SHIFT)
//
// The nonzeros of an item are dealt to the lane groups in equal shares of whole quads, wherever the rows end: a
// group emits the rows that lie inside its share, and the sums of rows that go on in the next group travel along
// the groups by shuffle, in order, at the end.  (Dealing whole rows to the groups left most lanes idle behind the
// longest one: R-MAT scale 20, k = 32, 0.44 ms against 0.26 ms.)  Row ends are kept in shared memory (`ends`,
// SPMM_ENDS ints per warp), indices and values come as quads that all lanes of a group read, requested one
// quad ahead; U x R dense vectors are in flight per lane.  No atomics on values: bitwise reproducible.
template <typename T, int NB, int G, int R, int U, bool EXACT, typename Emit>
__device__ __forceinline__ void spmm_warp_item(const int4 item, const long long* __restrict__ rowptr, long long nnz,
                                               const int* __restrict__ colidx, const T* val,
                                               const char* X, unsigned ldx_bytes, int nvec, bool aligned,
                                               const Emit& emit, const SpmmLong& lg, int* ends, int lane) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int SLOTS = 32 / G;            // G need not divide 32: the lanes of slot SLOTS have no share
    const int slot = lane / G, gl = lane % G;
    unsigned off[R];
    bool on[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {   // lanes past the row's last vector read it too and emit nothing
        const int v = gl + q * G;
        on[q] = EXACT || v < nvec;
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
            if ((q < R - 1 && R <= 4) || on[q]) emit(row, gl + q * G, v[q]);
    };
    const bool is_rows = item.w < 0;
    const int nr = is_rows ? item.y - item.x : 0;
    const long long p0 = !is_rows ? item.y : (item.z >= 0 ? item.z : __ldg(rowptr + item.x));
    const int n = is_rows ? -1 - item.w : item.z - item.y;
    // positions count from the 16-byte boundary at or before the first nonzero
    const int lead = (int)(p0 & 3), stop = lead + n;
    const int share = ((stop + 4 * SLOTS - 1) / (4 * SLOTS)) * 4;
    const int begin = slot < SLOTS ? slot * share : stop, end = begin + share < stop ? begin + share : stop;
    int row_end_lane = stop;                 // lane l: end of row l of the item
    if (lane < nr) row_end_lane = lead + (int)(__ldg(rowptr + item.x + lane + 1) - p0);
    const int* cp = colidx + (p0 - lead);
    const T* vp = val + (p0 - lead);
    const int avail = (int)(nnz - (p0 - lead) < 0x7fffffff ? nnz - (p0 - lead) : 0x7fffffff);
    Quad<int> c4;
    Quad<T> v4;
    if (begin < end) {
        c4 = quad_load(cp, begin, avail, aligned);
        v4 = quad_load(vp, begin, avail, aligned);
    }
    int r = 0;                               // row of the item this group is in
    if (is_rows) {
        ends[lane] = row_end_lane;
#pragma unroll
        for (int g = 1; g < SLOTS; ++g) {
            const unsigned done = __ballot_sync(FULL, lane < nr && row_end_lane <= g * share);
            if (slot == g) r = __popc(done);
        }
        __syncwarp();
    }
    int row_end = r < nr ? ends[r] : stop;
    const bool open = is_rows && slot > 0 && begin < end && (r == 0 ? lead : ends[r - 1]) < begin;   // began in an earlier group
    bool in_head = open;
    Row<T, NB> acc[R], first[R];             // first: this group's part of a row that began in an earlier group
    clear(acc);
    if (SLOTS > 1) clear(first);
    auto close = [&]() {                     // the current row ends here
        if (SLOTS > 1 && in_head) {
#pragma unroll
            for (int q = 0; q < R; ++q) first[q] = acc[q];
            in_head = false;
        } else {
            flush(item.x + r, acc);
        }
        clear(acc);
        ++r;
        row_end = ends[r];
    };
    for (int i = begin; i < end; i += 4) {
        int c[4];
        T v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) { c[u] = c4.v[u]; v[u] = v4.v[u]; }
        const bool whole = i >= lead && i + 4 <= end;      // no position of this quad lies outside the item
#pragma unroll
        for (int h = 0; h < 4; h += U) {
            Row<T, NB> x[U][R];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                // Positions outside the item are read too (their columns are those of the neighbouring items) and
                // left out below: with the loads under a condition the kernel took 0.71 ms instead of 0.65 ms
                // (R-MAT scale 20, k = 128).
                const char* row = X + (u64)(unsigned)c[h + u] * ldx_bytes;
#pragma unroll
                for (int q = 0; q < R; ++q) row_load(x[u][q], row + (off[q] - off[0]));
            }
            // the next quad is requested behind the rows of this one: loads come back in order, and the indices may
            // have to come from device memory (requested ahead of the rows: 0.84 ms instead of 0.66 ms at R-MAT
            // scale 20, k = 128)
            if (h == 0 && i + 4 < end) {
                c4 = quad_load(cp, i + 4, avail, aligned);
                v4 = quad_load(vp, i + 4, avail, aligned);
            }
            if (whole && i + h + U <= row_end) {
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int q = 0; q < R; ++q) row_fma(acc[q], v[h + u], x[u][q]);
            } else {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int p = i + h + u;
                    if (p >= lead && p < end) {
                        while (p >= row_end) close();
#pragma unroll
                        for (int q = 0; q < R; ++q) row_fma(acc[q], v[h + u], x[u][q]);
                    }
                }
            }
        }
    }
    if (is_rows) {
        // rows that end with this share, and the empty rows after them
        if (begin < end || (slot == 0 && n == 0))
            while (r < nr && ends[r] <= end) close();
        if (SLOTS > 1) {
            // A row that goes on: its sum so far (acc) moves to the next group.  in_head still set: the whole share
            // lies inside one row that began earlier and goes on.
            if (__any_sync(FULL, open)) {
                Row<T, NB> carry[R];
                clear(carry);
#pragma unroll
                for (int g = 1; g < SLOTS; ++g)
#pragma unroll
                    for (int q = 0; q < R; ++q)
#pragma unroll
                        for (int h = 0; h < Row<T, NB>::N; ++h) {
                            const auto sum = in_head ? e_add(carry[q].x[h], acc[q].x[h]) : acc[q].x[h];
                            const auto up = __shfl_up_sync(FULL, sum, G);
                            if (slot == g) carry[q].x[h] = up;
                        }
                if (open && !in_head) {
#pragma unroll
                    for (int q = 0; q < R; ++q) row_add(carry[q], first[q]);
                    int h = 0;           // the row in which this share begins
                    while (ends[h] <= begin) ++h;
                    flush(item.x + h, carry);
                }
            }
        }
        __syncwarp();
        return;
    }
    // piece of a long row: add up the groups, leave the sum in the carry; the last piece to arrive adds the carries
    // in order
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
    const int lr = item.w & ((1 << SPMM_PIECE_SHIFT) - 1);
    const int first_piece = __ldg(lg.first_piece + lr), np = __ldg(lg.npieces + lr);
    char* carry = static_cast<char*>(lg.carry);
    const long long ldc_bytes = lg.ldc * (long long)sizeof(T);
    if (slot == 0)
#pragma unroll
        for (int q = 0; q < R; ++q)
            if (on[q]) row_store(carry + (first_piece + (item.w >> SPMM_PIECE_SHIFT)) * ldc_bytes + (gl + q * G) * NB, acc[q]);
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
    if (slot == 0) flush(item.x, acc);
    if (lane == 0) lg.counters[lr] = 0;
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
__device__ __forceinline__ void after_previous_kernel() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __threadfence();
}

constexpr int MAX_DEVICES = 64;

// Blocks of `threads` threads of a persistent launch of `kernel`: all that fit at once, at most `needed` (0: no
// limit).  `cache` belongs to this kernel and keeps the answer for the dynamic shared memory asked for last: the
// occupancy query costs more than a launch.
struct ResidentCache { std::atomic<unsigned long long> last[MAX_DEVICES] = {}; };   // smem << 32 | blocks
template <typename K>
unsigned resident_blocks(K kernel, ResidentCache& cache, long long needed, int threads = 256, size_t smem = 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 1;
    unsigned long long v = dev < MAX_DEVICES ? cache.last[dev].load(std::memory_order_relaxed) : 0;
    if (v == 0 || v >> 32 != smem) {
        int sms = 0, per_sm = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
        const int b = sms * (per_sm > 0 ? per_sm : 1);
        v = (unsigned long long)smem << 32 | (unsigned)(b > 0 ? b : 1);
        if (dev < MAX_DEVICES) cache.last[dev].store(v, std::memory_order_relaxed);
    }
    const long long b = (long long)(v & 0xffffffffu);
    return (unsigned)(needed > 0 && needed < b ? needed : b);
}

// Lanes per row (G) and vectors per lane (R) for a row of `nvec` vectors, at most 256.
//   SDDMM  few lanes with several vectors each: every index shuffle and every step of the reduction then serves
//          32 / G nonzeros (R-MAT scale 20, fp32: k = 64 0.35 ms as 8 x 2, 0.38 as 16 x 1; k = 128 0.60 ms as
//          8 x 4, 0.71 as 32 x 1).  9 to 12 vectors go as 4 x 3 (R-MAT scale 17, k = 40: 39 us, 47 as 8 x 2, where a
//          third of the lanes idles); 13 to 16 do not fit 4 x 4 as well (k = 64, scale 20: 0.375 ms).
//   SpMM   as many lanes as the row has vectors: an accumulator costs R vectors of registers, and nothing is
//          reduced across lanes inside a row (k = 64: 0.40 ms as 16 x 1, 0.41 as 8 x 2).  Where that leaves a quarter
//          of the lanes idle, three vectors per lane (k = 96, R-MAT scale 17: 67 us as 8 x 3, 100 as 32 x 1;
//          Erdos-Renyi 1 M rows: 1.81 against 1.96 ms; k = 192: 110 us as 16 x 3, 140 as 32 x 2), and groups of 5, 6
//          or 10 lanes, which share a warp one group more than 8 or 16 do (k = 40: 41 us as 10 x 1, 51 as 16 x 1;
//          k = 20: 32 against 35 us; groups of 2 and 3 gained nothing over 4).  Rows of 25 to 32
//          vectors that come out of the L2 (`cached`) go as 16 x 2, half the instructions per row (k = 128, scale
//          17: 86 against 101 us); out of device memory the occupancy counts for more (scale 20: 0.74 against
//          0.69 ms).
inline void pick_shape(int nvec, int* G, int* R, bool spmm, bool cached = false) {
    int g = 4;
    const int top = spmm ? 32 : (nvec <= 32 ? 8 : (nvec <= 64 ? 16 : 32));
    while (g < top && g < nvec) g <<= 1;
    if (spmm) {
        if (nvec == 5 || nvec == 6) g = nvec;
        if (nvec == 9 || nvec == 10) g = 10;
        if (nvec > 16 && nvec <= 24) g = 8;
        if (nvec > 24 && nvec <= 32 && cached) g = 16;
        if (nvec > 32 && nvec <= 48) g = 16;
    } else if (nvec > 8 && nvec <= 12) {
        g = 4;
    }
    int r = (nvec + g - 1) / g;
    r = r <= 4 ? r : 8;
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
        case 10 * 16 + 1: MACRO(10, 1); break;                                                            \
        case 16 * 16 + 1: MACRO(16, 1); break; case 32 * 16 + 1: MACRO(32, 1); break;                     \
        case 8 * 16 + 3: MACRO(8, 3); break;   case 16 * 16 + 2: MACRO(16, 2); break;                     \
        case 16 * 16 + 3: MACRO(16, 3); break; case 32 * 16 + 2: MACRO(32, 2); break;                     \
        case 32 * 16 + 3: MACRO(32, 3); break; case 32 * 16 + 4: MACRO(32, 4); break;                     \
        default: MACRO(32, 8); break;                                                                     \
    }
// Dense vectors a lane has in flight (U nonzeros x R vectors) and blocks of 256 threads an SM should hold: about
// half of the registers belong to loads in flight; more would halve the warps, fewer leave the memory idle.
__host__ __device__ constexpr int spmm_unroll(int R) { return R <= 3 ? 4 : (R == 4 ? 2 : 1); }
__host__ __device__ constexpr int sddmm_unroll(int R) { return R <= 4 ? 4 : 2; }
__host__ __device__ constexpr int sddmm_min_blocks(int R) { return R == 1 ? 4 : (R == 2 ? 3 : (R <= 4 ? 2 : 1)); }
__host__ __device__ constexpr int spmm_min_blocks(int G, int R) { return R == 1 ? 4 : (R == 2 && G == 32 ? 3 : 2); }

}  // namespace sp3
