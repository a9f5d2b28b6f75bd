// SDDMM and SpMM of one matrix by one call: the step of a single GPU (bench.py's unit) and the attention chain.
//
// Small steps are bound by launches: the two kernels of 5 to 50 thousand nonzeros run 2 us each, and every launch costs
// the host about that much.  Where the SpMM does not read what the SDDMM writes, both run in one launch here, the SpMM in
// the first blocks and the SDDMM in the others; with larger matrices and in chains the call queues the two kernels.
//
// Reference: the two kernels back to back, miniapp/main_combined.cpp:165-281.
#include "sp3_calls.cuh"

namespace sp3 {

template <typename T> struct PairArgs {
    // SDDMM: a window per warp
    long long nnz;
    int wn;
    const int *rowidx, *colidx;
    RowsByStride arows;
    const char* B;
    unsigned ldb_bytes;
    StoreLocal<T> store;
    // SpMM
    int nitems, nrows;
    const int4* items;
    const long long* rowptr;
    const int* ci;
    const T* val;
    const char* X;
    unsigned ldx_bytes;
    EmitLocal<T, 16> emit;
    SpmmLong lg;
    // both
    int nvec;
    bool aligned_sddmm, aligned_spmm;
    unsigned spmm_blocks;
};

constexpr int pair_min_blocks(int RS, int RP, bool f32) {
    const int a = sddmm_min_blocks(RS, f32), b = spmm_min_blocks(RP);
    return a < b ? a : b;
}

template <typename T, int GS, int RS, int GP, int RP>
__global__ void __launch_bounds__(256, pair_min_blocks(RS, RP, sizeof(T) == 4)) pair_kernel(const PairArgs<T> a) {
    after_previous_kernel();
    struct Lists { int4 cols[256 / 32][WINDOW_MAX / 4], rows[256 / 32][WINDOW_MAX / 4]; };
    __shared__ union Scratch {
        __device__ Scratch() {}
        Lists lists;
        ItemSmem<T, 16, GP, RP> items[256 / 32];
    } sm;
    const int warp = threadIdx.x >> 5;
    if (blockIdx.x < a.spmm_blocks)
        spmm_items<T, 16, GP, RP, false>(blockIdx.x, a.spmm_blocks, a.nitems, a.items, a.nrows, a.rowptr, a.ci, a.val, a.X,
                                         a.ldx_bytes, a.nvec, a.aligned_spmm, a.emit, a.lg, sm.items[warp]);
    else
        sddmm_window<T, 16, GS, RS, sddmm_unroll(RS, sizeof(T) == 4), false>(
            (long long)(blockIdx.x - a.spmm_blocks) * (256 / 32) + warp, a.wn, a.nnz, a.rowidx, a.colidx, a.arows, a.B,
            a.ldb_bytes, a.nvec, a.aligned_sddmm, a.store, sm.lists.cols[warp], sm.lists.rows[warp], threadIdx.x & 31);
}

// Shapes of the pair for rows of `nvec` vectors (see pick_shape); `short_rows`: several rows per item, whose ends lie inside
// the shares of the groups (see launch_spmm_nb).
struct PairShape { int gs, rs, gp, rp; };
inline PairShape pair_shape(int nvec, bool short_rows) {
    PairShape s;
    pick_shape(nvec, &s.gs, &s.rs, false);
    pick_shape(nvec, &s.gp, &s.rp, true, true);
    if (short_rows && nvec > 10 && (nvec <= 16 || (nvec > 24 && nvec <= 32))) {
        s.gp = 16;
        s.rp = nvec <= 16 ? 1 : 2;
    }
    return s;
}
#define SP3_PAIR_SHAPES(MACRO)                                                                            \
    switch (((s.gs * 16 + s.rs) * 64 + s.gp) * 16 + s.rp) {                                               \
        case ((4 * 16 + 1) * 64 + 4) * 16 + 1: MACRO(4, 1, 4, 1); break;                                  \
        case ((8 * 16 + 1) * 64 + 5) * 16 + 1: MACRO(8, 1, 5, 1); break;                                  \
        case ((8 * 16 + 1) * 64 + 6) * 16 + 1: MACRO(8, 1, 6, 1); break;                                  \
        case ((8 * 16 + 1) * 64 + 8) * 16 + 1: MACRO(8, 1, 8, 1); break;                                  \
        case ((4 * 16 + 3) * 64 + 10) * 16 + 1: MACRO(4, 3, 10, 1); break;                                \
        case ((4 * 16 + 3) * 64 + 8) * 16 + 2: MACRO(4, 3, 8, 2); break;                                  \
        case ((4 * 16 + 3) * 64 + 16) * 16 + 1: MACRO(4, 3, 16, 1); break;                                \
        case ((8 * 16 + 2) * 64 + 8) * 16 + 2: MACRO(8, 2, 8, 2); break;                                  \
        case ((8 * 16 + 2) * 64 + 16) * 16 + 1: MACRO(8, 2, 16, 1); break;                                \
        case ((8 * 16 + 3) * 64 + 8) * 16 + 3: MACRO(8, 3, 8, 3); break;                                  \
        case ((8 * 16 + 4) * 64 + 8) * 16 + 4: MACRO(8, 4, 8, 4); break;                                  \
        case ((8 * 16 + 4) * 64 + 16) * 16 + 2: MACRO(8, 4, 16, 2); break;                                \
        case ((16 * 16 + 3) * 64 + 16) * 16 + 3: MACRO(16, 3, 16, 3); break;                              \
        case ((16 * 16 + 4) * 64 + 16) * 16 + 4: MACRO(16, 4, 16, 4); break;                              \
        default: break;                                                                                   \
    }

// Blocks of the kernel that are resident at once; 0: no kernel of that shape.
template <typename T> unsigned pair_resident(const PairShape& s) {
    unsigned b = 0;
#define SP3_PAIR(A, B, C, D)                                                                              \
    {                                                                                                     \
        static ResidentCache cache;                                                                       \
        b = resident_blocks(pair_kernel<T, A, B, C, D>, cache, 0);                                        \
    }
    SP3_PAIR_SHAPES(SP3_PAIR)
#undef SP3_PAIR
    return b;
}

// Whether the two calls can be one launch that pays; the shape, the blocks of the SpMM and the nonzeros per window of the
// SDDMM if so.  It saves a launch on the host (2.2 us of 7.4) and a ramp on the device, and loses where the SpMM alone has
// all its items in flight at once and has not beside the SDDMM, unless split rows make one long chain of it anyway.  One
// launch / two, us with the host:
//   fp32, k = 32    1 k rows of 4 5.5 / 7.4; 4 k of 16 5.4 / 7.2; 10 k of 10 (not in flight at once) 9.6 / 8.2;
//                   Zipf rows, 176 k nonzeros 10.0 / 13.0; R-MAT scale 14 (228 k) 12.2 / 14.4
//   fp32, k = 64    1 k of 4 5.5 / 7.1; 4 k of 16 (not at once) 8.7 / 7.3; Zipf 14.0 / 14.6; R-MAT 17.4 / 18.5
//   fp32, k = 128   5 k of 4 5.6 / 7.6; R-MAT scale 11 7.2 / 10.8
//   fp64, k = 32    1 k of 4 5.5 / 7.5; R-MAT scale 11 6.4 / 9.2; Zipf 176 k 19.0 / 15.9; R-MAT scale 14 20.7 / 19.7
constexpr long long PAIR_MAX_NNZ = 1 << 18;   // with split rows (half as many without, and with fp64)
template <typename T> bool pair_plan(const SddmmCall& d, const SpmmCall& p, PairShape* s, unsigned* spmm_blocks, int* wn) {
    const long long lda = d.lda * (long long)sizeof(T), ldb = d.ldb * (long long)sizeof(T), ldx = p.ldx * (long long)sizeof(T),
                    ldy = p.ldy * (long long)sizeof(T), bytes = (long long)d.k * sizeof(T);
    const unsigned long long bits = lda | ldb | ldx | ldy | bytes | (uintptr_t)d.A | (uintptr_t)d.B | (uintptr_t)p.X |
                                    (uintptr_t)p.Y | (p.carry ? (uintptr_t)p.carry | (unsigned long long)p.ldc * sizeof(T) : 0);
    if (d.f64 != p.f64 || d.k != p.k || p.k_out != p.k || bits % 16 != 0 || bytes == 0 || bytes > 64 * 16 || lda >= 1ll << 32 ||
        ldb >= 1ll << 32 || ldx >= 1ll << 32 || d.where || d.also || d.pack_a.src || d.pack_b.src || p.pack_x.src ||
        d.nnz <= 0 || p.nrows <= 0 || p.items == nullptr || d.nnz > (p.carry && !d.f64 ? PAIR_MAX_NNZ : PAIR_MAX_NNZ / 2))
        return false;
    *s = pair_shape((int)(bytes / 16), 2ll * p.nrows > 3ll * p.nitems);
    const unsigned all = pair_resident<T>(*s);
    if (all < 2) return false;
    const unsigned items = (unsigned)((p.nitems + 7) / 8), least = (unsigned)((d.nnz + 8 * WINDOW_MAX - 1) / (8 * WINDOW_MAX));
    const unsigned alone = all / pair_min_blocks(s->rs, s->rp, sizeof(T) == 4) * (bytes <= 32 * 16 ? 4 : 3);
    if (items + least > all && items <= alone && !p.carry) return false;
    unsigned half = all > least + all / 2 ? all - least : all / 2;
    *spmm_blocks = items < half ? items : half;
    *wn = window_nnz(d.nnz, (long long)(all - *spmm_blocks) * 8, 32 / s->gs);
    return true;
}

template <typename T> int launch_pair(const SddmmCall& d, const SpmmCall& p, cudaStream_t st, bool* done) {
    PairShape s;
    PairArgs<T> a;
    *done = pair_plan<T>(d, p, &s, &a.spmm_blocks, &a.wn);
    if (!*done) return 0;
    a.nnz = d.nnz;
    a.rowidx = d.ri; a.colidx = d.ci;
    a.arows.base = (const char*)d.A;
    a.arows.ld_bytes = (unsigned)(d.lda * sizeof(T));
    a.B = (const char*)d.B;
    a.ldb_bytes = (unsigned)(d.ldb * sizeof(T));
    a.store = {(T*)d.out, (const T*)d.sv, ((uintptr_t)d.out | (uintptr_t)d.sv) % 16 == 0};
    a.nitems = p.nitems; a.nrows = p.nrows;
    a.items = (const int4*)p.items;
    a.rowptr = p.rowptr; a.ci = p.ci; a.val = (const T*)p.val;
    a.X = (const char*)p.X;
    a.ldx_bytes = (unsigned)(p.ldx * sizeof(T));
    a.emit = {(char*)p.Y, p.ldy * (long long)sizeof(T), (T)p.beta};
    a.lg = {p.first_piece, p.npieces, p.counters, p.carry, p.ldc, p.ticket};
    a.nvec = (int)(d.k * sizeof(T) / 16);
    a.aligned_sddmm = ((uintptr_t)d.ri | (uintptr_t)d.ci) % 16 == 0;
    a.aligned_spmm = ((uintptr_t)p.ci | (uintptr_t)p.val) % 16 == 0;
    const unsigned blocks = a.spmm_blocks + (unsigned)((d.nnz + a.wn * 8ll - 1) / (a.wn * 8ll));
#define SP3_PAIR(A, B, C, D) return launch_early(pair_kernel<T, A, B, C, D>, blocks, 0, st, a)
    SP3_PAIR_SHAPES(SP3_PAIR)
#undef SP3_PAIR
    return (int)cudaErrorInvalidConfiguration;
}

}  // namespace sp3

using namespace sp3;

SP3_API int sp3_cuda_sddmm_call(const void* record, void* stream);
SP3_API int sp3_cuda_spmm_call(const void* record, void* stream);

// The SDDMM, then the SpMM.  independent: neither reads or writes what the other writes.
SP3_API int sp3_cuda_pair_call(const void* sddmm, const void* spmm, int independent, void* stream) {
    const SddmmCall& d = *static_cast<const SddmmCall*>(sddmm);
    const SpmmCall& p = *static_cast<const SpmmCall*>(spmm);
    if (independent) {
        bool done = false;
        const int rc = d.f64 ? launch_pair<double>(d, p, (cudaStream_t)stream, &done)
                             : launch_pair<float>(d, p, (cudaStream_t)stream, &done);
        if (rc != 0 || done) return rc;
    }
    const int rc = sp3_cuda_sddmm_call(sddmm, stream);
    return rc ? rc : sp3_cuda_spmm_call(spmm, stream);
}
// 1 where that is one launch, else 0.
SP3_API int sp3_cuda_pair_fuses(const void* sddmm, const void* spmm, int independent) {
    const SddmmCall& d = *static_cast<const SddmmCall*>(sddmm);
    const SpmmCall& p = *static_cast<const SpmmCall*>(spmm);
    PairShape s;
    unsigned blocks;
    int wn;
    return independent && (d.f64 ? pair_plan<double>(d, p, &s, &blocks, &wn) : pair_plan<float>(d, p, &s, &blocks, &wn));
}
