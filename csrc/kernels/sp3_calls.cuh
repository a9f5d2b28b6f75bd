// Records of the bound calls (see `_BoundCall` in ops/cuda_ops.py): the arguments of one SDDMM or SpMM, which the caller
// keeps between launches.
#pragma once
#include "sp3_kernels.cuh"

namespace sp3 {

// An operand with rows of k values that is copied to rows of whole 16-byte vectors first (see pack_rows_kernel).
struct PackRows {
    const void* src;     // null: nothing to pack
    long long ld;        // elements
    void* dst;
    long long rows;
    int k, nvec;
};

}  // namespace sp3

// Field order: ops/cuda_ops.py.  Converting some twenty arguments costs the Python front end more than a small kernel runs.
struct SddmmCall {
    long long nnz;
    const int *ri, *ci;
    const void *sv, *A;
    long long lda;
    const void* B;
    long long ldb;
    void* out;
    int k, f64;
    // null, or: ri and ci are sorted by chunk of columns, the dot products go to `dots`, and the value of nonzero i (row
    // order) is sv[i] * dots[where[i]]
    const int* where;
    void* dots;
    sp3::PackRows pack_a, pack_b;   // A and B are filled from here first
    void* also;                // null, or a second place for the values (scores that are values of the next kernel)
};
struct SpmmCall {
    int nrows, nitems;
    const void* items;
    const long long* rowptr;
    const int* ci;
    const void *val, *X;
    long long ldx;
    void* Y;
    long long ldy;
    const int *first_piece, *npieces;
    int* counters;
    void* carry;
    long long ldc;
    int* ticket;
    double beta;
    int k, f64;
    int k_out;              // columns of Y (k of X counts the padding of its rows)
    int x_rows;             // rows of X
    sp3::PackRows pack_x;        // X is filled from here first
    long long nnz;
};
