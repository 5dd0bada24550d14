// Host-side pass over a CSR matrix's arrays when a handle takes them in: validity and
// row classes (krylov.cuh's ClassOp).
#pragma once

#include <vector>

namespace cfm {

constexpr int CLS_MAX = 256, CLS_MAXLEN = 32;  // classes of a matrix, entries of a row

struct RowClasses {
    int kind = 0;                    // 0 none, 1 rows alike in their column offsets, 2 in their values too
    std::vector<unsigned char> cls;  // class of each row
    std::vector<int> reps;           // first row of each class, ascending
};

// Classes of the rows of a matrix with 0-based rowptr (col in either base): by offsets
// and values where those are at most CLS_MAX, else by offsets, else none; none as well
// when a row is longer than CLS_MAXLEN.  At most `threads` host threads (0: OpenMP's
// number); the result does not depend on it.
RowClasses find_row_classes(int n, const int *rowptr, const int *col, const double *val, int threads = 0);

// What is wrong with the arrays of a caller's matrix, or nullptr.
const char *csr_fault(int n, long long nnz, const int *rowptr, const int *col, int base);

// dst[i] = src[i] - base
void rebase(const int *src, long long count, int base, int *dst);

}  // namespace cfm
