// mg_group.cuh -- the multigrid-preconditioned CG of mg.cu as one cooperative launch per solve
// (mg_group.cu).
#pragma once

#include "mg.cuh"
#include "mg_setup.h"
#include "pcg_group.cuh"

namespace scdat {

constexpr int kMgGroupThreads = 512;
constexpr int kMgGroupRows = 32;  // rows a thread of the finest level has, at most
constexpr int kMgEllBatch = 14;   // entries of a row whose loads are in flight together
constexpr int kMgEllMax = 42;     // most entries of an operator or restriction row
constexpr int kMgEllTransfer = 8; // entries of a prolongation row (trilinear: 8 at most)

// Rows of a matrix side by side: entry k of row i at k * pad + i, short rows filled with zero
// entries, the width a multiple of kMgEllBatch (prolongations: kMgEllTransfer).
template <typename V>
struct EllDev {
    const V* val;
    const int32_t* col;
    int width;
    int pad;
};

template <typename V>
struct MgGroupLevel {
    int R;
    V omega;
    EllDev<V> A;        // off-diagonal entries
    const V* diag;
    const V* dinv;
    EllDev<V> P, Rt;    // to the next level: rows of P (this level's rows), rows of P^T (the next one's)
    V *b, *xa, *xb, *res, *xo;
};

// The launch's constant part: levels in global memory, the coarsest inverse.
template <typename V>
struct MgGroupPlan {
    const MgGroupLevel<V>* lv = nullptr;  // [levels]
    int levels = 0;
    const V* cinv = nullptr;
    int blocks = 0;  // 0: the hierarchy does not fit
};

// Rearranges CSR rows (R of them, values of type S) into an EllDev's arrays (pad = R).
template <typename S, typename V>
void launch_csr_to_ell(int R, int width, const int32_t* ptr, const int32_t* col, const S* val, V* ell_val,
                       int32_t* ell_col, cudaStream_t st);

// Solves A x = b on level 0 from x (zero_start: from x = 0, which it then need not read): r, z, p, q
// are R-vectors; rr, bb, iter and done (< 0: a barrier wait ran out) in sc.
template <typename V>
cudaError_t launch_mgpcg_group(const MgGroupPlan<V>& mg, const V* b, V* x, V* r, V* z, V* p, V* q, bool zero_start,
                               double rtol, int max_iter, PcgScalars* sc, double* slots, cudaStream_t st);

}  // namespace scdat
