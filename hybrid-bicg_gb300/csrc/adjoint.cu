// Gradient kernels of the adjoint of a shifted family.
//
// For J = sum_j w_j c^T x_j with (A + sigma_j I) x_j = b, and the adjoint
// solutions y_j of (A^T + sigma_j I) y_j = c (lambda_j = w_j y_j):
//   dJ/db        = sum_j lambda_j
//   dJ/dsigma_j  = -lambda_j . x_j
//   dJ/dA[i][k]  = -sum_j lambda_j[i] x_j[k]   (on A's pattern: one value per entry)
// The same kernels serve any upstream gradient: given X and Lambda (lambda_j
// solving (A^T + sigma_j I) lambda_j = g_j), they return the gradients with
// respect to the values, b and the shifts.  The reference has no adjoint; the
// formulas are the standard ones for a linear solve.  Dot products are
// deterministic (fixed per-block partials summed in order).
#include "hbk_device.cuh"

using namespace hbk;

namespace {

constexpr int DOT_GRID = 512;  // partial sums per shift

__global__ void __launch_bounds__(NT) k_entry_rows(unsigned n, const unsigned *__restrict__ ptr, unsigned *rows) {
    for (size_t r = blockIdx.x * (size_t)NT + threadIdx.x; r < n; r += (size_t)gridDim.x * NT)
        for (unsigned e = ptr[r]; e < ptr[r + 1]; ++e) rows[e] = (unsigned)r;
}

// part[j * DOT_GRID + b] = sum over block b's elements of a_j . x_j, where
// a_j = A[j] (a_shared: one vector for all j)
__global__ void __launch_bounds__(NT) k_shift_dots(unsigned n, const double *__restrict__ X, size_t ldx,
                                                   const double *__restrict__ Aa, size_t lda, int a_shared,
                                                   double *part) {
    __shared__ double red[NW];
    const int j = blockIdx.y;
    const double *x = X + (size_t)j * ldx;
    const double *a = Aa + (a_shared ? 0 : (size_t)j * lda);
    double acc = 0.0;
    for (size_t i = blockIdx.x * (size_t)NT + threadIdx.x; i < n; i += (size_t)gridDim.x * NT) acc = fma(a[i], x[i], acc);
    acc = block_sum(acc, red);
    if (threadIdx.x == 0) part[(size_t)j * gridDim.x + blockIdx.x] = acc;
}

// out[j] = scale * w_j * sum_b part[j][b], one warp per shift, in a fixed order
// (one thread per shift: 512 dependent adds of 64 clocks, 42 us; a warp: 5 us)
__global__ void __launch_bounds__(NT) k_sum_parts(int m, int g, const double *__restrict__ part,
                                                  const double *__restrict__ w, double scale, double *out) {
    const int j = blockIdx.x * NW + (threadIdx.x >> 5);
    if (j >= m) return;
    double s = 0.0;
    for (int b = threadIdx.x & 31; b < g; b += 32) s += part[(size_t)j * g + b];
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) out[j] = scale * (w ? w[j] : 1.0) * s;
}

// db[i] = sum_j w_j Y[j][i]
__global__ void __launch_bounds__(NT) k_grad_b(unsigned n, int m, const double *__restrict__ Y, size_t ldy,
                                               const double *__restrict__ w, double *db) {
    for (size_t i = blockIdx.x * (size_t)NT + threadIdx.x; i < n; i += (size_t)gridDim.x * NT) {
        double s = 0.0;
        for (int j = 0; j < m; ++j) s = fma(w ? w[j] : 1.0, Y[(size_t)j * ldy + i], s);
        db[i] = s;
    }
}

// The same as k_grad_val for rows of few entries: one thread per row, up to
// GRAD_E entries at a time in registers.  The sum is bound by the FP64 pipe:
// w_j Y[j][row] is formed once per row and shift instead of once per entry (a
// seven-point stencil: 8 instead of 14 operations per row and shift), Y is
// read once and coalesced, and two shifts have their loads in flight together
// (one or four: 2 % slower; more than two blocks per SM: up to 5 %).  128^3,
// 32 shifts: 2062 -> 1110 us, without the map from entries to rows (47 us);
// floor 740 us (one FMA per entry and shift).  An operation that no lane needs
// costs the pipe as much as any other, so a warp runs the code for the longest
// of its rows (with that for GRAD_E always, 1 M rows and 32 shifts took 785 us
// at one, two or three entries per row; k_grad_val 435, 548, 689).
constexpr int GRAD_E = 8;
struct GradRow {
    unsigned e0, cnt;  // the row's next entries
    size_t row;
    int m;
    const unsigned *__restrict__ col;
    const double *__restrict__ X, *__restrict__ Y, *__restrict__ w;
    size_t ldx, ldy;
    double *__restrict__ dval;
    template <int E>
    __device__ __forceinline__ void part() const {
        unsigned c[E];
        double s[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
            c[e] = (unsigned)e < cnt ? col[e0 + e] : 0u;
            s[e] = 0.0;
        }
        const double *xj = X, *yj = Y + row;
#pragma unroll 2
        for (int j = 0; j < m; ++j, xj += ldx, yj += ldy) {
            const double y = (w ? w[j] : 1.0) * *yj;
#pragma unroll
            for (int e = 0; e < E; ++e)
                if ((unsigned)e < cnt) s[e] = fma(y, xj[c[e]], s[e]);
        }
#pragma unroll
        for (int e = 0; e < E; ++e)
            if ((unsigned)e < cnt) dval[e0 + e] = -s[e];
    }
    // most: of cnt over the warp
    template <int E>
    __device__ __forceinline__ void parts(unsigned most) const {
        if constexpr (E > 1) {
            if (most < E) {
                parts<E - 1>(most);
                return;
            }
        }
        part<E>();
    }
};
__global__ void __launch_bounds__(NT, 2) k_grad_val_rows(unsigned n, const unsigned *__restrict__ ptr,
                                                      const unsigned *__restrict__ col, int m,
                                                      const double *__restrict__ X, size_t ldx,
                                                      const double *__restrict__ Y, size_t ldy,
                                                      const double *__restrict__ w, double *__restrict__ dval) {
    for (size_t i0 = blockIdx.x * (size_t)NT + (threadIdx.x & ~31u); i0 < n; i0 += (size_t)gridDim.x * NT) {
        const size_t i = i0 + (threadIdx.x & 31);
        GradRow g{0u, 0u, i < n ? i : n - 1, m, col, X, Y, w, ldx, ldy, dval};
        if (i < n) g.e0 = ptr[i], g.cnt = ptr[i + 1] - g.e0;
        for (;;) {  // (whole warps)
            const unsigned most = __reduce_max_sync(0xffffffffu, g.cnt);
            if (!most) break;
            g.parts<GRAD_E>(most);
            const unsigned done = g.cnt < GRAD_E ? g.cnt : GRAD_E;
            g.e0 += done, g.cnt -= done;
        }
    }
}

// dval[e] = -sum_j w_j Y[j][row(e)] X[j][col(e)]
__global__ void __launch_bounds__(NT) k_grad_val(unsigned nnz, const unsigned *__restrict__ rows,
                                                 const unsigned *__restrict__ col, int m, const double *__restrict__ X,
                                                 size_t ldx, const double *__restrict__ Y, size_t ldy,
                                                 const double *__restrict__ w, double *dval) {
    for (size_t e = blockIdx.x * (size_t)NT + threadIdx.x; e < nnz; e += (size_t)gridDim.x * NT) {
        const unsigned i = rows[e], k = col[e];
        double s = 0.0;
        for (int j = 0; j < m; ++j)
            s = fma((w ? w[j] : 1.0) * Y[(size_t)j * ldy + i], X[(size_t)j * ldx + k], s);
        dval[e] = -s;
    }
}

}  // namespace

extern "C" {

int hbk_entry_rows(unsigned n, const unsigned *ptr, unsigned *rows, cudaStream_t st) {
    k_entry_rows<<<grid_for(n ? n : 1, 4), NT, 0, st>>>(n, ptr, rows);
    return (int)cudaGetLastError();
}

size_t hbk_adjoint_tmp_bytes(int m) { return sizeof(double) * (size_t)(m > 0 ? m : 1) * DOT_GRID; }

// out[j] = scale * w_j * (a_j . x_j); device pointers; tmp of hbk_adjoint_tmp_bytes(m)
int hbk_shift_dots(unsigned n, int m, const double *X, size_t ldx, const double *a, size_t lda, int a_shared,
                   const double *w, double scale, double *out, void *tmp, cudaStream_t st) {
    if (m <= 0) return 0;
    k_shift_dots<<<dim3(DOT_GRID, m), NT, 0, st>>>(n, X, ldx, a, lda, a_shared, (double *)tmp);
    k_sum_parts<<<(m + NW - 1) / NW, NT, 0, st>>>(m, DOT_GRID, (const double *)tmp, w, scale, out);
    return (int)cudaGetLastError();
}

int hbk_grad_b(unsigned n, int m, const double *Y, size_t ldy, const double *w, double *db, cudaStream_t st) {
    k_grad_b<<<grid_for(n ? n : 1, 2), NT, 0, st>>>(n, m, Y, ldy, w, db);
    return (int)cudaGetLastError();
}

int hbk_grad_val_rows(unsigned n, const unsigned *ptr, const unsigned *col, int m, const double *X, size_t ldx,
                      const double *Y, size_t ldy, const double *w, double *dval, cudaStream_t st) {
    if (!n) return 0;
    k_grad_val_rows<<<wave_grid<k_grad_val_rows>((int)(((size_t)n + NT - 1) / NT)), NT, 0, st>>>(n, ptr, col, m, X, ldx, Y,
                                                                                              ldy, w, dval);
    return (int)cudaGetLastError();
}

int hbk_grad_val(unsigned nnz, const unsigned *rows, const unsigned *col, int m, const double *X, size_t ldx,
                 const double *Y, size_t ldy, const double *w, double *dval, cudaStream_t st) {
    k_grad_val<<<grid_for(nnz ? nnz : 1, 2), NT, 0, st>>>(nnz, rows, col, m, X, ldx, Y, ldy, w, dval);
    return (int)cudaGetLastError();
}

}  // extern "C"
