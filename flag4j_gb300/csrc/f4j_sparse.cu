// f4j_sparse.cu -- CSR products and sparse structure on sm_103a.
//
// Products follow the reference loops' per-element order exactly (storage
// order over a row's nonzeros, product and sum rounded separately), so the
// results are bit-identical to Flag4j:
//   SpMV  RealCsrDenseMatMult.standardVector
//         (src/main/java/org/flag4j/linalg/ops/dense_sparse/csr/real/RealCsrDenseMatMult.java:172-192)
//   SpMM  RealCsrDenseMatMult.standard (same file :55-82)
//   S^T X RealCsrOps.transpose + standard (…/sparse/csr/real/RealCsrOps.java:195-225)
//   S1 S2 RealCsrMatMult, RealComplexCsrMatMult, SemiringCsrMatMult (CSR x CSR)
// SpMV / SpMM also have an opt-in FMA mode (fused multiply-add in storage
// order, within 2 k u |S||X|); SDDMM (the sparse adjoint's dS) has no
// reference counterpart and meets the same bound.
// Structure (COO->CSR, stable COO sort, transpose permutation) is integer
// work done with histograms, scans, a row-bucketed sort and a stable LSD
// radix sort.
#include <vector>

#include "f4j_internal.cuh"
#include "f4j_ptx.cuh"

namespace {

// ------------------------------------------------------------------ SpMV
// Load-balanced lanes.  A warp owns rpw consecutive rows [w0, w1) with
// nonzeros [E0, E1).  Lane l owns the rows whose first nonzero lies in
// [E0 + ceil(l * span / 32), E0 + ceil((l + 1) * span / 32)), span = E1 - E0:
// consecutive rows holding about span / 32 nonzeros, found by a lower-bound
// search on the row pointers.  Rows of different lengths therefore share the
// warp's work evenly (a lane per row made every warp wait for its longest
// row: about 1.75 add steps per nonzero at Poisson(16) lengths).  Each lane
// walks its contiguous nonzeros 8 at a time, from a multiple of 8: column
// indices and values with 32-byte loads, one L2 sector each (VEC; a group's
// loads stay inside the arrays, entries outside the lane's range are loaded
// and ignored; two 16-byte loads per sector reached L2 about twice), the 8
// gathers of x in flight together, then the products and the running sum in
// storage order,
// storing y at each row end.  Each product and each sum is rounded as
// RealCsrDenseMatMult.standardVector rounds them (acc starts at +0.0), so y is
// bit-identical.  GB300's FP64 pipe (2 lane-operations per clock per SM, two
// per nonzero) bounds the exact mode; the random 8-byte gathers of x (one L2
// sector each) come next.  Gathering the next group's x under the current
// group's sums (two groups in registers, 2 to 4 blocks per SM) was slower, 147
// to 237 us against 116 at 2^20 rows x 16: the warps lost hide more.  No shared memory, so L1 keeps its full size for
// the gathers.
// FUSED (the opt-in FMA mode) accumulates fma(v, x, acc) in the same order,
// one FP64 instruction per nonzero, within the reference's componentwise bound.
constexpr int SPMV_RPW_MAX = 256;  // rows per warp for large matrices
constexpr int SPMV_BLOCK = 256;

// Blocks per SM: 4 (64 registers) in both modes; 5 (48) spill.  Exact mode at
// 2^20 rows x 16, us: separate multiplies and adds at 5 blocks 118-119, FMA
// forms (ExactOps) at 5 blocks 120-122, at 4 blocks 115-116.
constexpr int SPMV_BLOCKS = 4;

// 32-byte read-only loads (one sector): 8 column indices, 4 values.  The
// address must be 32-byte aligned.
__device__ __forceinline__ void ld_nc_v8_b32(const int* p, int (&c)[8]) {
    asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]), "=r"(c[4]), "=r"(c[5]), "=r"(c[6]), "=r"(c[7])
                 : "l"(p));
}
__device__ __forceinline__ void ld_nc_v4_f64(const double* p, double& a, double& b, double& c, double& d) {
    asm volatile("ld.global.nc.v4.f64 {%0,%1,%2,%3}, [%4];" : "=d"(a), "=d"(b), "=d"(c), "=d"(d) : "l"(p));
}

template <bool FUSED, bool VEC>
__global__ void __launch_bounds__(SPMV_BLOCK, SPMV_BLOCKS)
    k_spmv(int64_t rows, int64_t nnz, int rpw, const int* __restrict__ rowptr, const int* __restrict__ colidx,
           const double* __restrict__ vals, const double* __restrict__ x, double* __restrict__ y) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * SPMV_BLOCK + threadIdx.x) >> 5;
    const int64_t w0 = warp * rpw;
    if (w0 >= rows) return;
    const int64_t w1 = w0 + rpw < rows ? w0 + rpw : rows;
    const int64_t E0 = __ldg(rowptr + w0), span = (int64_t)__ldg(rowptr + w1) - E0;
    // first row whose first nonzero is at or after this lane's target
    const int64_t target = E0 + (span * lane + 31) / 32;
    int64_t lo = w0, hi = w1;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if ((int64_t)__ldg(rowptr + mid) >= target) hi = mid;
        else lo = mid + 1;
    }
    const int64_t a = lo;
    int64_t b = __shfl_down_sync(0xffffffffu, a, 1);
    if (lane == 31) b = w1;
    if (a >= b) return;
    const int qs = __ldg(rowptr + a), qe = __ldg(rowptr + b);
    // rend: end of row r; rnext: end of row r + 1, loaded one row ahead so that
    // a row end never waits for a load on the running sum's chain
    int64_t r = a;
    int rend = __ldg(rowptr + a + 1);
    int rnext = a + 1 < b ? __ldg(rowptr + a + 2) : qe;
    const ExactOps ops;
    double acc = 0.0;
    while (rend == qs) {  // empty rows before the lane's first nonzero
        y[r] = 0.0;
        if (++r == b) return;
        rend = rnext;
        rnext = r + 1 < b ? __ldg(rowptr + r + 2) : qe;
    }
    for (int qb = VEC ? (qs & ~7) : qs; qb < qe; qb += 8) {
        int c[8];
        double v[8];
        if (VEC && (int64_t)qb + 8 <= nnz) {
            // qb is a multiple of 8: one 32-byte sector of indices, two of values
            ld_nc_v8_b32(colidx + qb, c);
            ld_nc_v4_f64(vals + qb, v[0], v[1], v[2], v[3]);
            ld_nc_v4_f64(vals + qb + 4, v[4], v[5], v[6], v[7]);
        } else {
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const bool ok = qb + u < qe;
                c[u] = ok ? __ldg(colidx + qb + u) : 0;
                v[u] = ok ? __ldg(vals + qb + u) : 0.0;
            }
        }
        double xv[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int q = qb + u;
            xv[u] = (q >= qs && q < qe) ? __ldg(x + c[u]) : 0.0;
        }
        if (!FUSED) {
#pragma unroll
            for (int u = 0; u < 8; u++) v[u] = ops.mul(v[u], xv[u]);
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int q = qb + u;
            if (q < qs || q >= qe) continue;
            acc = FUSED ? __fma_rn(v[u], xv[u], acc) : ops.add(v[u], acc);
            while (q + 1 == rend) {  // row r ends here (and any empty rows after it)
                y[r] = acc;
                acc = 0.0;
                if (++r == b) break;
                rend = rnext;
                rnext = r + 1 < b ? __ldg(rowptr + r + 2) : qe;
            }
        }
    }
}

// ------------------------------------------------------------------ SpMM
// A group of G lanes owns one row; each lane owns a column, or two adjacent ones
// (VEC2: 128-bit loads of X rows), and sums over the row's nonzeros in storage
// order.  G need not divide a warp (launch_spmm).
// For S^T products the same kernel reads values through the transpose
// permutation and row indices from the cached S^T structure.
// FUSED (the opt-in FMA mode): one fma(v, x, acc) per nonzero and column, in
// storage order; within the reference's componentwise bound.  Its FP64 work
// is half the exact mode's, so the X gathers' latency decides its speed: it
// runs 8 blocks per SM (32 registers) to keep more of them in flight; the
// exact mode runs 6 (40 registers), its best balance of loads in flight per
// warp against warps.  Exact mode at 2^20 rows x 16 nonzeros, 32 columns: 1.79
// ms, 95 % of the FP64 pipe's two lanes per SM and clock (2.07 ms with DMUL
// and DADD for ExactOps); 64 columns 3.54 ms (4.02).
// MIXED (exact mode, rows of different lengths in a warp): a group of eight
// nonzeros that is not whole in every row still running goes under predicates, its
// sums in pairs that the warp leaves together, so a warp takes its longest row's
// FP64 instructions, where whole groups and a loop over the rest took the most of
// both: 2^20 rows x 16, us, 2 columns 228 / 181, 8 819 / 594, 16 1326 / 1069.  Groups
// whole in all of them go without predicates, which is what long rows take: 80 % of
// 4.2 M nonzeros in 1024 rows, 8 columns 694 with predicates throughout, 613 so.  5
// blocks an SM (48 registers; 6 spill, 2 % slower).  With one row a warp the
// predicated rest costs more than the loop (32 columns 1792 / 2225, without the pairs).
template <bool VEC2, bool PERM, bool FUSED = false, bool MIXED = false>
__global__ void __launch_bounds__(256, FUSED ? 8 : (MIXED ? 5 : 6))
    k_spmm(int64_t rows, int64_t ncols, int G, const int* __restrict__ rowptr, const int* __restrict__ colidx,
           const double* __restrict__ vals, const int* __restrict__ perm, const double* __restrict__ X,
           double* __restrict__ Y) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, row = t / G;
    const int lane = (int)(t - row * G);
    if (row >= rows) return;
    const ExactOps ops;
    const int q0 = rowptr[row], q1 = rowptr[row + 1];
    constexpr int W = VEC2 ? 2 : 1;
    for (int64_t cbase = (int64_t)lane * W; cbase < ncols; cbase += (int64_t)G * W) {
        double a0 = 0.0, a1 = 0.0;
        int q = q0;
        constexpr int UN = 8;  // nonzeros whose X rows are in flight together
        if constexpr (MIXED) {
            for (; q < q1; q += UN) {
                double v[UN], xv[UN];
                if (__all_sync(__activemask(), q + UN <= q1)) {
#pragma unroll
                    for (int u = 0; u < UN; u++) {
                        v[u] = PERM ? __ldg(&vals[__ldg(&perm[q + u])]) : __ldg(&vals[q + u]);
                        xv[u] = __ldg(X + (int64_t)__ldg(&colidx[q + u]) * ncols + cbase);
                    }
#pragma unroll
                    for (int u = 0; u < UN; u++) a0 = ops.add(ops.mul(v[u], xv[u]), a0);
                    continue;
                }
#pragma unroll
                for (int u = 0; u < UN; u++) {
                    v[u] = xv[u] = 0.0;
                    if (q + u < q1) {
                        v[u] = PERM ? __ldg(&vals[__ldg(&perm[q + u])]) : __ldg(&vals[q + u]);
                        xv[u] = __ldg(X + (int64_t)__ldg(&colidx[q + u]) * ncols + cbase);
                    }
                }
#pragma unroll
                for (int u = 0; u < UN; u += 2) {
                    if (q + u >= q1) break;
                    a0 = ops.add(ops.mul(v[u], xv[u]), a0);
                    if (q + u + 1 < q1) a0 = ops.add(ops.mul(v[u + 1], xv[u + 1]), a0);
                }
            }
            Y[row * ncols + cbase] = a0;
            continue;
        }
        for (; q + UN <= q1; q += UN) {
            int c[UN];
            double v[UN];
#pragma unroll
            for (int u = 0; u < UN; u++) {
                c[u] = __ldg(&colidx[q + u]);
                v[u] = PERM ? __ldg(&vals[__ldg(&perm[q + u])]) : __ldg(&vals[q + u]);
            }
            if (VEC2) {
                double2 xv[UN];
#pragma unroll
                for (int u = 0; u < UN; u++) xv[u] = __ldg(reinterpret_cast<const double2*>(X + (int64_t)c[u] * ncols + cbase));
#pragma unroll
                for (int u = 0; u < UN; u++) {
                    if (FUSED) {
                        a0 = __fma_rn(v[u], xv[u].x, a0);
                        a1 = __fma_rn(v[u], xv[u].y, a1);
                    } else {
                        a0 = ops.add(ops.mul(v[u], xv[u].x), a0);
                        a1 = ops.add(ops.mul(v[u], xv[u].y), a1);
                    }
                }
            } else {
                double xv[UN];
#pragma unroll
                for (int u = 0; u < UN; u++) xv[u] = __ldg(X + (int64_t)c[u] * ncols + cbase);
#pragma unroll
                for (int u = 0; u < UN; u++) a0 = FUSED ? __fma_rn(v[u], xv[u], a0) : ops.add(ops.mul(v[u], xv[u]), a0);
            }
        }
        for (; q < q1; q++) {
            const int c = __ldg(&colidx[q]);
            const double v = PERM ? __ldg(&vals[__ldg(&perm[q])]) : __ldg(&vals[q]);
            if (VEC2) {
                const double2 xv = __ldg(reinterpret_cast<const double2*>(X + (int64_t)c * ncols + cbase));
                a0 = FUSED ? __fma_rn(v, xv.x, a0) : ops.add(ops.mul(v, xv.x), a0);
                a1 = FUSED ? __fma_rn(v, xv.y, a1) : ops.add(ops.mul(v, xv.y), a1);
            } else {
                const double xe = __ldg(X + (int64_t)c * ncols + cbase);
                a0 = FUSED ? __fma_rn(v, xe, a0) : ops.add(ops.mul(v, xe), a0);
            }
        }
        if (VEC2) *reinterpret_cast<double2*>(Y + row * ncols + cbase) = make_double2(a0, a1);
        else Y[row * ncols + cbase] = a0;
    }
}

// Complex CSR x complex dense (CsrCMatrix.mult(CMatrix) ->
// DenseCsrSemiringMatMult.standard, src/main/java/org/flag4j/linalg/ops/
// dense_sparse/csr/semiring_ops/DenseCsrSemiringMatMult.java:59-98): a group
// of G lanes owns one row, a lane one complex column; per nonzero in storage
// order y += x * v with Complex128.mult's rounding (Complex128.java:336-341):
// pr = xr*vr - xi*vi, pi = xr*vi + xi*vr, each product and sum rounded.
__global__ void __launch_bounds__(256)
    k_zspmm(int64_t rows, int64_t ncols, int G, const int* __restrict__ rowptr, const int* __restrict__ colidx,
            const double2* __restrict__ vals, const double2* __restrict__ X, double2* __restrict__ Y) {
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
    const int lane = threadIdx.x % G;
    if (row >= rows) return;
    const ExactOps ops;
    const int q0 = rowptr[row], q1 = rowptr[row + 1];
    for (int64_t c0 = lane; c0 < ncols; c0 += G) {
        double ar = 0.0, ai = 0.0;
        int q = q0;
        constexpr int UN = 8;  // nonzeros whose X entries are in flight together
        for (; q + UN <= q1; q += UN) {
            double2 v[UN], x[UN];
#pragma unroll
            for (int u = 0; u < UN; u++) {
                v[u] = __ldg(&vals[q + u]);
                x[u] = __ldg(&X[(int64_t)__ldg(&colidx[q + u]) * ncols + c0]);
            }
#pragma unroll
            for (int u = 0; u < UN; u++) {
                const double pr = ops.sub(ops.mul(x[u].x, v[u].x), ops.mul(x[u].y, v[u].y));
                const double pi = ops.add(ops.mul(x[u].x, v[u].y), ops.mul(x[u].y, v[u].x));
                ar = ops.add(pr, ar);
                ai = ops.add(pi, ai);
            }
        }
        for (; q < q1; q++) {
            const double2 v = __ldg(&vals[q]);
            const double2 x = __ldg(&X[(int64_t)__ldg(&colidx[q]) * ncols + c0]);
            const double pr = ops.sub(ops.mul(x.x, v.x), ops.mul(x.y, v.y));
            const double pi = ops.add(ops.mul(x.x, v.y), ops.mul(x.y, v.x));
            ar = ops.add(pr, ar);
            ai = ops.add(pi, ai);
        }
        Y[row * ncols + c0] = make_double2(ar, ai);
    }
}

// ------------------------------------------------------------------ SDDMM
// Warp per row of S; half-warps take alternate nonzeros; a lane owns 4
// columns of each 64-column pass (sequential), then a 16-lane tree sum.
__global__ void __launch_bounds__(256)
    k_sddmm(int64_t rows, int64_t ncols, const int* __restrict__ rowptr, const int* __restrict__ colidx,
            const double* __restrict__ A, const double* __restrict__ B, double* __restrict__ out) {
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const int lane = threadIdx.x % 32, half = lane / 16, l16 = lane % 16;
    if (row >= rows) return;
    const int q0 = rowptr[row], q1 = rowptr[row + 1];
    const double* arow = A + row * ncols;
    for (int qb = q0; qb < q1; qb += 2) {
        const int q = qb + half;
        double s = 0.0;
        if (q < q1) {
            const double* brow = B + (int64_t)__ldg(&colidx[q]) * ncols;
            for (int64_t c0 = 0; c0 < ncols; c0 += 64) {
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int64_t c = c0 + l16 * 4 + u;
                    if (c < ncols) s = fma(__ldg(&arow[c]), __ldg(&brow[c]), s);
                }
            }
        }
        for (int off = 8; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (q < q1 && l16 == 0) out[q] = s;
    }
}

// SDDMM of up to 64 columns of rows ld entries apart (add: on top of the columns
// before), flat over the nonzeros: a warp takes SD_WARP consecutive nonzeros, eight at a time, a group of 4 lanes one nonzero.  A unit
// is a 16-byte pair of columns (PAIRS: an even number of columns, aligned
// operands) or one column; lane l4 of a group owns the units l4, l4 + 4, ..., at
// most U of them, so the group's four lanes read 64 (32) contiguous bytes a
// step.  The FP64 pipe bounds it: with 64 columns 16 FMAs a nonzero and lane and
// three adds for four nonzeros (their sums are exchanged so that each lane ends
// up with one; two adds each take 72 instructions for these 67).  What keeps the
// pipe fed: a unit of the next nonzero's row of B is loaded as soon as the current
// one has been used, its indices a step earlier, and nothing waits for a barrier.
// The rows of A come through L1 (rowidx is sorted: neighbouring groups read the
// same row; B does not allocate there).  Narrower rows add up in
// two sums a lane, from 33 columns in four: no larger an error than k_sddmm's 16
// sums (rms over 10^6 entries, 16, 32 and
// 48 columns: 3.93, 3.26 and 2.77e-17 for 4.09, 3.26 and 2.84e-17 of sum |a||b|).
// rowidx: the row of each nonzero, the first one's in rowidx[0].  A view of a larger
// pattern has rowptr[0] > 0, and its column indices and results stand from there;
// rows that hold fewer than nnz nonzeros leave the rest of out alone.
// Measured: 64 columns, 2^18 rows x 16, 0.50 ms at 3 or 4 blocks an SM, 0.55 at 2,
// 0.56 with A staged in shared memory by blocks of 64 nonzeros.  k_sddmm / this, us,
// 2^20 rows x 16: 1 column 4129 / 288, 4 3966 / 346, 8 3968 / 544, 16 3968 / 702, 32
// 3966 / 1135, 33 3966 / 2309, 48 3965 / 1861, 63 3966 / 2453, 66 5971 / 2810, 96 5761 /
// 3756, 128 5760 / 4925; 2^17 rows: 193 1256 / 1089, 200 1205 / 981, 256 1203 / 1255,
// 512 2116 / 2564: past SD_FLAT_COLS its parts' indexes and sums cost more than
// k_sddmm's tree.
constexpr int SD_WARP = 64, SD_FLAT_COLS = 200;
__device__ __forceinline__ double2 ld_nc_stream(const double2* p) {
    double2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ double ld_nc_stream(const double* p) {
    double v;
    asm volatile("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
// The nonzeros w0 .. w0 + SD_WARP - 1 of a view (see k_sddmm_flat), a warp on one at
// a time.
__device__ __noinline__ void sddmm_view(int64_t w0, int first, int held, int ncols, int64_t ld, bool add,
                                        const int* rowidx, const int* colidx, const double* A, const double* B,
                                        double* out) {
    for (int64_t i = w0; i < held && i < w0 + SD_WARP; i++) {
        const double *a = A + rowidx[i] * ld, *b = B + colidx[first + i] * ld;
        double s = 0.0;
        for (int c = threadIdx.x % 32; c < ncols; c += 32) s = fma(a[c], b[c], s);
        for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (threadIdx.x % 32 == 0) out[first + i] = add ? out[first + i] + s : s;
    }
}
template <int U, bool PAIRS>
__global__ void __launch_bounds__(256, 4)
    k_sddmm_flat(int64_t rows, int64_t nnz0, int ncols, int64_t ld, bool add, const int* __restrict__ rowptr,
                 const int* __restrict__ rowidx, const int* __restrict__ colidx, const double* __restrict__ A,
                 const double* __restrict__ B, double* __restrict__ out) {
    using V = typename std::conditional<PAIRS, double2, double>::type;
    constexpr bool WHOLE = PAIRS && U == 8;  // 64 columns, no unit left over (the launch sees to it)
    constexpr int SUMS = WHOLE || (!PAIRS && U == 1) ? 1 : (U > (PAIRS ? 4 : 8) ? 4 : 2);
    const int lane = threadIdx.x % 32, g = lane >> 2, l4 = lane & 3;
    const int units = WHOLE ? 32 : (PAIRS ? ncols / 2 : ncols);
    // 16 units a lane are short of registers: with 32-bit indices, or the view's
    // offsets in the loop, 63 columns take 2.6 to 2.8 ms for 2.4
    using Q = typename std::conditional<U == 16, int64_t, unsigned>::type;
    Q nnz = (Q)nnz0;  // below 2^31
    const Q w0 = ((Q)blockIdx.x * 8 + threadIdx.x / 32) * SD_WARP;
    if (w0 >= nnz) return;
    const int first = __ldg(rowptr);
    const Q held = (Q)(__ldg(rowptr + rows) - first);
    if constexpr (U == 16) {
        if (first != 0 || held != nnz) {
            sddmm_view(w0, first, (int)(held < nnz ? held : nnz), ncols, ld, add, rowidx, colidx, A, B, out);
            return;
        }
    } else {
        if (held < nnz) nnz = held;
        if (w0 >= nnz) return;
        colidx += first;
        out += first;
    }
    auto at = [&](int step) {  // past the end: the last nonzero again, not stored
        const Q q = w0 + step * 8 + g;
        return q < nnz ? q : nnz - 1;
    };
    auto row_of = [&](const double* X, int64_t i) {
        return reinterpret_cast<const V*>(X + i * ld) + l4;
    };
    auto mine = [&](int u) { return WHOLE || 4 * u + l4 < units; };
    const V* arow = row_of(A, __ldg(rowidx + at(0)));
    const V* brow = row_of(B, __ldg(colidx + at(0)));
    int rn = __ldg(rowidx + at(1)), cn = __ldg(colidx + at(1));
    V b[U];
#pragma unroll
    for (int u = 0; u < U; u++) b[u] = mine(u) ? ld_nc_stream(brow + 4 * u) : V{};
#pragma unroll 1
    for (int s0 = 0; s0 < SD_WARP / 8; s0 += 4) {
        double p[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int step = s0 + j;
            const V* an = row_of(A, rn);
            brow = row_of(B, cn);
            if (step + 2 < SD_WARP / 8) {
                rn = __ldg(rowidx + at(step + 2));
                cn = __ldg(colidx + at(step + 2));
            }
            double s[SUMS] = {};
#pragma unroll
            for (int u = 0; u < U; u++) {
                const V a = mine(u) ? __ldg(arow + 4 * u) : V{};
                if constexpr (PAIRS) {
                    double &x = s[2 * u % SUMS], &y = s[(2 * u + 1) % SUMS];
                    x = fma(a.x, b[u].x, x);
                    y = fma(a.y, b[u].y, y);
                } else {
                    double& x = s[u % SUMS];
                    x = fma(a, b[u], x);
                }
                if (step + 1 < SD_WARP / 8 && mine(u)) b[u] = ld_nc_stream(brow + 4 * u);
            }
            p[j] = s[0];
            if constexpr (SUMS == 2) p[j] = s[0] + s[1];
            if constexpr (SUMS == 4) p[j] = (s[0] + s[1]) + (s[2] + s[3]);
            arow = an;
        }
        // four sums of four lanes: lane l4 ends with the nonzero of step s0 + l4
        const bool h2 = l4 & 2, h1 = l4 & 1;
        const double u0 = __shfl_xor_sync(0xffffffffu, h2 ? p[0] : p[2], 2);
        const double u1 = __shfl_xor_sync(0xffffffffu, h2 ? p[1] : p[3], 2);
        const double t0 = (h2 ? p[2] : p[0]) + u0, t1 = (h2 ? p[3] : p[1]) + u1;
        const double r = (h1 ? t1 : t0) + __shfl_xor_sync(0xffffffffu, h1 ? t0 : t1, 1);
        const Q q = w0 + (s0 + l4) * 8 + g;
        if (q < nnz) out[q] = add ? out[q] + r : r;
    }
}

// ------------------------------------------------------------------ structure
__global__ void k_count(int64_t n, const int* __restrict__ idx, int* __restrict__ counts_plus1) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        atomicAdd(&counts_plus1[idx[i] + 1], 1);
}

// COO -> CSR row count with the row range check of SparseValidation.validateCoo:
// one count per in-range row index in counts_plus1[r + 1], and the first
// position of an out-of-range one in *first_bad.  A thread takes eight
// consecutive entries and adds each run of equal rows at once (COO input is
// usually row-sorted); neighbouring threads whose eight are all of one row add
// together, or the threads of a row of millions would queue at one counter.  16.8 M
// entries, us, one entry a lane with equal rows matched across the warp / eight a
// thread / this: 16 a row 71 / 16 / 19, all in one row 334 / 1313 / 48.  VEC: 16-byte
// loads.
template <bool VEC>
__global__ void k_count_rows_checked(int64_t n, const int* __restrict__ idx, int64_t limit,
                                     int* __restrict__ counts_plus1, int* __restrict__ first_bad) {
    const int lane = threadIdx.x & 31;
    const int64_t i0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
    const int m = n - i0 < 8 ? (n > i0 ? (int)(n - i0) : 0) : 8;
    int v[8];
    if (VEC && m == 8) {
        const int4 a = reinterpret_cast<const int4*>(idx + i0)[0], b = reinterpret_cast<const int4*>(idx + i0)[1];
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    } else {
#pragma unroll
        for (int u = 0; u < 8; u++) v[u] = u < m ? idx[i0 + u] : -1;
    }
    bool whole = m > 0 && v[0] >= 0 && v[0] < limit;  // one row
#pragma unroll
    for (int u = 1; u < 8; u++) whole = whole && (u >= m || v[u] == v[0]);
    const int before = __shfl_up_sync(0xffffffffu, whole ? v[0] : -1, 1);
    const bool joins = whole && lane > 0 && before == v[0];
    const unsigned later = __ballot_sync(0xffffffffu, !joins) & ~((2u << lane) - 1u);
    const int end = later ? __ffs((int)later) - 1 : 32;  // the lanes from this one on that join it end here
    const int last = __shfl_sync(0xffffffffu, m, end - 1);
    if (whole) {
        if (!joins) atomicAdd(&counts_plus1[v[0] + 1], 8 * (end - 1 - lane) + last);
        return;
    }
    int run = 0;
#pragma unroll
    for (int u = 0; u < 8; u++) {
        if (u >= m) break;
        if (v[u] < 0 || v[u] >= limit) {
            atomicMin(first_bad, (int)(i0 + u));
            continue;
        }
        run++;
        if (u + 1 >= m || v[u + 1] != v[u]) {
            atomicAdd(&counts_plus1[v[u] + 1], run);
            run = 0;
        }
    }
}

// Copy of COO column indices into the CSR with the column range check:
// the first offending position in *first_bad.  VEC: 16-byte loads and stores.
template <bool VEC>
__global__ void k_copy_cols_checked(int64_t n, const int* __restrict__ src, int64_t limit, int* __restrict__ dst,
                                    int* __restrict__ first_bad) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    int64_t done = 0;
    if (VEC) {
        const int64_t n4 = n / 4;
        for (int64_t j = t; j < n4; j += stride) {
            const int4 v = reinterpret_cast<const int4*>(src)[j];
            const int e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (e[q] < 0 || e[q] >= limit) atomicMin(first_bad, (int)(4 * j + q));
            reinterpret_cast<int4*>(dst)[j] = v;
        }
        done = 4 * n4;
    }
    for (int64_t i = done + t; i < n; i += stride) {
        const int v = src[i];
        if (v < 0 || v >= limit) atomicMin(first_bad, (int)i);
        dst[i] = v;
    }
}

// SparseValidation.validateCsr checks (src/main/java/org/flag4j/arrays/sparse/SparseValidation.java:151-206):
// first row with negative start or decreasing pointers, first bad column.
__global__ void k_validate_csr(int64_t rows, int64_t cols, int64_t nnz, const int* __restrict__ rowptr,
                               const int* __restrict__ colidx, int* __restrict__ bad_row,
                               int* __restrict__ bad_col) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += (int64_t)gridDim.x * blockDim.x) {
        int s = rowptr[i], e = rowptr[i + 1];
        if (s < 0 || s > e) {
            atomicMin(bad_row, (int)i);
            continue;
        }
        for (int q = s; q < e && q < nnz; q++) {
            int c = colidx[q];
            if (c < 0 || c >= cols) {
                atomicMin(bad_col, q);
                break;
            }
        }
    }
}

// Row of each of the nnz nonzeros, the first one's in rowidx[0] (rowptr[0] may be
// above 0).  A warp covers 32 consecutive rows: their nonzeros are written in order, each lane finding its row among the 32 by bisection over
// the lanes (a warp per row left half its lanes idle at 16 nonzeros a row and
// started 2^20 warps: 93 us for 16.8 M nonzeros).
__global__ void k_expand_rows(int64_t rows, int64_t nnz, const int* __restrict__ rowptr, int* __restrict__ rowidx) {
    const int64_t w0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32) * 32;
    const int lane = threadIdx.x % 32;
    if (w0 >= rows) return;
    const int64_t r = w0 + lane;
    const int end = __ldg(rowptr + (r < rows ? r + 1 : rows));  // rows past the last end where it ends
    const int first = __ldg(rowptr), q1 = __shfl_sync(0xffffffffu, end, 31);
    for (int base = __ldg(rowptr + w0); base < q1; base += 32) {
        const int q = base + lane;
        int lo = 0;  // first row of the 32 that ends after q
#pragma unroll
        for (int step = 16; step; step >>= 1) {
            const int e = __shfl_sync(0xffffffffu, end, lo + step - 1);
            if (e <= q) lo += step;
        }
        if (q < q1 && q - first < nnz) rowidx[q - first] = (int)(w0 + lo);
    }
}

__global__ void k_iota(int64_t n, int* __restrict__ v) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        v[i] = (int)i;
}

// keys[i] = src[perm ? perm[i] : i], with the sign bit flipped when `flip`
// (so unsigned order is signed int order)
__global__ void k_flip_copy(int64_t n, const int* __restrict__ perm, const int* __restrict__ src, bool flip,
                            unsigned* __restrict__ keys) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) keys[i] = (unsigned)src[perm ? perm[i] : i] ^ (flip ? 0x80000000u : 0u);
}

// perm and dst pass through once and are marked so, which leaves L2 to src.
template <typename T>
__global__ void k_gather(int64_t n, const int* __restrict__ perm, const T* __restrict__ src, T* __restrict__ dst) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        __stcs(dst + i, __ldg(src + __ldcs(perm + i)));
}

// ---------------- inclusive scan (int32), 1024 threads x 4 items per block
constexpr int SCAN_T = 1024, SCAN_IPT = 4, SCAN_TILE = SCAN_T * SCAN_IPT;

__device__ __forceinline__ int block_scan_incl(int v, int* sh) {
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    for (int off = 1; off < 32; off <<= 1) {
        int o = __shfl_up_sync(0xffffffffu, v, off);
        if (lane >= off) v += o;
    }
    if (lane == 31) sh[warp] = v;
    __syncthreads();
    if (warp == 0) {
        int w = sh[lane];
        for (int off = 1; off < 32; off <<= 1) {
            int o = __shfl_up_sync(0xffffffffu, w, off);
            if (lane >= off) w += o;
        }
        sh[lane] = w;
    }
    __syncthreads();
    if (warp > 0) v += sh[warp - 1];
    __syncthreads();
    return v;
}

__global__ void __launch_bounds__(SCAN_T) k_scan_tiles(int64_t n, int* __restrict__ data, int* __restrict__ sums) {
    __shared__ int sh[32];
    const int64_t base = (int64_t)blockIdx.x * SCAN_TILE + (int64_t)threadIdx.x * SCAN_IPT;
    int v[SCAN_IPT];
    int t = 0;
#pragma unroll
    for (int i = 0; i < SCAN_IPT; i++) {
        v[i] = (base + i < n) ? data[base + i] : 0;
        t += v[i];
    }
    int incl = block_scan_incl(t, sh);
    int run = incl - t;
#pragma unroll
    for (int i = 0; i < SCAN_IPT; i++) {
        run += v[i];
        if (base + i < n) data[base + i] = run;
    }
    if (threadIdx.x == SCAN_T - 1) sums[blockIdx.x] = incl;
}

__global__ void k_scan_add(int64_t n, int* __restrict__ data, const int* __restrict__ sums) {
    if (blockIdx.x == 0) return;
    const int add = sums[blockIdx.x - 1];
    const int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
    constexpr int U = 8;  // in flight a thread: one at a time, 2^20 entries took 11.5 us for 4.2
    for (int i = threadIdx.x; i < SCAN_TILE; i += U * blockDim.x) {
        int v[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int64_t at = base + i + u * (int)blockDim.x;
            v[u] = i + u * (int)blockDim.x < SCAN_TILE && at < n ? data[at] : 0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int64_t at = base + i + u * (int)blockDim.x;
            if (i + u * (int)blockDim.x < SCAN_TILE && at < n) data[at] = v[u] + add;
        }
    }
}

// ---------------- stable LSD radix sort of (key, value) pairs, 8-bit digits
constexpr int RS_T = 256, RS_SUB = 16, RS_TILE = RS_T * RS_SUB;  // 4096 items per block

__global__ void __launch_bounds__(RS_T) k_radix_hist(int64_t n, const unsigned* __restrict__ keys, int shift,
                                                     int* __restrict__ hist, int nblocks) {
    __shared__ int h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * RS_TILE;
    for (int i = threadIdx.x; i < RS_TILE; i += RS_T)
        if (base + i < n) atomicAdd(&h[(keys[base + i] >> shift) & 255], 1);
    __syncthreads();
    hist[(int64_t)threadIdx.x * nblocks + blockIdx.x] = h[threadIdx.x];
}

// hist holds inclusive scan over [digit][block]; block b's start for digit d
// is incl[d*nb + b] - count.  Items are ranked stably: sub-tile order, then
// warp order, then lane order.
__global__ void __launch_bounds__(RS_T) k_radix_scatter(int64_t n, const unsigned* __restrict__ keys_in,
                                                        const int* __restrict__ vals_in, int shift,
                                                        const int* __restrict__ incl, const int* __restrict__ cnt,
                                                        int nblocks, unsigned* __restrict__ keys_out,
                                                        int* __restrict__ vals_out) {
    __shared__ int run[256];       // running output position per digit
    __shared__ int wcount[8][256];  // per-warp digit counts of the current sub-tile
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    {
        const int64_t idx = (int64_t)threadIdx.x * nblocks + blockIdx.x;
        run[threadIdx.x] = incl[idx] - cnt[idx];
    }
    const int64_t base = (int64_t)blockIdx.x * RS_TILE;
    for (int sub = 0; sub < RS_SUB; sub++) {
        for (int w = 0; w < 8; w++) wcount[w][threadIdx.x] = 0;
        __syncthreads();
        const int64_t i = base + (int64_t)sub * RS_T + threadIdx.x;
        const bool valid = i < n;
        unsigned key = valid ? keys_in[i] : 0u;
        int val = valid ? vals_in[i] : 0;
        int d = valid ? (int)((key >> shift) & 255) : 256 + lane;  // invalid lanes get unique dummies
        unsigned peers = __match_any_sync(0xffffffffu, d);
        int rank_in_warp = __popc(peers & ((1u << lane) - 1));
        if (valid && rank_in_warp == 0) wcount[warp][d] = __popc(peers);
        __syncthreads();
        int pos = 0;
        if (valid) {
            int before = 0;
            for (int w = 0; w < warp; w++) before += wcount[w][d];
            pos = run[d] + before + rank_in_warp;
        }
        __syncthreads();
        {
            int tot = 0;
            for (int w = 0; w < 8; w++) tot += wcount[w][threadIdx.x];
            run[threadIdx.x] += tot;
        }
        if (valid) {
            keys_out[pos] = key;
            vals_out[pos] = val;
        }
        __syncthreads();
    }
}

// ---------------- transpose structure: stable order by column in two passes
// A stable sort of the nonzeros by column, most significant bits first.  Pass 1
// (k_tp_hist, a scan, k_tp_scatter) moves each nonzero, as one 64-bit word of
// its low column bits, row and source index, into at most TP_NB buckets of
// 2^shift columns, in storage order inside each; pass 2 (k_tp_bucket, a block
// per bucket) counts the bucket's columns, which gives its part of the row
// pointers, and orders it by column.  A bucket far above the others goes in
// segments, a block each (k_tp_segments).  Both rank stably the same way: each warp
// owns a contiguous part of the items and a counter per bucket (column); the
// counters are summed over the warps before, so a warp then only walks its own
// items in order.  The lanes holding equal keys are found with one ballot per
// key bit (__match_any_sync took ~130 clocks an SM for 32 mostly different
// keys).  Items are placed in shared memory and leave in runs: gathering them
// from global memory by their place instead took half of both passes.
// Against an LSD radix sort of (column, index) pairs, three passes of two random
// 4-byte writes at 2^20 columns, and the rows gathered after it: 2^20 rows and
// columns, 16.8 M nonzeros, 0.93 -> 0.39 ms (scatter 138, bucket 191, histogram
// and places 38, rows 19 us).  Both passes are instruction-bound (153 and 204 warp
// instructions per 32 items).  The kernels are a chain (chain_wait in f4j_ptx.cuh):
// 65536 rows and columns x 8, T() 105 -> 92 us.
constexpr int TP_NB = 1024, TP_BITS = 10;
constexpr int TP1_T = 256, TP1_WARPS = TP1_T / 32, TP1_TILE = 4096;  // pass 1: items per block
constexpr int TP2_T = 512, TP2_WARPS = TP2_T / 32;
constexpr int TP2_CNT = TP2_WARPS * TP_NB;
constexpr int TP2_CAP = 18432;           // bucket items that pass 2 places in shared memory
constexpr int TP2_SEG = 16384;           // items of a segment of a big bucket

// hist[block][bucket], rows of nbp (nb rounded up to a multiple of four).
__global__ void __launch_bounds__(512) k_tp_hist(int64_t n, const int* __restrict__ col, int shift, int nbp,
                                                 int* __restrict__ hist) {
    __shared__ int h[TP_NB];
    chain_trigger();
    for (int i = threadIdx.x; i < nbp; i += 512) h[i] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * TP1_TILE;
    const int cnt = (int)(n - base < TP1_TILE ? n - base : TP1_TILE);
#pragma unroll 8
    for (int i = threadIdx.x; i < cnt; i += 512) atomicAdd(&h[__ldg(col + base + i) >> shift], 1);
    __syncthreads();
    for (int i = threadIdx.x; i < nbp; i += 512) hist[(int64_t)blockIdx.x * nbp + i] = h[i];
}

// The places of pass 1 come from prefixes down the columns of hist: chunks of
// TP_CHUNK blocks here (in place, exclusive; the chunk's total to part), the
// chunks and the buckets in k_tp_starts.  Bucket-major counts and one scan over
// all of them wrote and read four bytes at a time: 2^20 columns, 16.8 M
// nonzeros, histogram and scan 69 us for 38,
// and the places read with them 12 us of k_tp_scatter's.
constexpr int TP_CHUNK = 64;
__global__ void __launch_bounds__(64) k_tp_chunks(int nblocks, int nbp, int* __restrict__ hist, int* __restrict__ part) {
    const int b = 4 * (64 * blockIdx.y + threadIdx.x), r0 = blockIdx.x * TP_CHUNK;
    chain_wait();
    chain_trigger();
    if (b >= nbp) return;
    const int r1 = r0 + TP_CHUNK < nblocks ? r0 + TP_CHUNK : nblocks;
    int4 run = make_int4(0, 0, 0, 0);
    constexpr int U = 16;
    for (int r = r0; r < r1; r += U) {
        int4 v[U];
#pragma unroll
        for (int u = 0; u < U; u++)
            v[u] = r + u < r1 ? *reinterpret_cast<const int4*>(hist + (int64_t)(r + u) * nbp + b) : make_int4(0, 0, 0, 0);
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (r + u < r1) *reinterpret_cast<int4*>(hist + (int64_t)(r + u) * nbp + b) = run;
            run.x += v[u].x, run.y += v[u].y, run.z += v[u].z, run.w += v[u].w;
        }
    }
    *reinterpret_cast<int4*>(part + (int64_t)blockIdx.x * nbp + b) = run;
}

// Exclusive prefix of v over the block's WARPS warps; *total their sum.
template <int WARPS>
__device__ __forceinline__ int tp_block_excl(int v, int* sh, int* total) {
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    int x = v;
    for (int off = 1; off < 32; off <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += o;
    }
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    int before = 0, all = 0;
    for (int w = 0; w < WARPS; w++) {
        if (w < warp) before += sh[w];
        all += sh[w];
    }
    __syncthreads();
    *total = all;
    return before + x - v;
}

// The buckets that go in segments, of more than `above` items: big[0 .. n), the segments of big[i] are
// seg0[i] .. seg0[i + 1) - 1 of all.
// done[i]: its segments whose columns are counted.
struct TpBig {
    int above;
    int *n, *big, *seg0, *done;
};

// part: exclusive prefix over the chunks, in place; start[b]: the bucket's first
// place, start[nb]: all items; the big buckets.  One block, a thread per bucket.
__global__ void __launch_bounds__(TP_NB) k_tp_starts(int chunks, int nb, int nbp, int* __restrict__ part,
                                                     int* __restrict__ start, const TpBig to) {
    __shared__ int sh[TP_NB / 32];
    const int b = threadIdx.x;
    chain_wait();
    chain_trigger();
    int run = 0;
    if (b < nbp) {
        constexpr int U = 16;
        for (int r = 0; r < chunks; r += U) {
            int v[U];
#pragma unroll
            for (int u = 0; u < U; u++) v[u] = r + u < chunks ? part[(int64_t)(r + u) * nbp + b] : 0;
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (r + u < chunks) part[(int64_t)(r + u) * nbp + b] = run;
                run += v[u];
            }
        }
    }
    int total;
    const int at = tp_block_excl<TP_NB / 32>(run, sh, &total);
    if (b < nb) start[b] = at;
    if (b == 0) start[nb] = total;
    // one scan for both counts: at most 2^18 segments, 2^10 big buckets
    const int segs = b < nb && run > to.above ? (run - 1) / TP2_SEG + 1 : 0;
    const int before = tp_block_excl<TP_NB / 32>(segs << 11 | (segs > 0), sh, &total);
    if (segs) {
        to.big[before & 2047] = b;
        to.seg0[before & 2047] = before >> 11;
        to.done[before & 2047] = 0;
    }
    if (b == 0) {
        *to.n = total & 2047;
        to.seg0[total & 2047] = total >> 11;
    }
}

// cnt[w * nkp + key]: how many of warp w's items have the key (nkp: keys rounded
// up to a multiple of four, the rest zero).  Turns it into the place of the
// warp's first one in (key, item) order; start(key, first) sees each key's first
// place.  A thread takes four adjacent keys, so that one
// block scan covers 4 x threads of them.
template <int WARPS, typename F>
__device__ __forceinline__ void tp_places(int* cnt, int nw, int nkp, int* sh, F start) {
    int run = 0;
    for (int k0 = 0; k0 < nkp; k0 += WARPS * 128) {
        const int key = k0 + 4 * (int)threadIdx.x;
        const bool in = key < nkp;
        int4 c = make_int4(0, 0, 0, 0);
        if (in)
            for (int w = 0; w < nw; w++) {
                const int4 t = *reinterpret_cast<const int4*>(cnt + w * nkp + key);
                c.x += t.x, c.y += t.y, c.z += t.z, c.w += t.w;
            }
        int total;
        int4 at;
        at.x = run + tp_block_excl<WARPS>(c.x + c.y + c.z + c.w, sh, &total);
        at.y = at.x + c.x, at.z = at.y + c.y, at.w = at.z + c.z;
        if (in) {
            start(key, at);
            for (int w = 0; w < nw; w++) {
                int4* p = reinterpret_cast<int4*>(cnt + w * nkp + key);
                const int4 t = *p;
                *p = at;
                at.x += t.x, at.y += t.y, at.z += t.z, at.w += t.w;
            }
        }
        run += total;
    }
    __syncthreads();
}

// The place of this lane's item (key < 0: none), stably after the warp's
// earlier items; all lanes call.  keys below 2^bits.
__device__ __forceinline__ int tp_rank(int* mine, int key, int bits) {
    const int lane = threadIdx.x % 32;
    unsigned peers = __ballot_sync(0xffffffffu, key >= 0);
    for (int b = 0; b < bits; b++) {
        const unsigned one = __ballot_sync(0xffffffffu, (key >> b) & 1);
        peers &= (key >> b) & 1 ? one : ~one;
    }
    int at = 0;
    if (key >= 0) at = mine[key];
    const int r = __popc(peers & ((1u << lane) - 1));
    __syncwarp();
    if (key >= 0 && r == 0) mine[key] = at + __popc(peers);
    __syncwarp();
    return at + r;
}

// What the passes write at each place of the order: source index and row, and for
// f4j_csr_transpose (col non-null) the transpose's own copy of the row.  The
// values stay with k_gather: read here, by the 16 warps an SM holds, they took
// 460 us for its 163.
struct TpOut {
    int *perm, *row, *col;
    __device__ __forceinline__ void put(int64_t at, int q, int r) const {
        perm[at] = q;
        row[at] = r;
        if (col) col[at] = r;
    }
};

// Item words: source index in the low qbits, row in the next rbits, column
// within the bucket above.
__global__ void __launch_bounds__(TP1_T) k_tp_scatter(int64_t n, const int* __restrict__ col,
                                                      const int* __restrict__ row, int shift, int nb, int qbits,
                                                      int rbits, const int* __restrict__ hist,
                                                      const int* __restrict__ part, const int* __restrict__ start,
                                                      unsigned long long* __restrict__ items, const TpOut to) {
    extern __shared__ unsigned long long tp_smem[];
    unsigned long long* place = tp_smem;                      // (column, row) at each place of the tile
    int* cnt = reinterpret_cast<int*>(place + TP1_TILE);       // [warp][bucket]
    int* delta = cnt + TP1_WARPS * TP_NB;                     // place in the output less place in the tile
    uint16_t* order = reinterpret_cast<uint16_t*>(delta + TP_NB);  // tile item at each place
    __shared__ int sh[TP1_WARPS];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int64_t base = (int64_t)blockIdx.x * TP1_TILE;
    const int m = (int)(n - base < TP1_TILE ? n - base : TP1_TILE);
    // a lane's items are loaded once, all in flight together
    constexpr int PART = TP1_TILE / TP1_WARPS, PER = PART / 32;
    const int nkp = (nb + 3) & ~3;
    int* mine = cnt + warp * nkp;
    const int i0 = warp * PART + lane;
    chain_wait();
    chain_trigger();
    // this block's first place of four buckets, for tp_places (nb <= 4 x threads; start has nbp entries)
    static_assert(TP_NB <= 4 * TP1_T, "four buckets a thread");
    int4 out = make_int4(0, 0, 0, 0);
    if (4 * (int)threadIdx.x < nkp) {
        const int4 x = reinterpret_cast<const int4*>(hist + (int64_t)blockIdx.x * nkp)[threadIdx.x];
        const int4 y = reinterpret_cast<const int4*>(part + (int64_t)(blockIdx.x / TP_CHUNK) * nkp)[threadIdx.x];
        const int4 z = reinterpret_cast<const int4*>(start)[threadIdx.x];
        out = make_int4(x.x + y.x + z.x, x.y + y.y + z.y, x.z + y.z + z.z, x.w + y.w + z.w);
    }
    int c[PER], r[PER];
#pragma unroll
    for (int u = 0; u < PER; u++) {
        const bool in = i0 + 32 * u < m;
        c[u] = in ? __ldg(col + base + i0 + 32 * u) : -1;
        r[u] = in ? __ldg(row + base + i0 + 32 * u) : 0;
    }
    for (int i = threadIdx.x; i < TP1_WARPS * nkp / 4; i += TP1_T)
        reinterpret_cast<int4*>(cnt)[i] = make_int4(0, 0, 0, 0);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < PER; u++)
        if (c[u] >= 0) atomicAdd(&mine[c[u] >> shift], 1);
    __syncthreads();
    tp_places<TP1_WARPS>(cnt, TP1_WARPS, nkp, sh, [&](int b, int4 first) {
        *reinterpret_cast<int4*>(delta + b) = make_int4(out.x - first.x, out.y - first.y, out.z - first.z, out.w - first.w);
    });
#pragma unroll
    for (int u = 0; u < PER; u++) {
        const int at = tp_rank(mine, c[u] >= 0 ? c[u] >> shift : -1, TP_BITS);
        if (c[u] >= 0) {
            place[at] = (unsigned long long)(unsigned)c[u] << 32 | (unsigned)r[u];
            order[at] = (uint16_t)(i0 + 32 * u);
        }
    }
    __syncthreads();
    for (int p = threadIdx.x; p < m; p += TP1_T) {
        const unsigned long long w = place[p];
        const int cc = (int)(w >> 32);
        const unsigned long long q = (unsigned long long)(base + order[p]);
        const int64_t dst = (int64_t)p + delta[cc >> shift];
        if (items) {
            items[dst] = q | (w & 0xffffffffull) << qbits |
                         (unsigned long long)(cc & ((1 << shift) - 1)) << (qbits + rbits);
        } else {  // one column a bucket: this is the whole order
            to.put(dst, (int)q, (int)w);
        }
    }
}

// Orders the m items at `in` by key, stably: put(place, item) for each; start(key,
// first) sees each key's first place before that.  nw warps (all of them up to 2^10
// columns a bucket) rank; each takes a multiple of 32 items.
template <typename F, typename G>
__device__ __forceinline__ void tp_order(const unsigned long long* __restrict__ in, int m, int up, int shift, int nw,
                                         int nkp, int* cnt, int* sh, F start, G put) {
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    for (int i = threadIdx.x; i < nw * nkp / 4; i += TP2_T) reinterpret_cast<int4*>(cnt)[i] = make_int4(0, 0, 0, 0);
    __syncthreads();
    const int part = ((m + nw - 1) / nw + 31) & ~31;
    int* mine = cnt + warp * nkp;
    const int i0 = warp < nw && warp * part < m ? warp * part : m;
    const int i1 = i0 + part < m ? i0 + part : m;
    constexpr int U = 8;  // loads in flight per lane
    for (int i = i0 + lane; i < i1; i += 32 * U) {
        int key[U];
#pragma unroll
        for (int u = 0; u < U; u++) key[u] = i + 32 * u < i1 ? (int)(__ldg(in + i + 32 * u) >> up) : -1;
#pragma unroll
        for (int u = 0; u < U; u++)
            if (key[u] >= 0) atomicAdd(&mine[key[u]], 1);
    }
    __syncthreads();
    tp_places<TP2_WARPS>(cnt, nw, nkp, sh, start);
    for (int i = i0; i < i1; i += 32 * U) {
        unsigned long long w[U];
#pragma unroll
        for (int u = 0; u < U; u++) w[u] = i + 32 * u + lane < i1 ? __ldg(in + i + 32 * u + lane) : ~0ull;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const bool has = i + 32 * u + lane < i1;
            const int at = tp_rank(mine, has ? (int)(w[u] >> up) : -1, shift);
            if (has) put(at, w[u]);
        }
    }
}

// Segment seg of all: its big bucket (an index of of.big) and its first item within that.
__device__ __forceinline__ int tp_segment(const TpBig& of, int seg, int64_t& at) {
    int lo = 0, hi = *of.n - 1;  // the last big bucket that starts at or before it
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (__ldg(of.seg0 + mid) <= seg) lo = mid;
        else hi = mid - 1;
    }
    at = (int64_t)(seg - __ldg(of.seg0 + lo)) * TP2_SEG;
    return lo;
}

// The places of big bucket i's segments, once all are counted: seg_cnt becomes, down
// each column, the exclusive prefix over them; the columns' totals give the bucket's
// row pointers.  A thread takes four adjacent columns of a row.
__device__ __forceinline__ void tp_seg_places(int64_t cols, int shift, const int* start, const TpBig& of, int i,
                                              int* seg_cnt, int* sh, int* t_rowptr) {
    const int nkp = ((1 << shift) + 3) & ~3;
    const int b = of.big[i], g0 = of.seg0[i], g1 = of.seg0[i + 1];
    int before = start[b];
    for (int k0 = 0; k0 < nkp; k0 += 4 * TP2_T) {
        const int c = k0 + 4 * (int)threadIdx.x;
        int4 run = make_int4(0, 0, 0, 0);
        if (c < nkp) {
            constexpr int U = 8;
            for (int g = g0; g < g1; g += U) {
                int4 v[U];
#pragma unroll
                for (int u = 0; u < U; u++)
                    v[u] = g + u < g1 ? __ldcg(reinterpret_cast<const int4*>(seg_cnt + (int64_t)(g + u) * nkp + c))
                                      : make_int4(0, 0, 0, 0);
#pragma unroll
                for (int u = 0; u < U; u++) {
                    if (g + u < g1) *reinterpret_cast<int4*>(seg_cnt + (int64_t)(g + u) * nkp + c) = run;
                    run.x += v[u].x, run.y += v[u].y, run.z += v[u].z, run.w += v[u].w;
                }
            }
        }
        int total;
        int at = before + tp_block_excl<TP2_WARPS>(run.x + run.y + run.z + run.w, sh, &total);
        before += total;
        const int each[4] = {run.x, run.y, run.z, run.w};
        const int64_t c0 = ((int64_t)b << shift) + c;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (c + u < 1 << shift && c0 + u < cols) t_rowptr[c0 + u] = at;
            at += each[u];
        }
    }
}

// The blocks of pass 2 after the buckets': they count the columns of the big
// buckets' segments, seg_cnt[segment][column], and the one that counts a bucket's
// last goes on to its places; k_tp_seg_order then moves the items.  A block a bucket
// left most of the work to one SM where the columns are skewed (a graph's vertices by
// degree, a dense band).  T() at 2^20 rows and columns, 16.8 M nonzeros, us, a radix
// sort / a block a bucket / this: 80 % of them in 1024 columns 2231 / 27785 / 745, in
// one column 9539 / 14892 / 657, columns by a power law 5708 / 20739 / 742; evenly
// spread 1478 / 604 / 611.
__device__ __forceinline__ void tp_segments(int first, int stride, int64_t cols, int shift, int up, const int* start,
                                            const unsigned long long* items, int* t_rowptr, const TpBig& of,
                                            int* seg_cnt, int* cnt, int* sh) {
    __shared__ int last;
    const int nkp = ((1 << shift) + 3) & ~3, segs = of.seg0[*of.n];
    for (int seg = first; seg < segs; seg += stride) {
        int64_t at;
        const int i = tp_segment(of, seg, at), b = of.big[i];
        const int64_t s0 = start[b] + at, s1 = start[b + 1];
        const int m = (int)(s1 - s0 < TP2_SEG ? s1 - s0 : TP2_SEG);
        for (int c = threadIdx.x; c < nkp; c += TP2_T) cnt[c] = 0;
        __syncthreads();
#pragma unroll 8
        for (int j = threadIdx.x; j < m; j += TP2_T) atomicAdd(&cnt[__ldg(items + s0 + j) >> up], 1);
        __syncthreads();
        for (int c = threadIdx.x; c < nkp; c += TP2_T) seg_cnt[(int64_t)seg * nkp + c] = cnt[c];
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) last = atomicAdd(of.done + i, 1) + 1 == of.seg0[i + 1] - of.seg0[i];
        __syncthreads();
        if (last) {
            __threadfence();
            tp_seg_places(cols, shift, start, of, i, seg_cnt, sh, t_rowptr);
        }
        __syncthreads();
    }
}

// Bucket b = blockIdx.x < nb: columns [b << shift, (b + 1) << shift), items
// [start[b], start[b + 1]) of the pass 1 output.  The blocks from nb on: tp_segments.
__global__ void __launch_bounds__(TP2_T) k_tp_bucket(int nb, int64_t cols, int shift, int qbits, int rbits, int nw,
                                                     const int* __restrict__ start,
                                                     const unsigned long long* __restrict__ items,
                                                     int* __restrict__ t_rowptr, const TpOut to, const TpBig of,
                                                     int* __restrict__ seg_cnt) {
    extern __shared__ unsigned long long tp_smem[];
    unsigned long long* place = tp_smem;                 // item at each place of the bucket
    int* cnt = reinterpret_cast<int*>(place + TP2_CAP);   // [warp][column]
    __shared__ int sh[TP2_WARPS];
    const int up = qbits + rbits;
    const int b = blockIdx.x;
    chain_wait();
    chain_trigger();
    if (b >= nb) {
        tp_segments(b - nb, gridDim.x - nb, cols, shift, up, start, items, t_rowptr, of, seg_cnt, cnt, sh);
        return;
    }
    const int64_t s0 = __ldg(start + b), s1 = __ldg(start + b + 1);
    if (b == nb - 1 && threadIdx.x == 0) t_rowptr[cols] = (int)s1;
    if (s1 - s0 > of.above) return;
    const int m = (int)(s1 - s0);
    const bool placed = m <= TP2_CAP;  // else more items than shared memory holds: straight to their places
    const int64_t c0 = (int64_t)b << shift;
    const int nk = (int)(cols - c0 < (1 << shift) ? cols - c0 : 1 << shift);
    const unsigned long long qmask = (1ull << qbits) - 1, rmask = (1ull << rbits) - 1;
    auto start_of = [&](int c, int4 first) {
        const int f[4] = {first.x, first.y, first.z, first.w};
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (c + u < nk) t_rowptr[c0 + c + u] = (int)s0 + f[u];
    };
    tp_order(items + s0, m, up, shift, nw, (nk + 3) & ~3, cnt, sh, start_of, [&](int at, unsigned long long w) {
        if (placed) place[at] = w;
        else to.put(s0 + at, (int)(w & qmask), (int)(w >> qbits & rmask));
    });
    if (!placed) return;
    __syncthreads();
    for (int p = threadIdx.x; p < m; p += TP2_T) {
        const unsigned long long w = place[p];
        to.put(s0 + p, (int)(w & qmask), (int)(w >> qbits & rmask));
    }
}

// The big buckets' segments, each ordered by a block and written to its places.
__global__ void __launch_bounds__(TP2_T) k_tp_seg_order(int64_t cols, int shift, int qbits, int rbits, int nw,
                                                        const int* __restrict__ start,
                                                        const unsigned long long* __restrict__ items,
                                                        const int* __restrict__ t_rowptr, const TpOut to, const TpBig of,
                                                        const int* __restrict__ seg_cnt) {
    extern __shared__ unsigned long long tp_smem[];
    unsigned long long* place = tp_smem;
    int* cnt = reinterpret_cast<int*>(place + TP2_SEG);
    int* delta = cnt + TP2_CNT;  // place in the output less place in the segment, by column
    __shared__ int sh[TP2_WARPS];
    chain_wait();
    const int nkp = ((1 << shift) + 3) & ~3, up = qbits + rbits, segs = of.seg0[*of.n];
    const unsigned long long qmask = (1ull << qbits) - 1, rmask = (1ull << rbits) - 1;
    for (int seg = blockIdx.x; seg < segs; seg += gridDim.x) {
        int64_t at;
        const int b = of.big[tp_segment(of, seg, at)];
        const int64_t s0 = __ldg(start + b) + at, s1 = __ldg(start + b + 1);
        const int m = (int)(s1 - s0 < TP2_SEG ? s1 - s0 : TP2_SEG);
        const int64_t c0 = (int64_t)b << shift;
        auto start_of = [&](int c, int4 first) {
            const int4 d = *reinterpret_cast<const int4*>(seg_cnt + (int64_t)seg * nkp + c);
            const int v[4] = {d.x - first.x, d.y - first.y, d.z - first.z, d.w - first.w};
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (c0 + c + u < cols) delta[c + u] = v[u] + t_rowptr[c0 + c + u];
        };
        tp_order(items + s0, m, up, shift, nw, nkp, cnt, sh, start_of,
                 [&](int p, unsigned long long w) { place[p] = w; });
        __syncthreads();
        for (int p = threadIdx.x; p < m; p += TP2_T) {
            const unsigned long long w = place[p];
            to.put((int64_t)p + delta[w >> up], (int)(w & qmask), (int)(w >> qbits & rmask));
        }
        __syncthreads();
    }
}

// Row pointers when every bucket is one column (shift 0).
__global__ void k_tp_rowptr(int nb, const int* __restrict__ start, int* __restrict__ t_rowptr) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c <= nb) t_rowptr[c] = start[c];
}

// ---------------- COO sort by (row, col), stable
// Sorting by (row, col) stably is sorting by the unique key (row, col, input
// index).  The triplets are bucketed by row through per-row atomic cursors
// (which leaves each row's order arbitrary), then each row's segment is
// sorted by (col, input index), packed as one 64-bit key, in registers (rows
// of up to 32 entries, a warp per row) or in shared memory (bitonic, up to
// SEG_CAP entries, a block per row).  The values follow through the input
// index.  Longer rows, and negative indices, take the radix path.
constexpr int SEG_CAP = 4096;

__global__ void k_coo_minmax(int64_t n, const int* __restrict__ r, const int* __restrict__ c, int* __restrict__ mm) {
    int lo = INT32_MAX, hr = INT32_MIN, hc = INT32_MIN;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int a = __ldg(&r[i]), b = __ldg(&c[i]);
        lo = min(lo, min(a, b));
        hr = max(hr, a);
        hc = max(hc, b);
    }
    for (int o = 16; o; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hr = max(hr, __shfl_xor_sync(0xffffffffu, hr, o));
        hc = max(hc, __shfl_xor_sync(0xffffffffu, hc, o));
    }
    if (threadIdx.x % 32 == 0) {
        atomicMin(&mm[0], lo);
        atomicMax(&mm[1], hr);
        atomicMax(&mm[2], hc);
    }
}

__global__ void k_count_rows(int64_t n, const int* __restrict__ r, int* __restrict__ cnt) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        atomicAdd(&cnt[__ldg(&r[i])], 1);
}

__global__ void k_max_int(int64_t n, const int* __restrict__ v, int* __restrict__ out) {
    int m = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        m = max(m, __ldg(&v[i]));
    for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x % 32 == 0) atomicMax(out, m);
}

// rp: exclusive row offsets (rows + 1); cur: per-row cursors, zeroed
__global__ void k_coo_bucket(int64_t n, const int* __restrict__ r, const int* __restrict__ c,
                             const int* __restrict__ rp, int* __restrict__ cur, unsigned long long* __restrict__ key) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int row = __ldg(&r[i]);
        const int pos = __ldg(&rp[row]) + atomicAdd(&cur[row], 1);
        key[pos] = ((unsigned long long)(unsigned)__ldg(&c[i]) << 32) | (unsigned)i;
    }
}

// writes one sorted entry: row, column, and the value of its input index
__device__ __forceinline__ void coo_emit(int64_t pos, int row, unsigned long long k, int* __restrict__ ro,
                                         int* __restrict__ co, const double* __restrict__ vin,
                                         double* __restrict__ vo, int* __restrict__ po) {
    ro[pos] = row;
    co[pos] = (int)(k >> 32);
    if (vo) vo[pos] = __ldg(&vin[(unsigned)k]);
    if (po) po[pos] = (int)(unsigned)k;
}

// a warp per row; rows of up to 64 entries are ranked in registers, two keys
// per lane (keys are unique, so the ranks are a permutation), longer ones are
// listed for k_coo_seg_block (nlong[0] counts them; nlong[3] is the longest row)
__global__ void k_coo_seg_warp(int64_t rows, const int* __restrict__ rp, const unsigned long long* __restrict__ key,
                               int* __restrict__ ro, int* __restrict__ co, const double* __restrict__ vin,
                               double* __restrict__ vo, int* __restrict__ po, int* __restrict__ longlist,
                               int* __restrict__ nlong) {
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const int lane = threadIdx.x % 32;
    // nlong[3]: the longest row; beyond SEG_CAP the host sorts by radix from
    // the untouched input instead
    if (row >= rows || nlong[3] > SEG_CAP) return;
    const int q0 = __ldg(&rp[row]), len = __ldg(&rp[row + 1]) - q0;
    if (len > 64) {
        if (lane == 0) longlist[atomicAdd(nlong, 1)] = (int)row;
        return;
    }
    const unsigned long long k0 = lane < len ? key[q0 + lane] : ~0ull;
    const unsigned long long k1 = lane + 32 < len ? key[q0 + 32 + lane] : ~0ull;
    const int n0 = len < 32 ? len : 32, n1 = len - n0;
    int r0 = 0, r1 = 0;
    for (int j = 0; j < n0; j++) {
        const unsigned long long x = __shfl_sync(0xffffffffu, k0, j);
        r0 += x < k0;
        r1 += x < k1;
    }
    for (int j = 0; j < n1; j++) {
        const unsigned long long x = __shfl_sync(0xffffffffu, k1, j);
        r0 += x < k0;
        r1 += x < k1;
    }
    if (lane < len) coo_emit(q0 + r0, (int)row, k0, ro, co, vin, vo, po);
    if (lane + 32 < len) coo_emit(q0 + r1, (int)row, k1, ro, co, vin, vo, po);
}

// a block per listed row (65 .. pmax entries, pmax a power of two up to
// SEG_CAP): bitonic sort in shared memory (pmax keys)
__global__ void __launch_bounds__(512) k_coo_seg_block(const int* __restrict__ longlist, const int* __restrict__ nlong,
                                                       const int* __restrict__ rp,
                                                       const unsigned long long* __restrict__ key,
                                                       int* __restrict__ ro, int* __restrict__ co,
                                                       const double* __restrict__ vin, double* __restrict__ vo,
                                                       int* __restrict__ po) {
    extern __shared__ unsigned long long sk[];
    const int nl = *nlong;
    for (int b = blockIdx.x; b < nl; b += gridDim.x) {
        const int row = longlist[b];
        const int q0 = rp[row], len = rp[row + 1] - q0;
        int P = 64;
        while (P < len) P <<= 1;
        for (int i = threadIdx.x; i < P; i += blockDim.x) sk[i] = i < len ? key[q0 + i] : ~0ull;
        __syncthreads();
        for (int size = 2; size <= P; size <<= 1) {
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int t = threadIdx.x; t < P / 2; t += blockDim.x) {
                    const int lo = 2 * t - (t & (stride - 1));
                    const int hi = lo + stride;
                    const bool up = (lo & size) == 0;
                    const unsigned long long a = sk[lo], c = sk[hi];
                    if ((a > c) == up) {
                        sk[lo] = c;
                        sk[hi] = a;
                    }
                }
                __syncthreads();
            }
        }
        for (int i = threadIdx.x; i < len; i += blockDim.x) coo_emit(q0 + i, row, sk[i], ro, co, vin, vo, po);
        __syncthreads();
    }
}

// ---------------- CSR x CSR (RealCsrMatMult, src/main/java/org/flag4j/linalg/
// ops/sparse/csr/real/RealCsrMatMult.java)
// Dense result (standard, :53-75): a warp per row i of A walks the row's
// nonzeros in storage order; for each, the lanes add a * B[k, :] into the
// dense row i of C (zeroed), each product and sum rounded.  A row of B holds
// distinct columns, so the lanes of one step touch distinct entries; the
// __syncwarp orders successive steps.
template <int AK, int BK>
__device__ __forceinline__ double2 spgemm_prod(const double* __restrict__ av, int64_t q,
                                               const double* __restrict__ bv, int64_t t) {
    // the product each variant adds: real b*a; bVal.mult(aVal) with a real
    // (RealComplexCsrMatMult.java:78) or complex a (SemiringCsrMatMult.java:81,
    // Complex128.java:336-341: b.re a.re - b.im a.im, b.re a.im + b.im a.re);
    // aVal.mult(bVal) with b real (RealComplexCsrMatMult.java:113)
    if (!AK && !BK) return make_double2(__dmul_rn(__ldg(&av[q]), __ldg(&bv[t])), 0.0);
    if (!AK) {
        const double a = __ldg(&av[q]);
        const double2 b = __ldg(reinterpret_cast<const double2*>(bv) + t);
        return make_double2(__dmul_rn(b.x, a), __dmul_rn(b.y, a));
    }
    const double2 a = __ldg(reinterpret_cast<const double2*>(av) + q);
    if (!BK) {
        const double b = __ldg(&bv[t]);
        return make_double2(__dmul_rn(a.x, b), __dmul_rn(a.y, b));
    }
    const double2 b = __ldg(reinterpret_cast<const double2*>(bv) + t);
    return make_double2(__dsub_rn(__dmul_rn(b.x, a.x), __dmul_rn(b.y, a.y)),
                        __dadd_rn(__dmul_rn(b.x, a.y), __dmul_rn(b.y, a.x)));
}

// AK / BK: 1 when A's / B's values are complex (interleaved); C is complex
// (interleaved) when either is.
template <int AK, int BK>
__global__ void k_spgemm_dense(int64_t rows, int64_t n2, const int* __restrict__ arp, const int* __restrict__ aci,
                               const double* __restrict__ av, const int* __restrict__ brp,
                               const int* __restrict__ bci, const double* __restrict__ bv, double* __restrict__ C) {
    constexpr int W = (AK || BK) ? 2 : 1;
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const int lane = threadIdx.x % 32;
    if (row >= rows) return;
    double* Cr = C + row * n2 * W;
    const int q1 = __ldg(&arp[row + 1]);
    for (int q = __ldg(&arp[row]); q < q1; q++) {
        const int k = __ldg(&aci[q]);
        const int t1 = __ldg(&brp[k + 1]);
        for (int t = __ldg(&brp[k]) + lane; t < t1; t += 32) {
            const int64_t j = __ldg(&bci[t]);
            const double2 p = spgemm_prod<AK, BK>(av, q, bv, t);
            Cr[W * j] = __dadd_rn(Cr[W * j], p.x);
            if (W == 2) Cr[W * j + 1] = __dadd_rn(Cr[W * j + 1], p.y);
        }
        __syncwarp();
    }
}

// CSR result (standardAsSparse, :92-131), expand-sort-compress: every product
// b * a is written out in the reference's loop order (rows of A, a row's
// nonzeros, then the nonzeros of B's row), stably sorted by (row, column),
// and each run of one (row, column) summed in order starting from its first
// product, as HashMap.merge(col, b * a, Double::sum) does.
__global__ void k_spgemm_len(int64_t annz, const int* __restrict__ aci, const int* __restrict__ brp,
                             int* __restrict__ len, unsigned long long* __restrict__ total) {
    const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long l = 0;
    if (q < annz) {
        const int k = __ldg(&aci[q]);
        l = (unsigned long long)(__ldg(&brp[k + 1]) - __ldg(&brp[k]));
        len[q] = (int)l;
    }
    for (int o = 16; o; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if (threadIdx.x % 32 == 0 && l) atomicAdd(total, l);
}

// off: inclusive scan of the expansion lengths, one per nonzero of A; ev
// holds W values per product (interleaved when complex)
template <int AK, int BK>
__global__ void k_spgemm_expand(int64_t rows, const int* __restrict__ arp, const int* __restrict__ aci,
                                const double* __restrict__ av, const int* __restrict__ brp,
                                const int* __restrict__ bci, const double* __restrict__ bv,
                                const int* __restrict__ off, int* __restrict__ er, int* __restrict__ ec,
                                double* __restrict__ ev) {
    constexpr int W = (AK || BK) ? 2 : 1;
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const int lane = threadIdx.x % 32;
    if (row >= rows) return;
    const int q1 = __ldg(&arp[row + 1]);
    for (int q = __ldg(&arp[row]); q < q1; q++) {
        const int k = __ldg(&aci[q]);
        const int t0 = __ldg(&brp[k]), t1 = __ldg(&brp[k + 1]);
        const int64_t base = (int64_t)(q ? __ldg(&off[q - 1]) : 0) - t0;
        for (int t = t0 + lane; t < t1; t += 32) {
            er[base + t] = (int)row;
            ec[base + t] = __ldg(&bci[t]);
            const double2 p = spgemm_prod<AK, BK>(av, q, bv, t);
            ev[W * (base + t)] = p.x;
            if (W == 2) ev[W * (base + t) + 1] = p.y;
        }
    }
}

// complex products gathered into sorted order: dst[i] = src[perm[i]]
__global__ void k_gather_z(int64_t n, const int* __restrict__ perm, const double2* __restrict__ src,
                           double2* __restrict__ dst) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = src[perm[i]];
}

// fs: inclusive scan of the run-start flags of the sorted expansion
__global__ void k_run_flags(int64_t n, const int* __restrict__ r, const int* __restrict__ c, int* __restrict__ f) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < n) f[e] = (e == 0 || r[e] != r[e - 1] || c[e] != c[e - 1]) ? 1 : 0;
}

__global__ void k_run_starts(int64_t n, const int* __restrict__ fs, int* __restrict__ starts) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < n && (e == 0 || fs[e] != fs[e - 1])) starts[fs[e] - 1] = (int)e;
}

template <int W>
__global__ void k_run_sum(int64_t runs, int64_t n, const int* __restrict__ starts, const int* __restrict__ r,
                          const int* __restrict__ c, const double* __restrict__ v, int* __restrict__ oc,
                          double* __restrict__ ov, int* __restrict__ rowcnt) {
    const int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= runs) return;
    const int s0 = starts[u];
    const int64_t s1 = u + 1 < runs ? starts[u + 1] : n;
    double acc0 = v[W * (int64_t)s0], acc1 = W == 2 ? v[W * (int64_t)s0 + 1] : 0.0;
    for (int64_t e = s0 + 1; e < s1; e++) {
        acc0 = __dadd_rn(acc0, v[W * e]);
        if (W == 2) acc1 = __dadd_rn(acc1, v[W * e + 1]);
    }
    oc[u] = c[s0];
    ov[W * u] = acc0;
    if (W == 2) ov[W * u + 1] = acc1;
    atomicAdd(&rowcnt[r[s0]], 1);
}

}  // namespace

// ------------------------------------------------------------------ host helpers
static int grid1(int64_t n, int t = 256) {
    int64_t b = (n + t - 1) / t;
    if (b < 1) b = 1;
    if (b > 1 << 20) b = 1 << 20;
    return (int)b;
}

// In-place inclusive scan of int32 data[n] (recursive over tile sums).
static int scan_inclusive(f4j_ctx* ctx, int* data, int64_t n) {
    if (n <= 0) return F4J_OK;
    const int64_t tiles = f4j_cdiv(n, SCAN_TILE);
    int* sums = nullptr;
    int rc = f4j_dev_alloc(ctx, (size_t)tiles * sizeof(int), (void**)&sums);
    if (rc) return rc;
    k_scan_tiles<<<(unsigned)tiles, SCAN_T, 0, ctx->stream>>>(n, data, sums);
    F4J_LAUNCHED(ctx);
    if (tiles > 1) {
        rc = scan_inclusive(ctx, sums, tiles);
        if (rc) {
            f4j_dev_free(ctx, sums);
            return rc;
        }
        k_scan_add<<<(unsigned)tiles, 256, 0, ctx->stream>>>(n, data, sums);
        F4J_LAUNCHED(ctx);
    }
    f4j_dev_free(ctx, sums);
    return F4J_OK;
}

// Stable sort of (keys, vals) by the low `bits` bits of keys; result in place.
static int radix_sort_pairs(f4j_ctx* ctx, unsigned* keys, int* vals, int64_t n, int bits) {
    if (n <= 1 || bits <= 0) return F4J_OK;
    const int nb = (int)f4j_cdiv(n, RS_TILE);
    unsigned* k2 = nullptr;
    int* v2 = nullptr;
    int *hist = nullptr, *cnt = nullptr;
    int rc = f4j_dev_alloc(ctx, (size_t)n * 4, (void**)&k2);
    if (!rc) rc = f4j_dev_alloc(ctx, (size_t)n * 4, (void**)&v2);
    if (!rc) rc = f4j_dev_alloc(ctx, (size_t)256 * nb * 4, (void**)&hist);
    if (!rc) rc = f4j_dev_alloc(ctx, (size_t)256 * nb * 4, (void**)&cnt);
    unsigned *ka = keys, *kb = k2;
    int *va = vals, *vb = v2;
    for (int shift = 0; !rc && shift < bits; shift += 8) {
        k_radix_hist<<<nb, RS_T, 0, ctx->stream>>>(n, ka, shift, hist, nb);
        F4J_LAUNCHED(ctx);
        cudaMemcpyAsync(cnt, hist, (size_t)256 * nb * 4, cudaMemcpyDeviceToDevice, ctx->stream);
        rc = scan_inclusive(ctx, hist, (int64_t)256 * nb);
        if (rc) break;
        k_radix_scatter<<<nb, RS_T, 0, ctx->stream>>>(n, ka, va, shift, hist, cnt, nb, kb, vb);
        F4J_LAUNCHED(ctx);
        unsigned* tk = ka; ka = kb; kb = tk;
        int* tv = va; va = vb; vb = tv;
    }
    if (!rc && ka != keys) {
        cudaMemcpyAsync(keys, ka, (size_t)n * 4, cudaMemcpyDeviceToDevice, ctx->stream);
        cudaMemcpyAsync(vals, va, (size_t)n * 4, cudaMemcpyDeviceToDevice, ctx->stream);
    }
    f4j_dev_free(ctx, k2);
    f4j_dev_free(ctx, v2);
    f4j_dev_free(ctx, hist);
    f4j_dev_free(ctx, cnt);
    return rc;
}

static int bits_for(int64_t maxval) {
    int b = 0;
    while (b < 31 && (1ll << b) <= maxval) b++;
    return b;
}

// Stable order of S's nonzeros by column and its row pointers, by
// most-significant-bits-first buckets (see k_tp_scatter); shift: columns per
// bucket, qbits / rbits: bits of a source index and of a row.
static int transpose_buckets(f4j_ctx* ctx, f4j_csr S, int shift, int qbits, int rbits, const int* rowidx, int* trp,
                             const TpOut& to) {
    const int64_t nnz = S->nnz, cols = S->cols;
    const int* col = (const int*)S->colidx->ptr;
    const int nb = (int)((cols - 1) >> shift) + 1;
    const int nblocks = (int)f4j_cdiv(nnz, TP1_TILE);
    const size_t smem1 = (size_t)TP1_TILE * 10 + (size_t)(TP1_WARPS + 1) * TP_NB * 4;
    const size_t smem2 = (size_t)TP2_CAP * 8 + (size_t)TP2_CNT * 4;
    F4J_CUDA(cudaFuncSetAttribute(k_tp_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1));
    const size_t smem3 = (size_t)TP2_SEG * 8 + (size_t)(TP2_CNT + (4 << TP_BITS)) * 4;
    F4J_CUDA(cudaFuncSetAttribute(k_tp_bucket, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem2));
    F4J_CUDA(cudaFuncSetAttribute(k_tp_seg_order, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem3));
    int* hist = nullptr;
    unsigned long long* items = nullptr;
    const int nbp = (nb + 3) & ~3, chunks = (int)f4j_cdiv(nblocks, TP_CHUNK);
    // big buckets: of more items than shared memory places and twice the others' mean (evenly filled
    // ones are as fast whole: 2^20 rows x 20, us, whole / in segments: 3000 columns 687 / 825, 2^20 998 /
    // 1044; x 64 2519 / 2771, 4587 / 3265).  At most this many, and segments of them, whose counts take
    // the place of hist, which is done with by then
    int64_t above = f4j_cdiv(2 * nnz, nb) > TP2_CAP ? f4j_cdiv(2 * nnz, nb) : TP2_CAP;
    above = above < INT32_MAX ? above : INT32_MAX;
    const int64_t bigs = shift ? nnz / (above + 1) : 0, segs = bigs ? nnz / TP2_SEG + bigs : 0;
    const size_t rows_hist = (size_t)nblocks * nbp, rows_seg = (size_t)segs * (((1 << shift) + 3) & ~3);
    const size_t head = rows_hist > rows_seg ? rows_hist : rows_seg;
    int rc = f4j_dev_alloc(ctx, (head + (size_t)(chunks + 4) * nbp + 12) * 4, (void**)&hist);
    if (!rc && shift) rc = f4j_dev_alloc(ctx, (size_t)nnz * 8, (void**)&items);
    if (!rc) {
        int *part = hist + head, *start = part + (size_t)chunks * nbp;
        const TpBig big{(int)above, start + nbp + 4, start + nbp + 8, start + 2 * nbp + 8, start + 3 * nbp + 12};
        k_tp_hist<<<nblocks, 512, 0, ctx->stream>>>(nnz, col, shift, nbp, hist);
        f4j_launch(true, k_tp_chunks, dim3(chunks, (unsigned)f4j_cdiv(nbp, 256)), 64, 0, ctx->stream, nblocks, nbp, hist, part);
        f4j_launch(true, k_tp_starts, 1, TP_NB, 0, ctx->stream, chunks, nb, nbp, part, start, big);
        f4j_launch(true, k_tp_scatter, nblocks, TP1_T, smem1, ctx->stream, nnz, col, rowidx, shift, nb, qbits, rbits, hist,
                   part, start, items, to);
        if (shift) {
            const int nw = TP2_WARPS < TP2_CNT >> shift ? TP2_WARPS : TP2_CNT >> shift;
            const int most = (int)(segs < ctx->sm_count ? segs : ctx->sm_count);
            f4j_launch(true, k_tp_bucket, nb + most, TP2_T, smem2, ctx->stream, nb, cols, shift, qbits, rbits, nw, start,
                       items, trp, to, big, hist);
            if (most) {
                f4j_launch(true, k_tp_seg_order, most, TP2_T, smem3, ctx->stream, cols, shift, qbits, rbits, nw, start, items,
                           trp, to, big, hist);
                ctx->launches++;
            }
        } else {
            k_tp_rowptr<<<grid1(nb + 1), 256, 0, ctx->stream>>>(nb, start, trp);
        }
        ctx->launches += 5;
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) rc = f4j_cuda_fail(e, "transpose structure");
    }
    f4j_dev_free(ctx, hist);
    f4j_dev_free(ctx, items);
    return rc;
}

// The same by an LSD radix sort of (column, index) pairs: past 2^22 columns
// (4096 a bucket), where a block's counters leave fewer than four warps to rank,
// and where an item does not fit 64 bits.
static int transpose_radix(f4j_ctx* ctx, f4j_csr S, const int* rowidx, int* trp, int* perm, int* trow) {
    const int64_t nnz = S->nnz, cols = S->cols;
    unsigned* keys = nullptr;
    int rc = f4j_dev_alloc(ctx, (size_t)nnz * 4, (void**)&keys);
    if (rc) return rc;
    // pointers of S^T: column counts, inclusive scan (as RealCsrOps.transpose :203-211)
    cudaMemsetAsync(trp, 0, (size_t)(cols + 1) * 4, ctx->stream);
    k_count<<<grid1(nnz), 256, 0, ctx->stream>>>(nnz, (const int*)S->colidx->ptr, trp);
    ctx->launches++;
    rc = scan_inclusive(ctx, trp + 1, cols);
    if (!rc) {
        // stable order by column == scatter in storage order (:216-222)
        cudaMemcpyAsync(keys, S->colidx->ptr, (size_t)nnz * 4, cudaMemcpyDeviceToDevice, ctx->stream);
        k_iota<<<grid1(nnz), 256, 0, ctx->stream>>>(nnz, perm);
        ctx->launches++;
        rc = radix_sort_pairs(ctx, keys, perm, nnz, bits_for(cols - 1));
    }
    if (!rc) {
        k_gather<int><<<grid1(nnz), 256, 0, ctx->stream>>>(nnz, perm, rowidx, trow);
        ctx->launches++;
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) rc = f4j_cuda_fail(e, "transpose structure");
    }
    f4j_dev_free(ctx, keys);
    return rc;
}

// Whether calls on the context's stream become part of a graph.  What the stream
// allocates then belongs to the graph and holds nothing until the graph runs, so
// no handle may keep it.
static int in_capture(f4j_ctx* ctx, bool* captured) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    F4J_CUDA(cudaStreamIsCapturing(ctx->stream, &st));
    *captured = st != cudaStreamCaptureStatusNone;
    return F4J_OK;
}

// Frees a structure that ensure_transpose made for this call alone.
static void drop_transpose(f4j_ctx* ctx, f4j_csr S, bool once) {
    if (!once) return;
    f4j_dev_free(ctx, S->t_rowptr);
    f4j_dev_free(ctx, S->t_perm);
    f4j_dev_free(ctx, S->t_rowidx);
    S->t_rowptr = S->t_perm = S->t_rowidx = nullptr;
}

// Builds the cached transpose structure of S (RealCsrOps.transpose order).  *once:
// in a stream capture it is for this call alone, which drops it (drop_transpose)
// behind its last use: the graph then makes and frees it each time it runs.  t_col:
// an array for a copy of its column indices, made on the way where that can be
// (*copied).
static int ensure_transpose(f4j_ctx* ctx, f4j_csr S, bool* once, int* t_col = nullptr, bool* copied = nullptr) {
    *once = false;
    if (S->t_perm) return F4J_OK;
    int rc = in_capture(ctx, once);
    if (rc) return rc;
    const int64_t nnz = S->nnz, rows = S->rows, cols = S->cols;
    int *trp = nullptr, *perm = nullptr, *trow = nullptr, *ri = nullptr;
    rc = f4j_dev_alloc(ctx, (size_t)(cols + 1) * 4, (void**)&trp);
    if (!rc) rc = f4j_dev_alloc(ctx, (size_t)nnz * 4, (void**)&perm);
    if (!rc) rc = f4j_dev_alloc(ctx, (size_t)nnz * 4, (void**)&trow);
    if (!rc && nnz == 0) {
        const cudaError_t e = cudaMemsetAsync(trp, 0, (size_t)(cols + 1) * 4, ctx->stream);
        if (e != cudaSuccess) rc = f4j_cuda_fail(e, "transpose structure");
    } else if (!rc) {
        const int* rowidx = (const int*)S->rowidx;  // cached by f4j_sddmm, or made here
        if (!rowidx) {
            rc = f4j_dev_alloc(ctx, (size_t)nnz * 4, (void**)&ri);
            if (!rc) {
                k_expand_rows<<<(unsigned)f4j_cdiv(rows, 256), 256, 0, ctx->stream>>>(rows, nnz, (const int*)S->rowptr->ptr, ri);
                ctx->launches++;
            }
            rowidx = ri;
        }
        int shift = 0;
        while (((cols - 1) >> shift) >= TP_NB) shift++;
        const int qbits = bits_for(nnz - 1), rbits = bits_for(rows - 1);
        const bool buckets = shift <= 12 && qbits + rbits + shift <= 64;
        if (!rc)
            rc = buckets ? transpose_buckets(ctx, S, shift, qbits, rbits, rowidx, trp, TpOut{perm, trow, t_col})
                         : transpose_radix(ctx, S, rowidx, trp, perm, trow);
        if (!rc && t_col) *copied = buckets;
        f4j_dev_free(ctx, ri);
    }
    if (rc) {
        f4j_dev_free(ctx, trp);
        f4j_dev_free(ctx, perm);
        f4j_dev_free(ctx, trow);
        return rc;
    }
    S->t_rowptr = trp;
    S->t_perm = perm;
    S->t_rowidx = trow;
    return F4J_OK;
}

// Row of each nonzero, cached in the handle.
static int ensure_rowidx(f4j_ctx* ctx, f4j_csr S) {
    if (S->rowidx || S->nnz == 0) return F4J_OK;
    int* ri = nullptr;
    int rc = f4j_dev_alloc(ctx, (size_t)S->nnz * 4, (void**)&ri);
    if (rc) return rc;
    k_expand_rows<<<(unsigned)f4j_cdiv(S->rows, 256), 256, 0, ctx->stream>>>(S->rows, S->nnz,
                                                                             (const int*)S->rowptr->ptr, ri);
    F4J_LAUNCHED(ctx);
    S->rowidx = ri;
    return F4J_OK;
}

static int launch_spmm(f4j_ctx* ctx, int64_t rows, int64_t nnz, int64_t ncols, const int* rp, const int* ci,
                       const double* v, const int* perm, const double* X, double* Y, bool fused = false) {
    if (rows == 0 || ncols == 0) return F4J_OK;
    // Lanes of a row: a power of two up to a warp, two columns a lane (128-bit X
    // loads) above 32 columns, or one lane a column, rows straddling warps, where
    // that power of two (64 columns a pass) would leave too many lanes idle.  2^20 rows
    // x 16, us, power of two / a lane a column: exact mode 5 columns 625 / 416, 9 1119 /
    // 691, 15 1121 / 1115, 17 1792 / 1246, 24 1792 / 1628, 28 1793 / 1943, 33 3562 / 2217, 48
    // 3538 / 2997, 52 3536 / 3405, 56 3538 / 3617, 72 7054 / 4486, 112 7054 / 6964; FMA mode
    // 5 423 / 284, 13 683 / 655, 15 685 / 738, 17 927 / 812, 20 931 / 899, 22 935 / 984, 33
    // 1820 / 1370, 48 1807 / 1621, 52 1808 / 1887, 96 3591 / 2812.  Rows of mostly less
    // than two nonzeros (the transpose of a wide matrix) are writes of zeros, for
    // which more lanes and predicates are only work: S^T of 19026 x 593791 x 6, 76
    // columns, with its SDDMM 201 / 352.
    const bool filled = nnz >= 2 * rows;
    int64_t lanes = 1;  // what the first form occupies
    while (lanes < 32 && lanes < ncols) lanes *= 2;
    if (ncols > 32) lanes = f4j_cdiv(ncols, 64) * 64;
    const bool flat = filled &&
                      (fused ? ncols <= 14 || (ncols <= 32 ? ncols * 8 <= lanes * 5 : ncols * 4 <= lanes * 3)
                             : ncols <= 16 || ncols * 4 <= lanes * 3) &&
                      f4j_cdiv(rows * ncols, 256) <= INT32_MAX;
    const bool vec2 = !flat && ncols > 32 && (ncols % 2 == 0) && f4j_aligned16(X) && f4j_aligned16(Y);
    const int G = (int)(flat ? ncols : (lanes < 32 ? lanes : 32));
    const int64_t threads = rows * G;
    const unsigned blocks = (unsigned)f4j_cdiv(threads, 256);
    f4j_prof_begin(ctx);
    if (fused) {
        // the FMA mode (products with no reference order to keep): no transpose variant
        if (vec2) k_spmm<true, false, true><<<blocks, 256, 0, ctx->stream>>>(rows, ncols, G, rp, ci, v, perm, X, Y);
        else k_spmm<false, false, true><<<blocks, 256, 0, ctx->stream>>>(rows, ncols, G, rp, ci, v, perm, X, Y);
    } else if (vec2) {
        if (perm) k_spmm<true, true><<<blocks, 256, 0, ctx->stream>>>(rows, ncols, G, rp, ci, v, perm, X, Y);
        else k_spmm<true, false><<<blocks, 256, 0, ctx->stream>>>(rows, ncols, G, rp, ci, v, perm, X, Y);
    } else {
        if (filled && G % 32) {  // a warp holds rows of different lengths
            if (perm) k_spmm<false, true, false, true><<<blocks, 256, 0, ctx->stream>>>(rows, ncols, G, rp, ci, v, perm, X, Y);
            else k_spmm<false, false, false, true><<<blocks, 256, 0, ctx->stream>>>(rows, ncols, G, rp, ci, v, perm, X, Y);
        } else if (perm) k_spmm<false, true><<<blocks, 256, 0, ctx->stream>>>(rows, ncols, G, rp, ci, v, perm, X, Y);
        else k_spmm<false, false><<<blocks, 256, 0, ctx->stream>>>(rows, ncols, G, rp, ci, v, perm, X, Y);
    }
    f4j_prof_end(ctx);
    F4J_LAUNCHED(ctx);
    return F4J_OK;
}

// ------------------------------------------------------------------ C ABI
extern "C" int f4j_csr_wrap(f4j_ctx* ctx, int64_t rows, int64_t cols, int64_t nnz, f4j_buf rowptr, f4j_buf colidx,
                            f4j_buf vals, int validate, f4j_csr* out) {
    F4J_LOCK(ctx);
    F4J_CHECK_CTX(ctx);
    if (!out) return f4j_fail(F4J_ERR_ARG, "null output pointer");
    *out = nullptr;
    if (!rowptr || !colidx || !vals) return f4j_fail(F4J_ERR_ARG, "null CSR buffer");
    if (rows < 0 || cols < 0 || nnz < 0) return f4j_fail(F4J_ERR_ARG, "negative CSR size");
    if (rows > INT32_MAX || cols > INT32_MAX || nnz > INT32_MAX)
        return f4j_fail(F4J_ERR_ARG, "CSR sizes exceed Flag4j's int range");
    if ((int64_t)rows * cols < nnz)
        return f4j_fail(F4J_ERR_CSR,
                        "The number of non-zero entries cannot be greater than the total number of entries in the "
                        "matrix but got nnz=%lld and totalEntries=%lld",
                        (long long)nnz, (long long)(rows * cols));
    if (rowptr->bytes < (size_t)(rows + 1) * 4)
        return f4j_fail(F4J_ERR_CSR, "Expecting rowPointers to have length (numRows + 1)=%lld", (long long)(rows + 1));
    if (colidx->bytes < (size_t)nnz * 4 || vals->bytes < (size_t)nnz * 8)
        return f4j_fail(F4J_ERR_CSR, "column index / value buffers shorter than nnz=%lld", (long long)nnz);
    if (!f4j_aligned(rowptr->ptr, 4) || !f4j_aligned(colidx->ptr, 4) || !f4j_aligned(vals->ptr, 8))
        return f4j_fail(F4J_ERR_ARG, "CSR buffers must be aligned to their element size");
    F4J_CUDA(cudaSetDevice(ctx->device));
    if (validate) {
        void* ws;
        int rc = f4j_workspace(ctx, 2, 64, &ws);
        if (rc) return rc;
        int h[4] = {INT32_MAX, INT32_MAX, 0, 0};
        F4J_CUDA(cudaMemcpyAsync(ws, h, 8, cudaMemcpyHostToDevice, ctx->stream));
        if (rows) {
            k_validate_csr<<<grid1(rows), 256, 0, ctx->stream>>>(rows, cols, nnz, (const int*)rowptr->ptr,
                                                                 (const int*)colidx->ptr, (int*)ws, (int*)ws + 1);
            F4J_LAUNCHED(ctx);
        }
        int first_last[2] = {0, 0};
        F4J_CUDA(cudaMemcpyAsync(h, ws, 8, cudaMemcpyDeviceToHost, ctx->stream));
        F4J_CUDA(cudaMemcpyAsync(&first_last[0], rowptr->ptr, 4, cudaMemcpyDeviceToHost, ctx->stream));
        F4J_CUDA(cudaMemcpyAsync(&first_last[1], (int*)rowptr->ptr + rows, 4, cudaMemcpyDeviceToHost, ctx->stream));
        F4J_CUDA(cudaStreamSynchronize(ctx->stream));
        if (h[0] != INT32_MAX) {
            int p[2];
            cudaMemcpy(p, (int*)rowptr->ptr + h[0], 8, cudaMemcpyDeviceToHost);
            if (p[0] < 0)
                return f4j_fail(F4J_ERR_CSR, "All rowPointers must be positive but got %d at index %d.", p[0], h[0]);
            return f4j_fail(F4J_ERR_CSR,
                            "rowPointers must be monotonically increasing but got values %d and %d at indices %d "
                            "and %d.",
                            p[0], p[1], h[0], h[0] + 1);
        }
        if (h[1] != INT32_MAX) {
            int c = 0;
            cudaMemcpy(&c, (int*)colidx->ptr + h[1], 4, cudaMemcpyDeviceToHost);
            return f4j_fail(F4J_ERR_CSR, "Invalid column index [%d] encountered for CSR matrix of shape (%lld, %lld)", c,
                            (long long)rows, (long long)cols);
        }
        if ((int64_t)first_last[1] - first_last[0] != nnz)
            return f4j_fail(F4J_ERR_CSR, "rowIndices specifies %lld elements but nnz=%lld. These values must be equal.",
                            (long long)((int64_t)first_last[1] - first_last[0]), (long long)nnz);
    }
    *out = new f4j_csr_s{rows, cols, nnz, rowptr, colidx, vals, false, nullptr, nullptr, nullptr, nullptr};
    return F4J_OK;
}

extern "C" int f4j_csr_free(f4j_ctx* ctx, f4j_csr S) {
    F4J_LOCK(ctx);
    F4J_CHECK_CTX(ctx);
    if (!S) return F4J_OK;
    F4J_CUDA(cudaStreamSynchronize(ctx->stream));
    cudaFree(S->t_rowptr);
    cudaFree(S->t_perm);
    cudaFree(S->t_rowidx);
    cudaFree(S->rowidx);
    if (S->owns) {
        f4j_buf_free(ctx, S->rowptr);
        f4j_buf_free(ctx, S->colidx);
        f4j_buf_free(ctx, S->vals);
    }
    delete S;
    return F4J_OK;
}

extern "C" int f4j_csr_info(f4j_csr S, int64_t* rows, int64_t* cols, int64_t* nnz) {
    if (!S) return f4j_fail(F4J_ERR_ARG, "null CSR handle");
    if (rows) *rows = S->rows;
    if (cols) *cols = S->cols;
    if (nnz) *nnz = S->nnz;
    return F4J_OK;
}

extern "C" int f4j_csr_buffers(f4j_csr S, f4j_buf* rowptr, f4j_buf* colidx, f4j_buf* vals) {
    if (!S) return f4j_fail(F4J_ERR_ARG, "null CSR handle");
    if (rowptr) *rowptr = S->rowptr;
    if (colidx) *colidx = S->colidx;
    if (vals) *vals = S->vals;
    return F4J_OK;
}

static int alloc_owned_csr(f4j_ctx* ctx, int64_t rows, int64_t cols, int64_t nnz, f4j_csr* out, int vw = 1) {
    f4j_buf rp = nullptr, ci = nullptr, v = nullptr;
    int rc = f4j_buf_alloc_pooled(ctx, (size_t)(rows + 1) * 4, &rp);
    if (!rc) rc = f4j_buf_alloc_pooled(ctx, (size_t)nnz * 4, &ci);
    if (!rc) rc = f4j_buf_alloc_pooled(ctx, (size_t)nnz * 8 * vw, &v);
    if (rc) {
        f4j_buf_free(ctx, rp);
        f4j_buf_free(ctx, ci);
        f4j_buf_free(ctx, v);
        return rc;
    }
    *out = new f4j_csr_s{rows, cols, nnz, rp, ci, v, true, nullptr, nullptr, nullptr, nullptr};
    return F4J_OK;
}

extern "C" int f4j_csr_from_coo(f4j_ctx* ctx, int64_t rows, int64_t cols, int64_t nnz, f4j_buf rowidx, f4j_buf colidx,
                                f4j_buf vals, f4j_csr* out) {
    F4J_LOCK(ctx);
    F4J_CHECK_CTX(ctx);
    if (!out) return f4j_fail(F4J_ERR_ARG, "null output pointer");
    *out = nullptr;
    if (!rowidx || !colidx || !vals) return f4j_fail(F4J_ERR_ARG, "null COO buffer");
    if (rows < 0 || cols < 0 || nnz < 0 || rows > INT32_MAX || cols > INT32_MAX || nnz > INT32_MAX)
        return f4j_fail(F4J_ERR_ARG, "bad COO sizes");
    if (rowidx->bytes < (size_t)nnz * 4 || colidx->bytes < (size_t)nnz * 4 || vals->bytes < (size_t)nnz * 8)
        return f4j_fail(F4J_ERR_CSR,
                        "The number of non-zero entries must match the number of row and column indices");
    if ((int64_t)rows * cols < nnz)
        return f4j_fail(F4J_ERR_CSR, "The number of non-zero entries cannot be greater than the total number of entries");
    F4J_CUDA(cudaSetDevice(ctx->device));
    // SparseValidation.validateCoo (…/SparseValidation.java:70-98): indices in
    // range, checked by the count and the column copy themselves; the handle is
    // returned only after both checks have passed (one wait, at the end)
    void* ws;
    int rc = f4j_workspace(ctx, 2, 64, &ws);
    if (rc) return rc;
    int h[2] = {INT32_MAX, INT32_MAX};
    F4J_CUDA(cudaMemcpyAsync(ws, h, 8, cudaMemcpyHostToDevice, ctx->stream));
    f4j_csr S;
    rc = alloc_owned_csr(ctx, rows, cols, nnz, &S);
    if (rc) return rc;
    int* rp = (int*)S->rowptr->ptr;
    // CooMatrix.toCsr (…/CooMatrix.java:457-470): count per row into rp[r+1],
    // inclusive scan; column indices and values copied unchanged
    F4J_CUDA(cudaMemsetAsync(rp, 0, (size_t)(rows + 1) * 4, ctx->stream));
    if (nnz) {
        (f4j_aligned16(rowidx->ptr) ? k_count_rows_checked<true> : k_count_rows_checked<false>)
            <<<grid1(f4j_cdiv(nnz, 8)), 256, 0, ctx->stream>>>(nnz, (const int*)rowidx->ptr, rows, rp, (int*)ws);
        F4J_LAUNCHED(ctx);
        const bool vec = ((reinterpret_cast<uintptr_t>(colidx->ptr) | reinterpret_cast<uintptr_t>(S->colidx->ptr)) &
                          15) == 0;
        if (vec)
            k_copy_cols_checked<true><<<grid1(f4j_cdiv(nnz, 4)), 256, 0, ctx->stream>>>(
                nnz, (const int*)colidx->ptr, cols, (int*)S->colidx->ptr, (int*)ws + 1);
        else
            k_copy_cols_checked<false><<<grid1(nnz), 256, 0, ctx->stream>>>(
                nnz, (const int*)colidx->ptr, cols, (int*)S->colidx->ptr, (int*)ws + 1);
        F4J_LAUNCHED(ctx);
    }
    rc = scan_inclusive(ctx, rp + 1, rows);
    if (rc) {
        f4j_csr_free(ctx, S);
        return rc;
    }
    F4J_CUDA(cudaMemcpyAsync(S->vals->ptr, vals->ptr, (size_t)nnz * 8, cudaMemcpyDeviceToDevice, ctx->stream));
    F4J_CUDA(cudaMemcpyAsync(h, ws, 8, cudaMemcpyDeviceToHost, ctx->stream));
    F4J_CUDA(cudaStreamSynchronize(ctx->stream));
    if (h[0] != INT32_MAX || h[1] != INT32_MAX) {
        f4j_csr_free(ctx, S);
        int at = h[0] < h[1] ? h[0] : h[1];
        int rc2[2];
        cudaMemcpy(&rc2[0], (int*)rowidx->ptr + at, 4, cudaMemcpyDeviceToHost);
        cudaMemcpy(&rc2[1], (int*)colidx->ptr + at, 4, cudaMemcpyDeviceToHost);
        return f4j_fail(F4J_ERR_CSR, "Invalid index [%d, %d] encountered for COO matrix of shape (%lld, %lld)", rc2[0],
                        rc2[1], (long long)rows, (long long)cols);
    }
    *out = S;
    return F4J_OK;
}

// Radix path of f4j_coo_sort: stable LSD by column, then by row, over the
// keys' significant bits (all 32 with a sign flip when an index is negative,
// so negative indices order first as the reference's int comparison has them).
static int coo_sort_radix(f4j_ctx* ctx, int64_t nnz, int* rowidx, int* colidx, double* vals, int rbits, int cbits,
                          bool flip, int* perm_out) {
    unsigned* keys = nullptr;
    int *perm = nullptr, *tmp = nullptr;
    double* vtmp = nullptr;
    int rc = f4j_dev_alloc(ctx, (size_t)nnz * 4, (void**)&keys);
    if (!rc) rc = f4j_dev_alloc(ctx, (size_t)nnz * 4, (void**)&perm);
    if (!rc) rc = f4j_dev_alloc(ctx, (size_t)nnz * 4, (void**)&tmp);
    if (!rc && vals) rc = f4j_dev_alloc(ctx, (size_t)nnz * 8, (void**)&vtmp);
    if (!rc) {
        k_iota<<<grid1(nnz), 256, 0, ctx->stream>>>(nnz, perm);
        k_flip_copy<<<grid1(nnz), 256, 0, ctx->stream>>>(nnz, nullptr, colidx, flip, keys);
        ctx->launches += 2;
        rc = radix_sort_pairs(ctx, keys, perm, nnz, cbits);
    }
    if (!rc) {
        k_flip_copy<<<grid1(nnz), 256, 0, ctx->stream>>>(nnz, perm, rowidx, flip, keys);
        ctx->launches++;
        rc = radix_sort_pairs(ctx, keys, perm, nnz, rbits);
    }
    if (!rc) {
        k_gather<int><<<grid1(nnz), 256, 0, ctx->stream>>>(nnz, perm, rowidx, tmp);
        cudaMemcpyAsync(rowidx, tmp, (size_t)nnz * 4, cudaMemcpyDeviceToDevice, ctx->stream);
        k_gather<int><<<grid1(nnz), 256, 0, ctx->stream>>>(nnz, perm, colidx, tmp);
        cudaMemcpyAsync(colidx, tmp, (size_t)nnz * 4, cudaMemcpyDeviceToDevice, ctx->stream);
        if (vals) {
            k_gather<double><<<grid1(nnz), 256, 0, ctx->stream>>>(nnz, perm, vals, vtmp);
            cudaMemcpyAsync(vals, vtmp, (size_t)nnz * 8, cudaMemcpyDeviceToDevice, ctx->stream);
        }
        ctx->launches += vals ? 3 : 2;
        if (perm_out) cudaMemcpyAsync(perm_out, perm, (size_t)nnz * 4, cudaMemcpyDeviceToDevice, ctx->stream);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) rc = f4j_cuda_fail(e, "coo sort");
    }
    f4j_dev_free(ctx, keys);
    f4j_dev_free(ctx, perm);
    f4j_dev_free(ctx, tmp);
    f4j_dev_free(ctx, vtmp);
    return rc;
}

// Stable sort of n device triplets by (row, col), in place (v may be null);
// perm_out (may be null) receives the input index of every sorted position.
static int coo_sort_dev(f4j_ctx* ctx, int64_t nnz, int* r, int* c, double* v, int* perm_out = nullptr) {
    if (nnz <= 1) {
        if (nnz == 1 && perm_out) F4J_CUDA(cudaMemsetAsync(perm_out, 0, 4, ctx->stream));
        return F4J_OK;
    }
    const unsigned red_grid = (unsigned)std::min<int64_t>(grid1(nnz), (int64_t)ctx->sm_count * 8);

    // index range: mm = {min of rows and columns, max row, max column, longest row}
    int* mm = nullptr;
    int rc = f4j_dev_alloc(ctx, 16, (void**)&mm);
    if (rc) return rc;
    const int mm0[4] = {INT32_MAX, INT32_MIN, INT32_MIN, 0};
    F4J_CUDA(cudaMemcpyAsync(mm, mm0, 16, cudaMemcpyHostToDevice, ctx->stream));
    k_coo_minmax<<<red_grid, 256, 0, ctx->stream>>>(nnz, r, c, mm);
    ctx->launches++;
    int hm[4];
    F4J_CUDA(cudaMemcpyAsync(hm, mm, 16, cudaMemcpyDeviceToHost, ctx->stream));
    F4J_CUDA(cudaStreamSynchronize(ctx->stream));
    if (hm[0] < 0) {
        f4j_dev_free(ctx, mm);
        return coo_sort_radix(ctx, nnz, r, c, v, 32, 32, true, perm_out);
    }
    const int64_t rows = (int64_t)hm[1] + 1;
    if (rows > 4 * nnz + 4096) {  // row offsets would outweigh the triplets
        f4j_dev_free(ctx, mm);
        int rb = 0, cb = 0;
        while (rb < 31 && (1ll << rb) <= hm[1]) rb++;
        while (cb < 31 && (1ll << cb) <= hm[2]) cb++;
        return coo_sort_radix(ctx, nnz, r, c, v, rb, cb, false, perm_out);
    }

    // row offsets and the longest row
    int *rp = nullptr, *cur = nullptr;
    rc = f4j_dev_alloc(ctx, (size_t)(rows + 1) * 4, (void**)&rp);
    if (!rc) rc = f4j_dev_alloc(ctx, (size_t)rows * 4, (void**)&cur);
    if (!rc) {
        F4J_CUDA(cudaMemsetAsync(rp, 0, (size_t)(rows + 1) * 4, ctx->stream));
        k_count_rows<<<red_grid, 256, 0, ctx->stream>>>(nnz, r, rp + 1);
        k_max_int<<<(unsigned)std::min<int64_t>(grid1(rows), (int64_t)ctx->sm_count * 8), 256, 0, ctx->stream>>>(
            rows, rp + 1, mm + 3);
        ctx->launches += 2;
        rc = scan_inclusive(ctx, rp + 1, rows);
    }
    // buckets and the warp segment sort are queued before the host reads the
    // longest row, so the GPU never waits on the host between them; the warp
    // kernel leaves the input untouched when a row exceeds SEG_CAP
    unsigned long long* key = nullptr;
    double* vin = nullptr;
    int* longlist = nullptr;
    const int64_t maxlong = std::min<int64_t>(rows, nnz / 65 + 1);
    if (!rc) rc = f4j_dev_alloc(ctx, (size_t)nnz * 8, (void**)&key);
    if (!rc && v) rc = f4j_dev_alloc(ctx, (size_t)nnz * 8, (void**)&vin);
    if (!rc) rc = f4j_dev_alloc(ctx, (size_t)maxlong * 4, (void**)&longlist);
    if (!rc) {
        F4J_CUDA(cudaMemsetAsync(cur, 0, (size_t)rows * 4, ctx->stream));
        F4J_CUDA(cudaMemsetAsync(mm, 0, 4, ctx->stream));  // mm[0]: count of listed long rows
        if (v) F4J_CUDA(cudaMemcpyAsync(vin, v, (size_t)nnz * 8, cudaMemcpyDeviceToDevice, ctx->stream));
        k_coo_bucket<<<red_grid, 256, 0, ctx->stream>>>(nnz, r, c, rp, cur, key);
        k_coo_seg_warp<<<(unsigned)f4j_cdiv(rows * 32, 256), 256, 0, ctx->stream>>>(rows, rp, key, r, c, vin, v,
                                                                                   perm_out, longlist, mm);
        ctx->launches += 2;
        F4J_CUDA(cudaMemcpyAsync(&hm[3], mm + 3, 4, cudaMemcpyDeviceToHost, ctx->stream));
        F4J_CUDA(cudaStreamSynchronize(ctx->stream));
        if (hm[3] > SEG_CAP) {
            f4j_dev_free(ctx, key);
            f4j_dev_free(ctx, vin);
            f4j_dev_free(ctx, longlist);
            f4j_dev_free(ctx, rp);
            f4j_dev_free(ctx, cur);
            f4j_dev_free(ctx, mm);
            int rb = 0, cb = 0;
            while (rb < 31 && (1ll << rb) <= hm[1]) rb++;
            while (cb < 31 && (1ll << cb) <= hm[2]) cb++;
            return coo_sort_radix(ctx, nnz, r, c, v, rb, cb, false, perm_out);
        }
        if (hm[3] > 64) {
            // block path sized to the longest row: pmax keys of shared memory, pmax / 2 threads
            int pmax = 128;
            while (pmax < hm[3]) pmax <<= 1;
            const int bthreads = pmax / 2 < 512 ? pmax / 2 : 512;
            const unsigned bgrid = (unsigned)std::min<int64_t>(maxlong, (int64_t)ctx->sm_count * 32);
            k_coo_seg_block<<<bgrid, bthreads, (size_t)pmax * 8, ctx->stream>>>(longlist, mm, rp, key, r, c, vin, v,
                                                                                perm_out);
            ctx->launches++;
        }
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) rc = f4j_cuda_fail(e, "coo sort");
    }
    f4j_dev_free(ctx, key);
    f4j_dev_free(ctx, vin);
    f4j_dev_free(ctx, longlist);
    f4j_dev_free(ctx, rp);
    f4j_dev_free(ctx, cur);
    f4j_dev_free(ctx, mm);
    return rc;
}

extern "C" int f4j_coo_sort(f4j_ctx* ctx, int64_t nnz, f4j_buf rowidx, f4j_buf colidx, f4j_buf vals) {
    F4J_LOCK(ctx);
    F4J_CHECK_CTX(ctx);
    if (!rowidx || !colidx) return f4j_fail(F4J_ERR_ARG, "null COO buffer");
    if (nnz < 0 || nnz > INT32_MAX) return f4j_fail(F4J_ERR_ARG, "bad nnz");
    if (rowidx->bytes < (size_t)nnz * 4 || colidx->bytes < (size_t)nnz * 4 || (vals && vals->bytes < (size_t)nnz * 8))
        return f4j_fail(F4J_ERR_ARG, "COO buffers shorter than nnz");
    if (nnz <= 1) return F4J_OK;
    F4J_CUDA(cudaSetDevice(ctx->device));
    return coo_sort_dev(ctx, nnz, (int*)rowidx->ptr, (int*)colidx->ptr, vals ? (double*)vals->ptr : nullptr);
}

// ------------------------------------------------------------------ CSR x CSR
// The value kinds of A and B select the variant: real x real (RealCsrMatMult),
// real x complex and complex x real (RealComplexCsrMatMult), complex x complex
// (SemiringCsrMatMult over Complex128).
static int check_csr_values(f4j_csr S, int cplx) {
    if (cplx && (S->vals->bytes < (size_t)S->nnz * 16 || !f4j_aligned16(S->vals->ptr)))
        return f4j_fail(F4J_ERR_ARG, "complex CSR values need 16 * nnz bytes, 16-byte aligned");
    return F4J_OK;
}

template <int AK, int BK>
static void launch_spgemm_dense(f4j_ctx* ctx, f4j_csr A, f4j_csr B, double* C) {
    k_spgemm_dense<AK, BK><<<(unsigned)f4j_cdiv(A->rows * 32, 256), 256, 0, ctx->stream>>>(
        A->rows, B->cols, (const int*)A->rowptr->ptr, (const int*)A->colidx->ptr, (const double*)A->vals->ptr,
        (const int*)B->rowptr->ptr, (const int*)B->colidx->ptr, (const double*)B->vals->ptr, C);
}

extern "C" int f4j_csr_mult_dense_ex(f4j_ctx* ctx, f4j_csr A, int a_complex, f4j_csr B, int b_complex, f4j_buf C,
                                     f4j_report* rep) {
    F4J_LOCK(ctx);
    F4J_CHECK_CTX(ctx);
    if (!A || !B || !C) return f4j_fail(F4J_ERR_ARG, "null argument");
    if (A->cols != B->rows) return f4j_shape_error(A->rows, A->cols, B->rows, B->cols);
    int rc = check_csr_values(A, a_complex);
    if (!rc) rc = check_csr_values(B, b_complex);
    if (rc) return rc;
    const int W = (a_complex || b_complex) ? 2 : 1;
    if (C->bytes < (size_t)(A->rows * B->cols) * 8 * W) return f4j_fail(F4J_ERR_ARG, "C buffer too small");
    F4J_CUDA(cudaSetDevice(ctx->device));
    int64_t l0 = ctx->launches;
    if (A->rows * B->cols > 0) {
        F4J_CUDA(cudaMemsetAsync(C->ptr, 0, (size_t)(A->rows * B->cols) * 8 * W, ctx->stream));
        double* Cp = (double*)C->ptr;
        f4j_prof_begin(ctx);
        if (a_complex && b_complex) launch_spgemm_dense<1, 1>(ctx, A, B, Cp);
        else if (a_complex) launch_spgemm_dense<1, 0>(ctx, A, B, Cp);
        else if (b_complex) launch_spgemm_dense<0, 1>(ctx, A, B, Cp);
        else launch_spgemm_dense<0, 0>(ctx, A, B, Cp);
        f4j_prof_end(ctx);
        F4J_LAUNCHED(ctx);
    }
    if (rep) {
        *rep = f4j_report{};
        rep->launches = (int32_t)(ctx->launches - l0);
    }
    return F4J_OK;
}

extern "C" int f4j_csr_mult_dense(f4j_ctx* ctx, f4j_csr A, f4j_csr B, f4j_buf C, f4j_report* rep) {
    F4J_LOCK(ctx);
    return f4j_csr_mult_dense_ex(ctx, A, 0, B, 0, C, rep);
}

template <int AK, int BK>
static void launch_spgemm_expand(f4j_ctx* ctx, f4j_csr A, f4j_csr B, const int* off, int* er, int* ec, double* ev) {
    k_spgemm_expand<AK, BK><<<(unsigned)f4j_cdiv(A->rows * 32, 256), 256, 0, ctx->stream>>>(
        A->rows, (const int*)A->rowptr->ptr, (const int*)A->colidx->ptr, (const double*)A->vals->ptr,
        (const int*)B->rowptr->ptr, (const int*)B->colidx->ptr, (const double*)B->vals->ptr, off, er, ec, ev);
}

extern "C" int f4j_csr_mult_csr_ex(f4j_ctx* ctx, f4j_csr A, int a_complex, f4j_csr B, int b_complex, f4j_csr* out,
                                   f4j_report* rep) {
    F4J_LOCK(ctx);
    F4J_CHECK_CTX(ctx);
    if (!A || !B || !out) return f4j_fail(F4J_ERR_ARG, "null argument");
    *out = nullptr;
    if (A->cols != B->rows) return f4j_shape_error(A->rows, A->cols, B->rows, B->cols);
    int rc = check_csr_values(A, a_complex);
    if (!rc) rc = check_csr_values(B, b_complex);
    if (rc) return rc;
    const int W = (a_complex || b_complex) ? 2 : 1;
    F4J_CUDA(cudaSetDevice(ctx->device));
    int64_t l0 = ctx->launches;
    const int64_t annz = A->nnz, rows = A->rows;
    const int* aci = (const int*)A->colidx->ptr;
    const int* brp = (const int*)B->rowptr->ptr;

    // expansion size
    int* len = nullptr;
    unsigned long long* total = nullptr;
    unsigned long long E = 0;
    rc = f4j_dev_alloc(ctx, (size_t)(annz > 0 ? annz : 1) * 4, (void**)&len);
    if (!rc) rc = f4j_dev_alloc(ctx, 8, (void**)&total);
    if (!rc && annz > 0) {
        F4J_CUDA(cudaMemsetAsync(total, 0, 8, ctx->stream));
        k_spgemm_len<<<(unsigned)f4j_cdiv(annz, 256), 256, 0, ctx->stream>>>(annz, aci, brp, len, total);
        ctx->launches++;
        F4J_CUDA(cudaMemcpyAsync(&E, total, 8, cudaMemcpyDeviceToHost, ctx->stream));
        F4J_CUDA(cudaStreamSynchronize(ctx->stream));
        if (E > (unsigned long long)INT32_MAX)
            rc = f4j_fail(F4J_ERR_UNSUPPORTED, "CSR product expands to %llu products, over 2^31 - 1", E);
    }
    int *er = nullptr, *ec = nullptr, *fs = nullptr, *starts = nullptr, *perm = nullptr;
    double *ev = nullptr, *evs = nullptr;
    int64_t runs = 0;
    if (!rc && E > 0) {
        rc = scan_inclusive(ctx, len, annz);
        if (!rc) rc = f4j_dev_alloc(ctx, E * 4, (void**)&er);
        if (!rc) rc = f4j_dev_alloc(ctx, E * 4, (void**)&ec);
        if (!rc) rc = f4j_dev_alloc(ctx, E * 8 * W, (void**)&ev);
        if (!rc) {
            if (a_complex && b_complex) launch_spgemm_expand<1, 1>(ctx, A, B, len, er, ec, ev);
            else if (a_complex) launch_spgemm_expand<1, 0>(ctx, A, B, len, er, ec, ev);
            else if (b_complex) launch_spgemm_expand<0, 1>(ctx, A, B, len, er, ec, ev);
            else launch_spgemm_expand<0, 0>(ctx, A, B, len, er, ec, ev);
            ctx->launches++;
            if (W == 1) {
                rc = coo_sort_dev(ctx, (int64_t)E, er, ec, ev);
            } else {
                // complex products follow the sort through its permutation
                rc = f4j_dev_alloc(ctx, E * 4, (void**)&perm);
                if (!rc) rc = coo_sort_dev(ctx, (int64_t)E, er, ec, nullptr, perm);
                if (!rc) rc = f4j_dev_alloc(ctx, E * 16, (void**)&evs);
                if (!rc) {
                    k_gather_z<<<(unsigned)f4j_cdiv(E, 256), 256, 0, ctx->stream>>>(
                        (int64_t)E, perm, (const double2*)ev, (double2*)evs);
                    ctx->launches++;
                    double* t = ev;
                    ev = evs;
                    evs = t;
                }
            }
        }
        if (!rc) rc = f4j_dev_alloc(ctx, E * 4, (void**)&fs);
        if (!rc) {
            k_run_flags<<<(unsigned)f4j_cdiv(E, 256), 256, 0, ctx->stream>>>((int64_t)E, er, ec, fs);
            ctx->launches++;
            rc = scan_inclusive(ctx, fs, (int64_t)E);
        }
        if (!rc) {
            int last = 0;
            F4J_CUDA(cudaMemcpyAsync(&last, fs + E - 1, 4, cudaMemcpyDeviceToHost, ctx->stream));
            F4J_CUDA(cudaStreamSynchronize(ctx->stream));
            runs = last;
            rc = f4j_dev_alloc(ctx, (size_t)runs * 4, (void**)&starts);
        }
        if (!rc) {
            k_run_starts<<<(unsigned)f4j_cdiv(E, 256), 256, 0, ctx->stream>>>((int64_t)E, fs, starts);
            ctx->launches++;
        }
    }
    f4j_csr T = nullptr;
    if (!rc) rc = alloc_owned_csr(ctx, rows, B->cols, runs, &T, W);
    if (!rc) {
        int* trp = (int*)T->rowptr->ptr;
        F4J_CUDA(cudaMemsetAsync(trp, 0, (size_t)(rows + 1) * 4, ctx->stream));
        if (runs > 0) {
            const unsigned g = (unsigned)f4j_cdiv(runs, 256);
            if (W == 2)
                k_run_sum<2><<<g, 256, 0, ctx->stream>>>(runs, (int64_t)E, starts, er, ec, ev, (int*)T->colidx->ptr,
                                                         (double*)T->vals->ptr, trp + 1);
            else
                k_run_sum<1><<<g, 256, 0, ctx->stream>>>(runs, (int64_t)E, starts, er, ec, ev, (int*)T->colidx->ptr,
                                                         (double*)T->vals->ptr, trp + 1);
            ctx->launches++;
            rc = scan_inclusive(ctx, trp + 1, rows);
        }
        cudaError_t e = cudaGetLastError();
        if (!rc && e != cudaSuccess) rc = f4j_cuda_fail(e, "CSR x CSR");
    }
    f4j_dev_free(ctx, len);
    f4j_dev_free(ctx, total);
    f4j_dev_free(ctx, er);
    f4j_dev_free(ctx, ec);
    f4j_dev_free(ctx, ev);
    f4j_dev_free(ctx, evs);
    f4j_dev_free(ctx, perm);
    f4j_dev_free(ctx, fs);
    f4j_dev_free(ctx, starts);
    if (rc) {
        if (T) f4j_csr_free(ctx, T);
        return rc;
    }
    *out = T;
    if (rep) {
        *rep = f4j_report{};
        rep->launches = (int32_t)(ctx->launches - l0);
    }
    return F4J_OK;
}

extern "C" int f4j_csr_mult_csr(f4j_ctx* ctx, f4j_csr A, f4j_csr B, f4j_csr* out, f4j_report* rep) {
    F4J_LOCK(ctx);
    return f4j_csr_mult_csr_ex(ctx, A, 0, B, 0, out, rep);
}

extern "C" int f4j_csr_transpose(f4j_ctx* ctx, f4j_csr S, f4j_csr* out) {
    F4J_LOCK(ctx);
    F4J_CHECK_CTX(ctx);
    if (!S || !out) return f4j_fail(F4J_ERR_ARG, "null argument");
    F4J_CUDA(cudaSetDevice(ctx->device));
    f4j_csr T;
    int rc = alloc_owned_csr(ctx, S->cols, S->rows, S->nnz, &T);
    if (rc) return rc;
    bool once = false, copied = false;
    rc = ensure_transpose(ctx, S, &once, (int*)T->colidx->ptr, &copied);
    if (rc) {
        f4j_csr_free(ctx, T);
        return rc;
    }
    F4J_CUDA(cudaMemcpyAsync(T->rowptr->ptr, S->t_rowptr, (size_t)(S->cols + 1) * 4, cudaMemcpyDeviceToDevice,
                             ctx->stream));
    if (!copied)
        F4J_CUDA(cudaMemcpyAsync(T->colidx->ptr, S->t_rowidx, (size_t)S->nnz * 4, cudaMemcpyDeviceToDevice, ctx->stream));
    if (S->nnz) {
        k_gather<double><<<grid1(S->nnz), 256, 0, ctx->stream>>>(S->nnz, (const int*)S->t_perm,
                                                                 (const double*)S->vals->ptr, (double*)T->vals->ptr);
        F4J_LAUNCHED(ctx);
    }
    drop_transpose(ctx, S, once);
    *out = T;
    return F4J_OK;
}

extern "C" int f4j_csr_transpose_perm(f4j_ctx* ctx, f4j_csr S, f4j_buf perm_out) {
    F4J_LOCK(ctx);
    F4J_CHECK_CTX(ctx);
    if (!S || !perm_out) return f4j_fail(F4J_ERR_ARG, "null argument");
    if (perm_out->bytes < (size_t)S->nnz * 4) return f4j_fail(F4J_ERR_ARG, "perm buffer too small");
    F4J_CUDA(cudaSetDevice(ctx->device));
    bool once = false;
    int rc = ensure_transpose(ctx, S, &once);
    if (rc) return rc;
    F4J_CUDA(cudaMemcpyAsync(perm_out->ptr, S->t_perm, (size_t)S->nnz * 4, cudaMemcpyDeviceToDevice, ctx->stream));
    drop_transpose(ctx, S, once);
    return F4J_OK;
}

extern "C" int f4j_spmv_ex(f4j_ctx* ctx, f4j_csr S, f4j_buf x, f4j_buf y, int mode, f4j_report* rep) {
    F4J_LOCK(ctx);
    F4J_CHECK_CTX(ctx);
    if (mode != F4J_SPARSE_EXACT && mode != F4J_SPARSE_FMA) return f4j_fail(F4J_ERR_ARG, "unknown sparse mode %d", mode);
    if (!S || !x || !y) return f4j_fail(F4J_ERR_ARG, "null argument");
    if (x->bytes < (size_t)S->cols * 8)
        return f4j_fail(F4J_ERR_ARG, "Expecting values to be equal but got: [%lld, %lld]", (long long)S->cols,
                        (long long)(x->bytes / 8));
    if (y->bytes < (size_t)S->rows * 8) return f4j_fail(F4J_ERR_ARG, "y buffer too small");
    if (!f4j_aligned(x->ptr, 8) || !f4j_aligned(y->ptr, 8)) return f4j_fail(F4J_ERR_ARG, "x and y must be 8-byte aligned");
    F4J_CUDA(cudaSetDevice(ctx->device));
    int64_t l0 = ctx->launches;
    if (S->rows) {
        // rows per warp: as many as fill every SM's resident blocks of 8 warps
        // once (216 at 2^20 rows), so the SMs finish together;
        // more rows per warp balance the lanes better, up to 256; at least 32
        const int64_t slots = (int64_t)ctx->sm_count * SPMV_BLOCKS * (SPMV_BLOCK / 32);
        int64_t rpw64 = f4j_cdiv(S->rows, slots);
        const int rpw = (int)(rpw64 < 32 ? 32 : (rpw64 > SPMV_RPW_MAX ? SPMV_RPW_MAX : rpw64));
        const unsigned blocks = (unsigned)f4j_cdiv(f4j_cdiv(S->rows, rpw), SPMV_BLOCK / 32);
        const bool fused = mode == F4J_SPARSE_FMA;
        // 32-byte loads of column indices and values when both arrays start 32-byte aligned
        const bool vec = f4j_aligned(S->colidx->ptr, 32) && f4j_aligned(S->vals->ptr, 32);
        auto kern = fused ? (vec ? k_spmv<true, true> : k_spmv<true, false>)
                          : (vec ? k_spmv<false, true> : k_spmv<false, false>);
        f4j_prof_begin(ctx);
        kern<<<blocks, SPMV_BLOCK, 0, ctx->stream>>>(S->rows, S->nnz, rpw, (const int*)S->rowptr->ptr,
                                                     (const int*)S->colidx->ptr, (const double*)S->vals->ptr,
                                                     (const double*)x->ptr, (double*)y->ptr);
        f4j_prof_end(ctx);
        F4J_LAUNCHED(ctx);
    }
    if (rep) {
        *rep = f4j_report{};
        rep->flops = 2.0 * S->nnz;
        rep->bytes = 12.0 * S->nnz + 4.0 * (S->rows + 1) + 8.0 * S->cols + 8.0 * S->rows;
        rep->launches = (int32_t)(ctx->launches - l0);
    }
    return F4J_OK;
}

extern "C" int f4j_spmv(f4j_ctx* ctx, f4j_csr S, f4j_buf x, f4j_buf y, f4j_report* rep) {
    F4J_LOCK(ctx);
    return f4j_spmv_ex(ctx, S, x, y, F4J_SPARSE_EXACT, rep);
}

extern "C" int f4j_spmm_ex(f4j_ctx* ctx, f4j_csr S, f4j_buf X, int64_t ncols, f4j_buf Y, int mode,
                           f4j_report* rep) {
    F4J_LOCK(ctx);
    F4J_CHECK_CTX(ctx);
    if (mode != F4J_SPARSE_EXACT && mode != F4J_SPARSE_FMA) return f4j_fail(F4J_ERR_ARG, "unknown sparse mode %d", mode);
    if (!S || !X || !Y) return f4j_fail(F4J_ERR_ARG, "null argument");
    if (ncols < 0) return f4j_fail(F4J_ERR_ARG, "negative column count");
    if (X->bytes < (size_t)S->cols * ncols * 8) return f4j_fail(F4J_ERR_ARG, "X buffer too small");
    if (Y->bytes < (size_t)S->rows * ncols * 8) return f4j_fail(F4J_ERR_ARG, "Y buffer too small");
    if (!f4j_aligned(X->ptr, 8) || !f4j_aligned(Y->ptr, 8)) return f4j_fail(F4J_ERR_ARG, "X and Y must be 8-byte aligned");
    F4J_CUDA(cudaSetDevice(ctx->device));
    int64_t l0 = ctx->launches;
    int rc = launch_spmm(ctx, S->rows, S->nnz, ncols, (const int*)S->rowptr->ptr, (const int*)S->colidx->ptr,
                         (const double*)S->vals->ptr, nullptr, (const double*)X->ptr, (double*)Y->ptr,
                         mode == F4J_SPARSE_FMA);
    if (rc) return rc;
    if (rep) {
        *rep = f4j_report{};
        rep->flops = 2.0 * S->nnz * ncols;
        rep->bytes = 12.0 * S->nnz + 4.0 * (S->rows + 1) + 8.0 * ncols * (S->cols + S->rows);
        rep->launches = (int32_t)(ctx->launches - l0);
    }
    return F4J_OK;
}

extern "C" int f4j_spmm(f4j_ctx* ctx, f4j_csr S, f4j_buf X, int64_t ncols, f4j_buf Y, f4j_report* rep) {
    F4J_LOCK(ctx);
    return f4j_spmm_ex(ctx, S, X, ncols, Y, F4J_SPARSE_EXACT, rep);
}

extern "C" int f4j_zspmm(f4j_ctx* ctx, f4j_csr S, f4j_buf X, int64_t ncols, f4j_buf Y, f4j_report* rep) {
    F4J_LOCK(ctx);
    F4J_CHECK_CTX(ctx);
    if (!S || !X || !Y) return f4j_fail(F4J_ERR_ARG, "null argument");
    if (ncols < 0) return f4j_fail(F4J_ERR_ARG, "negative column count");
    if (S->vals->bytes < (size_t)S->nnz * 16)
        return f4j_fail(F4J_ERR_ARG, "complex CSR values need 16 bytes per nonzero (nnz=%lld)", (long long)S->nnz);
    if (X->bytes < (size_t)S->cols * ncols * 16) return f4j_fail(F4J_ERR_ARG, "X buffer too small");
    if (Y->bytes < (size_t)S->rows * ncols * 16) return f4j_fail(F4J_ERR_ARG, "Y buffer too small");
    if (!f4j_aligned16(S->vals->ptr) || !f4j_aligned16(X->ptr) || !f4j_aligned16(Y->ptr))
        return f4j_fail(F4J_ERR_ARG, "complex buffers must be 16-byte aligned");
    F4J_CUDA(cudaSetDevice(ctx->device));
    int64_t l0 = ctx->launches;
    if (S->rows && ncols) {
        int G = 1;
        while (G < 32 && G < ncols) G *= 2;
        f4j_prof_begin(ctx);
        k_zspmm<<<(unsigned)f4j_cdiv(S->rows * G, 256), 256, 0, ctx->stream>>>(
            S->rows, ncols, G, (const int*)S->rowptr->ptr, (const int*)S->colidx->ptr, (const double2*)S->vals->ptr,
            (const double2*)X->ptr, (double2*)Y->ptr);
        f4j_prof_end(ctx);
        F4J_LAUNCHED(ctx);
    }
    if (rep) {
        *rep = f4j_report{};
        rep->flops = 8.0 * S->nnz * ncols;
        rep->bytes = 20.0 * S->nnz + 4.0 * (S->rows + 1) + 16.0 * ncols * (S->cols + S->rows);
        rep->launches = (int32_t)(ctx->launches - l0);
    }
    return F4J_OK;
}

extern "C" int f4j_spmm_t(f4j_ctx* ctx, f4j_csr S, f4j_buf dC, int64_t ncols, f4j_buf dX, f4j_report* rep) {
    F4J_LOCK(ctx);
    F4J_CHECK_CTX(ctx);
    if (!S || !dC || !dX) return f4j_fail(F4J_ERR_ARG, "null argument");
    if (ncols < 0) return f4j_fail(F4J_ERR_ARG, "negative column count");
    if (dC->bytes < (size_t)S->rows * ncols * 8) return f4j_fail(F4J_ERR_ARG, "dC buffer too small");
    if (dX->bytes < (size_t)S->cols * ncols * 8) return f4j_fail(F4J_ERR_ARG, "dX buffer too small");
    F4J_CUDA(cudaSetDevice(ctx->device));
    int64_t l0 = ctx->launches;
    bool once = false;
    int rc = ensure_transpose(ctx, S, &once);
    if (rc) return rc;
    rc = launch_spmm(ctx, S->cols, S->nnz, ncols, (const int*)S->t_rowptr, (const int*)S->t_rowidx,
                     (const double*)S->vals->ptr, (const int*)S->t_perm, (const double*)dC->ptr, (double*)dX->ptr);
    drop_transpose(ctx, S, once);
    if (rc) return rc;
    if (rep) {
        *rep = f4j_report{};
        rep->flops = 2.0 * S->nnz * ncols;
        rep->bytes = 16.0 * S->nnz + 4.0 * (S->cols + 1) + 8.0 * ncols * (S->cols + S->rows);
        rep->launches = (int32_t)(ctx->launches - l0);
    }
    return F4J_OK;
}

extern "C" int f4j_sddmm(f4j_ctx* ctx, f4j_csr S, f4j_buf A, f4j_buf B, int64_t ncols, f4j_buf out,
                         f4j_report* rep) {
    F4J_LOCK(ctx);
    F4J_CHECK_CTX(ctx);
    if (!S || !A || !B || !out) return f4j_fail(F4J_ERR_ARG, "null argument");
    if (ncols < 0) return f4j_fail(F4J_ERR_ARG, "negative column count");
    if (A->bytes < (size_t)S->rows * ncols * 8) return f4j_fail(F4J_ERR_ARG, "A buffer too small");
    if (B->bytes < (size_t)S->cols * ncols * 8) return f4j_fail(F4J_ERR_ARG, "B buffer too small");
    if (out->bytes < (size_t)S->nnz * 8) return f4j_fail(F4J_ERR_ARG, "output buffer too small");
    F4J_CUDA(cudaSetDevice(ctx->device));
    int64_t l0 = ctx->launches;
    if (S->rows && S->nnz) {
        f4j_prof_begin(ctx);
        // no room for the row of each nonzero, or a stream capture, which an allocation
        // kept in the handle must not be part of: k_sddmm, which needs none
        bool captured = false;
        int rc = S->rowidx ? F4J_OK : in_capture(ctx, &captured);
        if (!rc) rc = ncols >= 1 && ncols <= SD_FLAT_COLS && !captured ? ensure_rowidx(ctx, S) : F4J_ERR_OOM;
        if (rc && rc != F4J_ERR_OOM) return rc;
        if (rc == F4J_OK) {
            using Kernel = void (*)(int64_t, int64_t, int, int64_t, bool, const int*, const int*, const int*,
                                    const double*, const double*, double*);
            static const Kernel pairs[8] = {k_sddmm_flat<1, true>, k_sddmm_flat<2, true>, k_sddmm_flat<3, true>,
                                            k_sddmm_flat<4, true>, k_sddmm_flat<5, true>, k_sddmm_flat<6, true>,
                                            k_sddmm_flat<7, true>, k_sddmm_flat<8, true>};
            static const Kernel ones[5] = {k_sddmm_flat<1, false>, k_sddmm_flat<2, false>, k_sddmm_flat<4, false>,
                                           k_sddmm_flat<8, false>, k_sddmm_flat<16, false>};
            const double *a = (const double*)A->ptr, *b = (const double*)B->ptr;
            const bool even = ncols % 2 == 0 && f4j_aligned16(a) && f4j_aligned16(b);
            // more than 64 columns: equal parts of at most 56, whose sums k_sddmm_flat
            // keeps in four, added up in order.  57 to 63 columns go singly: eight
            // pairs a lane are built for 64 alone, where no unit is left over
            const int64_t part = ncols <= 64 ? 64 : f4j_cdiv(f4j_cdiv(ncols, f4j_cdiv(ncols, 56)), 8) * 8;
            for (int64_t c0 = 0; c0 < ncols; c0 += part) {
                const int w = (int)(ncols - c0 < part ? ncols - c0 : part);
                Kernel k;
                if (even && w > 4 && (w <= 56 || w == 64)) {  // up to four columns: a lane's pair leaves lanes idle
                    k = pairs[(w + 7) / 8 - 1];
                } else {
                    int i = 0;
                    while ((4 << i) < w) i++;
                    k = ones[i];
                }
                k<<<(unsigned)f4j_cdiv(S->nnz, 8 * SD_WARP), 256, 0, ctx->stream>>>(
                    S->rows, S->nnz, w, ncols, c0 > 0, (const int*)S->rowptr->ptr, (const int*)S->rowidx,
                    (const int*)S->colidx->ptr, a + c0, b + c0, (double*)out->ptr);
                if (c0 + part < ncols) ctx->launches++;
            }
        } else {
            k_sddmm<<<(unsigned)f4j_cdiv(S->rows * 32, 256), 256, 0, ctx->stream>>>(
                S->rows, ncols, (const int*)S->rowptr->ptr, (const int*)S->colidx->ptr, (const double*)A->ptr,
                (const double*)B->ptr, (double*)out->ptr);
        }
        f4j_prof_end(ctx);
        F4J_LAUNCHED(ctx);
    }
    if (rep) {
        *rep = f4j_report{};
        rep->flops = 2.0 * S->nnz * ncols;
        rep->bytes = 12.0 * S->nnz + 4.0 * (S->rows + 1) + 8.0 * ncols * (S->rows + S->cols);
        rep->launches = (int32_t)(ctx->launches - l0);
    }
    return F4J_OK;
}
