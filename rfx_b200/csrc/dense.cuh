// Small dense FP64 linear algebra run inside one CTA (matrices of at most
// 128 x 128 held in shared memory): Cholesky with the inverse of its factor and
// a cyclic Jacobi eigensolver.  Used for the s x s Gram / Rayleigh-Ritz
// problems of the MDS and low-rank paths.
#pragma once
#include <cuda_runtime.h>

namespace rfx {

// Sum of part[q * stride], q = lane, lane + 32, ... < nparts, in that order,
// then a fixed shuffle tree over the warp; SUM_BATCH loads in flight at a time
// (a loop of one load and one add waits for each).
constexpr int SUM_BATCH = 20;
template <typename T>
__device__ __forceinline__ T warp_part_sum(const T* part, int nparts, size_t stride, int lane) {
    T v = 0;
    for (int q0 = lane; q0 < nparts; q0 += 32 * SUM_BATCH) {
        T x[SUM_BATCH];
#pragma unroll
        for (int u = 0; u < SUM_BATCH; ++u) x[u] = q0 + 32 * u < nparts ? part[(size_t)(q0 + 32 * u) * stride] : (T)0;
#pragma unroll
        for (int u = 0; u < SUM_BATCH; ++u)
            if (q0 + 32 * u < nparts) v += x[u];
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}

// Cholesky G = L L^T of the s x s SPD matrix in G (row-major, leading dim ld;
// L is left in the lower triangle) and the inverse of L in Linv (lower, zeros
// above).  Returns false (in every thread) if a pivot is not positive.  A
// finished column of L is subtracted from everything right of it at once, and
// a finished row of the inverse from the rows below, so a step's chain is one
// square root, one division and one product; the inverse runs one column
// behind on the second half of the threads.  Every entry takes its products in
// the order k = 0, 1, ....  blockDim.x is a multiple of 64.
__device__ inline bool cta_cholesky_inverse(double* G, double* Linv, int s, int ld, double* flag) {
    const int nt = blockDim.x / 2;
    const bool chol = (int)threadIdx.x < nt;
    const int tid = chol ? threadIdx.x : threadIdx.x - nt;
    for (int e = threadIdx.x; e < s * s; e += 2 * nt) Linv[(e / s) * ld + e % s] = e / s == e % s ? 1.0 : 0.0;
    if (threadIdx.x == 0) *flag = 1.0;
    __syncthreads();
    for (int j = 0; j <= s; ++j) {
        const int k = j - 1;  // the inverse's row
        double djj = 0.0;
        if (chol) {
            if (j < s) {
                const double d = G[j * ld + j];
                const bool good = d > 0.0;
                djj = sqrt(good ? d : 1.0);
                if (tid == 0 && !good) *flag = 0.0;
                for (int i = j + 1 + tid; i < s; i += nt) G[i * ld + j] = G[i * ld + j] / djj;
            }
        } else if (k >= 0) {
            const double lkk = G[k * ld + k];
            for (int c = tid; c <= k; c += nt) Linv[k * ld + c] = Linv[k * ld + c] / lkk;
        }
        __syncthreads();
        if (chol) {
            if (j < s) {
                if (tid == 0) G[j * ld + j] = djj;
                // 16 x (nt / 16) threads over the remaining lower triangle
                for (int i = j + 1 + tid / 16; i < s; i += nt / 16) {
                    const double lij = G[i * ld + j];
                    for (int q = j + 1 + tid % 16; q <= i; q += 16)
                        G[i * ld + q] = fma(-lij, G[q * ld + j], G[i * ld + q]);
                }
            }
        } else if (k >= 0) {
            for (int r = k + 1 + tid / 16; r < s; r += nt / 16) {
                const double lrk = G[r * ld + k];
                for (int c = tid % 16; c <= k; c += 16)
                    Linv[r * ld + c] = fma(-lrk, Linv[k * ld + c], Linv[r * ld + c]);
            }
        }
        __syncthreads();
    }
    return *flag > 0.5;
}

// Cyclic Jacobi eigendecomposition of the symmetric s x s matrix A (destroyed;
// s even):
// eigenvalues on the diagonal of A, eigenvectors in the columns of V.
// Rotations of disjoint index pairs are applied in parallel (round-robin
// ordering); at most `sweeps` full sweeps, fewer once every off-diagonal entry
// is at FP64 rounding relative to its diagonal pair, or (abs_tol > 0) below
// abs_tol times the largest diagonal magnitude: the absolute stop ends a
// spectrum with eigenvalues near zero, whose relative test rounding keeps
// open, and leaves the large eigenpairs accurate to abs_tol.  A leading
// dimension ld = s + 1 keeps the column passes free of shared-memory bank
// conflicts.
__device__ inline void cta_jacobi(double* A, double* V, int s, int ld, int sweeps, int* pairs, double abs_tol = 0.0) {
    const int tid = threadIdx.x, nt = blockDim.x;
    for (int e = tid; e < s * s; e += nt) V[(e / s) * ld + (e % s)] = ((e / s) == (e % s)) ? 1.0 : 0.0;
    __syncthreads();
    const int m = s;  // round-robin over an even count
    __shared__ double cs[64][2];
    for (int sw = 0; sw < sweeps; ++sw) {
        // converged when every off-diagonal entry is negligible against its
        // diagonal pair, |a_pq| <= 1e-16 sqrt(|a_pp a_qq|) (the relative
        // criterion, which keeps small eigenvalues accurate)
        double floor2 = 0.0;
        if (abs_tol > 0.0) {
            double dmax = 0.0;
            for (int r = 0; r < s; ++r) dmax = fmax(dmax, fabs(A[r * ld + r]));
            floor2 = (abs_tol * dmax) * (abs_tol * dmax);
        }
        int active = 0;
        for (int e = tid; e < s * s; e += nt) {
            const int r = e / s, q = e % s;
            if (r < q) {
                const double v = A[r * ld + q];
                if (v * v > 1e-32 * fabs(A[r * ld + r] * A[q * ld + q]) && v * v > floor2) active = 1;
            }
        }
        if (!__syncthreads_or(active)) break;
        for (int round = 0; round < m - 1; ++round) {
            // round-robin tournament: index 0 stays, indices 1..m-1 rotate;
            // pair k joins positions k and m-1-k
            // (the thread that numbers pair k also computes its rotation; the
            // barrier below publishes both)
            int rot = 0;
            for (int k = tid; k < m / 2; k += nt) {
                const int pa = k, pb = m - 1 - k;
                const int a = (pa == 0) ? 0 : ((pa - 1 + round) % (m - 1)) + 1;
                const int b = ((pb - 1 + round) % (m - 1)) + 1;
                const int p = min(a, b), q = max(a, b);
                pairs[2 * k] = p;
                pairs[2 * k + 1] = q;
                double c = 1.0, sn = 0.0;
                {
                    const double apq = A[p * ld + q];
                    // entries already below the stop test are not rotated
                    if (fabs(apq) > 1e-300 && apq * apq > 1e-32 * fabs(A[p * ld + p] * A[q * ld + q]) &&
                        apq * apq > floor2) {
                        rot = 1;
                        const double app = A[p * ld + p], aqq = A[q * ld + q];
                        const double tau = (aqq - app) / (2.0 * apq);
                        const double t = (tau >= 0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
                        c = 1.0 / sqrt(1.0 + t * t);
                        sn = t * c;
                    }
                }
                cs[k][0] = c;
                cs[k][1] = sn;
            }
            // a round without a rotation leaves A and V as they are
            if (!__syncthreads_or(rot)) continue;
            // A <- J^T A J by 2 x 2 blocks (rows of pair k1, columns of pair
            // k2): the row rotation, then the column rotation, each entry
            // loaded and stored once; V <- V J in the same pass
            const int h = m / 2, nw = nt >> 5, w = tid >> 5, lane = tid & 31;
            for (int task = w; task < 2 * h; task += nw) {
                const int k1 = task < h ? task : task - h;
                const int p1 = pairs[2 * k1], q1 = pairs[2 * k1 + 1];
                const double c1 = cs[k1][0], s1 = cs[k1][1];
                if (task < h) {
                    for (int k2 = lane; k2 < h; k2 += 32) {
                        const int p2 = pairs[2 * k2], q2 = pairs[2 * k2 + 1];
                        const double c2 = cs[k2][0], s2 = cs[k2][1];
                        const double pp = A[p1 * ld + p2], qp = A[q1 * ld + p2];
                        const double pq = A[p1 * ld + q2], qq = A[q1 * ld + q2];
                        const double rpp = c1 * pp - s1 * qp, rqp = s1 * pp + c1 * qp;
                        const double rpq = c1 * pq - s1 * qq, rqq = s1 * pq + c1 * qq;
                        A[p1 * ld + p2] = c2 * rpp - s2 * rpq;
                        A[p1 * ld + q2] = s2 * rpp + c2 * rpq;
                        A[q1 * ld + p2] = c2 * rqp - s2 * rqq;
                        A[q1 * ld + q2] = s2 * rqp + c2 * rqq;
                    }
                } else {
                    for (int r = lane; r < s; r += 32) {
                        const double vp = V[r * ld + p1], vq = V[r * ld + q1];
                        V[r * ld + p1] = c1 * vp - s1 * vq;
                        V[r * ld + q1] = s1 * vp + c1 * vq;
                    }
                }
            }
            __syncthreads();
        }
    }
}

}  // namespace rfx
