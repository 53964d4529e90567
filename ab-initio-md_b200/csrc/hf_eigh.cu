// Symmetric eigenproblem of the SCF loop for small molecules (n <= 64), by
// cyclic Jacobi rotations in one CTA (Golub & Van Loan, Matrix Computations,
// 8.5: parallel ordering, n/2 disjoint rotations a round).
//
// The library solver's tridiagonalisation and back-transformation are some
// hundred dependent launches at n = 50 (0.85 ms an SCF iteration of methanol
// 6-31G**, where the Fock build takes 0.3 ms). Here the matrix and the vectors
// stay in shared memory for all sweeps, and an iteration may start from the
// eigenvectors of the one before, in whose basis the matrix is nearly diagonal:
// two or three sweeps then, six or seven from scratch: SCF and gradient of
// methanol at two frames, 20 iterations, 39.5 -> 28.2 ms on one B200. Bound by the latency of
// a round (two barriers, a square root, shared-memory passes over both
// matrices). Above n = 64 a round's passes grow past what one SM does faster
// than the library.
#include <cstdio>

#include "../../include/aimd_b200.h"
#include "hf_eigh.h"

namespace {

constexpr int EIGH_THREADS = 512;
constexpr int EIGH_MAX_SWEEPS = 30;     // (a NaN matrix ends here)

__device__ double block_sum(double v, double* red) {
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    for (int w = 0; w < EIGH_THREADS / 32; ++w) t += red[w];
    return t;
}

// A: lower triangle of the matrix [n][n]; V [n][n]: eigenvectors in columns,
// ascending eigenvalues w; warm: V holds the starting vectors (orthonormal).
__global__ void __launch_bounds__(EIGH_THREADS) jacobi_kernel(int n, const double* __restrict__ Ain, double* V, double* w,
                                                              int warm) {
    extern __shared__ double sm[];
    __shared__ double red[EIGH_THREADS / 32], cs[AIMD_EIGH_MAX / 2], sn[AIMD_EIGH_MAX / 2];
    __shared__ int pi[AIMD_EIGH_MAX / 2], pj[AIMD_EIGH_MAX / 2];
    const int m = (n + 1) & ~1, ld = m + 1, h = m / 2;      // odd n: one idle row and column of zeros
    double *A = sm, *U = sm + m * ld, *T = sm + 2 * m * ld;
    for (int e = threadIdx.x; e < m * m; e += EIGH_THREADS) {
        const int i = e / m, j = e % m;
        const bool in = i < n && j < n;
        A[i * ld + j] = in ? Ain[(i > j ? i : j) * n + (i > j ? j : i)] : 0.0;
        U[i * ld + j] = in && warm ? V[i * n + j] : (i == j ? 1.0 : 0.0);
    }
    __syncthreads();
    if (warm) {         // A <- U^T A U
        for (int e = threadIdx.x; e < n * n; e += EIGH_THREADS) {
            const int i = e / n, j = e % n;
            double s = 0.0;
            for (int k = 0; k < n; ++k) s += A[i * ld + k] * U[k * ld + j];
            T[i * ld + j] = s;
        }
        __syncthreads();
        for (int e = threadIdx.x; e < n * n; e += EIGH_THREADS) {
            const int i = e / n, j = e % n;
            if (j > i) continue;
            double s = 0.0;
            for (int k = 0; k < n; ++k) s += U[k * ld + i] * T[k * ld + j];
            A[i * ld + j] = A[j * ld + i] = s;
        }
        __syncthreads();
    }
    double norm = 0.0;
    for (int e = threadIdx.x; e < m * m; e += EIGH_THREADS) norm += A[e / m * ld + e % m] * A[e / m * ld + e % m];
    norm = block_sum(norm, red);
    for (int sweep = 0; sweep < EIGH_MAX_SWEEPS; ++sweep) {
        double off = 0.0;
        for (int e = threadIdx.x; e < m * m; e += EIGH_THREADS) {
            const int i = e / m, j = e % m;
            if (i != j) off += A[i * ld + j] * A[i * ld + j];
        }
        off = block_sum(off, red);
        // convergence is quadratic: one sweep from 1e-13 of the norm ends at
        // rounding (uniform: every thread sums alike)
        if (off <= n * 1e-31 * norm) break;
        const bool last = off <= 1e-26 * norm;
        for (int r = 0; r < m - 1; ++r) {
            if (threadIdx.x < h) {
                const int p = threadIdx.x;
                int i = p == 0 ? m - 1 : (r + p) % (m - 1), j = p == 0 ? r : (r - p + m - 1) % (m - 1);
                if (i > j) {
                    const int t = i;
                    i = j;
                    j = t;
                }
                double c = 1.0, s = 0.0;
                const double aij = A[i * ld + j];
                if (j < n && fabs(aij) > 1e-300) {
                    const double th = (A[j * ld + j] - A[i * ld + i]) / (2.0 * aij);
                    const double t = copysign(1.0 / (fabs(th) + sqrt(1.0 + th * th)), th);
                    c = 1.0 / sqrt(1.0 + t * t);
                    s = t * c;
                }
                cs[p] = c;
                sn[p] = s;
                pi[p] = i;
                pj[p] = j;
            }
            __syncthreads();
            // one 2 x 2 block of A per pair of rotations, both sides at once
            for (int e = threadIdx.x; e < h * h; e += EIGH_THREADS) {
                const int p = e / h, q = e % h;
                const int i = pi[p] * ld, j = pj[p] * ld, k = pi[q], l = pj[q];
                const double c = cs[q], s = sn[q], a0 = A[i + k], a1 = A[i + l], b0 = A[j + k], b1 = A[j + l];
                const double x0 = c * a0 - s * a1, x1 = s * a0 + c * a1, y0 = c * b0 - s * b1, y1 = s * b0 + c * b1;
                const double d = cs[p], t = sn[p];
                A[i + k] = d * x0 - t * y0;
                A[i + l] = d * x1 - t * y1;
                A[j + k] = t * x0 + d * y0;
                A[j + l] = t * x1 + d * y1;
            }
            for (int e = threadIdx.x; e < n * h; e += EIGH_THREADS) {
                const int q = e % h;
                double* u = U + e / h * ld;
                const double c = cs[q], s = sn[q], u0 = u[pi[q]], u1 = u[pj[q]];
                u[pi[q]] = c * u0 - s * u1;
                u[pj[q]] = s * u0 + c * u1;
            }
            __syncthreads();
        }
        if (last) break;
    }
    // ascending order: the rank of each eigenvalue
    for (int i = threadIdx.x; i < n; i += EIGH_THREADS) {
        const double x = A[i * ld + i];
        int rank = 0;
        for (int k = 0; k < n; ++k) {
            const double y = A[k * ld + k];
            rank += y < x || (y == x && k < i);
        }
        T[i] = rank;
        w[rank] = x;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < n * n; e += EIGH_THREADS) V[e / n * n + (int)T[e % n]] = U[e / n * ld + e % n];
}

}  // namespace

namespace hf {
cudaError_t launch_eigh(int n, const double* A, double* V, double* w, int warm, cudaStream_t st) {
    const int m = (n + 1) & ~1;
    const size_t smem = sizeof(double) * 3 * m * (m + 1);
    static_assert(sizeof(double) * 3 * AIMD_EIGH_MAX * (AIMD_EIGH_MAX + 1) <= 227 * 1024 - 4096, "shared memory of a CTA");
    const cudaError_t r = cudaFuncSetAttribute(jacobi_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)(sizeof(double) * 3 * AIMD_EIGH_MAX * (AIMD_EIGH_MAX + 1)));
    if (r != cudaSuccess) return r;
    jacobi_kernel<<<1, EIGH_THREADS, smem, st>>>(n, A, V, w, warm);
    return cudaGetLastError();
}
}  // namespace hf
