// Symmetric eigenproblem of the SCF loop for small molecules (n <= 64), by
// cyclic Jacobi rotations in one CTA (Golub & Van Loan, Matrix Computations,
// 8.5: parallel ordering, n/2 disjoint rotations a round).
//
// The library solver's tridiagonalisation and back-transformation are some
// hundred dependent launches at n = 50 (0.85 ms an SCF iteration of methanol
// 6-31G**, where the Fock build takes 0.3 ms). Here the matrix and the vectors
// stay in shared memory for all sweeps, and an iteration may start from the
// eigenvectors of the one before, in whose basis the matrix is nearly diagonal:
// two or three sweeps then, seven or eight from scratch: SCF and gradient of
// methanol at two frames, 20 iterations, 39.5 -> 28.2 ms on one B200. Bound by the
// latency of a round (two barriers, a square root, shared-memory passes over both
// matrices). The limit of 64 is where a start from scratch meets the library, and
// one block of rotations a thread fills the CTA (us, one B200, from nearby vectors
// / from scratch / library): n = 16 56 / 98 / 198, 32 113 / 236 / 283,
// 48 217 / 461 / 776, 64 354 / 846 / 936.
#include <cstdio>

#include "../../include/aimd_b200.h"
#include "hf_eigh.h"

namespace {

// Pair p of the m/2 disjoint pairs of a round (the circle method on m players,
// m - 1 rounds): pair 0 is player m - 1 against the round's number, the others
// move on by one each round, so that a thread needs no index arithmetic and no
// shared table to follow its pair.
struct Pair {
    int i, j;
    __device__ Pair(int p, int m) : i(p == 0 ? m - 1 : p), j(p == 0 ? 0 : m - 1 - p) {}
    __device__ void advance(int m) {
        if (i != m - 1) i = i + 1 == m - 1 ? 0 : i + 1;
        j = j + 1 == m - 1 ? 0 : j + 1;
    }
};

constexpr int EIGH_THREADS = 1024;     // one 2 x 2 block of rotations a thread at n = 64
constexpr int EIGH_MAX_SWEEPS = 30;     // (random matrices of n = 64 take 8)
constexpr double ROT_SMALL = 1e-5;      // sine of a rotation that does not disturb the others of its sweep

__device__ double block_sum(double v, double* red) {
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    for (int w = 0; w < EIGH_THREADS / 32; ++w) t += red[w];
    return t;
}

__device__ double block_max(double v, double* red) {
    for (int d = 16; d > 0; d >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, d));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    for (int w = 0; w < EIGH_THREADS / 32; ++w) t = fmax(t, red[w]);
    return t;
}

// A: lower triangle of the matrix [n][n]; V [n][n]: eigenvectors in columns,
// ascending eigenvalues w; warm: V holds the starting vectors (orthonormal).
// All of V and w are NaN if an element of A or of the starting vectors is not
// finite, or if the sweeps do not end.
__global__ void __launch_bounds__(EIGH_THREADS) jacobi_kernel(int n, const double* __restrict__ Ain, double* V, double* w,
                                                              int warm) {
    extern __shared__ double sm[];
    __shared__ double red[EIGH_THREADS / 32];
    __shared__ double2 rot[AIMD_EIGH_MAX / 2];              // (cos, sin) of the round's rotations
    const int m = (n + 1) & ~1, ld = m + 1, h = m / 2;      // odd n: one idle row and column of zeros
    static_assert(AIMD_EIGH_MAX * AIMD_EIGH_MAX / 2 <= 2 * EIGH_THREADS, "two rotations of the vectors a thread");
    const int e0 = threadIdx.x, e1 = threadIdx.x + EIGH_THREADS;
    auto rotate = [](double* u, const Pair& q, double2 g) {
        const double u0 = u[q.i], u1 = u[q.j];
        u[q.i] = g.x * u0 - g.y * u1;
        u[q.j] = g.y * u0 + g.x * u1;
    };
    double *A = sm, *U = sm + m * ld, *T = sm + 2 * m * ld;
    bool finite = true;
    double big = 0.0;
    for (int e = threadIdx.x; e < m * m; e += EIGH_THREADS) {
        const int i = e / m, j = e % m;
        const bool in = i < n && j < n;
        const double a = in ? Ain[(i > j ? i : j) * n + (i > j ? j : i)] : 0.0;
        const double u = in && warm ? V[i * n + j] : (i == j ? 1.0 : 0.0);
        finite &= isfinite(a) && isfinite(u);
        big = fmax(big, fabs(a));
        A[i * ld + j] = a;
        U[i * ld + j] = u;
    }
    auto fail = [&] {
        for (int e = threadIdx.x; e < n * n; e += EIGH_THREADS) V[e] = nan("");
        for (int i = threadIdx.x; i < n; i += EIGH_THREADS) w[i] = nan("");
    };
    if (__syncthreads_or(!finite)) return fail();
    // elements up to 1 by a power of two (exact): their squares stay in range
    int ex;
    frexp(block_max(big, red), &ex);
    for (int e = threadIdx.x; e < m * m; e += EIGH_THREADS) A[e / m * ld + e % m] = scalbn(A[e / m * ld + e % m], -ex);
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
    for (int sweep = 0;; ++sweep) {
        if (sweep == EIGH_MAX_SWEEPS) return fail();
        double off = 0.0;
        for (int e = threadIdx.x; e < m * m; e += EIGH_THREADS) {
            const int i = e / m, j = e % m;
            if (i != j) off += A[i * ld + j] * A[i * ld + j];
        }
        off = block_sum(off, red);
        if (off <= n * 1e-31 * norm) break;     // at rounding (uniform: every thread sums alike)
        // A sweep of rotations by at most ROT_SMALL leaves n ROT_SMALL times
        // what it met: from 1e-13 of the norm on that is below rounding, and
        // another sum of the squares is saved. Larger rotations at such an off
        // are those of eigenvalues as close as the off-diagonal elements; they
        // fill in what the sweep had cleared, so it is tested again
        // (I + 1e-13 R, n = 64: residual 6e-14 of the norm without the test).
        const bool small = off <= 1e-26 * norm;
        bool turned = false;
        Pair rp(threadIdx.x < h ? threadIdx.x : 0, m), bp(e0 < h * h ? e0 / h : 0, m), bq(e0 % h, m), v0(e0 % h, m), v1(e1 % h, m);
        for (int r = 0; r < m - 1; ++r) {
            if (threadIdx.x < h) {
                const int i = rp.i, j = rp.j;
                double c = 1.0, s = 0.0;
                const double aij = A[i * ld + j];
                if (i < n && j < n && fabs(aij) > 1e-300) {
                    const double th = (A[j * ld + j] - A[i * ld + i]) / (2.0 * aij);
                    const double t = copysign(1.0 / (fabs(th) + sqrt(1.0 + th * th)), th);
                    c = 1.0 / sqrt(1.0 + t * t);
                    s = t * c;
                    turned |= fabs(s) > ROT_SMALL;
                }
                rot[threadIdx.x] = make_double2(c, s);
            }
            __syncthreads();
            // one 2 x 2 block of A per pair of rotations, both sides at once
            if (e0 < h * h) {
                const int i = bp.i * ld, j = bp.j * ld, k = bq.i, l = bq.j;
                const double2 q = rot[e0 % h], p = rot[e0 / h];
                const double a0 = A[i + k], a1 = A[i + l], b0 = A[j + k], b1 = A[j + l];
                const double x0 = q.x * a0 - q.y * a1, x1 = q.y * a0 + q.x * a1, y0 = q.x * b0 - q.y * b1, y1 = q.y * b0 + q.x * b1;
                A[i + k] = p.x * x0 - p.y * y0;
                A[i + l] = p.x * x1 - p.y * y1;
                A[j + k] = p.y * x0 + p.x * y0;
                A[j + l] = p.y * x1 + p.x * y1;
                // the rotated element itself is zero: its rounding, relative to
                // the diagonal, would keep off above the limit
                if (bp.i == bq.i) A[i + l] = A[j + k] = 0.0;
            }
            if (e0 < n * h) rotate(U + e0 / h * ld, v0, rot[e0 % h]);
            if (e1 < n * h) rotate(U + e1 / h * ld, v1, rot[e1 % h]);
            rp.advance(m);
            bp.advance(m);
            bq.advance(m);
            v0.advance(m);
            v1.advance(m);
            __syncthreads();
        }
        if (!__syncthreads_or(turned) && small) break;
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
        w[rank] = scalbn(x, ex);
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
