// One-electron integrals and their nuclear-derivative contractions.
//
// One warp per segmented shell pair (si >= sj), class-templated on
// (l_i, l_j). Overlap-type integrals use t = 0 Hermite coefficients
// (E^{ij}_0 sqrt(pi/p) per direction), kinetic energy the 1-D second
// derivative identity, the dipole E^{ij}_1 + X_PO E^{ij}_0, and the nuclear
// attraction the Hermite Coulomb integrals R_tuv(p, P - C).
// (The reference's _overlap_type_kernel, _nuclear_kernel,
// _overlap_kinetic_grad_kernel and _nuclear_grad_kernel,
// aimd/qc/integrals.py:155-501.)
//
// The lanes share a pair's primitive pairs (overlap, kinetic, dipole), and its
// (primitive pair, nucleus) combinations (attraction): a pair of contracted s
// shells carries up to 64 primitive pairs times every nucleus, which one
// thread a pair worked through alone while the device waited for it; and the
// nuclei's forces went through compare-and-swap loops on one address a warp.
// Bound by FP64 issue now; the Boys function comes from the shared table. (H2O)32 cc-pVDZ on one B200, all six classes:
// integrals 5.0 -> 1.0 ms, gradient 23.5 -> 1.6 ms.
#pragma once
#include "hf_eri.cuh"

namespace hf {

struct ShellView {
    int nshell, natm, nao;
    const int* atom;
    const int* l;
    const int* ao;
    const int* p0;      // first primitive
    const int* np;      // primitive count
    const double* exps;
    const double* coefs;
    const double* pos;  // [natm][3]
    const double* charges;
    const int* pair_i;  // shell pairs (si >= sj), grouped by class (li, lj) with li >= lj
    const int* pair_j;
    const double* boys; // Boys tables of all orders
};

// -1/2 <i| d^2/dx^2 |j> from overlap factors e[i][j][0] (j up to J+2 present)
template <int IM, int JM>
__device__ __forceinline__ double kin1d(const double (&e)[IM + 1][JM + 1][IM + JM + 1], int i, int j, double b) {
    double v = -2.0 * b * (2 * j + 1) * e[i][j][0] + 4.0 * b * b * e[i][j + 2][0];
    if (j >= 2) v += j * (j - 1) * e[i][j - 2][0];
    return -0.5 * v;
}

constexpr int ONEE_THREADS = 128;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}

// Lanes of a warp over (primitive pair, nucleus): al lanes along the nuclei
// (the power of two from natm on, at most 32), 32 / al along the primitives.
__device__ __forceinline__ int atom_lanes(int natm) {
    int al = 1;
    while (al < natm && al < 32) al <<= 1;
    return al;
}

// S, T, dipole (about origin o) and V for shell pairs of class (LI, LJ);
// pairs [p_begin, p_end) of the class-sorted shell-pair list.
template <int LI, int LJ>
__global__ void __launch_bounds__(ONEE_THREADS) onee_kernel(ShellView sv, int p_begin, int p_end, double ox, double oy,
                                                            double oz, double* S, double* T, double* M, double* V) {
    constexpr int NI = ncart(LI), NJ = ncart(LJ), L = LI + LJ;
    using Boys = BoysOf<L, double, true>;
    extern __shared__ __align__(16) double smem[];      // Boys table
    Boys::stage(sv.boys, smem);
    __syncthreads();
    const auto boys = Boys::get(smem);
    const int lane = threadIdx.x & 31, nwarp = gridDim.x * (ONEE_THREADS / 32);
    const int al = atom_lanes(sv.natm), c0 = lane & (al - 1), k0 = lane / al, kl = 32 / al;
    const double sqpi = sqrt(PI);
    for (int ip = p_begin + blockIdx.x * (ONEE_THREADS / 32) + (threadIdx.x >> 5); ip < p_end; ip += nwarp) {
        const int si = sv.pair_i[ip], sj = sv.pair_j[ip];
        const int ai = sv.atom[si], aj = sv.atom[sj];
        const double Ax = sv.pos[3 * ai], Ay = sv.pos[3 * ai + 1], Az = sv.pos[3 * ai + 2];
        const double Bx = sv.pos[3 * aj], By = sv.pos[3 * aj + 1], Bz = sv.pos[3 * aj + 2];
        const double ABx = Ax - Bx, ABy = Ay - By, ABz = Az - Bz;
        const int nb = sv.np[sj], np = sv.np[si] * nb;
        double s[NI][NJ] = {}, t[NI][NJ] = {}, mx[NI][NJ] = {}, my[NI][NJ] = {}, mz[NI][NJ] = {}, vv[NI][NJ] = {};
        for (int k = lane; k < np; k += 32) {
            const int ka = sv.p0[si] + k / nb, kb = sv.p0[sj] + k % nb;
            const double a = sv.exps[ka], b = sv.exps[kb], p = a + b, mu = a * b / p, oo2p = 0.5 / p, bp = b / p, ap = a / p;
            const double cc = sv.coefs[ka] * sv.coefs[kb];
            const double sq = sqpi / sqrt(p);
            double ex[LI + 1][LJ + 3][L + 3], ey[LI + 1][LJ + 3][L + 3], ez[LI + 1][LJ + 3][L + 3];
            hermite_e<LI, LJ + 2>(-bp * ABx, ap * ABx, oo2p, exp(-mu * ABx * ABx) * sq * cc, ex);
            hermite_e<LI, LJ + 2>(-bp * ABy, ap * ABy, oo2p, exp(-mu * ABy * ABy) * sq, ey);
            hermite_e<LI, LJ + 2>(-bp * ABz, ap * ABz, oo2p, exp(-mu * ABz * ABz) * sq, ez);
            const double Px = (a * Ax + b * Bx) / p - ox, Py = (a * Ay + b * By) / p - oy, Pz = (a * Az + b * Bz) / p - oz;
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const int ix = cart_x(LI, i), iy = cart_y(LI, i), iz = cart_z(LI, i);
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    const int jx = cart_x(LJ, j), jy = cart_y(LJ, j), jz = cart_z(LJ, j);
                    const double sx = ex[ix][jx][0], sy = ey[iy][jy][0], sz = ez[iz][jz][0];
                    s[i][j] += sx * sy * sz;
                    t[i][j] += kin1d<LI, LJ + 2>(ex, ix, jx, b) * sy * sz + sx * kin1d<LI, LJ + 2>(ey, iy, jy, b) * sz +
                               sx * sy * kin1d<LI, LJ + 2>(ez, iz, jz, b);
                    mx[i][j] += (ex[ix][jx][1] + Px * sx) * sy * sz;
                    my[i][j] += sx * (ey[iy][jy][1] + Py * sy) * sz;
                    mz[i][j] += sx * sy * (ez[iz][jz][1] + Pz * sz);
                }
            }
        }
        for (int k = k0; k < np; k += kl) {
            const int ka = sv.p0[si] + k / nb, kb = sv.p0[sj] + k % nb;
            const double a = sv.exps[ka], b = sv.exps[kb], p = a + b, ip_ = 1.0 / p, mu = a * b * ip_, bp = b * ip_,
                         ap = a * ip_;
            // nuclear attraction: rsum_h = sum_C (-Z_C 2 pi / p) R_h(p, P - C) over this lane's nuclei
            double rsum[nherm(L)];
#pragma unroll
            for (int h = 0; h < nherm(L); ++h) rsum[h] = 0.0;
            for (int c = c0; c < sv.natm; c += al) {
                double R[nherm(L)];
                hermite_r<L>(p, (Ax - sv.pos[3 * c]) - bp * ABx, (Ay - sv.pos[3 * c + 1]) - bp * ABy,
                             (Az - sv.pos[3 * c + 2]) - bp * ABz, R, boys);
                const double w = -sv.charges[c] * 2.0 * PI * ip_;
#pragma unroll
                for (int h = 0; h < nherm(L); ++h) rsum[h] += w * R[h];
            }
            double ex[LI + 1][LJ + 1][L + 1], ey[LI + 1][LJ + 1][L + 1], ez[LI + 1][LJ + 1][L + 1];
            const double e00 = exp(-mu * (ABx * ABx + ABy * ABy + ABz * ABz)) * sv.coefs[ka] * sv.coefs[kb];
            hermite_e<LI, LJ>(-bp * ABx, ap * ABx, 0.5 * ip_, e00, ex);
            hermite_e<LI, LJ>(-bp * ABy, ap * ABy, 0.5 * ip_, 1.0, ey);
            hermite_e<LI, LJ>(-bp * ABz, ap * ABz, 0.5 * ip_, 1.0, ez);
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const int ix = cart_x(LI, i), iy = cart_y(LI, i), iz = cart_z(LI, i);
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    const int jx = cart_x(LJ, j), jy = cart_y(LJ, j), jz = cart_z(LJ, j);
                    double acc = 0.0;
#pragma unroll
                    for (int tt = 0; tt <= ix + jx; ++tt)
#pragma unroll
                        for (int uu = 0; uu <= iy + jy; ++uu) {
                            const double exy = ex[ix][jx][tt] * ey[iy][jy][uu];
#pragma unroll
                            for (int ww = 0; ww <= iz + jz; ++ww) acc += exy * ez[iz][jz][ww] * rsum[hidx(tt, uu, ww)];
                        }
                    vv[i][j] += acc;
                }
            }
        }
        const int n = sv.nao, oi = sv.ao[si], oj = sv.ao[sj];
        const size_t nn = (size_t)n * n;
#pragma unroll
        for (int i = 0; i < NI; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const double f = cart_norm(cart_x(LI, i), cart_y(LI, i), cart_z(LI, i)) *
                                 cart_norm(cart_x(LJ, j), cart_y(LJ, j), cart_z(LJ, j));
                const size_t a1 = (size_t)(oi + i) * n + oj + j, a2 = (size_t)(oj + j) * n + oi + i;
                const double o[6] = {f * warp_sum(s[i][j]),  f * warp_sum(t[i][j]),  f * warp_sum(mx[i][j]),
                                     f * warp_sum(my[i][j]), f * warp_sum(mz[i][j]), f * warp_sum(vv[i][j])};
                // a diagonal block holds both (i, j) and (j, i) already
                if (lane == 0 || (lane == 1 && si != sj)) {
                    const size_t at = lane == 0 ? a1 : a2;
                    S[at] = o[0];
                    T[at] = o[1];
                    M[at] = o[2];
                    M[nn + at] = o[3];
                    M[2 * nn + at] = o[4];
                    V[at] = o[5];
                }
            }
    }
}

// d/dR [ sum W S + sum D T ] (W with the sign the caller wants) and
// d/dR sum D V for shell pairs of class (LI, LJ); CTA-shared accumulator.
// Attraction: with Y the density-contracted Hermite vector of a primitive pair
// and dY its derivative at X = A - B (hermite_de), per nucleus C
//   G = w sum_h Y_h R_{h+1}(P - C),  U = w sum_h dY_h R_h
//   dA = (a/p) G + U,  dB = (b/p) G - U,  dC = -G.
template <int LI, int LJ>
__global__ void __launch_bounds__(ONEE_THREADS) onee_grad_kernel(ShellView sv, int p_begin, int p_end,
                                                                 const double* W, const double* Dm, facc* grad) {
    using Boys = BoysOf<LI + LJ + 1, double, true>;
    extern __shared__ __align__(16) double smem[];      // Boys table, then the accumulator
    unsigned* gsh = reinterpret_cast<unsigned*>(smem + Boys::elems);    // low words [natm][3], then the high words
    const int n3 = 3 * sv.natm;
    for (int i = threadIdx.x; i < 2 * n3; i += blockDim.x) gsh[i] = 0u;
    Boys::stage(sv.boys, smem);
    __syncthreads();
    const auto boys = Boys::get(smem);
    auto gadd = [&](int i, double v) { sadd(gsh + i, gsh + n3 + i, v, FIX_G); };
    constexpr int NI = ncart(LI), NJ = ncart(LJ), L = LI + LJ, NH = nherm(L);
    const int lane = threadIdx.x & 31, nwarp = gridDim.x * (ONEE_THREADS / 32);
    const int al = atom_lanes(sv.natm), c0 = lane & (al - 1), k0 = lane / al, kl = 32 / al;
    const double sqpi = sqrt(PI);
    for (int ip = p_begin + blockIdx.x * (ONEE_THREADS / 32) + (threadIdx.x >> 5); ip < p_end; ip += nwarp) {
        const int si = sv.pair_i[ip], sj = sv.pair_j[ip];
        const int ai = sv.atom[si], aj = sv.atom[sj];
        const int n = sv.nao, oi = sv.ao[si], oj = sv.ao[sj];
        const double Ax = sv.pos[3 * ai], Ay = sv.pos[3 * ai + 1], Az = sv.pos[3 * ai + 2];
        const double ABx = Ax - sv.pos[3 * aj], ABy = Ay - sv.pos[3 * aj + 1], ABz = Az - sv.pos[3 * aj + 2];
        const double sym = si != sj ? 2.0 : 1.0;
        const int nb = sv.np[sj], np = sv.np[si] * nb;
        double dv[NI][NJ];
#pragma unroll
        for (int i = 0; i < NI; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const double f = cart_norm(cart_x(LI, i), cart_y(LI, i), cart_z(LI, i)) *
                                 cart_norm(cart_x(LJ, j), cart_y(LJ, j), cart_z(LJ, j));
                dv[i][j] = f * Dm[(size_t)(oi + i) * n + oj + j];
            }
        double gA[3] = {0.0, 0.0, 0.0}, gB[3] = {0.0, 0.0, 0.0};
        // overlap and kinetic (only between different atoms; pairs si > sj)
        if (ai != aj) {
            for (int k = lane; k < np; k += 32) {
                const int ka = sv.p0[si] + k / nb, kb = sv.p0[sj] + k % nb;
                const double a = sv.exps[ka], b = sv.exps[kb], p = a + b, mu = a * b / p, oo2p = 0.5 / p, bp = b / p,
                             ap = a / p;
                const double cc = sv.coefs[ka] * sv.coefs[kb];
                const double sq = sqpi / sqrt(p);
                double ex[LI + 2][LJ + 3][L + 4], ey[LI + 2][LJ + 3][L + 4], ez[LI + 2][LJ + 3][L + 4];
                hermite_e<LI + 1, LJ + 2>(-bp * ABx, ap * ABx, oo2p, exp(-mu * ABx * ABx) * sq * cc, ex);
                hermite_e<LI + 1, LJ + 2>(-bp * ABy, ap * ABy, oo2p, exp(-mu * ABy * ABy) * sq, ey);
                hermite_e<LI + 1, LJ + 2>(-bp * ABz, ap * ABz, oo2p, exp(-mu * ABz * ABz) * sq, ez);
                double g[3] = {0.0, 0.0, 0.0};
#pragma unroll
                for (int i = 0; i < NI; ++i)
#pragma unroll
                    for (int j = 0; j < NJ; ++j) {
                        const int I3[3] = {cart_x(LI, i), cart_y(LI, i), cart_z(LI, i)};
                        const int J3[3] = {cart_x(LJ, j), cart_y(LJ, j), cart_z(LJ, j)};
                        const double f = cart_norm(I3[0], I3[1], I3[2]) * cart_norm(J3[0], J3[1], J3[2]);
                        double S1[3], K1[3], dS[3], dK[3];
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            const auto& e = d == 0 ? ex : (d == 1 ? ey : ez);
                            const int ii = I3[d], jj = J3[d];
                            S1[d] = e[ii][jj][0];
                            K1[d] = kin1d<LI + 1, LJ + 2>(e, ii, jj, b);
                            dS[d] = 2.0 * a * e[ii + 1][jj][0];
                            dK[d] = 2.0 * a * kin1d<LI + 1, LJ + 2>(e, ii + 1, jj, b);
                            if (ii > 0) {
                                dS[d] -= ii * e[ii - 1][jj][0];
                                dK[d] -= ii * kin1d<LI + 1, LJ + 2>(e, ii - 1, jj, b);
                            }
                        }
                        const double w2 = 2.0 * f * W[(size_t)(oi + i) * n + oj + j], d2 = 2.0 * dv[i][j];
                        g[0] += w2 * dS[0] * S1[1] * S1[2] + d2 * (dK[0] * S1[1] * S1[2] + dS[0] * (K1[1] * S1[2] + S1[1] * K1[2]));
                        g[1] += w2 * S1[0] * dS[1] * S1[2] + d2 * (dK[1] * S1[0] * S1[2] + dS[1] * (K1[0] * S1[2] + S1[0] * K1[2]));
                        g[2] += w2 * S1[0] * S1[1] * dS[2] + d2 * (dK[2] * S1[0] * S1[1] + dS[2] * (K1[0] * S1[1] + S1[0] * K1[1]));
                    }
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    gA[d] += g[d];
                    gB[d] -= g[d];
                }
            }
        }
        // nuclear attraction
        for (int k = k0; k < np; k += kl) {
            const int ka = sv.p0[si] + k / nb, kb = sv.p0[sj] + k % nb;
            const double a = sv.exps[ka], b = sv.exps[kb], p = a + b, ip_ = 1.0 / p, mu = a * b * ip_, bp = b * ip_,
                         ap = a * ip_;
            double Y[NH], U[3][NH];
            {
                double e[3][LI + 1][LJ + 1][L + 1], de[3][LI + 1][LJ + 1][L + 1];
                const double e00 = exp(-mu * (ABx * ABx + ABy * ABy + ABz * ABz)) * sv.coefs[ka] * sv.coefs[kb] * sym;
                const double AB[3] = {ABx, ABy, ABz};
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    hermite_e<LI, LJ>(-bp * AB[d], ap * AB[d], 0.5 * ip_, d == 0 ? e00 : 1.0, e[d]);
                    hermite_de<LI, LJ>(-bp * AB[d], ap * AB[d], 0.5 * ip_, bp, ap, 2.0 * mu * AB[d], e[d], de[d]);
                }
#pragma unroll
                for (int h = 0; h < NH; ++h) Y[h] = U[0][h] = U[1][h] = U[2][h] = 0.0;
#pragma unroll
                for (int i = 0; i < NI; ++i)
#pragma unroll
                    for (int j = 0; j < NJ; ++j) {
                        const int ix = cart_x(LI, i), iy = cart_y(LI, i), iz = cart_z(LI, i);
                        const int jx = cart_x(LJ, j), jy = cart_y(LJ, j), jz = cart_z(LJ, j);
#pragma unroll
                        for (int tt = 0; tt <= ix + jx; ++tt) {
                            const double wx = dv[i][j] * e[0][ix][jx][tt], wf = dv[i][j] * de[0][ix][jx][tt];
#pragma unroll
                            for (int uu = 0; uu <= iy + jy; ++uu) {
                                const double wxy = wx * e[1][iy][jy][uu], wfy = wf * e[1][iy][jy][uu],
                                             wxf = wx * de[1][iy][jy][uu];
#pragma unroll
                                for (int ww = 0; ww <= iz + jz; ++ww) {
                                    const int h = hidx(tt, uu, ww);
                                    Y[h] += wxy * e[2][iz][jz][ww];
                                    U[0][h] += wfy * e[2][iz][jz][ww];
                                    U[1][h] += wxf * e[2][iz][jz][ww];
                                    U[2][h] += wxy * de[2][iz][jz][ww];
                                }
                            }
                        }
                    }
            }
            double G[3] = {0.0, 0.0, 0.0}, u[3] = {0.0, 0.0, 0.0};
            for (int c = c0; c < sv.natm; c += al) {
                double R[nherm(L + 1)];
                hermite_r<L + 1>(p, (Ax - sv.pos[3 * c]) - bp * ABx, (Ay - sv.pos[3 * c + 1]) - bp * ABy,
                                 (Az - sv.pos[3 * c + 2]) - bp * ABz, R, boys);
                const double w = -sv.charges[c] * 2.0 * PI * ip_;
                double g[3] = {0.0, 0.0, 0.0};
#pragma unroll
                for (int tt = 0; tt <= L; ++tt)
#pragma unroll
                    for (int uu = 0; uu <= L - tt; ++uu)
#pragma unroll
                        for (int ww = 0; ww <= L - tt - uu; ++ww) {
                            const int h = hidx(tt, uu, ww);
                            g[0] += Y[h] * R[hidx(tt + 1, uu, ww)];
                            g[1] += Y[h] * R[hidx(tt, uu + 1, ww)];
                            g[2] += Y[h] * R[hidx(tt, uu, ww + 1)];
                            const double wr = w * R[h];
                            u[0] += U[0][h] * wr;
                            u[1] += U[1][h] * wr;
                            u[2] += U[2][h] * wr;
                        }
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    g[d] *= w;
                    G[d] += g[d];
                    gadd(3 * c + d, -g[d]);
                }
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                gA[d] += ap * G[d] + u[d];
                gB[d] += bp * G[d] - u[d];
            }
        }
        // the pair's two centres: lanes 0-2 add A's sums, lanes 3-5 B's
        double mine = 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double sa = warp_sum(gA[d]), sb = warp_sum(gB[d]);
            if (lane == d) mine = sa;
            if (lane == 3 + d) mine = sb;
        }
        if (lane < 6) gadd(lane < 3 ? 3 * ai + lane : 3 * aj + lane - 3, mine);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n3; i += blockDim.x) {
        const facc v = join_planes(gsh[i], gsh[n3 + i]);
        if (v != 0) atomicAdd(&grad[i], v);
    }
}

}  // namespace hf
