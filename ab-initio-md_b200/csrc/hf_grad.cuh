// Integral-direct two-electron gradient 1/2 sum Gamma d(mn|ls)/dR.
//
// Same decomposition as the J/K build: chunks of one bra block pair each, one
// thread item per (ket pair, ket component pair cd). The quartet list is
// enumerated at thr / Gamma_bound, so every quartet the exact test can keep
// is visited; each item applies the reference's test Q1 Q2 max|Gamma| < thr
// (aimd/qc/integrals.py:1329) to its column of Gamma.
//
//   Gamma_{mnls} = deg [Dc_mn Dc_ls - k/2 sum_x (Dx_ml Dx_ns + Dx_ms Dx_nl)],
//   deg = 1/2 x (2 if A != B) x (2 if C != D) x (2 if P1 != P2)
// (aimd/qc/integrals.py:1298-1328).
//
// A primitive quartet's part of the energy is
//   sum_{h,k} Y_h e_k (-1)^|k| R_{h+k}(P - Q),
// with Y the bra's Hermite expansion contracted with Gamma and e the column's
// ket expansion. The centres enter through P and Q, where d/dP_x raises h by
// one (and d/dQ = -d/dP), and through the expansions, which depend on
// X_AB = A - B and X_CD = C - D alone:
//   G = sum Y_h e_k (-1)^|k| R_{h+k+1},  U, V = the same sum with dY/dX_AB, de/dX_CD
//   dA = (a/p) G + U,  dB = (b/p) G - U,  dC = -(c/q) G + V,  dD = -(d/q) G - V
// (D from translational invariance, -(A + B + C), per column). So one sum over
// the column's box, X_h = sum_k e_k (-1)^|k| R_{h+k} to |h| = LAB + 1, gives
// G = sum Y_h X_{h+1} and U = sum (dY)_h X_h, and Z_k = sum_h Y_h R_{h+k}, from
// the same R values, gives V. The reference (and an earlier form of this file)
// instead raises and lowers each Gaussian, 2a E^{i+1} - i E^{i-1}, with every
// bra row's box widened by one in each direction (aimd/qc/integrals.py:
// 1049-1244): for pp|pp some 900 multiply-adds a primitive quartet and column
// in that step, against 180 here, and ten times the code: the kernels of a
// small molecule are bound by fetching each instruction once. One B200, raised
// form -> this one: methanol 6-31G** 16.4 -> 1.67 ms, (H2O)8 cc-pVDZ 73.1 ->
// 10.2 ms, (H2O)32 1095 -> 178 ms; with the Boys table, the rows of Dx in shared
// memory and the pair data by sorted position 0.63, 7.1 and 155 ms.
#pragma once
#include "hf_eri.cuh"

namespace hf {

struct GradArgs {
    QuartetArgs q;
    const double* Dc;       // [nao][nao] symmetric
    const double* Dx;       // [nx][nao][nao] symmetric
    int nx;
    double kfac;
    double thr;             // exact screening threshold on Q1 Q2 max|Gamma|
    facc* grad;             // [natm][3] (fixed point, FIX_G)
    int natm;
    size_t rbuf;            // elements of the kernel's staged-R buffer (set per launch)
    const double* bmc;      // [nblock][nblock] max |Dc| per block pair
    const double* bmx;      // [nblock][nblock] max over x of |Dx| per block pair (nx > 0)
    int nblock;
    int dglobal;            // 1: the bra functions' rows of Dx are read from Dx itself, 0: staged in shared memory (set per launch)
    WorkPlan plan;          // chunks of the launch (set per launch)
};

// Two-stage items (R_tuv to L + 1 staged per primitive quartet) for the
// gradient of class pair (CX, CY): the same classes as the J/K build.
template <int CX, int CY>
constexpr bool grad_rsmem() { return QClass<CX, CY>::RSMEM; }

// Of the other classes, those with more than 20 R_tuv (to L + 1) keep each
// thread's in shared memory while the box pass runs: R is the largest array of
// the gradient body, and in registers it pushes the body into local memory.
// Up to 84 values (L + 1 = 6, 172 KB for the eight warps of an SM); an odd
// stride, so that a warp's accesses to one element spread over the banks.
template <int CX, int CY>
constexpr bool grad_rcol() {
    constexpr int NH = nherm(QClass<CX, CY>::L + 1);
    return !grad_rsmem<CX, CY>() && NH > 20 && NH <= 84;
}
template <int CX, int CY>
constexpr int grad_rstride() { return nherm(QClass<CX, CY>::L + 1) | 1; }

// E and dE/dX_AB of one bra pair's primitives, in the same layout (st.E, st.D).
template <int LA, int LB, typename RT>
__device__ __forceinline__ void stage_bra_de(const BraStageT<RT>& st) {
    using BE = BraE<LA, LB>;
    for (int w = threadIdx.x; w < st.i.nbp * 3; w += blockDim.x) {
        const int ib = w / 3, d = w % 3;
        const double* b = st.i.rec + (size_t)ib * PPW;
        const double ip = 1.0 / (b[0] + b[1]), pa = b[6 + d], pb = b[9 + d];
        double e[LA + 1][LB + 1][LA + LB + 1], de[LA + 1][LB + 1][LA + LB + 1];
        hermite_e<LA, LB>(pa, pb, 0.5 * ip, 1.0, e);        // K is in the scalars
        hermite_de<LA, LB>(pa, pb, 0.5 * ip, b[1] * ip, b[0] * ip, 2.0 * b[0] * b[1] * ip * (pb - pa), e, de);
        // exp(-mu |A - B|^2) is in the scalars; each direction's table carries
        // its derivative through de[0][0][0]
        RT* out = st.E + (size_t)ib * BE::SIZE;
        RT* dout = st.D + (size_t)ib * BE::SIZE;
#pragma unroll
        for (int i = 0; i <= LA; ++i)
#pragma unroll
            for (int j = 0; j <= LB; ++j)
#pragma unroll
                for (int t = 0; t <= LA + LB; ++t) {
                    out[BE::at(d, i, j, t)] = static_cast<RT>(e[i][j][t]);
                    dout[BE::at(d, i, j, t)] = static_cast<RT>(de[i][j][t]);
                }
    }
    stage_bra_scalars(st);
}

// Primitive loops of one gradient column (bra primitives [ib0, ib1)): bra
// primitives outer, so that Y (the bra's E contracted with the Gamma column)
// and the U sum, linear in X, are formed once per bra primitive.
template <int CX, int CY, typename RT, bool RS, typename Boys>
__device__ __forceinline__ void grad_prims(const BraStageT<RT>& st, const RT (&Gr)[QClass<CX, CY>::NROW][QClass<CX, CY>::KG],
                                           const double* __restrict__ rk, int nkp, int ic, int id, int kg,
                                           RT (&dA)[3], RT (&dB)[3], RT (&dC)[3], const RT* __restrict__ Rs,
                                           RT* Rcol, int ib0, int ib1, int nk, Boys boys) {
    using Q = QClass<CX, CY>;
    using BE = BraE<Q::LA, Q::LB>;
    constexpr int LA = Q::LA, LB = Q::LB, LC = Q::LC, LD = Q::LD, LAB = Q::LAB, LCD = Q::LCD, L = Q::L + 1;
    constexpr int NHB = Q::NHB, NH1 = nherm(LAB + 1);
    constexpr int KG = Q::KG;
    const int cx = cart_x(LC, ic), cy = cart_y(LC, ic), cz = cart_z(LC, ic);
    const int dx = cart_x(LD, id), dy = cart_y(LD, id), dz = cart_z(LD, id);
    const RT fcd = cart_norm(cx, cy, cz) * cart_norm(dx, dy, dz);
    const int nab = st.i.nA * st.i.nB;
    for (int ib = ib0; ib < ib1; ++ib) {
        const RT* sb = st.SB + ib * SBW;
        const RT* E = st.E + (size_t)ib * BE::SIZE;
        const RT* DE = st.D + (size_t)ib * BE::SIZE;
        // Gamma of row ab contracted with this bra primitive's coefficients and f_ab
        auto gq = [&](int ia, int jb, int kk) {
            const RT fab = cart_norm(cart_x(LA, ia), cart_y(LA, ia), cart_z(LA, ia)) *
                           cart_norm(cart_x(LB, jb), cart_y(LB, jb), cart_z(LB, jb));
            RT s = RT(0);
#pragma unroll
            for (int kab = 0; kab < Q::KAB; ++kab)
                if (kab == 0 || kab < nab) s += sb[8 + kab] * Gr[kab * Q::NAB + ia * Q::NB + jb][kk];
            return s * fab;
        };
        RT Y[KG][NHB], Xs[KG][NHB];
#pragma unroll
        for (int kk = 0; kk < KG; ++kk)
#pragma unroll
            for (int h = 0; h < NHB; ++h) Y[kk][h] = Xs[kk][h] = RT(0);
        // one direction at a time, as bra_rows: per (az, bz) the x and y
        // factors into W, then the z factor
#pragma unroll
        for (int az = 0; az <= LA; ++az)
#pragma unroll
            for (int bz = 0; bz <= LB; ++bz) {
                RT W[KG][ncart(LAB)];
#pragma unroll
                for (int kk = 0; kk < KG; ++kk)
#pragma unroll
                    for (int i = 0; i < ncart(LAB); ++i) W[kk][i] = RT(0);
#pragma unroll
                for (int ay = 0; ay <= LA - az; ++ay)
#pragma unroll
                    for (int by = 0; by <= LB - bz; ++by) {
                        const int ax = LA - az - ay, bx = LB - bz - by;
#pragma unroll
                        for (int kk = 0; kk < KG; ++kk) {
                            if (kk > 0 && kk >= nk) continue;
                            const RT g = gq(cart_index(ay, az), cart_index(by, bz), kk);
#pragma unroll
                            for (int t = 0; t <= ax + bx; ++t) {
                                const RT ge = ax + bx > 0 ? g * E[BE::at(0, ax, bx, t)] : g;
#pragma unroll
                                for (int u = 0; u <= ay + by; ++u)
                                    W[kk][cart_index(t, u)] += ay + by > 0 ? ge * E[BE::at(1, ay, by, u)] : ge;
                            }
                        }
                    }
#pragma unroll
                for (int kk = 0; kk < KG; ++kk) {
                    if (kk > 0 && kk >= nk) continue;
#pragma unroll
                    for (int t = 0; t <= LAB - az - bz; ++t)
#pragma unroll
                        for (int u = 0; u <= LAB - az - bz - t; ++u)
#pragma unroll
                            for (int w = 0; w <= az + bz; ++w)
                                Y[kk][hidx(t, u, w)] += az + bz > 0 ? E[BE::at(2, az, bz, w)] * W[kk][cart_index(t, u)]
                                                                    : W[kk][cart_index(t, u)];
                }
            }
        RT gG[3] = {RT(0), RT(0), RT(0)};       // G summed over the ket primitives
        for (int ik = 0; ik < nkp; ++ik) {
            const KetRecT<RT> k = load_ket<RT>(rk + (size_t)ik * PPW);
            const RT q = k.a + k.b, iq = RT(1) / q, oo2q = RT(0.5) * iq, cq = k.a * iq, dq = k.b * iq;
            RT ex[LCD + 1], ey[LCD + 1], ez[LCD + 1], fx[LCD + 1], fy[LCD + 1], fz[LCD + 1];
            {
                RT e[LC + 1][LD + 1][LCD + 1], de[LC + 1][LD + 1][LCD + 1];
                const RT m2 = RT(2) * k.a * dq;
                hermite_e<LC, LD>(k.QAx, k.QBx, oo2q, RT(1), e);
                hermite_de<LC, LD>(k.QAx, k.QBx, oo2q, dq, cq, m2 * (k.QBx - k.QAx), e, de);
                select_row<LC, LD, LCD>(e, cx, dx, ex);
                select_row<LC, LD, LCD>(de, cx, dx, fx);
                hermite_e<LC, LD>(k.QAy, k.QBy, oo2q, RT(1), e);
                hermite_de<LC, LD>(k.QAy, k.QBy, oo2q, dq, cq, m2 * (k.QBy - k.QAy), e, de);
                select_row<LC, LD, LCD>(e, cy, dy, ey);
                select_row<LC, LD, LCD>(de, cy, dy, fy);
                hermite_e<LC, LD>(k.QAz, k.QBz, oo2q, RT(1), e);
                hermite_de<LC, LD>(k.QAz, k.QBz, oo2q, dq, cq, m2 * (k.QBz - k.QAz), e, de);
                select_row<LC, LD, LCD>(e, cz, dz, ez);
                select_row<LC, LD, LCD>(de, cz, dz, fz);
            }
            auto body = [&](const auto& R) {
                RT sc[KG], Yc[NHB];
                const RT fk = fcd * k.K * iq;
#pragma unroll
                for (int i = 0; i < KG; ++i) {
                    RT c = k.c[0];
#pragma unroll
                    for (int j = 1; j < Q::KCD; ++j)
                        if (j == kg * KG + i) c = k.c[j];
                    sc[i] = c * fk;
                }
#pragma unroll
                for (int h = 0; h < NHB; ++h) Yc[h] = sc[0] * Y[0][h];
#pragma unroll
                for (int kk = 1; kk < KG; ++kk) {
                    if (kk >= nk) continue;
#pragma unroll
                    for (int h = 0; h < NHB; ++h) Yc[h] += sc[kk] * Y[kk][h];
                }
                // one pass over the box: X_h and Z_k from the same R values
                RT X[NH1], vx = RT(0), vy = RT(0), vz = RT(0);
#pragma unroll
                for (int h = 0; h < NH1; ++h) X[h] = RT(0);
#pragma unroll
                for (int t2 = 0; t2 <= LCD; ++t2) {
                    if (t2 > cx + dx) continue;
#pragma unroll
                    for (int u2 = 0; u2 <= LCD - t2; ++u2) {
                        if (u2 > cy + dy) continue;
                        const RT exy = ((t2 + u2) & 1) ? -ex[t2] * ey[u2] : ex[t2] * ey[u2];
                        const RT fxy = ((t2 + u2) & 1) ? -fx[t2] * ey[u2] : fx[t2] * ey[u2];
                        const RT exf = ((t2 + u2) & 1) ? -ex[t2] * fy[u2] : ex[t2] * fy[u2];
#pragma unroll
                        for (int v2 = 0; v2 <= LCD - t2 - u2; ++v2) {
                            if (v2 > cz + dz) continue;
                            const RT s = (v2 & 1) ? -ez[v2] : ez[v2];
                            const RT e = exy * s;
                            RT z = RT(0);
#pragma unroll
                            for (int t = 0; t <= LAB + 1; ++t)
#pragma unroll
                                for (int u = 0; u <= LAB + 1 - t; ++u)
#pragma unroll
                                    for (int w = 0; w <= LAB + 1 - t - u; ++w) {
                                        const RT r = R[hidx(t + t2, u + u2, w + v2)];
                                        X[hidx(t, u, w)] += e * r;
                                        if (t + u + w <= LAB) z += Yc[hidx(t, u, w)] * r;
                                    }
                            vx += fxy * s * z;
                            vy += exf * s * z;
                            vz += ((v2 & 1) ? -exy : exy) * fz[v2] * z;
                        }
                    }
                }
                RT gx = RT(0), gy = RT(0), gz = RT(0);
#pragma unroll
                for (int t = 0; t <= LAB; ++t)
#pragma unroll
                    for (int u = 0; u <= LAB - t; ++u)
#pragma unroll
                        for (int w = 0; w <= LAB - t - u; ++w) {
                            const RT y = Yc[hidx(t, u, w)];
                            gx += y * X[hidx(t + 1, u, w)];
                            gy += y * X[hidx(t, u + 1, w)];
                            gz += y * X[hidx(t, u, w + 1)];
                        }
#pragma unroll
                for (int kk = 0; kk < KG; ++kk) {
                    if (kk > 0 && kk >= nk) continue;
#pragma unroll
                    for (int h = 0; h < NHB; ++h) Xs[kk][h] += sc[kk] * X[h];
                }
                gG[0] += gx;
                gG[1] += gy;
                gG[2] += gz;
                dC[0] += vx - cq * gx;
                dC[1] += vy - cq * gy;
                dC[2] += vz - cq * gz;
            };
            if constexpr (RS) {
                body(Rs + (size_t)(ik * st.i.nbp + ib) * nherm(L));
            } else {
                const BraPrim<RT> b = load_bra(sb);
                const RT rs = rsqrt_t(b.p + q);
                RT R[nherm(L)];
                hermite_r_scaled<L>(b.p * q * (rs * rs), b.X - k.Qx, b.Y - k.Qy, b.Z - k.Qz, rs, R, boys);
                if constexpr (grad_rcol<CX, CY>()) {
#pragma unroll
                    for (int i = 0; i < nherm(L); ++i) Rcol[i] = R[i];
                    body(Rcol);
                } else {
                    body(R);
                }
            }
        }
        // U on the summed X, once per bra primitive
        RT ux = RT(0), uy = RT(0), uz = RT(0);
#pragma unroll
        for (int az = 0; az <= LA; ++az)
#pragma unroll
            for (int bz = 0; bz <= LB; ++bz) {
#pragma unroll
                for (int kk = 0; kk < KG; ++kk) {
                    if (kk > 0 && kk >= nk) continue;
                    RT W[ncart(LAB)], Wz[ncart(LAB)];       // E_z and dE_z applied
#pragma unroll
                    for (int t = 0; t <= LAB - az - bz; ++t)
#pragma unroll
                        for (int u = 0; u <= LAB - az - bz - t; ++u) {
                            RT s = Xs[kk][hidx(t, u, 0)], sz = RT(0);
                            if (az + bz > 0) {
                                s *= E[BE::at(2, az, bz, 0)];
#pragma unroll
                                for (int w = 1; w <= az + bz; ++w) s += E[BE::at(2, az, bz, w)] * Xs[kk][hidx(t, u, w)];
                            }
#pragma unroll
                            for (int w = 0; w <= az + bz; ++w) sz += DE[BE::at(2, az, bz, w)] * Xs[kk][hidx(t, u, w)];
                            W[cart_index(t, u)] = s;
                            Wz[cart_index(t, u)] = sz;
                        }
#pragma unroll
                    for (int ay = 0; ay <= LA - az; ++ay)
#pragma unroll
                        for (int by = 0; by <= LB - bz; ++by) {
                            const int ax = LA - az - ay, bx = LB - bz - by;
                            const RT g = gq(cart_index(ay, az), cart_index(by, bz), kk);
#pragma unroll
                            for (int t = 0; t <= ax + bx; ++t) {
                                RT s = W[cart_index(t, 0)], sy = RT(0), sz = Wz[cart_index(t, 0)];
                                if (ay + by > 0) {
                                    s *= E[BE::at(1, ay, by, 0)];
                                    sz *= E[BE::at(1, ay, by, 0)];
#pragma unroll
                                    for (int u = 1; u <= ay + by; ++u) {
                                        s += E[BE::at(1, ay, by, u)] * W[cart_index(t, u)];
                                        sz += E[BE::at(1, ay, by, u)] * Wz[cart_index(t, u)];
                                    }
                                }
#pragma unroll
                                for (int u = 0; u <= ay + by; ++u) sy += DE[BE::at(1, ay, by, u)] * W[cart_index(t, u)];
                                const RT ge = ax + bx > 0 ? g * E[BE::at(0, ax, bx, t)] : g;
                                ux += g * DE[BE::at(0, ax, bx, t)] * s;
                                uy += ge * sy;
                                uz += ge * sz;
                            }
                        }
                }
            }
        const RT ap = sb[4], bp = sb[5];
        dA[0] += ap * gG[0] + ux;
        dA[1] += ap * gG[1] + uy;
        dA[2] += ap * gG[2] + uz;
        dB[0] += bp * gG[0] - ux;
        dB[1] += bp * gG[1] - uy;
        dB[2] += bp * gG[2] - uz;
    }
}

// Gradient contribution of one column; adds A, B parts to gab and C, D
// parts to the shared accumulator gsh (low words [natm][3], then the high words). RS: R_tuv / sqrt(p + q) (to L + 1)
// of the ket pair's primitive quartets staged in Rs ([ik][ib][NH(L + 1)]).
template <int CX, int CY, typename RT, bool RS, typename Boys>
__device__ __forceinline__ void grad_column(const GradArgs& a, const BraStageT<RT>& st, const PairMeta& ket, double QQ, int ic,
                                            int id, int kg, double (&gab)[6], unsigned* gsh,
                                            const RT* __restrict__ Rs, RT* Rcol, int ib0, int ib1,
                                            int nk, Boys boys, const double* Dsm) {
    using Q = QClass<CX, CY>;
    const int aC = ket.aA, aD = ket.aB;
    if (st.i.aA == st.i.aB && st.i.aB == aC && aC == aD) return;          // one-centre: invariant
    const int nC = ket.nA, nD = ket.nB, oC = ket.oA, oD = ket.oB;
    const int n = a.q.nao;
    const size_t nn = (size_t)n * n;
    const double deg = 0.5 * (st.i.A != st.i.B ? 2.0 : 1.0) * (ket.A != ket.B ? 2.0 : 1.0) * (st.i.P1 != ket.P ? 2.0 : 1.0);
    // Gamma column
    double G[Q::NROW][Q::KG];
    double gmax = 0.0;
#pragma unroll
    for (int kk = 0; kk < Q::KG; ++kk) {
        const int kq = kg * Q::KG + kk;
        const bool cv = kq < nC * nD;
        const int kc = cv ? kq / nD : 0, kd = cv ? kq % nD : 0;
        const size_t l = oC + kc * Q::NC + ic, sg = oD + kd * Q::ND + id;
#pragma unroll
        for (int r = 0; r < Q::NROW; ++r) {
            const int kab = r / Q::NAB, ab = r % Q::NAB, ka = kab / st.i.nB, kb = kab % st.i.nB;
            double val = 0.0;
            if (cv && kab < st.i.nA * st.i.nB) {
                const int m = ka * Q::NA + ab / Q::NB, nb_ = kb * Q::NB + ab % Q::NB;
                val = __ldg(a.Dc + (size_t)(st.i.oA + m) * n + st.i.oB + nb_) * __ldg(a.Dc + l * n + sg);
                for (int x = 0; x < a.nx; ++x) {
                    constexpr int NFA = Q::KA * Q::NA, NF = NFA + Q::KB * Q::NB;
                    const double* Xm = (a.dglobal ? a.Dx + x * nn + (size_t)st.i.oA * n : Dsm + (size_t)x * NF * n) + (size_t)m * n;
                    const double* Xn = (a.dglobal ? a.Dx + x * nn + (size_t)st.i.oB * n : Dsm + (size_t)(x * NF + NFA) * n) + (size_t)nb_ * n;
                    val -= 0.5 * a.kfac * (Xm[l] * Xn[sg] + Xm[sg] * Xn[l]);
                }
                val *= deg;
            }
            G[r][kk] = val;
            gmax = fmax(gmax, fabs(val));
        }
    }
    if (QQ == 0.0 || QQ * gmax < a.thr) return;
    // the Gamma column in the arithmetic type of the quartet
    RT Gr[Q::NROW][Q::KG];
#pragma unroll
    for (int r = 0; r < Q::NROW; ++r)
#pragma unroll
        for (int kk = 0; kk < Q::KG; ++kk) Gr[r][kk] = static_cast<RT>(G[r][kk]);
    RT dA[3] = {0.0, 0.0, 0.0}, dB[3] = {0.0, 0.0, 0.0}, dC[3] = {0.0, 0.0, 0.0};
    grad_prims<CX, CY, RT, RS>(st, Gr, ket.rec, ket.npp, ic, id, kg, dA, dB, dC, Rs,
                               Rcol, ib0, ib1, nk, boys);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double da = dA[d], db = dB[d], dc = dC[d];
        gab[d] += da;
        gab[3 + d] += db;
        sadd(gsh + 3 * aC + d, gsh + 3 * (a.natm + aC) + d, dc, FIX_G);
        sadd(gsh + 3 * aD + d, gsh + 3 * (a.natm + aD) + d, -(da + db + dc), FIX_G);
    }
}

// Ket pairs pass the queue when the block bound of Gamma over the whole
// block quartet, deg [|Dc|_AB |Dc|_CD + |k|/2 nx (|Dx|_AC |Dx|_BD +
// |Dx|_AD |Dx|_BC)] >= max|Gamma|, can reach the threshold and the quartet
// is not one-centre; the exact per-column test follows in grad_column.

template <int CX, int CY, typename RT, typename Boys>
__device__ __forceinline__ void grad_ket_class(const GradArgs& a, const BraStageT<RT>& st, int spos, double (&gab)[6],
                                               unsigned* gsh, FlatItems& f, KetQueueR* kq, int* queue, RT* Rbuf,
                                               Boys boys, const double* Dsm) {
    using Q = QClass<CX, CY>;
    constexpr bool RS = grad_rsmem<CX, CY>();
    const double q1 = a.q.sortedQ[spos];
    const int nb = a.nblock;
    const double xf = 0.5 * fabs(a.kfac) * a.nx;
    auto keep = [&](int pos) {
        const PairMeta k = load_meta(a.q, pos);
        const int C = k.A, Dd = k.B, aC = k.aA, aD = k.aB;
        if (st.i.aA == st.i.aB && st.i.aB == aC && aC == aD) return false;
        double gb = a.bmc[st.i.A * nb + st.i.B] * a.bmc[C * nb + Dd];
        if (a.nx > 0)
            gb += xf * (a.bmx[st.i.A * nb + C] * a.bmx[st.i.B * nb + Dd] + a.bmx[st.i.A * nb + Dd] * a.bmx[st.i.B * nb + C]);
        const double deg = 0.5 * (st.i.A != st.i.B ? 2.0 : 1.0) * (C != Dd ? 2.0 : 1.0) * (st.i.P1 != k.P ? 2.0 : 1.0);
        return q1 * a.q.sortedQ[pos] * deg * gb >= a.thr;
    };
    // item r = (contraction group, bra-primitive split, column)
    auto work = [&](int sub, int pos, int r, const RT* Rs) {
        const int nkg = seg_groups<Q::KG, Q::NKG>(sub), nsp = bra_splits(st.i.nbp, sub, f.item_pq);
        const int kg = r % nkg, sp = (r / nkg) % nsp, cd = r / (nkg * nsp);
        grad_column<CX, CY, RT, RS>(a, st, load_meta(a.q, pos), q1 * a.q.sortedQ[pos], cd / Q::ND, cd % Q::ND, kg, gab,
                                    gsh, Rs, Rbuf + threadIdx.x * grad_rstride<CX, CY>(), st.i.nbp * sp / nsp, st.i.nbp * (sp + 1) / nsp,
                                    group_combos<Q::KG>(sub, kg), boys, Dsm);
    };
    if constexpr (RS) {
        int rot = 0;
        for (int sub = 0; sub < NSUB; ++sub)
            if (f.kcnt[sub] > 0)
                ket_items_r<Q::L + 1>(f.nper[sub], f.kj0[sub], f.kcnt[sub], *kq, rot, st, a.q, Rbuf, keep,
                                      [&](int pos, int r, const RT* Rs) { work(sub, pos, r, Rs); });
    } else {
        flat_items(f, true, queue, keep,
                   [&](int sub, int pos, int r) { work(sub, pos, r, static_cast<const RT*>(nullptr)); });
    }
}

// The Boys function of the (CX, CY) gradient kernel: from the table up to
// order L + 1 = 5, by series above (whose R columns leave no room for it).
template <int CX, int CY, typename RT>
using GradBoys = BoysOf<QClass<CX, CY>::L + 1, RT, (QClass<CX, CY>::L + 1 <= 5)>;

// One kernel per (bra class, ket class), persistent: a CTA runs chunks
// (bra pair of class CX, window of its ket pairs of class CY) of the
// launch's work plan until it is used up. Dynamic shared memory: gradient
// accumulator [natm][3] (one per CTA, flushed at the end), Boys table, D rows, staged R, bra E
// and dE/dX_AB tables.
// RT = double: the FP64 quartets; RT = float: the FP32 quartets of the
// mixed-precision path (accumulated in FP64).
template <int CX, int CY, typename RT>
__global__ void __launch_bounds__(CLASS_THREADS) grad2e_bra_kernel(GradArgs a) {
    using Q0 = QClass<CX, 0>;
    using Q = QClass<CX, CY>;
    using Boys = GradBoys<CX, CY, RT>;
    extern __shared__ __align__(16) double smem[];
    double* btab = smem;                                                // Boys table
    unsigned* gsh = reinterpret_cast<unsigned*>(btab + Boys::elems);    // low words [natm][3], then the high words
    constexpr int NFA = Q::KA * Q::NA, NF = NFA + Q::KB * Q::NB;
    const int n = a.q.nao;
    double* Dsm = btab + Boys::elems + even(3 * a.natm);                // the bra functions' rows of Dx [nx][NF][nao]
    RT* Rbuf = reinterpret_cast<RT*>(Dsm + (a.dglobal ? 0 : even((size_t)a.nx * NF * n)));
    RT* Esm = Rbuf + a.rbuf;
    __shared__ BraInfo info;
    __shared__ FlatItems f;
    __shared__ QueueOf<grad_rsmem<CX, CY>()> kq;
    __shared__ int sh[2];
    const int nbra = a.q.cls_start[CX + 1] - a.q.cls_start[CX];
    const int total = a.plan.off[nbra];
    for (int i = threadIdx.x; i < 6 * a.natm; i += blockDim.x) gsh[i] = 0u;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) f.item_pq = *a.plan.pq;           // (read after the first barrier)
    bool staged = false;        // the Boys table is in shared memory
    auto gadd = [&](int i, double v) { sadd(gsh + i, gsh + 3 * a.natm + i, v, FIX_G); };
    for (;;) {
        if (warp == 0) {
            int c, b;
            next_chunk(a.plan, nbra, total, c, b);
            if (lane == 0) {
                sh[0] = c;
                sh[1] = b;
                if (c >= 0) load_info(load_meta(a.q, a.q.cls_start[CX] + b), info);
            }
        }
        __syncthreads();                                        // (also orders the zeroing)
        const int c = sh[0], b = sh[1];
        if (c < 0) break;                                       // uniform: c is shared
        const int spos = a.q.cls_start[CX] + b;
        if (!staged) {
            Boys::stage(a.q.boys, btab);
            staged = true;
        }
        const BraStageT<RT> st = stage_view(info, Esm, BraE<Q0::LA, Q0::LB>::SIZE);
        if (warp == 0) {
            const int sub = lane < NSUB ? lane : 0;
            plan_window<CX, CY, RT>(a.q, spos, st.i.nbp, c - a.plan.off[b], a.plan.off[b + 1] - a.plan.off[b], Q::NCD,
                                    seg_groups<Q::KG, Q::NKG>(sub), bra_splits(st.i.nbp, sub, f.item_pq), f);
        }
        stage_bra_de<Q0::LA, Q0::LB>(st);
        if (!a.dglobal) {
            const int na = info.nA * Q::NA * n, nb = info.nB * Q::NB * n;
            for (int x = 0; x < a.nx; ++x) {
                const double* X = a.Dx + (size_t)x * n * n;
#pragma unroll 4
                for (int i = threadIdx.x; i < na; i += blockDim.x) Dsm[(size_t)x * NF * n + i] = __ldg(X + (size_t)info.oA * n + i);
#pragma unroll 4
                for (int i = threadIdx.x; i < nb; i += blockDim.x) Dsm[((size_t)x * NF + NFA) * n + i] = __ldg(X + (size_t)info.oB * n + i);
            }
        }
        __syncthreads();
        double gab[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        grad_ket_class<CX, CY, RT>(a, st, spos, gab, gsh, f, kq.r(), kq.flat(), Rbuf, Boys::get(btab), Dsm);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (gab[d] != 0.0) gadd(3 * st.i.aA + d, gab[d]);
            if (gab[3 + d] != 0.0) gadd(3 * st.i.aB + d, gab[3 + d]);
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < 3 * a.natm; i += blockDim.x) {
        const facc v = join_planes(gsh[i], gsh[3 * a.natm + i]);
        if (v != 0) atomicAdd(a.grad + i, v);
    }
}

// Elements of the staged-R buffer of the (CX, CY) gradient kernel (the
// two-stage classes), or of its threads' R columns.
template <int CX, int CY, typename RT>
size_t grad_rbuf_elems(int threads, int max_bra_prims, int max_ket_prims) {
    if constexpr (grad_rsmem<CX, CY>())
        return fours(rsmem_bytes<QClass<CX, CY>::L + 1, RT>(max_bra_prims, max_ket_prims) / sizeof(RT));
    if constexpr (grad_rcol<CX, CY>()) return fours((size_t)grad_rstride<CX, CY>() * threads);
    return 0;
}

template <int CX, int CY, typename RT>
size_t grad_smem_bytes(int natm, int nx, int nao, int max_bra_prims, size_t rbuf_elems, bool dglobal) {
    using Q0 = QClass<CX, 0>;
    constexpr size_t NF = Q0::KA * Q0::NA + Q0::KB * Q0::NB;
    return sizeof(double) * (even(3 * (size_t)natm) + GradBoys<CX, CY, RT>::elems + (dglobal ? 0 : even(nx * NF * nao))) +
           sizeof(RT) * (rbuf_elems + (size_t)max_bra_prims * (2 * BraE<Q0::LA, Q0::LB>::SIZE + SBW));
}

}  // namespace hf
