// Contracted block-quartet ERIs and their integral-direct J/K digestion.
//
// Work decomposition (one launch per bra class X and ket class Y <= X):
//   * a chunk = (bra block pair P1, window of its ket list), taken by a CTA;
//   * the ket block pairs P2 of class Y that pass Q1 Q2 >= thr are, in each
//     segment, a prefix of its Q-sorted list (cut at P1's own position for
//     Y == X, so each unordered pair of pairs is visited once);
//   * one thread item = (ket pair P2, ket Cartesian component pair cd): it
//     computes the column (ab|cd) for every bra row ab and every contraction
//     combination, by McMurchie-Davidson: per primitive quartet R_tuv up to
//     L = l_a+l_b+l_c+l_d, the ket Hermite->Cartesian step for its own cd,
//     and the bra step (the reference's _eri_block,
//     aimd/qc/integrals.py:777-842, reorganised by column).
// The bra pair's primitive E tables are staged once per chunk in shared
// memory. Digestion: every exchange image of the 8-fold symmetry lands in a
// row of the bra pair's functions, so K rows are accumulated in shared
// memory and flushed once per chunk; J_ab accumulates in per-thread shared
// slots; only J_cd goes straight to global memory.
//
// What bounds these kernels is instruction issue (FP64 chains at 8 warps per
// SM) and, for small molecules, fetching the unrolled code of each kernel
// once; DRAM traffic is negligible. Hence one pass over a column's box with
// its conditions tested per box entry, no code for the entries that no column
// reaches (t + u + v > LCD), and the bra step one direction at a time. With
// those and the flat item lists, one B200: water 6-31G* 2.67 -> 0.37 ms,
// (H2O)8 difference build 11.5 -> 4.4 ms, (H2O)32 cc-pVDZ 266 -> 118 ms.
// Digestion took as long as the integrals (dp|ps 4.9 of 6.8 ms, pp|ps 6.5 of
// 9.4, ps|ss 5.3 of 16.3): the bra functions' rows of D, read at the scattered
// columns of a warp's ket pairs, were a cache line a lane and load. With the
// rows in shared memory and the columns of an item digested together:
// (H2O)32 93 -> 70 ms, (H2O)8 difference build 3.25 -> 1.95 ms. Water now takes
// 0.14 ms.
#pragma once
#include <type_traits>

#include "hf_device.cuh"

namespace hf {

template <int CX, int CY>
struct QClass {
    static constexpr int LA = cls_la(CX), LB = cls_lb(CX), LC = cls_la(CY), LD = cls_lb(CY);
    static constexpr int LAB = LA + LB, LCD = LC + LD, L = LAB + LCD;
    static constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
    static constexpr int NAB = NA * NB, NCD = NC * ND;
    static constexpr int KA = ncon_cap(LA), KB = ncon_cap(LB), KC = ncon_cap(LC), KD = ncon_cap(LD);
    static constexpr int KAB = KA * KB, KCD = KC * KD;
    static constexpr int NROW = KAB * NAB;
    // ket contraction combinations per thread item: all of them unless the
    // per-thread accumulator v[NROW][KG] would exceed 24 doubles
    static constexpr int KG = NROW * KCD <= 24 ? KCD : ((KCD % 2 == 0 && NROW * 2 <= 24) ? 2 : 1);
    static constexpr int NKG = KCD / KG;
    static constexpr int NHB = nherm(LAB);
    // R_tuv staged once per primitive quartet for all columns of a ket pair
    // (two-stage items): for dd bras against dp and dd kets, whose pairs have
    // one to three primitive pairs, 18-36 columns and L = 7-8, so that the
    // staged sub-chunks hold many items (measured: staging the classes with
    // many-primitive pairs starved the sub-chunks and was slower)
    static constexpr bool RSMEM = CX == 5 && CY >= 4;
    // Column-blocked items: one item covers the NC columns (ic, id) of one
    // id, so R_tuv of a primitive quartet is computed once for NC columns
    // instead of once per column; for the s/p bra classes against p kets,
    // where the NC x NROW x KG accumulators fit in registers
    static constexpr bool CBLK = (CX == 1 || CX == 2) && CY >= 1;
    static constexpr int NCB = CBLK ? NC : 1;       // columns per item
    static constexpr int NITEM = NCD / NCB;         // column items per ket pair and contraction group
};

// E table of one bra primitive.
template <int LA, int LB>
struct BraE {
    static constexpr int I = LA + 1, J = LB + 1, T = LA + LB + 1;
    static constexpr int SIZE = 3 * I * J * T;
    __device__ static int at(int d, int i, int j, int t) { return ((d * I + i) * J + j) * T + t; }
};

// Shared-memory stage of one bra pair. The E tables and per-primitive
// scalars are held in the arithmetic type RT of the kernel that reads them
// (double, or float for the mixed-precision quartets); they are computed in
// FP64 either way.
// per bra primitive: p, Px, Py, Pz, a/p, b/p, -, -, then c0..c3, the contraction
// products times 2 pi^(5/2) K / p (K = exp(-mu |A - B|^2)); 16-byte aligned
constexpr int SBW = 12;
struct BraInfo {
    int P1, A, B, nbp, aA, aB;
    int nA, nB, oA, oB;
    const double* rec;      // bra primitive records (global)
};
// Each thread's view: the pair's integers in shared memory, and pointers
// derived from the kernel's shared array (held in registers, not in shared
// memory, so that the compiler knows their address space).
template <typename RT>
struct BraStageT {
    const BraInfo& i;
    RT* SB;                 // [nbp][SBW] (shared)
    RT* E;                  // [nbp][BraE::SIZE] (shared)
    RT* D;                  // gradients: dE/dX_AB in the same layout (shared)
};

template <typename RT>
__device__ __forceinline__ void stage_bra_scalars(const BraStageT<RT>& st) {
    for (int ib = threadIdx.x; ib < st.i.nbp; ib += blockDim.x) {
        const double* b = st.i.rec + (size_t)ib * PPW;
        RT* o = st.SB + (size_t)ib * SBW;
        const double p = b[0] + b[1], ip = 1.0 / p, f = TWO_PI_2_5 * b[2] * ip;
        const double vals[SBW] = {p, b[3], b[4], b[5], b[0] * ip, b[1] * ip, 0.0, 0.0,
                                  f * b[12], f * b[13], f * b[14], f * b[15]};
#pragma unroll
        for (int i = 0; i < SBW; ++i) o[i] = static_cast<RT>(vals[i]);
    }
}

// Fill the shared stage (E tables and scalars) for all bra primitives. An ss
// bra has no table: E^{00}_0 = 1 (K is in the scalars), which bra_rows knows.
// Without it the longest s contraction that a J/K launch takes beside the Boys
// table is 45 primitives (41 with it).
template <int LA, int LB>
constexpr int bra_e_size() { return LA + LB > 0 ? BraE<LA, LB>::SIZE : 0; }
template <int LA, int LB, typename RT>
__device__ __forceinline__ void stage_bra_e(const BraStageT<RT>& st) {
    using BE = BraE<LA, LB>;
    for (int w = threadIdx.x; w < (LA + LB > 0 ? st.i.nbp * 3 : 0); w += blockDim.x) {
        const int ib = w / 3, d = w % 3;
        const double* b = st.i.rec + (size_t)ib * PPW;
        const double p = b[0] + b[1];
        double e[LA + 1][LB + 1][LA + LB + 1];
        hermite_e<LA, LB>(b[6 + d], b[9 + d], 0.5 / p, 1.0, e);      // K is in the scalars
        RT* out = st.E + (size_t)ib * BE::SIZE;
#pragma unroll
        for (int i = 0; i < LA + 1; ++i)
#pragma unroll
            for (int j = 0; j < LB + 1; ++j)
#pragma unroll
                for (int t = 0; t < LA + LB + 1; ++t) out[BE::at(d, i, j, t)] = static_cast<RT>(e[i][j][t]);
    }
    stage_bra_scalars(st);
}

// The bra primitive's exponent sum and centre, in vector loads.
template <typename RT>
struct BraPrim {
    RT p, X, Y, Z;
};
__device__ __forceinline__ BraPrim<double> load_bra(const double* sb) {
    const double2 u = *reinterpret_cast<const double2*>(sb), v = *reinterpret_cast<const double2*>(sb + 2);
    return BraPrim<double>{u.x, u.y, v.x, v.y};
}
__device__ __forceinline__ BraPrim<float> load_bra(const float* sb) {
    const float4 u = *reinterpret_cast<const float4*>(sb);
    return BraPrim<float>{u.x, u.y, u.z, u.w};
}

// One primitive-pair record of a ket pair (16 doubles, 128-byte aligned),
// loaded with 16-byte vector loads, held in the kernel's arithmetic type.
template <typename RT>
struct KetRecT {
    RT a, b, K, Qx, Qy, Qz, QAx, QAy, QAz, QBx, QBy, QBz, c[4];
};
template <typename RT>
__device__ __forceinline__ KetRecT<RT> load_ket(const double* __restrict__ rec) {
    const double2* r2 = reinterpret_cast<const double2*>(rec);
    KetRecT<RT> k;
    double2 v = __ldg(r2 + 0); k.a = (RT)v.x; k.b = (RT)v.y;
    v = __ldg(r2 + 1); k.K = (RT)v.x; k.Qx = (RT)v.y;
    v = __ldg(r2 + 2); k.Qy = (RT)v.x; k.Qz = (RT)v.y;
    v = __ldg(r2 + 3); k.QAx = (RT)v.x; k.QAy = (RT)v.y;
    v = __ldg(r2 + 4); k.QAz = (RT)v.x; k.QBx = (RT)v.y;
    v = __ldg(r2 + 5); k.QBy = (RT)v.x; k.QBz = (RT)v.y;
    v = __ldg(r2 + 6); k.c[0] = (RT)v.x; k.c[1] = (RT)v.y;
    v = __ldg(r2 + 7); k.c[2] = (RT)v.x; k.c[3] = (RT)v.y;
    return k;
}

__device__ __forceinline__ double rsqrt_t(double x) { return rsqrt(x); }
__device__ __forceinline__ float rsqrt_t(float x) { return rsqrtf(x); }

// out[t] = e[i][j][t] for runtime (i, j), by predicated copies (no local memory).
template <int IM, int JM, int T, typename RT>
__device__ __forceinline__ void select_row(const RT (&e)[IM + 1][JM + 1][T + 1], int i, int j, RT (&out)[T + 1]) {
#pragma unroll
    for (int t = 0; t <= T; ++t) out[t] = RT(0);
#pragma unroll
    for (int ii = 0; ii <= IM; ++ii)
#pragma unroll
        for (int jj = 0; jj <= JM; ++jj)
            if (ii == i && jj == j)
#pragma unroll
                for (int t = 0; t <= T; ++t) out[t] = e[ii][jj][t];
}

// out[i][t] = e[i][j][t] for every i (runtime j), by predicated copies.
template <int IM, int JM, int T, typename RT>
__device__ __forceinline__ void select_j(const RT (&e)[IM + 1][JM + 1][T + 1], int j, RT (&out)[IM + 1][T + 1]) {
#pragma unroll
    for (int i = 0; i <= IM; ++i)
#pragma unroll
        for (int t = 0; t <= T; ++t) {
            RT x = e[i][0][t];
#pragma unroll
            for (int jj = 1; jj <= JM; ++jj)
                if (jj == j) x = e[i][jj][t];
            out[i][t] = x;
        }
}

// Bra Hermite -> Cartesian step of one bra primitive, one direction at a time:
// row(ia, jb, s) receives s[kk] = f_ab sum_{tuw} E^{ab}_tuw X[kk]_tuw for every
// component pair (ia, jb). For each (az, bz) the sum over w is taken once for
// all (t, u) (W), then the sums over u and t of its (ay, by): some 440
// multiply-adds for dd, against three products for each of the 400 entries of
// the rows' boxes.
template <int LA, int LB, int KG, typename RT, typename Row>
__device__ __forceinline__ void bra_rows(const RT* E, const RT (&X)[KG][nherm(LA + LB)], Row row) {
    using BE = BraE<LA, LB>;
#pragma unroll
    for (int az = 0; az <= LA; ++az)
#pragma unroll
        for (int bz = 0; bz <= LB; ++bz) {
            RT W[KG][ncart(LA + LB)];
#pragma unroll
            for (int t = 0; t <= LA + LB - az - bz; ++t)
#pragma unroll
                for (int u = 0; u <= LA + LB - az - bz - t; ++u)
#pragma unroll
                    for (int kk = 0; kk < KG; ++kk) {
                        RT s = X[kk][hidx(t, u, 0)];                // (E^{00}_0 = 1)
                        if (az + bz > 0) {
                            s *= E[BE::at(2, az, bz, 0)];
#pragma unroll
                            for (int w = 1; w <= az + bz; ++w) s += E[BE::at(2, az, bz, w)] * X[kk][hidx(t, u, w)];
                        }
                        W[kk][cart_index(t, u)] = s;
                    }
#pragma unroll
            for (int ay = 0; ay <= LA - az; ++ay)
#pragma unroll
                for (int by = 0; by <= LB - bz; ++by) {
                    const int ax = LA - az - ay, bx = LB - bz - by;
                    const RT fab = static_cast<RT>(cart_norm(ax, ay, az) * cart_norm(bx, by, bz));
                    RT s[KG];
#pragma unroll
                    for (int kk = 0; kk < KG; ++kk) {
                        s[kk] = RT(0);
#pragma unroll
                        for (int t = 0; t <= ax + bx; ++t) {
                            RT y = W[kk][cart_index(t, 0)];
                            if (ay + by > 0) {
                                y *= E[BE::at(1, ay, by, 0)];
#pragma unroll
                                for (int u = 1; u <= ay + by; ++u) y += E[BE::at(1, ay, by, u)] * W[kk][cart_index(t, u)];
                            }
                            s[kk] += ax + bx > 0 ? E[BE::at(0, ax, bx, t)] * y : y;
                        }
                        s[kk] *= fab;
                    }
                    row(cart_index(ay, az), cart_index(by, bz), s);
                }
        }
}

// v[r][kk] = (row r | cd, contraction kk) of the quartet (staged bra pair,
// ket pair records rk with nkp primitive pairs); r = (ka*nB + kb)*NAB +
// ia*NB + jb, kk = kc*nD + kd - kg*KG (compact contraction indices over the
// blocks' actual counts).
// Loop order: bra primitives outer; for each, the ket primitives inner,
// where the ket step X_tuv (bra Hermite index tuv) of every primitive
// quartet is summed with its ket contraction coefficients,
// Xs[kk]_tuv = sum_ik c_ik[kk] X_tuv(ib, ik); the bra Hermite->Cartesian
// step, linear in X, then runs once per bra primitive instead of once per
// primitive quartet (the reference applies it per primitive quartet,
// aimd/qc/integrals.py:777-842).
// RS = false: R_tuv of each primitive quartet is computed here; RS = true:
// it is read from Rs, [ik][ib][NH(L)] R_tuv / sqrt(p + q) staged by the CTA
// (stage_r below) once for all the columns of the ket pair.
template <int CX, int CY, typename RT, bool RS, typename Boys>
__device__ __forceinline__ void eri_column_bra_outer(const BraStageT<RT>& st, const double* __restrict__ rk, int nkp, int ic,
                                           int id, int kg, RT (&v)[QClass<CX, CY>::NROW][QClass<CX, CY>::KG],
                                           const RT* __restrict__ Rs, int ib0, int ib1, int nk, Boys boys) {
    using Q = QClass<CX, CY>;
    using BE = BraE<Q::LA, Q::LB>;
    constexpr int LA = Q::LA, LB = Q::LB, LC = Q::LC, LD = Q::LD, LAB = Q::LAB, LCD = Q::LCD, L = Q::L;
    const int cx = cart_x(LC, ic), cy = cart_y(LC, ic), cz = cart_z(LC, ic);
    const int dx = cart_x(LD, id), dy = cart_y(LD, id), dz = cart_z(LD, id);
    const RT fcd = static_cast<RT>(cart_norm(cx, cy, cz) * cart_norm(dx, dy, dz));
#pragma unroll
    for (int r = 0; r < Q::NROW; ++r)
#pragma unroll
        for (int k = 0; k < Q::KG; ++k) v[r][k] = RT(0);
    for (int ib = ib0; ib < ib1; ++ib) {
        const RT* sb = st.SB + ib * SBW;
        RT Xs[Q::KG][Q::NHB];
#pragma unroll
        for (int k = 0; k < Q::KG; ++k)
#pragma unroll
            for (int h = 0; h < Q::NHB; ++h) Xs[k][h] = RT(0);
        for (int ik = 0; ik < nkp; ++ik) {
            const KetRecT<RT> k = load_ket<RT>(rk + (size_t)ik * PPW);
            const RT q = k.a + k.b, oo2q = RT(0.5) / q;
            // ket E coefficients of this column only (box t2 <= cx+dx, ...)
            RT ex[LCD + 1], ey[LCD + 1], ez[LCD + 1];
            {
                RT e[LC + 1][LD + 1][LCD + 1];
                hermite_e<LC, LD>(k.QAx, k.QBx, oo2q, RT(1), e);
                select_row<LC, LD, LCD>(e, cx, dx, ex);
                hermite_e<LC, LD>(k.QAy, k.QBy, oo2q, RT(1), e);
                select_row<LC, LD, LCD>(e, cy, dy, ey);
                hermite_e<LC, LD>(k.QAz, k.QBz, oo2q, RT(1), e);
                select_row<LC, LD, LCD>(e, cz, dz, ez);
            }
            RT ck[Q::KG];
#pragma unroll
            for (int i = 0; i < Q::KG; ++i) {
                RT c = k.c[0];
#pragma unroll
                for (int j = 1; j < Q::KCD; ++j)
                    if (j == kg * Q::KG + i) c = k.c[j];
                ck[i] = c * (fcd * k.K * (RT(2) * oo2q));
            }
            // ket step: Xs[kk]_h += ck[kk] sum_{k in box(cd)} (-1)^|k| E^{cd}_k R_{h+k},
            // box entries outer, so that a column's box conditions are tested
            // once per entry and not once per (entry, h); with several
            // contraction combinations the sum is formed once and then scaled
            auto ket_step = [&](const auto& R) {
                RT X[Q::NHB];
#pragma unroll
                for (int h = 0; h < Q::NHB; ++h) X[h] = Q::KG > 1 ? RT(0) : Xs[0][h];
                const RT sc = Q::KG > 1 ? RT(1) : ck[0];
#pragma unroll
                for (int t2 = 0; t2 <= LCD; ++t2) {
                    if (t2 > cx + dx) continue;
#pragma unroll
                    for (int u2 = 0; u2 <= LCD - t2; ++u2) {
                        if (u2 > cy + dy) continue;
                        const RT exy = sc * (((t2 + u2) & 1) ? -ex[t2] * ey[u2] : ex[t2] * ey[u2]);
#pragma unroll
                        for (int v2 = 0; v2 <= LCD - t2 - u2; ++v2) {
                            if (v2 > cz + dz) continue;
                            const RT e = (v2 & 1) ? -exy * ez[v2] : exy * ez[v2];
#pragma unroll
                            for (int t = 0; t <= LAB; ++t)
#pragma unroll
                                for (int u = 0; u <= LAB - t; ++u)
#pragma unroll
                                    for (int w = 0; w <= LAB - t - u; ++w)
                                        X[hidx(t, u, w)] += e * R[hidx(t + t2, u + u2, w + v2)];
                        }
                    }
                }
#pragma unroll
                for (int h = 0; h < Q::NHB; ++h) {
                    if constexpr (Q::KG > 1) Xs[0][h] += ck[0] * X[h];
                    else Xs[0][h] = X[h];
                }
#pragma unroll
                for (int kk = 1; kk < Q::KG; ++kk) {
                    if (kk >= nk) continue;
#pragma unroll
                    for (int h = 0; h < Q::NHB; ++h) Xs[kk][h] += ck[kk] * X[h];
                }
            };
            if constexpr (RS) {
                ket_step(Rs + (size_t)(ik * st.i.nbp + ib) * nherm(L));
            } else {
                const BraPrim<RT> b = load_bra(sb);
                const RT rs = rsqrt_t(b.p + q);
                RT R[nherm(L)];
                hermite_r_scaled<L>(b.p * q * (rs * rs), b.X - k.Qx, b.Y - k.Qy, b.Z - k.Qz, rs, R, boys);
                ket_step(R);
            }
        }
        // bra step, once per bra primitive:
        // v[(ka,kb),ab][kk] += C[ka,kb] f_ab sum_box E^{ab}_tuv Xs[kk]_tuv
        bra_rows<LA, LB, Q::KG>(st.E + (size_t)ib * BE::SIZE, Xs, [&](int ia, int jb, const RT (&s)[Q::KG]) {
#pragma unroll
            for (int kab = 0; kab < Q::KAB; ++kab)
#pragma unroll
                for (int kk = 0; kk < Q::KG; ++kk) v[kab * Q::NAB + ia * Q::NB + jb][kk] += sb[8 + kab] * s[kk];
        });
    }
}

// Ket ss: one column, R_tuv is the ket step itself. Ket primitives outermost,
// bra primitives inner, the bra step per primitive quartet: the order for bra
// pairs with many primitives (ss, ps, pp). The bra-contracted rows A of one
// ket primitive meet its nk contraction combinations once.
template <int CX, int CY, typename RT, typename Boys>
__device__ __forceinline__ void eri_column_ket_outer(const BraStageT<RT>& st, const double* __restrict__ rk, int nkp,
                                                     int kg, RT (&v)[QClass<CX, CY>::NROW][QClass<CX, CY>::KG],
                                                     int ib0, int ib1, int nk, Boys boys) {
    using Q = QClass<CX, CY>;
    using BE = BraE<Q::LA, Q::LB>;
    constexpr int LA = Q::LA, LB = Q::LB, L = Q::L;
    static_assert(Q::LCD == 0, "ket ss");
    const int nab = st.i.nA * st.i.nB;
#pragma unroll
    for (int r = 0; r < Q::NROW; ++r)
#pragma unroll
        for (int k = 0; k < Q::KG; ++k) v[r][k] = RT(0);
    for (int ik = 0; ik < nkp; ++ik) {
        const KetRecT<RT> k = load_ket<RT>(rk + (size_t)ik * PPW);
        const RT q = k.a + k.b;
        RT A[Q::NROW];
#pragma unroll
        for (int r = 0; r < Q::NROW; ++r) A[r] = RT(0);
        for (int ib = ib0; ib < ib1; ++ib) {
            const RT* sb = st.SB + ib * SBW;
            const BraPrim<RT> b = load_bra(sb);
            const RT rs = rsqrt_t(b.p + q);
            RT R[1][nherm(L)];
            hermite_r_scaled<L>(b.p * q * (rs * rs), b.X - k.Qx, b.Y - k.Qy, b.Z - k.Qz, rs, R[0], boys);
            bra_rows<LA, LB, 1>(st.E + (size_t)ib * BE::SIZE, R, [&](int ia, int jb, const RT (&s)[1]) {
#pragma unroll
                for (int kab = 0; kab < Q::KAB; ++kab)
                    if (kab == 0 || kab < nab) A[kab * Q::NAB + ia * Q::NB + jb] += sb[8 + kab] * s[0];
            });
        }
        const RT ck0 = k.K / q;
#pragma unroll
        for (int kk = 0; kk < Q::KG; ++kk) {
            if (kk > 0 && kk >= nk) continue;
            RT c = k.c[0];
#pragma unroll
            for (int j = 1; j < Q::KCD; ++j)
                if (j == kg * Q::KG + kk) c = k.c[j];
            c *= ck0;
#pragma unroll
            for (int r = 0; r < Q::NROW; ++r) v[r][kk] += A[r] * c;
        }
    }
}

// v[ic][r][kk] = (row r | ic id, contraction kk) for the NC columns of one
// id (column-blocked items): the ket-outer order with R_tuv of each
// primitive quartet computed once and applied to every column; the ket E
// rows of a column come from the per-primitive table at compile-time ic.
template <int CX, int CY, typename RT, typename Boys>
__device__ __forceinline__ void eri_cols_ket_outer(const BraStageT<RT>& st, const double* __restrict__ rk, int nkp,
                                                   int id, int kg,
                                                   RT (&v)[QClass<CX, CY>::NC][QClass<CX, CY>::NROW][QClass<CX, CY>::KG],
                                                   int ib0, int ib1, int nk, Boys boys) {
    using Q = QClass<CX, CY>;
    using BE = BraE<Q::LA, Q::LB>;
    constexpr int LA = Q::LA, LB = Q::LB, LC = Q::LC, LD = Q::LD, LAB = Q::LAB, LCD = Q::LCD, L = Q::L;
    const int dx = LD ? cart_x(LD, id) : 0, dy = LD ? cart_y(LD, id) : 0, dz = LD ? cart_z(LD, id) : 0;
    const RT fd = static_cast<RT>(cart_norm(dx, dy, dz));
    const int nab = st.i.nA * st.i.nB;
#pragma unroll
    for (int c = 0; c < Q::NC; ++c)
#pragma unroll
        for (int r = 0; r < Q::NROW; ++r)
#pragma unroll
            for (int k = 0; k < Q::KG; ++k) v[c][r][k] = RT(0);
    for (int ik = 0; ik < nkp; ++ik) {
        const KetRecT<RT> k = load_ket<RT>(rk + (size_t)ik * PPW);
        const RT q = k.a + k.b, oo2q = RT(0.5) / q;
        // ket E of this id: ex[i][t] = E^{i, dx}_t for every i <= LC
        RT ex[LC + 1][LCD + 1], ey[LC + 1][LCD + 1], ez[LC + 1][LCD + 1];
        {
            RT e[LC + 1][LD + 1][LCD + 1];
            hermite_e<LC, LD>(k.QAx, k.QBx, oo2q, RT(1), e);
            select_j<LC, LD, LCD>(e, dx, ex);
            hermite_e<LC, LD>(k.QAy, k.QBy, oo2q, RT(1), e);
            select_j<LC, LD, LCD>(e, dy, ey);
            hermite_e<LC, LD>(k.QAz, k.QBz, oo2q, RT(1), e);
            select_j<LC, LD, LCD>(e, dz, ez);
        }
        RT ck[Q::KG];
#pragma unroll
        for (int i = 0; i < Q::KG; ++i) {
            RT c = k.c[0];
#pragma unroll
            for (int j = 1; j < Q::KCD; ++j)
                if (j == kg * Q::KG + i) c = k.c[j];
            ck[i] = c * (fd * k.K * (RT(2) * oo2q));
        }
        for (int ib = ib0; ib < ib1; ++ib) {
            const RT* sb = st.SB + ib * SBW;
            const BraPrim<RT> b = load_bra(sb);
            const RT rs = rsqrt_t(b.p + q);
            RT R[nherm(L)];
            hermite_r_scaled<L>(b.p * q * (rs * rs), b.X - k.Qx, b.Y - k.Qy, b.Z - k.Qz, rs, R, boys);
            const RT* E = st.E + (size_t)ib * BE::SIZE;
#pragma unroll
            for (int ic = 0; ic < Q::NC; ++ic) {
                const int cx = cart_x(LC, ic), cy = cart_y(LC, ic), cz = cart_z(LC, ic);
                const RT fc = static_cast<RT>(cart_norm(cx, cy, cz));
                RT X[1][Q::NHB];
#pragma unroll
                for (int h = 0; h < Q::NHB; ++h) X[0][h] = RT(0);
#pragma unroll
                for (int t2 = 0; t2 <= LCD; ++t2) {
                    if (t2 > cx + dx) continue;
#pragma unroll
                    for (int u2 = 0; u2 <= LCD - t2; ++u2) {
                        if (u2 > cy + dy) continue;
                        const RT exy = fc * (((t2 + u2) & 1) ? -ex[cx][t2] * ey[cy][u2] : ex[cx][t2] * ey[cy][u2]);
#pragma unroll
                        for (int v2 = 0; v2 <= LCD - t2 - u2; ++v2) {
                            if (v2 > cz + dz) continue;
                            const RT e = (v2 & 1) ? -exy * ez[cz][v2] : exy * ez[cz][v2];
#pragma unroll
                            for (int t = 0; t <= LAB; ++t)
#pragma unroll
                                for (int u = 0; u <= LAB - t; ++u)
#pragma unroll
                                    for (int w = 0; w <= LAB - t - u; ++w)
                                        X[0][hidx(t, u, w)] += e * R[hidx(t + t2, u + u2, w + v2)];
                        }
                    }
                }
                // bra step of column ic
                bra_rows<LA, LB, 1>(E, X, [&](int ia, int jb, const RT (&s)[1]) {
#pragma unroll
                    for (int kab = 0; kab < Q::KAB; ++kab) {
                        if (kab > 0 && kab >= nab) continue;
                        const RT c = sb[8 + kab] * s[0];
#pragma unroll
                        for (int kk = 0; kk < Q::KG; ++kk)
                            if (kk == 0 || kk < nk) v[ic][kab * Q::NAB + ia * Q::NB + jb][kk] += c * ck[kk];
                    }
                });
            }
        }
    }
}

// (row r | cd) of a quartet column, nk contraction combinations of the ket:
// bra-outer order (the bra step once per bra primitive) for the d-shell bra
// classes, whose pairs have few primitives; ket-outer order for ss, ps and pp
// bras against ss kets (against p kets: column blocks, and here the diagonal
// quartets of the Schwarz bounds).
template <int CX, int CY, typename RT, bool RS = false, typename Boys = BoysSeries>
__device__ __forceinline__ void eri_column(const BraStageT<RT>& st, const double* __restrict__ rk, int nkp, int ic,
                                           int id, int kg, RT (&v)[QClass<CX, CY>::NROW][QClass<CX, CY>::KG],
                                           const RT* __restrict__ Rs, int ib0, int ib1, int nk, Boys boys = Boys()) {
    if constexpr (RS || CX >= 3 || CY > 0)
        eri_column_bra_outer<CX, CY, RT, RS>(st, rk, nkp, ic, id, kg, v, Rs, ib0, ib1, nk, boys);
    else
        eri_column_ket_outer<CX, CY, RT>(st, rk, nkp, kg, v, ib0, ib1, nk, boys);
}

// Everything the quartet kernels share.
struct QuartetArgs {
    PairView pv;
    BlockView bv;
    const double* sortedQ;      // [npair]
    const int64_t* counts;      // [NSEG][npair + 1] kept ket prefix length per (ket segment, bra position)
    // mixed precision: [NSEG][npair + 1] prefix with Q1 Q2 >= the FP32
    // cutoff (evaluated in FP64); the rest of the kept prefix runs in FP32.
    // nullptr: everything in FP64.
    const int64_t* counts_hi;
    const int* seg_start;       // [NSEG + 1] sorted position of each segment (device)
    const int4* meta;           // [3][npair] what an item needs of the pair at a sorted position (PairMeta)
    const double* boys;         // Boys tables of all orders (device)
    int npair;
    int cls_start[NCLS + 1];    // sorted positions of each angular class (geometry independent)
    int nao;
};

// One pair by its sorted position: three 16-byte loads, neighbouring positions
// side by side, where pair index -> blocks -> contractions, AOs and atoms was a
// chain of three dependent loads at the start of every item.
struct PairMeta {
    int P, npp, nA, nB, oA, oB, aA, aB, A, B;
    const double* rec;      // primitive records
};
__device__ __forceinline__ PairMeta load_meta(const QuartetArgs& a, int pos) {
    const int4 u = __ldg(a.meta + pos), v = __ldg(a.meta + a.npair + pos), w = __ldg(a.meta + 2 * a.npair + pos);
    const int64_t slot = static_cast<int64_t>((static_cast<uint64_t>(static_cast<unsigned>(w.w)) << 32) | static_cast<unsigned>(w.z));
    return PairMeta{u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w, w.x, w.y, a.pv.rec + slot * PPW};
}

// Ket range [b, e) of segment seg for bra position spos that the kernels of
// arithmetic type RT evaluate: the FP64 prefix, or the FP32 tail.
template <typename RT>
__device__ __forceinline__ void ket_range(const QuartetArgs& a, int seg, int spos, int64_t& b, int64_t& e) {
    const size_t i = (size_t)seg * (a.npair + 1) + spos;
    const int64_t cnt = a.counts[i];
    int64_t hi = cnt;
    if (a.counts_hi) hi = a.counts_hi[i] < cnt ? a.counts_hi[i] : cnt;
    if constexpr (sizeof(RT) == sizeof(double)) {
        b = 0;
        e = hi;
    } else {
        b = hi;
        e = a.counts_hi ? cnt : hi;
    }
}

// ---------------------------------------------------------------- work plan
// The class kernels are persistent: their CTAs take chunks of (bra pair,
// ket window) from a device counter until the launch's plan is used up, so
// that the few heavy bras (many primitives, long ket lists) are spread over
// many CTAs instead of setting the kernel's duration. A plan holds, per bra
// of the class, the exclusive prefix of its chunk counts; chunk j of nch
// covers the bra's work units [W j / nch, W (j + 1) / nch) in ket segment
// order. Work of a ket pair of segment sub: bra primitive pairs x twice
// the segment's typical ket primitive pairs x the column items per pair.
struct WorkPlan {
    const int* off;     // [nbra + 1] chunk prefix over the bras of the class (off[nbra]: chunks)
    int* next;          // chunk counter of the launch (zeroed with the plan)
    const int* pq;      // primitive quartets per split column item of the launch
};

__host__ __device__ constexpr int ket_prims2(int ppb) {
    return ppb == 0 ? 2 : ppb == 1 ? 5 : ppb == 2 ? 11 : ppb == 3 ? 23 : ppb == 4 ? 47 : 80;
}

template <int CX, int CY>
__device__ __forceinline__ int64_t ket_work(int sub);

// Work units of bra position spos against ket class CY in the FP64 (w[0]) and
// FP32 (w[1]) ket ranges.
template <int CX, int CY>
__device__ void bra_work(const QuartetArgs& q, int spos, int64_t (&w)[2]) {
    w[0] = w[1] = 0;
    for (int sub = 0; sub < NSUB; ++sub) {
        const size_t i = (size_t)(CY * NSUB + sub) * (q.npair + 1) + spos;
        const int64_t cnt = q.counts[i], hi = q.counts_hi && q.counts_hi[i] < cnt ? q.counts_hi[i] : cnt;
        const int64_t unit = ket_work<CX, CY>(sub);
        w[0] += hi * unit;
        w[1] += (cnt - hi) * unit;
    }
    const int npp = load_meta(q, spos).npp;
    w[0] *= npp;
    w[1] *= npp;
}

// Kets [k0, k1) of a segment of len kets, each of weight wk, whose work
// starts inside the window [w0, w1) (acc: work of the segments before).
__device__ __forceinline__ void window_kets(int64_t w0, int64_t w1, int64_t acc, int64_t wk, int64_t len,
                                            int64_t& k0, int64_t& k1) {
    auto first = [&](int64_t x) { return x <= 0 ? int64_t(0) : ((x + wk - 1) / wk < len ? (x + wk - 1) / wk : len); };
    k0 = first(w0 - acc);
    k1 = first(w1 - acc);
}

// Chunk j of nch of a bra of W work units: [W j / nch, W (j + 1) / nch),
// without forming W j.
__device__ __forceinline__ int64_t chunk_edge(int64_t W, int j, int nch) {
    const int64_t q = W / nch, r = W % nch;
    return q * j + (r * j) / nch;
}

// The next chunk of the launch for this CTA (warp 0 calls it): lane 0 takes
// it from the counter, the lanes search its bra together, 32 entries a step
// (last b with off[b] <= c; a lone thread's binary search was a chain of a
// dozen loads that the CTA waited for, once a chunk). c = -1 when the plan is
// used up. Chunks are taken from the last on: bras of many primitives come
// last in the order, and the long chunks should not be the launch's tail.
__device__ __forceinline__ void next_chunk(const WorkPlan& plan, int nbra, int total, int& c, int& b) {
    const int lane = threadIdx.x & 31;
    int cc = 0;
    if (lane == 0) cc = atomicAdd(plan.next, 1);
    cc = __shfl_sync(0xffffffffu, cc, 0);
    c = cc < total ? total - 1 - cc : -1;
    int lo = 0, hi = nbra;                              // off[lo] <= c < off[hi]
    while (c >= 0 && hi - lo > 1) {
        const int step = (hi - lo + 31) / 32, at = lo + lane * step;
        const unsigned le = __ballot_sync(0xffffffffu, at < hi && plan.off[at] <= c);
        lo += (31 - __clz(le)) * step;                  // lane 0 always holds: le != 0
        hi = lo + step < hi ? lo + step : hi;
    }
    b = lo;
}

__device__ __forceinline__ void load_info(const PairMeta& m, BraInfo& st) {
    st.P1 = m.P;
    st.A = m.A;
    st.B = m.B;
    st.nbp = m.npp;
    st.rec = m.rec;
    st.aA = m.aA;
    st.aB = m.aB;
    st.nA = m.nA;
    st.nB = m.nB;
    st.oA = m.oA;
    st.oB = m.oB;
}
// by pair index (the Schwarz bounds, before the pairs are sorted)
__device__ __forceinline__ void load_info(const QuartetArgs& a, int P1, BraInfo& st) {
    st.P1 = P1;
    st.A = a.pv.pa_blk[P1];
    st.B = a.pv.pb_blk[P1];
    st.nbp = a.pv.npp[P1];
    st.rec = a.pv.rec + a.pv.slot[P1] * PPW;
    st.aA = a.bv.atom[st.A];
    st.aB = a.bv.atom[st.B];
    st.nA = a.bv.ncon[st.A];
    st.nB = a.bv.ncon[st.B];
    st.oA = a.bv.ao[st.A];
    st.oB = a.bv.ao[st.B];
}
// The stage in the shared array E: [nbp][SBW] scalars, then the E tables of
// `size` elements a primitive, then (gradients) the dE/dX_AB tables.
template <typename RT>
__device__ __forceinline__ BraStageT<RT> stage_view(const BraInfo& info, RT* E, int size) {
    RT* e = E + info.nbp * SBW;
    return BraStageT<RT>{info, E, e, e + info.nbp * size};
}

// The bra stage holds vectors of 16 bytes: what lies before it in shared memory
// is rounded up to a multiple of four elements (of either type).
__host__ __device__ constexpr size_t even(size_t n) { return (n + 1) & ~(size_t)1; }
__host__ __device__ constexpr size_t fours(size_t n) { return (n + 3) & ~(size_t)3; }

// How the quartets of one kernel evaluate the Boys function of order L: from
// the shared table (copied by the CTA before its first chunk) or by series.
template <int L, typename RT, bool TABLE>
struct BoysOf {
    static constexpr bool table = TABLE && sizeof(RT) == sizeof(double);
    static_assert(!table || L <= BOYS_MAX_N, "order without a table");
    using type = std::conditional_t<table, BoysShared, BoysSeries>;
    static constexpr int elems = table ? BOYS_COLS * boys_rows(L) : 0;      // doubles of shared memory
    __device__ static type get(const double* shared) {
        if constexpr (table) return type{shared};
        else return type{};
    }
    __device__ static void stage(const double* tables, double* shared) {
        if constexpr (table) {
            const double2* src = reinterpret_cast<const double2*>(tables + boys_offset(L));
#pragma unroll 4
            for (int i = threadIdx.x; i < elems / 2; i += blockDim.x) reinterpret_cast<double2*>(shared)[i] = __ldg(src + i);
        }
    }
};

// CTA sizes. The class kernels hold up to 255 registers a thread, so that an
// SM runs eight of their warps: as two CTAs of four or one of eight
// (class_shape picks per context). Small CTAs wait less for one
// another and for the start and end of a chunk; large ones share one copy of
// the K rows, the D rows and the Boys table, which together pass half of an
// SM's shared memory at 800 AOs.
constexpr int CLASS_THREADS = 256;      // the largest

struct JKArgs {
    QuartetArgs q;
    const double* D;    // [nao][nao], symmetric
    facc* J;            // un-symmetrised accumulators, same shape (fixed point)
    facc* K;
    const double* dmax; // device scalar max |D|: the fixed-point scale of J and K is jk_fix_for(*dmax)
    // density-weighted screening (difference densities): skip a quartet when
    // Q1 Q2 max|D| over its six density blocks < dthr; bmax = nullptr: off
    const double* bmax; // [nblock][nblock] max |D| per block pair (all sets)
    int nblock;
    double dthr;
    size_t rbuf;        // elements of the kernel's staged-R buffer (set per launch)
    // 1: the K rows of the bra functions accumulate in global memory (set per
    // launch when the per-CTA shared rows, NF x nao doubles, would not fit)
    int kglobal;
    // 1: the bra functions' rows of D are read from D itself (set per launch
    // when they would not fit beside the K rows), 0: staged in shared memory
    int dglobal;
    WorkPlan plan;      // chunks of the launch (set per launch)
};

// Digest the NCB columns (ic0 + c, id) of a quartet (all ket contractions kk).
// Each tensor element the block reaches is visited
// n_gen = (A==B ? 2:1)(C==D ? 2:1)(P1==P2 ? 2:1) times under the 8 index maps,
// so each image carries g = 1/n_gen:
//   J[m,n] += 2g v D[l,s],  J[l,s] += 2g v D[m,n]
//   K[m,l] += g v D[n,s],   K[n,l] += g v D[m,s],  K[m,s] += g v D[n,l],  K[n,s] += g v D[m,l]
// (m in A, n in B, l in C, s in D); the host forms J + J^T and K + K^T.
// K rows m, n belong to the bra pair: Ksm[slot][col], slot < KA*NA for
// A's functions, then B's; so do the rows of D that K needs, which DA and DB
// point to (staged in shared memory, or D itself where they do not fit). The
// columns of one block of an item share their s: their parts of K[., s] and
// J_ab are summed first.
template <int CX, int CY, bool KGLOBAL, int NCB, typename ST, typename RT>
__device__ __forceinline__ void jk_digest(const JKArgs& a, const ST& st, const PairMeta& ket, int ic0, int id, int kg,
                                          const RT (&v)[NCB][QClass<CX, CY>::NROW][QClass<CX, CY>::KG], double* Jt,
                                          unsigned* Ksm, const double* DA, const double* DB, double fx) {
    using Q = QClass<CX, CY>;
    const int nC = ket.nA, nD = ket.nB, oC = ket.oA, oD = ket.oB;
    const double g = (st.i.A == st.i.B ? 0.5 : 1.0) * (ket.A == ket.B ? 0.5 : 1.0) * (st.i.P1 == ket.P ? 0.5 : 1.0);
    const double gf = g * fx;               // scaled to fixed point (a power of two: exact)
    const int n = a.q.nao;
    constexpr int NFA = Q::KA * Q::NA;      // A slots, then B slots
    constexpr int NF = NFA + Q::KB * Q::NB;
    const double* __restrict__ D = a.D;
    // K rows of the bra functions: shared accumulator, or the global K
    // itself (KGLOBAL, for bra classes whose rows would not fit)
    const bool kgl = KGLOBAL || a.kglobal;
    auto kadd = [&](int f, int row, int col, double val) {      // row f of the shared rows is that row of K
        if (kgl) {
            fadd(a.K + (size_t)row * n + col, val, 1.0);
        } else {
            unsigned* p = Ksm + (size_t)f * n + col;
            sadd(p, p + (size_t)NF * n, val, 1.0);
        }
    };
#pragma unroll
    for (int kk = 0; kk < Q::KG; ++kk) {
        const int kq = kg * Q::KG + kk;
        if (kq >= nC * nD) continue;
        const int kc = kq / nD, kd = kq % nD;
        const int l = oC + kc * Q::NC + ic0, sg = oD + kd * Q::ND + id;     // columns l + c
        double dls[NCB], jcd[NCB];
#pragma unroll
        for (int c = 0; c < NCB; ++c) {
            dls[c] = 2.0 * g * __ldg(D + (size_t)(l + c) * n + sg);
            jcd[c] = 0.0;
        }
#pragma unroll
        for (int ka = 0; ka < Q::KA; ++ka)
#pragma unroll
            for (int kb = 0; kb < Q::KB; ++kb) {
                if (ka >= st.i.nA || kb >= st.i.nB) continue;
#pragma unroll
                for (int ia = 0; ia < Q::NA; ++ia)
#pragma unroll
                    for (int jb = 0; jb < Q::NB; ++jb) {
                        const int r = (ka * st.i.nB + kb) * Q::NAB + ia * Q::NB + jb;
                        const int m = ka * Q::NA + ia, nb_ = st.i.oB + kb * Q::NB + jb;
                        const double dmn = DA[(size_t)m * n + nb_];
                        double jab = 0.0;
#pragma unroll
                        for (int c = 0; c < NCB; ++c) {
                            jcd[c] += (double)v[c][r][kk] * dmn;
                            jab += (double)v[c][r][kk] * dls[c];
                        }
                        Jt[r * blockDim.x + threadIdx.x] += jab;
                    }
            }
#pragma unroll
        for (int c = 0; c < NCB; ++c) fadd(a.J + (size_t)(l + c) * n + sg, 2.0 * gf * jcd[c], 1.0);
        // K[m, l] and K[m, sg]: rows of A's functions
#pragma unroll
        for (int ka = 0; ka < Q::KA; ++ka)
#pragma unroll
            for (int ia = 0; ia < Q::NA; ++ia) {
                if (ka >= st.i.nA) continue;
                double s1[NCB], s2 = 0.0;
#pragma unroll
                for (int c = 0; c < NCB; ++c) s1[c] = 0.0;
#pragma unroll
                for (int kb = 0; kb < Q::KB; ++kb)
#pragma unroll
                    for (int jb = 0; jb < Q::NB; ++jb) {
                        if (kb >= st.i.nB) continue;
                        const int r = (ka * st.i.nB + kb) * Q::NAB + ia * Q::NB + jb;
                        const double* row = DB + (size_t)(kb * Q::NB + jb) * n;
                        const double ds = row[sg];
#pragma unroll
                        for (int c = 0; c < NCB; ++c) {
                            s1[c] += (double)v[c][r][kk] * ds;
                            s2 += (double)v[c][r][kk] * row[l + c];
                        }
                    }
                const int f = ka * Q::NA + ia;
#pragma unroll
                for (int c = 0; c < NCB; ++c) kadd(f, st.i.oA + f, l + c, gf * s1[c]);
                kadd(f, st.i.oA + f, sg, gf * s2);
            }
        // K[n, l] and K[n, sg]: rows of B's functions
#pragma unroll
        for (int kb = 0; kb < Q::KB; ++kb)
#pragma unroll
            for (int jb = 0; jb < Q::NB; ++jb) {
                if (kb >= st.i.nB) continue;
                double s1[NCB], s2 = 0.0;
#pragma unroll
                for (int c = 0; c < NCB; ++c) s1[c] = 0.0;
#pragma unroll
                for (int ka = 0; ka < Q::KA; ++ka)
#pragma unroll
                    for (int ia = 0; ia < Q::NA; ++ia) {
                        if (ka >= st.i.nA) continue;
                        const int r = (ka * st.i.nB + kb) * Q::NAB + ia * Q::NB + jb;
                        const double* row = DA + (size_t)(ka * Q::NA + ia) * n;
                        const double ds = row[sg];
#pragma unroll
                        for (int c = 0; c < NCB; ++c) {
                            s1[c] += (double)v[c][r][kk] * ds;
                            s2 += (double)v[c][r][kk] * row[l + c];
                        }
                    }
                const int f = kb * Q::NB + jb;
#pragma unroll
                for (int c = 0; c < NCB; ++c) kadd(NFA + f, st.i.oB + f, l + c, gf * s1[c]);
                kadd(NFA + f, st.i.oB + f, sg, gf * s2);
            }
    }
}

// Queue chunk of the two-stage items (ket_items_r below).
constexpr int KQ_CAP = 256;

// Ket contraction groups of KG combinations that a segment's pairs need: its
// pairs carry 1, 2 or 4 contraction combinations (sub-class contraction
// bucket), stored first in the compact index, so groups past them are empty.
template <int KG, int NKG>
__device__ __forceinline__ int seg_groups(int sub) {
    const int cb = sub % NCONB;
    const int ncs = cb == 0 ? 1 : (cb == 1 ? 2 : 4);
    const int g = (ncs + KG - 1) / KG;
    return g < NKG ? g : NKG;
}
// contraction combinations of a segment's pairs in their group kg
template <int KG>
__device__ __forceinline__ int group_combos(int sub, int kg) {
    const int cb = sub % NCONB, n = (cb == 0 ? 1 : (cb == 1 ? 2 : 4)) - kg * KG;
    return n < KG ? n : KG;
}
template <int CX, int CY>
__device__ __forceinline__ int64_t ket_work(int sub) {
    using Q = QClass<CX, CY>;
    return (int64_t)ket_prims2(sub / NCONB) * Q::NCD * seg_groups<Q::KG, Q::NKG>(sub);
}

// Bra-primitive splits of the column items of a ket segment: an item of a
// pair of many primitive quartets would run them all in one thread while
// the rest of the CTA waits at the next barrier, so such items are split
// over ranges of the bra primitives (about item_pq quartets each: split_length
// of the launch; the partial columns are linear in the quartets and are
// digested one by one).
__device__ __forceinline__ int bra_splits(int nbp, int sub, int item_pq) {
    const int s = nbp * ket_prims2(sub / NCONB) / (2 * item_pq);
    return s < 1 ? 1 : (s > nbp ? nbp : s);
}

// Compact the positions p0 .. p0+m-1 that pass keep() into q.pos[0 .. q.n)
// in position order (per-warp ballots, warps in index order), so that the
// queue, the item dealing and every per-thread partial sum are the same on
// every run. store(slot, pos) records what the caller needs per entry.
template <typename Queue, typename Keep, typename Store>
__device__ __forceinline__ void compact(Queue& q, int p0, int m, Keep keep, Store store) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    int n = 0;
    for (int i0 = 0; i0 < m; i0 += blockDim.x) {
        const int i = i0 + threadIdx.x;
        const bool k = i < m && keep(p0 + i);
        const unsigned mask = __ballot_sync(0xffffffffu, k);
        if (lane == 0) q.wcnt[warp] = __popc(mask);
        __syncthreads();
        int before = n, total = 0;
        for (int w = 0; w < nwarps; ++w) {
            const int c = q.wcnt[w];
            if (w < warp) before += c;
            total += c;
        }
        if (k) store(before + __popc(mask & ((1u << lane) - 1u)), p0 + i);
        n += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) q.n = n;
    __syncthreads();
}

// ---- Flat items
// The column items of one chunk, over all segments of its ket class, are one
// list: item i belongs to the segment sub with pre[sub] <= i < pre[sub + 1],
// and within it to ket pair (i - pre[sub]) % cnt[sub] (column-major:
// neighbouring lanes take the same column of different ket pairs, so that the
// column's box conditions are warp-uniform). Threads walk the list with stride
// blockDim.x and meet no barrier on the way. One list per segment, with a
// barrier after each, left threads idle: at (H2O)32 a bra pair has some 50 ket
// pairs in a segment, and 128 threads share them.
// Where ket pairs are tested (difference builds, gradients), the list runs
// over the pairs that passed, queued eight a thread at a time.
constexpr int LQ_CAP = 8 * 256;     // queue entries: eight a thread
template <typename T>
__device__ __forceinline__ T warp_incl(T v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const T u = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += u;
    }
    return v;
}
struct FlatItems {
    int64_t pre[NSUB + 1];      // items before each segment of the class (of the queued pairs)
    int cnt[NSUB];              // ket pairs of the chunk's window in each segment (of the queued ones)
    int j0[NSUB];               // sorted position (queue slot) of the first of them
    int kcnt[NSUB], kj0[NSUB];  // the whole window: pairs and first sorted position
    int kpre[NSUB + 1];         // pairs before each segment
    int nper[NSUB];             // items per ket pair
    int wsum[32];
    int item_pq;                // primitive quartets per split item of the launch
};

// The window of chunk j of nch of bra position spos (warp 0 calls it, one lane
// per segment): kcnt, kj0, kpre, nper, and the item list over the whole window.
template <int CX, int CY, typename RT>
__device__ __forceinline__ void plan_window(const QuartetArgs& q, int spos, int nbp, int j, int nch, int ncols,
                                            int nkg, int nsp, FlatItems& f) {
    const int sub = threadIdx.x & 31;
    int64_t kb = 0, len = 0, wk = 1;
    if (sub < NSUB) {
        int64_t ke;
        ket_range<RT>(q, CY * NSUB + sub, spos, kb, ke);
        len = ke > kb ? ke - kb : 0;
        wk = ket_work<CX, CY>(sub) * nbp;
    }
    const int64_t incl = warp_incl(len * wk), W = __shfl_sync(0xffffffffu, incl, 31);
    int64_t k0 = 0, k1 = 0;
    if (len > 0)
        window_kets(chunk_edge(W, j, nch), chunk_edge(W, j + 1, nch), incl - len * wk, wk, len, k0, k1);
    const int cnt = k1 > k0 ? static_cast<int>(k1 - k0) : 0;
    const int nper = ncols * nkg * nsp;
    const int kincl = warp_incl(cnt);
    const int64_t iincl = warp_incl(static_cast<int64_t>(cnt) * nper);
    if (sub < NSUB) {
        f.cnt[sub] = f.kcnt[sub] = cnt;
        f.j0[sub] = f.kj0[sub] = q.seg_start[CY * NSUB + sub] + static_cast<int>(kb + k0);
        f.nper[sub] = nper;
        f.kpre[sub + 1] = kincl;
        f.pre[sub + 1] = iincl;
    }
    if (sub == 0) {
        f.kpre[0] = 0;
        f.pre[0] = 0;
    }
}

// Every item of the window: work(sub, pos, r) with pos the ket's sorted
// position and r < nper[sub]. QUEUED: only the ket pairs that pass keep(pos)
// (kept in order, so that items, threads and partial sums are the same on
// every run); queue holds LQ_CAP ints. All threads of the CTA call this.
template <typename Keep, typename Work>
__device__ __forceinline__ void flat_items(FlatItems& f, bool queued, int* queue, Keep keep, Work work) {
    constexpr int PER = 8;                              // pairs a thread tests at a time
    const int cap = PER * static_cast<int>(blockDim.x);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int total = f.kpre[NSUB];
    for (int base = 0; base < total; base += queued ? cap : total) {
        if (queued) {
            if (threadIdx.x < NSUB) f.cnt[threadIdx.x] = 0;
            // PER consecutive pairs a thread
            unsigned mask = 0;
            int s = 0, pos[PER];
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                const int i = base + static_cast<int>(threadIdx.x) * PER + k;
                if (i >= total) continue;
                while (i >= f.kpre[s + 1]) ++s;
                pos[k] = f.kj0[s] + i - f.kpre[s];
                if (keep(pos[k])) mask |= 1u << k;
            }
            const int c = __popc(mask), incl = warp_incl(c);
            if (lane == 31) f.wsum[warp] = incl;
            __syncthreads();
            int slot = incl - c;
            for (int w = 0; w < warp; ++w) slot += f.wsum[w];
            s = 0;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                const int i = base + static_cast<int>(threadIdx.x) * PER + k;
                if (!(mask >> k & 1u)) continue;
                while (i >= f.kpre[s + 1]) ++s;
                queue[slot++] = pos[k];
                atomicAdd(&f.cnt[s], 1);
            }
            __syncthreads();
            if (warp == 0) {
                const int n = lane < NSUB ? f.cnt[lane] : 0;
                const int ni = warp_incl(n);
                const int64_t ii = warp_incl(static_cast<int64_t>(n) * (lane < NSUB ? f.nper[lane] : 0));
                if (lane < NSUB) {
                    f.j0[lane] = ni - n;
                    f.pre[lane + 1] = ii;
                }
            }
            __syncthreads();
        }
        // from the last segment (pairs of the most primitives) to the first, so
        // that the threads part at short items
        int s = NSUB - 1;
        for (int64_t it = f.pre[NSUB] - 1 - threadIdx.x; it >= 0; it -= blockDim.x) {
            while (it < f.pre[s]) --s;
            const unsigned loc = static_cast<unsigned>(it - f.pre[s]), nq = f.cnt[s];
            const unsigned r = loc / nq;
            const int at = f.j0[s] + static_cast<int>(loc - r * nq);
            work(s, queued ? queue[at] : at, static_cast<int>(r));
        }
        if (queued) __syncthreads();
    }
}

// ---- Two-stage items: R_tuv staged in shared memory
// A ket pair of class Y carries NCD Cartesian columns (x contraction
// groups), each one work item; R_tuv of a primitive quartet is the same for
// all of them. For the classes where recomputing it per item costs
// (QClass::RSMEM), each queue chunk is cut into sub-chunks whose primitive quartets
// fit RB_PQ slots of a shared buffer (plus the largest single ket pair),
// and per sub-chunk:
//   stage 1: one thread per primitive quartet (ket pair i, ket primitive ik,
//            bra primitive ib) writes R_tuv / sqrt(p + q) into the buffer;
//   stage 2: the column items of the sub-chunk's ket pairs read it.
template <int L, typename RT>
struct RSmem {
    static constexpr int NH = nherm(L);
    // slots per sub-chunk: about 32 KB of R (FP64; 16 KB of FP32 R)
    static constexpr int RB_PQ = (4096 + NH - 1) / NH;
    // R level recursion in shared memory instead of registers from this L on
    // (it would hold NH(L) values in registers for the whole kernel)
    static constexpr bool INPLACE = L >= 6;
};
template <int L, typename RT>
__host__ __device__ constexpr size_t rsmem_bytes(int max_bra_prims, int max_ket_prims) {
    return sizeof(RT) * (size_t)nherm(L) * (RSmem<L, RT>::RB_PQ + (size_t)max_bra_prims * max_ket_prims);
}

struct KetQueueR {
    int pos[KQ_CAP];
    int wcnt[32];           // per-warp counts of one compaction step
    int pq[KQ_CAP + 1];     // exclusive prefix of primitive quartets over the chunk's entries
    int sc[KQ_CAP];         // sub-chunk of each entry
    int n;
};

// The queue a kernel needs: of the two-stage items, or of the flat ones.
template <bool TWO>
struct QueueOf {
    KetQueueR q;
    __device__ KetQueueR* r() { return &q; }
    __device__ int* flat() { return nullptr; }
};
template <>
struct QueueOf<false> {
    int q[LQ_CAP];
    __device__ KetQueueR* r() { return nullptr; }
    __device__ int* flat() { return q; }
};

// first index in [lo, hi) with a[i] >= key (a non-decreasing)
__device__ __forceinline__ int lower_bound_i(const int* a, int lo, int hi, int key) {
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (a[mid] < key) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// R_tuv / sqrt(p + q) of primitive quartet (bra primitive ib of the stage, ket
// primitive record kr) into out[NH(L)] (shared memory).
template <int L, typename RT>
__device__ __forceinline__ void stage_r(const BraStageT<RT>& st, int ib, const double* __restrict__ kr, RT* out) {
    const double2* r2 = reinterpret_cast<const double2*>(kr);
    const double2 ab = __ldg(r2 + 0), kq = __ldg(r2 + 1), qyz = __ldg(r2 + 2);
    const BraPrim<RT> b = load_bra(st.SB + ib * SBW);
    const RT q = static_cast<RT>(ab.x) + static_cast<RT>(ab.y);
    const RT rs = rsqrt_t(b.p + q), alpha = b.p * q * (rs * rs);
    const RT X = b.X - static_cast<RT>(kq.y), Y = b.Y - static_cast<RT>(qyz.x), Z = b.Z - static_cast<RT>(qyz.y);
    if constexpr (RSmem<L, RT>::INPLACE) {
        hermite_r_scaled<L>(alpha, X, Y, Z, rs, out);
    } else {
        RT R[nherm(L)];
        hermite_r_scaled<L>(alpha, X, Y, Z, rs, R);
#pragma unroll
        for (int h = 0; h < nherm(L); ++h) out[h] = R[h];
    }
}

// The column items of a segment's ket pairs [j0, j0 + cnt) that pass keep(pos),
// r < nper of each; work(pos, r, Rs) receives the ket pair's staged R
// ([ik][ib][NH(L)]). Rbuf holds rsmem_bytes(...) bytes.
template <int L, typename RT, typename Keep, typename Work>
__device__ __forceinline__ void ket_items_r(int nper, int j0, int64_t cnt, KetQueueR& q, int& rot,
                                            const BraStageT<RT>& st, const QuartetArgs& qa, RT* Rbuf, Keep keep,
                                            Work work) {
    constexpr int NH = nherm(L);
    constexpr int B = RSmem<L, RT>::RB_PQ;
    const int lane = threadIdx.x & 31;
    const int nbp = st.i.nbp;
    for (int64_t base = 0; base < cnt; base += KQ_CAP) {
        const int m = static_cast<int>(cnt - base < KQ_CAP ? cnt - base : KQ_CAP);
        compact(q, j0 + static_cast<int>(base), m, keep, [&](int slot, int pos) {
            q.pos[slot] = pos;
            q.pq[slot] = load_meta(qa, pos).npp * nbp;              // primitive quartets of the entry
        });
        const int ne = q.n;
        if (ne == 0) continue;                                      // uniform: q.n is shared
        // warp 0: exclusive prefix of the entries' primitive quartets and
        // their sub-chunks (an entry belongs to the sub-chunk of its last slot)
        if (threadIdx.x < 32) {
            constexpr int PER = KQ_CAP / 32;
            int c[PER], local = 0;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                const int i = lane * PER + k;
                c[k] = i < ne ? q.pq[i] : 0;
                local += c[k];
            }
            int incl = local;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += v;
            }
            __syncwarp();
            int run = incl - local;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                const int i = lane * PER + k;
                if (i < ne) {
                    q.pq[i] = run;
                    q.sc[i] = (run + (c[k] > 0 ? c[k] : 1) - 1) / B;
                    run += c[k];
                }
            }
            if (lane == 31) q.pq[ne] = incl;
        }
        __syncthreads();
        const int k0 = q.sc[0], k1 = q.sc[ne - 1];
        for (int kc = k0; kc <= k1; ++kc) {
            const int f = lower_bound_i(q.sc, 0, ne, kc), l = lower_bound_i(q.sc, f, ne, kc + 1);
            if (f == l) continue;                                   // uniform across the CTA
            const int pq0 = q.pq[f], npq = q.pq[l] - pq0;
            // stage 1: R of every primitive quartet of the sub-chunk
            for (int w = threadIdx.x; w < npq; w += blockDim.x) {
                const int i = lower_bound_i(q.pq, f, l + 1, pq0 + w + 1) - 1;   // last entry with pq <= pq0 + w
                const int rem = pq0 + w - q.pq[i];
                const int ik = rem / nbp, ib = rem - ik * nbp;
                stage_r<L>(st, ib, load_meta(qa, q.pos[i]).rec + (size_t)ik * PPW, Rbuf + (size_t)w * NH);
            }
            __syncthreads();
            // stage 2: the column items of the sub-chunk, column-major as in flat_items
            const int nsc = l - f;
            const int items = nsc * nper;
            int it = static_cast<int>(threadIdx.x) - rot;
            if (it < 0) it += blockDim.x;
            for (; it < items; it += blockDim.x) {
                const int i = f + it % nsc;
                work(q.pos[i], it / nsc, Rbuf + (size_t)(q.pq[i] - pq0) * NH);
            }
            rot = (rot + items) % static_cast<int>(blockDim.x);
            __syncthreads();
        }
    }
}

// The items of the staged bra pair (position spos) in the window that f holds.
template <int CX, int CY, bool KGLOBAL, typename RT, typename Boys>
__device__ __forceinline__ void jk_ket_class(const JKArgs& a, const BraStageT<RT>& st, int spos, double* Jt,
                                             unsigned* Ksm, FlatItems& f, KetQueueR* kq, int* queue, RT* Rbuf,
                                             Boys boys, const double* DA, const double* DB, double fx) {
    using Q = QClass<CX, CY>;
    const double q1 = a.q.sortedQ[spos];
    const double* bm = a.bmax;
    const int nb = a.nblock;
    // difference densities: density-weighted test on the six block pairs
    auto keep = [&](int pos) {
        if (!bm) return true;
        const PairMeta k = load_meta(a.q, pos);
        const int C = k.A, Dd = k.B;
        const double dm = fmax(fmax(bm[st.i.A * nb + st.i.B], bm[C * nb + Dd]),
                               fmax(fmax(bm[st.i.A * nb + C], bm[st.i.A * nb + Dd]),
                                    fmax(bm[st.i.B * nb + C], bm[st.i.B * nb + Dd])));
        return q1 * a.q.sortedQ[pos] * dm >= a.dthr;
    };
    // item r = (contraction group that the segment's pairs carry, bra-primitive split, column block)
    auto work = [&](int sub, int pos, int r, const RT* Rs) {
        const int nkg = seg_groups<Q::KG, Q::NKG>(sub), nsp = bra_splits(st.i.nbp, sub, f.item_pq);
        const int kg = r % nkg, sp = (r / nkg) % nsp, cd = r / (nkg * nsp);
        const int ib0 = st.i.nbp * sp / nsp, ib1 = st.i.nbp * (sp + 1) / nsp;
        const int nk = group_combos<Q::KG>(sub, kg);
        const PairMeta k = load_meta(a.q, pos);
        if constexpr (Q::CBLK) {
            // item = the NC columns of one id
            RT v[Q::NC][Q::NROW][Q::KG];
            eri_cols_ket_outer<CX, CY, RT>(st, k.rec, k.npp, cd, kg, v, ib0, ib1, nk, boys);
            jk_digest<CX, CY, KGLOBAL, Q::NC>(a, st, k, 0, cd, kg, v, Jt, Ksm, DA, DB, fx);
        } else {
            RT v[1][Q::NROW][Q::KG];
            eri_column<CX, CY, RT, Q::RSMEM>(st, k.rec, k.npp, cd / Q::ND, cd % Q::ND, kg, v[0], Rs, ib0, ib1, nk, boys);
            jk_digest<CX, CY, KGLOBAL, 1>(a, st, k, cd / Q::ND, cd % Q::ND, kg, v, Jt, Ksm, DA, DB, fx);
        }
    };
    if constexpr (Q::RSMEM) {
        int rot = 0;
        for (int sub = 0; sub < NSUB; ++sub)
            if (f.kcnt[sub] > 0)
                ket_items_r<Q::L>(f.nper[sub], f.kj0[sub], f.kcnt[sub], *kq, rot, st, a.q, Rbuf, keep,
                                  [&](int pos, int r, const RT* Rs) { work(sub, pos, r, Rs); });
    } else {
        flat_items(f, bm != nullptr, queue, keep,
                   [&](int sub, int pos, int r) { work(sub, pos, r, static_cast<const RT*>(nullptr)); });
    }
}

template <int CX>
struct JKKernel {
    using Q0 = QClass<CX, 0>;
    static constexpr int NROW = Q0::NROW;
    static constexpr int NF = Q0::KA * Q0::NA + Q0::KB * Q0::NB;
    static constexpr int ESIZE = bra_e_size<Q0::LA, Q0::LB>();
    // bra classes above ss: one kernel per ket class, so that each kernel
    // holds the code of one ket class only and the CTAs resident on an SM
    // share their instructions; dd bras accumulate K in global memory
    static constexpr bool SPLIT = CX >= 1;
    static constexpr bool KGLOBAL = CX == 5;
    static constexpr int KROWS = KGLOBAL ? 0 : NF;
};

// The Boys function of the (CX, Y) J/K kernel: from the table, except for the
// two-stage classes (a few per cent of a cc-pVDZ build, with R staged).
template <int CX, int Y, typename RT>
using JKBoys = BoysOf<QClass<CX, Y>::L, RT, !QClass<CX, Y>::RSMEM>;

// Dynamic shared memory: Boys table, per-thread J_ab slots
// [NROW][blockDim], K rows [NF][nao] (unless KGLOBAL), D rows
// [NF][nao] (unless dglobal), staged R, bra stage.

// RT = double: the FP64 quartets; RT = float: the FP32 quartets of the
// mixed-precision path (their J/K contributions still accumulate in FP64).
// YK = ket class of this kernel (-1: the ss bras, whose only ket class is ss).
// Persistent: a CTA runs chunks of the launch's work plan until it is used up.
template <int CX, typename RT, int YK>
__global__ void __launch_bounds__(CLASS_THREADS) jk_bra_kernel(JKArgs a) {
    using KK = JKKernel<CX>;
    using Q0 = QClass<CX, 0>;
    constexpr int Y = YK < 0 ? 0 : YK;      // the unsplit kernel (CX = 0) has one ket class too
    static_assert(YK >= 0 || CX == 0, "bra classes above ss are split by ket class");
    extern __shared__ __align__(16) double smem[];
    const int n = a.q.nao;
    const int krows = a.kglobal ? 0 : KK::KROWS;
    using QY = QClass<CX, Y>;
    using Boys = JKBoys<CX, Y, RT>;
    const int nt = blockDim.x;
    double* btab = smem;                                    // Boys table
    double* Jt = btab + Boys::elems;                        // per-thread J_ab slots
    unsigned* Ksm = reinterpret_cast<unsigned*>(Jt + KK::NROW * nt);   // low words of the K rows, then the high words
    double* Dsm = Jt + KK::NROW * nt + even((size_t)krows * n);       // the bra functions' rows of D
    RT* Rbuf = reinterpret_cast<RT*>(Dsm + (a.dglobal ? 0 : even((size_t)KK::NF * n)));
    RT* Esm = Rbuf + a.rbuf;
    __shared__ BraInfo info;
    __shared__ FlatItems f;
    __shared__ QueueOf<QY::RSMEM> kq;
    __shared__ int sh[2];
    const int nbra = a.q.cls_start[CX + 1] - a.q.cls_start[CX];
    const int total = a.plan.off[nbra];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double fx = jk_fix_for(__ldg(a.dmax));
    if (threadIdx.x == 0) f.item_pq = *a.plan.pq;               // (read after the first barrier)
    bool staged = false;        // the Boys table is in shared memory, and the accumulators are zero
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
        __syncthreads();
        const int c = sh[0], b = sh[1];
        if (c < 0) break;                                       // uniform: c is shared
        const int spos = a.q.cls_start[CX] + b;
        if (!staged) {
            Boys::stage(a.q.boys, btab);
            for (int i = threadIdx.x; i < krows * n + KK::NROW * nt; i += blockDim.x) Jt[i] = 0.0;
            staged = true;
        }
        const BraStageT<RT> st = stage_view(info, Esm, KK::ESIZE);
        if (warp == 0) {
            const int sub = lane < NSUB ? lane : 0;
            plan_window<CX, Y, RT>(a.q, spos, st.i.nbp, c - a.plan.off[b], a.plan.off[b + 1] - a.plan.off[b], QY::NITEM,
                                   seg_groups<QY::KG, QY::NKG>(sub), bra_splits(st.i.nbp, sub, f.item_pq), f);
        }
        stage_bra_e<Q0::LA, Q0::LB>(st);
        const double *DA = a.D + (size_t)info.oA * n, *DB = a.D + (size_t)info.oB * n;
        if (!a.dglobal) {
            constexpr int NFA = Q0::KA * Q0::NA;
            const int na = info.nA * Q0::NA * n, nb = info.nB * Q0::NB * n;
#pragma unroll 4
            for (int i = threadIdx.x; i < na; i += nt) Dsm[i] = __ldg(DA + i);
#pragma unroll 4
            for (int i = threadIdx.x; i < nb; i += nt) Dsm[NFA * n + i] = __ldg(DB + i);
            DA = Dsm;
            DB = Dsm + NFA * n;
        }
        __syncthreads();
        jk_ket_class<CX, Y, KK::KGLOBAL, RT>(a, st, spos, Jt, Ksm, f, kq.r(), kq.flat(), Rbuf,
                                                 Boys::get(btab), DA, DB, fx);
        __syncthreads();
        // flush J_ab: a warp a row sums the threads' slots (in a fixed
        // order) and clears them
        for (int r = warp; r < KK::NROW; r += nt / 32) {
            double val = 0.0;
            for (int t = 0; t < nt; t += 32) {
                val += Jt[r * nt + t + lane];
                Jt[r * nt + t + lane] = 0.0;
            }
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) val += __shfl_xor_sync(0xffffffffu, val, d);
            if (lane != 0 || val == 0.0) continue;
            const int kab = r / Q0::NAB, ab = r % Q0::NAB;
            const int ka = kab / st.i.nB, kb = kab % st.i.nB;
            const int m = st.i.oA + ka * Q0::NA + ab / Q0::NB, nb_ = st.i.oB + kb * Q0::NB + ab % Q0::NB;
            fadd(a.J + (size_t)m * n + nb_, val, fx);
        }
        // flush and clear the K rows
        if (krows > 0) {
            constexpr int NFA = Q0::KA * Q0::NA;
            for (int i = threadIdx.x; i < krows * n; i += blockDim.x) {
                const facc val = join_planes(Ksm[i], Ksm[krows * n + i]);
                if (val == 0) continue;
                Ksm[i] = Ksm[krows * n + i] = 0u;
                const int col = i % n, f_ = i / n;
                const int row = f_ < NFA ? st.i.oA + f_ : st.i.oB + (f_ - NFA);
                atomicAdd(a.K + (size_t)row * n + col, val);     // integer: order-independent
            }
        }
        __syncthreads();
    }
}

// Elements of the staged-R buffer of the (CX, YK) kernel (0 unless two-stage).
template <int CX, int YK, typename RT>
size_t jk_rbuf_elems(int max_bra_prims, int max_ket_prims) {
    if constexpr (YK >= 0) {
        using Q = QClass<CX, YK>;
        if constexpr (Q::RSMEM) return fours(rsmem_bytes<Q::L, RT>(max_bra_prims, max_ket_prims) / sizeof(RT));
    }
    return 0;
}

template <int CX, int Y, typename RT>
size_t jk_smem_bytes(int threads, int nao, int max_bra_prims, size_t rbuf_elems, bool kglobal, bool dglobal) {
    using KK = JKKernel<CX>;
    const size_t krows = kglobal ? 0 : KK::KROWS;
    return sizeof(double) * (even(krows * nao) + (dglobal ? 0 : even((size_t)KK::NF * nao)) +
                             (size_t)KK::NROW * threads + JKBoys<CX, Y, RT>::elems) +
           sizeof(RT) * (rbuf_elems + (size_t)max_bra_prims * (KK::ESIZE + SBW));
}

// ---------------------------------------------------------- Schwarz

// Q[P] = max_ab |(ab|ab)|^(1/2) (the reference's _schwarz_kernel,
// aimd/qc/integrals.py:864-883): one CTA per pair, its threads over (column,
// range of the bra primitives). With one thread a column, a pair of
// contracted s blocks (64 primitive pairs, one column) ran its 4096 primitive
// quartets in one thread.
constexpr int SCHWARZ_THREADS = 64;
template <int CX>
__global__ void __launch_bounds__(SCHWARZ_THREADS) schwarz_kernel(QuartetArgs a, const int* pairs_of_class, double* Qout) {
    using Q = QClass<CX, CX>;
    extern __shared__ __align__(16) double smem[];
    __shared__ BraInfo info;
    __shared__ double diag[Q::KAB][SCHWARZ_THREADS];    // partial (ab|ab) of each contraction combination
    __shared__ unsigned long long qmax;
    const int P = pairs_of_class[blockIdx.x];
    if (threadIdx.x == 0) {
        load_info(a, P, info);
        qmax = 0ull;
    }
    __syncthreads();
    const BraStageT<double> st = stage_view(info, smem, bra_e_size<Q::LA, Q::LB>());
    stage_bra_e<Q::LA, Q::LB>(st);
    __syncthreads();
    static_assert(Q::KG == Q::KCD, "diagonal quartets keep all contraction combinations in one item");
    constexpr int NSP = SCHWARZ_THREADS / Q::NCD;       // ranges of the bra primitives
    const int cd = threadIdx.x % Q::NCD, sp = threadIdx.x / Q::NCD;
    const int ib0 = st.i.nbp * sp / NSP, ib1 = st.i.nbp * (sp + 1) / NSP;
    if (sp < NSP) {
        double m[Q::KAB];
#pragma unroll
        for (int kk = 0; kk < Q::KAB; ++kk) m[kk] = 0.0;
        if (ib1 > ib0) {
            double v[Q::NROW][Q::KCD];
            eri_column<CX, CX>(st, st.i.rec, st.i.nbp, cd / Q::ND, cd % Q::ND, 0, v, static_cast<const double*>(nullptr),
                               ib0, ib1, Q::KCD);
#pragma unroll
            for (int kk = 0; kk < Q::KAB; ++kk)
#pragma unroll
                for (int r = 0; r < Q::NROW; ++r)
                    if (r == kk * Q::NAB + cd) m[kk] = v[r][kk];
        }
#pragma unroll
        for (int kk = 0; kk < Q::KAB; ++kk) diag[kk][threadIdx.x] = m[kk];
    }
    __syncthreads();
    // one thread per (combination, column) sums its ranges in order
    for (int i = threadIdx.x; i < st.i.nA * st.i.nB * Q::NCD; i += SCHWARZ_THREADS) {
        const int kk = i / Q::NCD, c = i % Q::NCD;
        double m = 0.0;
        for (int s = 0; s < NSP; ++s) m += diag[kk][s * Q::NCD + c];
        atomicMax(&qmax, (unsigned long long)__double_as_longlong(fabs(m)));   // bit order = value order
    }
    __syncthreads();
    if (threadIdx.x == 0) Qout[P] = sqrt(__longlong_as_double((long long)qmax));
}

}  // namespace hf
