// One-electron integrals on the device: overlap S, kinetic T and nuclear
// attraction V (nuclei plus optional external point charges, the QM/MM case).
//
// Replaces the CPU get1e path and the reference's getOEI_kernel
// (src/modules/quick_oei_module.f90:69-257, src/gpu/gpu_oei.cu:194,
// src/gpu/gpu_oei.h:193) for closed-shell SCF set-up.  Integrals use the
// McMurchie-Davidson Hermite expansion over QUICK's normalize_basis
// representation (aexp/dcoeff/itype/ncenter, src/modules/quick_basis_module.f90:385-424).
// S and T take one thread per basis-function pair (mu >= nu).  V takes one block per
// shell pair and chunk of charges (oei_shell_kernel); bases whose shells do not have
// QUICK's component order take one thread per function pair and chunk (oei_kernel).
// Results are symmetric and bit-reproducible.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <vector>

#include "quick_b200.h"
#include "common.cuh"

namespace qk {

constexpr int kOeiLmax = 3;              // per function (f)

struct OeiArgs {
    int nbasis, maxcontract, ncharge;
    const int* ncontract;
    const int* itype;      // 3 x nbasis
    const double* aexp;    // maxcontract x nbasis
    const double* dcoeff;  // maxcontract x nbasis
    const int* ncenter;    // 1-based atom index
    const double* xyz;     // 3 x natom
    const double* cxyz;    // 3 x ncharge (nuclei first, then external charges)
    const double* cq;      // ncharge
    const double* boys;
    double *S, *T, *V;     // nbasis^2
};

// Flat index of (t, u, v) among the triples with t + u + v <= 2 * kOeiLmax,
// ordered by total degree, then t descending, then u descending.
constexpr int kTuvMax = (2 * kOeiLmax + 1) * (2 * kOeiLmax + 2) * (2 * kOeiLmax + 3) / 6;
__device__ __forceinline__ int tuv_index(int t, int u, int v) {
    const int L = t + u + v;
    const int before = L * (L + 1) * (L + 2) / 6;           // triples of lower degree
    const int r = L - t;                                     // u + v
    return before + r * (r + 1) / 2 + v;
}

// The triple of a flat index, the index of a triple, and a loop whose index is a
// compile-time constant in its body (the R recursion keeps its values in registers only
// if every index is one).
struct Tuv { int t, u, v; };
__host__ __device__ constexpr int tuv_flat(int t, int u, int v) {
    const int L = t + u + v, r = u + v;
    return L * (L + 1) * (L + 2) / 6 + r * (r + 1) / 2 + v;
}
__host__ __device__ constexpr Tuv tuv_of(int i) {
    for (int L = 0;; ++L)
        for (int t = L; t >= 0; --t)
            for (int u = L - t; u >= 0; --u)
                if (tuv_flat(t, u, L - t - u) == i) return {t, u, L - t - u};
}
template <int N, int I = 0, typename Fn>
__device__ __forceinline__ void unroll_up(Fn&& f) {
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        unroll_up<N, I + 1>(f);
    }
}

// 1-D Hermite coefficients E[i][j][t], i <= li, j <= lj, t <= i + j, for one Cartesian axis.
__device__ __forceinline__ void hermite_E(int li, int lj, double XPA, double XPB, double oo2p, double E0,
                                          double E[kOeiLmax + 1][kOeiLmax + 1][2 * kOeiLmax + 1]) {
    E[0][0][0] = E0;
    for (int i = 0; i <= li; ++i) {
        for (int j = 0; j <= lj; ++j) {
            if (i == 0 && j == 0) continue;
            for (int t = 0; t <= i + j; ++t) {
                double v;
                if (j == 0) {
                    const double a = t > 0 ? E[i - 1][0][t - 1] : 0.0;
                    const double b = t <= i - 1 ? E[i - 1][0][t] : 0.0;
                    const double c = t + 1 <= i - 1 ? E[i - 1][0][t + 1] : 0.0;
                    v = oo2p * a + XPA * b + (t + 1) * c;
                } else {
                    const int tm = i + j - 1;
                    const double a = t > 0 ? E[i][j - 1][t - 1] : 0.0;
                    const double b = t <= tm ? E[i][j - 1][t] : 0.0;
                    const double c = t + 1 <= tm ? E[i][j - 1][t + 1] : 0.0;
                    v = oo2p * a + XPB * b + (t + 1) * c;
                }
                E[i][j][t] = v;
            }
        }
    }
}

// Gaussian products beyond this exponent (exp(-75) = 2.7e-33) contribute nothing that
// a 64-bit sum could show; an element that has no others is 0.
constexpr double kOeiExpMax = 75.0;

// Overlap and kinetic energy of one function pair per thread, from the 1-d overlaps
// s(i, j) = <x_A^i | x_B^j> by s(i+1, j) = PA s(i, j) + (i s(i-1, j) + j s(i, j-1)) / 2p.
__global__ void __launch_bounds__(128) oei_st_kernel(OeiArgs a) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = a.nbasis;
    if (t >= n * (n + 1) / 2) return;
    int mu = (int)((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
    while (mu * (mu + 1) / 2 > t) --mu;
    while ((mu + 1) * (mu + 2) / 2 <= t) ++mu;
    const int nu = t - mu * (mu + 1) / 2;
    const double* A = a.xyz + 3 * (a.ncenter[mu] - 1);
    const double* B = a.xyz + 3 * (a.ncenter[nu] - 1);
    const double AB[3] = {A[0] - B[0], A[1] - B[1], A[2] - B[2]};
    const double r2 = AB[0] * AB[0] + AB[1] * AB[1] + AB[2] * AB[2];
    double s = 0.0, tk = 0.0;
    for (int p = 0; p < a.ncontract[mu]; ++p) {
        const double al = a.aexp[p + a.maxcontract * mu], ca = a.dcoeff[p + a.maxcontract * mu];
        for (int q = 0; q < a.ncontract[nu]; ++q) {
            const double be = a.aexp[q + a.maxcontract * nu];
            const double pz = al + be, oo2p = 0.5 / pz, arg = al * be / pz * r2;
            if (arg > kOeiExpMax) continue;
            double S1[3], T1[3];
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                const int i0 = a.itype[3 * mu + x], j0 = a.itype[3 * nu + x];
                const double PA = -be / pz * AB[x], PB = al / pz * AB[x];
                constexpr int NJ = kOeiLmax + 3;   // j up to l + 2
                double row[NJ], prev[NJ];   // s(i, .) and s(i-1, .)
                row[0] = 1.0;
                for (int j = 1; j <= j0 + 2; ++j) row[j] = PB * row[j - 1] + (j > 1 ? (j - 1) * oo2p * row[j - 2] : 0.0);
                for (int i = 0; i < i0; ++i) {
                    double next[NJ];
                    for (int j = 0; j <= j0 + 2; ++j)
                        next[j] = PA * row[j] + oo2p * ((i ? i * prev[j] : 0.0) + (j ? j * row[j - 1] : 0.0));
                    for (int j = 0; j <= j0 + 2; ++j) { prev[j] = row[j]; row[j] = next[j]; }
                }
                S1[x] = row[j0];
                T1[x] = be * (2 * j0 + 1) * row[j0] - 2.0 * be * be * row[j0 + 2] -
                        (j0 > 1 ? 0.5 * j0 * (j0 - 1) * row[j0 - 2] : 0.0);
            }
            const double sq = sqrt(M_PI / pz);
            const double c = ca * a.dcoeff[q + a.maxcontract * nu] * exp(-arg) * sq * sq * sq;
            s += c * S1[0] * S1[1] * S1[2];
            tk += c * (T1[0] * S1[1] * S1[2] + S1[0] * T1[1] * S1[2] + S1[0] * S1[1] * T1[2]);
        }
    }
    a.S[(size_t)mu * n + nu] = s; a.S[(size_t)nu * n + mu] = s;
    a.T[(size_t)mu * n + nu] = tk; a.T[(size_t)nu * n + mu] = tk;
}

// grid (pairs / 128, charge chunks): chunk y sums the attraction of charges
// [y * chunk, (y + 1) * chunk) into Vpart[y][pair].
__global__ void oei_kernel(OeiArgs a, int chunk, double* __restrict__ Vpart) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = a.nbasis;
    const int npair = n * (n + 1) / 2;
    if (t >= npair) return;
    const int c0 = blockIdx.y * chunk;
    const int c1 = min(a.ncharge, c0 + chunk);
    // t -> (mu, nu), mu >= nu
    int mu = (int)((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
    while (mu * (mu + 1) / 2 > t) --mu;
    while ((mu + 1) * (mu + 2) / 2 <= t) ++mu;
    const int nu = t - mu * (mu + 1) / 2;
    const int la[3] = {a.itype[3 * mu], a.itype[3 * mu + 1], a.itype[3 * mu + 2]};
    const int lb[3] = {a.itype[3 * nu], a.itype[3 * nu + 1], a.itype[3 * nu + 2]};
    const double* A = a.xyz + 3 * (a.ncenter[mu] - 1);
    const double* B = a.xyz + 3 * (a.ncenter[nu] - 1);
    const int Lsum = la[0] + la[1] + la[2] + lb[0] + lb[1] + lb[2];
    double v = 0.0;
    double E[3][kOeiLmax + 1][kOeiLmax + 1][2 * kOeiLmax + 1];
    for (int p = 0; p < a.ncontract[mu]; ++p) {
        const double al = a.aexp[p + a.maxcontract * mu];
        const double ca = a.dcoeff[p + a.maxcontract * mu];
        for (int q = 0; q < a.ncontract[nu]; ++q) {
            const double be = a.aexp[q + a.maxcontract * nu];
            const double cb = a.dcoeff[q + a.maxcontract * nu];
            const double pz = al + be, oo2p = 0.5 / pz, mu_r = al * be / pz;
            double P[3];
            for (int x = 0; x < 3; ++x) {
                P[x] = (al * A[x] + be * B[x]) / pz;
                const double XAB = A[x] - B[x];
                hermite_E(la[x], lb[x], P[x] - A[x], P[x] - B[x], oo2p, exp(-mu_r * XAB * XAB), E[x]);
            }
            const double cc = ca * cb;
            // nuclear attraction: (2 pi / p) sum_tuv E_t E_u E_v R_tuv, with the
            // Hermite Coulomb integrals R built level by level (k = Lsum .. 0) in
            // two flat arrays over t + u + v <= Lsum - k
            const double pref = cc * 2.0 * M_PI / pz;
            const int lx = la[0] + lb[0], ly = la[1] + lb[1], lz = la[2] + lb[2];
            double Ex[2 * kOeiLmax + 1], Ey[2 * kOeiLmax + 1], Ez[2 * kOeiLmax + 1];
            for (int q2 = 0; q2 <= 2 * kOeiLmax; ++q2) {
                Ex[q2] = q2 <= lx ? E[0][la[0]][lb[0]][q2] : 0.0;
                Ey[q2] = q2 <= ly ? E[1][la[1]][lb[1]][q2] : 0.0;
                Ez[q2] = q2 <= lz ? E[2][la[2]][lb[2]][q2] : 0.0;
            }
            double m2p[2 * kOeiLmax + 1];   // (-2p)^k
            m2p[0] = 1.0;
            for (int k = 1; k <= 2 * kOeiLmax; ++k) m2p[k] = m2p[k - 1] * (-2.0 * pz);
            for (int c = c0; c < c1; ++c) {
                const double PC[3] = {P[0] - a.cxyz[3 * c], P[1] - a.cxyz[3 * c + 1], P[2] - a.cxyz[3 * c + 2]};
                const double r2 = PC[0] * PC[0] + PC[1] * PC[1] + PC[2] * PC[2];
                double F[2 * kOeiLmax + 1];
                boys_scaled<2 * kOeiLmax>(pz * r2, 1.0, a.boys, F);
                double Ra[kTuvMax], Rb[kTuvMax];
                double* Rn = Ra;   // level k + 1
                double* Rc = Rb;   // level k
                Rn[0] = m2p[Lsum] * F[Lsum];
                for (int k = Lsum - 1; k >= 0; --k) {
                    const int L = Lsum - k;
                    Rc[0] = m2p[k] * F[k];
                    for (int tt = 0; tt <= L; ++tt)
                        for (int uu = 0; uu <= L - tt; ++uu)
                            for (int vv = 0; vv <= L - tt - uu; ++vv) {
                                if (tt + uu + vv == 0) continue;
                                double r;
                                if (tt > 0) {
                                    r = PC[0] * Rn[tuv_index(tt - 1, uu, vv)];
                                    if (tt > 1) r += (tt - 1) * Rn[tuv_index(tt - 2, uu, vv)];
                                } else if (uu > 0) {
                                    r = PC[1] * Rn[tuv_index(tt, uu - 1, vv)];
                                    if (uu > 1) r += (uu - 1) * Rn[tuv_index(tt, uu - 2, vv)];
                                } else {
                                    r = PC[2] * Rn[tuv_index(tt, uu, vv - 1)];
                                    if (vv > 1) r += (vv - 1) * Rn[tuv_index(tt, uu, vv - 2)];
                                }
                                Rc[tuv_index(tt, uu, vv)] = r;
                            }
                    double* tmp = Rn; Rn = Rc; Rc = tmp;
                }
                // Rn holds level 0
                double vc = 0.0;
                for (int tt = 0; tt <= lx; ++tt)
                    for (int uu = 0; uu <= ly; ++uu)
                        for (int vv = 0; vv <= lz; ++vv) vc += Ex[tt] * Ey[uu] * Ez[vv] * Rn[tuv_index(tt, uu, vv)];
                v -= a.cq[c] * pref * vc;
            }
        }
    }
    Vpart[(size_t)blockIdx.y * npair + t] = v;
}

// exponent along `axis` of Cartesian component i of an L shell in QUICK's order (z
// exponent ascending, then y)
__host__ __device__ constexpr int cart_exp(int L, int i, int axis) {
    int k = 0;
    for (int z = 0; z <= L; ++z)
        for (int y = 0; y <= L - z; ++y, ++k)
            if (k == i) return axis == 0 ? L - y - z : axis == 1 ? y : z;
    return 0;
}

template <int LI, int LJ>
__device__ __forceinline__ void hermite_E_fixed(double XPA, double XPB, double oo2p, double E0,
                                                double (&E)[LI + 1][LJ + 1][LI + LJ + 1]) {
#pragma unroll
    for (int i = 0; i <= LI; ++i)
#pragma unroll
        for (int j = 0; j <= LJ; ++j)
#pragma unroll
            for (int t = 0; t <= LI + LJ; ++t) E[i][j][t] = 0.0;
    E[0][0][0] = E0;
#pragma unroll
    for (int i = 0; i <= LI; ++i)
#pragma unroll
        for (int j = 0; j <= LJ; ++j) {
            if (i == 0 && j == 0) continue;
#pragma unroll
            for (int t = 0; t <= i + j; ++t) {
                double v;
                if (j == 0) {
                    const double a = t > 0 ? E[i - 1][0][t - 1] : 0.0;
                    const double b = t <= i - 1 ? E[i - 1][0][t] : 0.0;
                    const double c = t + 1 <= i - 1 ? E[i - 1][0][t + 1] : 0.0;
                    v = oo2p * a + XPA * b + (t + 1) * c;
                } else {
                    const int tm = i + j - 1;
                    const double a = t > 0 ? E[i][j - 1][t - 1] : 0.0;
                    const double b = t <= tm ? E[i][j - 1][t] : 0.0;
                    const double c = t + 1 <= tm ? E[i][j - 1][t + 1] : 0.0;
                    v = oo2p * a + XPB * b + (t + 1) * c;
                }
                E[i][j][t] = v;
            }
        }
}

// Attraction to the nuclei and point charges, one block per shell pair and chunk of
// charges, the threads over the charges.  Per primitive pair a thread sums q_c R_tuv(c)
// over its charges -- the Hermite coefficients do not depend on the charge, so they are
// applied once to the sums and not to every charge -- and the block adds the threads'
// sums in a fixed order.  A charge costs its Boys function and the R recursion (about
// 60 + 3 NT operations); the reduction, 10 NT shuffles a warp, is small beside the
// 32 charges a thread has of 4000.  All threads work on one primitive pair, so a pair
// whose Gaussian product vanishes is left out by the whole block (52 to 55% of them for
// twenty waters).  20 H2O / 6-31G* with 4000 charges, whole call: 2.0 ms, against 12.2
// with a thread per shell pair that contracted charge by charge and a thread per
// function pair for the nuclei.
template <int LA, int LB>
__global__ void __launch_bounds__(128)
oei_shell_kernel(OeiArgs a, const int4* __restrict__ pairs, int chunk, const double2* __restrict__ rows,
                 double* __restrict__ Vpart) {
    constexpr int NA = (LA + 1) * (LA + 2) / 2, NB = (LB + 1) * (LB + 2) / 2, L = LA + LB;
    constexpr int NT = (L + 1) * (L + 2) * (L + 3) / 6, NOUT = (NA * NB + 31) / 32;
    __shared__ double E[3][LA + 1][LB + 1][L + 1];
    __shared__ double H[4][NT];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarps = blockDim.x >> 5;
    const int4 sp = pairs[blockIdx.x];   // first functions of the shells (L = LA, LB), same-shell flag
    const int fa0 = sp.x, fb0 = sp.y;
    const int c0 = blockIdx.y * chunk, c1 = min(a.ncharge, c0 + chunk);
    const int n = a.nbasis;
    const double* A = a.xyz + 3 * (a.ncenter[fa0] - 1);
    const double* B = a.xyz + 3 * (a.ncenter[fb0] - 1);
    const double AB[3] = {A[0] - B[0], A[1] - B[1], A[2] - B[2]};
    const double r2 = AB[0] * AB[0] + AB[1] * AB[1] + AB[2] * AB[2];
    const double2* bt = rows + boys_rows_at(L) / 2;
    double acc[NOUT];
#pragma unroll
    for (int k = 0; k < NOUT; ++k) acc[k] = 0.0;
    for (int p = 0; p < a.ncontract[fa0]; ++p) {
        const double al = a.aexp[p + a.maxcontract * fa0];
        for (int q = 0; q < a.ncontract[fb0]; ++q) {
            const double be = a.aexp[q + a.maxcontract * fb0];
            const double pz = al + be, oo2p = 0.5 / pz, mu_r = al * be / pz;
            if (mu_r * r2 > kOeiExpMax) continue;   // the whole block
            const double P[3] = {(al * A[0] + be * B[0]) / pz, (al * A[1] + be * B[1]) / pz,
                                 (al * A[2] + be * B[2]) / pz};
            if (tid < 3)
                hermite_E_fixed<LA, LB>(-be / pz * AB[tid], al / pz * AB[tid], oo2p, exp(-mu_r * AB[tid] * AB[tid]),
                                        E[tid]);
            double h[NT];
#pragma unroll
            for (int k = 0; k < NT; ++k) h[k] = 0.0;
            for (int c = c0 + tid; c < c1; c += blockDim.x) {
                const double X = P[0] - a.cxyz[3 * c], Y = P[1] - a.cxyz[3 * c + 1], Z = P[2] - a.cxyz[3 * c + 2];
                double F[L + 1];
                boys_scaled_rows<L>(pz * (X * X + Y * Y + Z * Z), a.cq[c], bt, F);
                double m2p = 1.0;   // (-2p)^k
#pragma unroll
                for (int k = 1; k <= L; ++k) {
                    m2p *= -2.0 * pz;
                    F[k] *= m2p;
                }
                double R[NT];
                R[0] = F[L];
                unroll_up<L>([&](auto step) {
                    constexpr int k = L - 1 - decltype(step)::value;   // level k from level k + 1
                    constexpr int NK = (L - k + 1) * (L - k + 2) * (L - k + 3) / 6;
                    // degree by degree downwards, so that the recursion runs in place
                    unroll_up<NK>([&](auto down) {
                        constexpr int i = NK - 1 - decltype(down)::value;
                        constexpr Tuv w = tuv_of(i);
                        constexpr int ax = w.t > 0 ? 0 : w.u > 0 ? 1 : 2, m = ax == 0 ? w.t : ax == 1 ? w.u : w.v;
                        if constexpr (i == 0) {
                            R[0] = F[k];
                        } else {
                            constexpr int i1 = tuv_flat(w.t - (ax == 0), w.u - (ax == 1), w.v - (ax == 2));
                            double r = (ax == 0 ? X : ax == 1 ? Y : Z) * R[i1];
                            if constexpr (m > 1) {
                                constexpr int i2 = tuv_flat(w.t - 2 * (ax == 0), w.u - 2 * (ax == 1), w.v - 2 * (ax == 2));
                                r = fma((double)(m - 1), R[i2], r);
                            }
                            R[i] = r;
                        }
                    });
                });
#pragma unroll
                for (int k = 0; k < NT; ++k) h[k] += R[k];
            }
#pragma unroll
            for (int k = 0; k < NT; ++k) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) h[k] += __shfl_xor_sync(0xffffffffu, h[k], o);
                if (lane == 0) H[warp][k] = h[k];
            }
            __syncthreads();
            for (int k = tid; k < NT; k += blockDim.x)
                for (int w = 1; w < nwarps; ++w) H[0][k] += H[w][k];
            __syncthreads();
#pragma unroll
            for (int k = 0; k < NOUT; ++k) {
                const int ij = tid + k * blockDim.x;
                if (ij >= NA * NB) break;
                const int i = ij / NB, j = ij % NB;
                const int ax = cart_exp(LA, i, 0), ay = cart_exp(LA, i, 1), az = cart_exp(LA, i, 2);
                const int bx = cart_exp(LB, j, 0), by = cart_exp(LB, j, 1), bz = cart_exp(LB, j, 2);
                double vc = 0.0;
                for (int tt = 0; tt <= ax + bx; ++tt)
                    for (int uu = 0; uu <= ay + by; ++uu)
                        for (int vv = 0; vv <= az + bz; ++vv)
                            vc += E[0][ax][bx][tt] * E[1][ay][by][uu] * E[2][az][bz][vv] *
                                  H[0][tuv_index(tt, uu, vv)];
                acc[k] -= a.dcoeff[p + a.maxcontract * (fa0 + i)] * a.dcoeff[q + a.maxcontract * (fb0 + j)] *
                          (2.0 * M_PI / pz) * vc;
            }
            __syncthreads();   // E and H are written again
        }
    }
    double* out = Vpart + (size_t)blockIdx.y * n * (n + 1) / 2;
#pragma unroll
    for (int k = 0; k < NOUT; ++k) {
        const int ij = tid + k * blockDim.x;
        if (ij >= NA * NB) break;
        const int f = fa0 + ij / NB, g = fb0 + ij % NB;
        if (sp.z != 0 && f < g) continue;
        const int mu = f > g ? f : g, nu = f > g ? g : f;
        out[(size_t)mu * (mu + 1) / 2 + nu] = acc[k];
    }
}

// V = sum of the chunks' partial sums, in chunk order (bit-reproducible).
__global__ void oei_reduce_kernel(OeiArgs a, int nchunk, const double* __restrict__ Vpart) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = a.nbasis;
    const int npair = n * (n + 1) / 2;
    if (t >= npair) return;
    int mu = (int)((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
    while (mu * (mu + 1) / 2 > t) --mu;
    while ((mu + 1) * (mu + 2) / 2 <= t) ++mu;
    const int nu = t - mu * (mu + 1) / 2;
    double v = 0.0;
    for (int k = 0; k < nchunk; ++k) v += Vpart[(size_t)k * npair + t];
    a.V[(size_t)mu * n + nu] = v;
    a.V[(size_t)nu * n + mu] = v;
}

// One non-blocking stream per device for the one-electron set-up, so that it
// neither waits for nor holds up work on other streams (no device-wide syncs:
// stream-ordered allocation, copies and a stream synchronisation only).
static cudaStream_t oei_stream(int device) {
    static std::mutex mu;
    static cudaStream_t streams[64] = {};
    std::lock_guard<std::mutex> g(mu);
    if (device < 0 || device >= 64) return nullptr;
    if (!streams[device]) {
        // highest priority, as the contexts' set-up streams (see qk_create)
        int lo = 0, hi = 0;
        cudaDeviceGetStreamPriorityRange(&lo, &hi);
        cudaStreamCreateWithPriority(&streams[device], cudaStreamNonBlocking, hi);
    }
    return streams[device];
}

// Per device, made at the first call and kept: a memory pool of its own for the calls'
// work buffers, which keeps up to 256 MB between calls instead of giving the pages back
// to the driver at every synchronisation.  All but 32 MB (one of the driver's pages) go back
// with the device's last context; without those a program that has one context at a time
// would map them anew for each molecule, 0.3 ms of the 3 ms that setting one up takes.
static std::mutex g_pool_mu;
static cudaMemPool_t g_pools[64] = {};
static cudaMemPool_t oei_pool(int device) {
    if (device < 0 || device >= 64) return nullptr;
    std::lock_guard<std::mutex> g(g_pool_mu);
    if (!g_pools[device]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        unsigned long long keep = 256ull << 20;
        cudaMemPool_t p = nullptr;
        if (cudaMemPoolCreate(&p, &props) != cudaSuccess) return nullptr;
        if (cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
            cudaMemPoolDestroy(p);
            return nullptr;
        }
        g_pools[device] = p;
    }
    return g_pools[device];
}
void oei_give_back(int device) {
    std::lock_guard<std::mutex> g(g_pool_mu);
    if (g_pools[device]) cudaMemPoolTrimTo(g_pools[device], 32ull << 20);   // blocks in use stay
}

}  // namespace qk

extern "C" int qk_oei_host(int device, int natom, const double* xyz, const double* Z, int nbasis, int maxcontract,
                           const int* ncontract, const int* itype, const double* aexp, const double* dcoeff,
                           const int* ncenter, int next, const double* ext_xyz, const double* ext_q,
                           double* S, double* T, double* V) {
    using namespace qk;
    if (natom <= 0 || nbasis <= 0 || maxcontract <= 0 || !xyz || !Z || !ncontract || !itype || !aexp ||
        !dcoeff || !ncenter || !S || !T || !V || next < 0 || (next > 0 && (!ext_xyz || !ext_q)))
        return QK_ERR_INVALID_ARG;
    for (int i = 0; i < nbasis; ++i) {   // the kernels' arrays hold a function of degree kOeiLmax
        const int* t = itype + 3 * (size_t)i;
        for (int x = 0; x < 3; ++x)
            if (t[x] < 0 || t[x] > kOeiLmax) return QK_ERR_UNSUPPORTED;
        if (t[0] + t[1] + t[2] > kOeiLmax) return QK_ERR_UNSUPPORTED;
    }
    for (int i = 0; i < nbasis; ++i)
        if (ncenter[i] < 1 || ncenter[i] > natom || ncontract[i] < 1 || ncontract[i] > maxcontract)
            return QK_ERR_INVALID_ARG;
    if (cudaSetDevice(device) != cudaSuccess) return QK_ERR_CUDA;
    const int nq = natom + next;
    std::vector<double> cxyz(3 * (size_t)nq), cq(nq);
    for (int i = 0; i < natom; ++i) {
        for (int k = 0; k < 3; ++k) cxyz[3 * i + k] = xyz[3 * i + k];
        cq[i] = Z[i];
    }
    for (int i = 0; i < next; ++i) {
        for (int k = 0; k < 3; ++k) cxyz[3 * (natom + i) + k] = ext_xyz[3 * i + k];
        cq[natom + i] = ext_q[i];
    }
    const size_t nn = (size_t)nbasis * nbasis;
    const long long npair = (long long)nbasis * (nbasis + 1) / 2;
    // charge chunks: enough blocks for about 4 waves of the GPU, at least 32 charges a chunk
    const long long want = std::max<long long>(1, (4LL * 148 * 2048 + npair - 1) / npair);
    // the shell-pair kernel takes the charges when every shell has QUICK's component
    // order; the function-pair kernel otherwise
    std::vector<int4> sp_list[kOeiLmax + 1][kOeiLmax + 1];
    bool shells = true;
    {
        std::vector<int> f0, Ls;
        for (int f = 0; f < nbasis && shells;) {
            const int L = itype[3 * f] + itype[3 * f + 1] + itype[3 * f + 2];
            const int nc = (L + 1) * (L + 2) / 2;
            if (f + nc > nbasis) { shells = false; break; }
            for (int k = 0; k < nc && shells; ++k) {
                const int g = f + k;
                shells = itype[3 * g] == cart_exp(L, k, 0) && itype[3 * g + 1] == cart_exp(L, k, 1) &&
                         itype[3 * g + 2] == cart_exp(L, k, 2) && ncenter[g] == ncenter[f] &&
                         ncontract[g] == ncontract[f];
                for (int p = 0; p < ncontract[f] && shells; ++p)
                    shells = aexp[p + (size_t)maxcontract * g] == aexp[p + (size_t)maxcontract * f];
            }
            f0.push_back(f);
            Ls.push_back(L);
            f += nc;
        }
        if (shells)
            for (int i = 0; i < (int)f0.size(); ++i)
                for (int j = 0; j <= i; ++j) {
                    const bool swap = Ls[j] > Ls[i];
                    const int a0 = swap ? f0[j] : f0[i], b0 = swap ? f0[i] : f0[j];
                    const int la = swap ? Ls[j] : Ls[i], lb = swap ? Ls[i] : Ls[j];
                    sp_list[la][lb].push_back(make_int4(a0, b0, i == j ? 1 : 0, 0));
                }
    }
    long long nsp = 0;
    for (auto& row : sp_list)
        for (auto& v : row) nsp += (long long)v.size();
    int nchunk, chunk, threads = 32;
    if (shells) {
        // a warp per block for the nuclei alone, four where a thread has charges enough;
        // chunks only where the shell pairs are too few for the GPU
        threads = nq >= 512 ? 128 : 32;
        const long long fill = (148LL * 16 + nsp - 1) / std::max<long long>(nsp, 1);
        nchunk = (int)std::max<long long>(1, std::min<long long>({fill, (nq + 4 * threads - 1) / (4 * threads), 65535LL}));
    } else {
        nchunk = (int)std::max<long long>(1, std::min<long long>({want, (nq + 31) / 32, 65535LL}));
    }
    chunk = (nq + nchunk - 1) / nchunk;
    cudaStream_t s = oei_stream(device);
    if (!s) return QK_ERR_CUDA;
    const double *boys = nullptr, *rows = nullptr;
    if (device_boys_tables(device, s, &boys, &rows) != cudaSuccess) return QK_ERR_CUDA;
    cudaMemPool_t pool = oei_pool(device);
    if (!pool) return QK_ERR_CUDA;
    int st = QK_OK;
    // one device block: inputs (packed on the host, one copy), then S T V, then the
    // partial sums
    std::vector<int4> sp_all;
    size_t sp_off[kOeiLmax + 1][kOeiLmax + 1] = {};
    for (int la = 0; la <= kOeiLmax; ++la)
        for (int lb = 0; lb <= kOeiLmax; ++lb) {
            sp_off[la][lb] = sp_all.size();
            sp_all.insert(sp_all.end(), sp_list[la][lb].begin(), sp_list[la][lb].end());
        }
    const size_t sizes[10] = {nbasis * sizeof(int), 3 * nbasis * sizeof(int), (size_t)maxcontract * nbasis * 8,
                              (size_t)maxcontract * nbasis * 8, nbasis * sizeof(int), 3 * (size_t)natom * 8,
                              cxyz.size() * 8, cq.size() * 8, sp_all.size() * sizeof(int4), 3 * nn * 8};
    const void* src[9] = {ncontract, itype, aexp, dcoeff, ncenter, xyz, cxyz.data(), cq.data(), sp_all.data()};
    size_t off[11];
    off[0] = 0;
    for (int i = 0; i < 10; ++i) off[i + 1] = off[i] + ((sizes[i] + 255) & ~size_t(255));
    const size_t total = off[10] + (size_t)nchunk * npair * 8;
    std::vector<char> packed(off[9]);
    for (int i = 0; i < 9; ++i)
        if (sizes[i] > 0) std::memcpy(packed.data() + off[i], src[i], sizes[i]);
    char* base = nullptr;
    if (cudaMallocFromPoolAsync((void**)&base, total, pool, s) != cudaSuccess) return QK_ERR_OUT_OF_MEMORY;
    if (cudaMemcpyAsync(base, packed.data(), packed.size(), cudaMemcpyHostToDevice, s) != cudaSuccess) st = QK_ERR_CUDA;
    if (st == QK_OK) {
        OeiArgs a;
        a.nbasis = nbasis; a.maxcontract = maxcontract; a.ncharge = nq;
        a.ncontract = (const int*)(base + off[0]); a.itype = (const int*)(base + off[1]);
        a.aexp = (const double*)(base + off[2]); a.dcoeff = (const double*)(base + off[3]);
        a.ncenter = (const int*)(base + off[4]); a.xyz = (const double*)(base + off[5]);
        a.cxyz = (const double*)(base + off[6]); a.cq = (const double*)(base + off[7]);
        a.boys = boys;
        a.S = (double*)(base + off[9]); a.T = a.S + nn; a.V = a.T + nn;
        double* Vpart = (double*)(base + off[10]);
        const int gx = (int)((npair + 127) / 128);
        oei_st_kernel<<<gx, 128, 0, s>>>(a);
        if (shells) {
            const int4* dsp = (const int4*)(base + off[8]);
#define QK_OEI_SP(LA, LB)                                                                              \
            if (!sp_list[LA][LB].empty())                                                              \
                oei_shell_kernel<LA, LB><<<dim3((unsigned)sp_list[LA][LB].size(), nchunk), threads, 0, s>>>( \
                    a, dsp + sp_off[LA][LB], chunk, (const double2*)rows, Vpart);
            // the longest blocks first
            QK_OEI_SP(3, 3) QK_OEI_SP(3, 2) QK_OEI_SP(3, 1) QK_OEI_SP(2, 2) QK_OEI_SP(3, 0) QK_OEI_SP(2, 1)
            QK_OEI_SP(2, 0) QK_OEI_SP(1, 1) QK_OEI_SP(1, 0) QK_OEI_SP(0, 0)
#undef QK_OEI_SP
        } else {
            oei_kernel<<<dim3(gx, nchunk), 128, 0, s>>>(a, chunk, Vpart);
        }
        oei_reduce_kernel<<<gx, 128, 0, s>>>(a, nchunk, Vpart);
        if (cudaGetLastError() != cudaSuccess) st = QK_ERR_CUDA;
        if (st == QK_OK && (cudaMemcpyAsync(S, a.S, nn * 8, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
                            cudaMemcpyAsync(T, a.T, nn * 8, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
                            cudaMemcpyAsync(V, a.V, nn * 8, cudaMemcpyDeviceToHost, s) != cudaSuccess))
            st = QK_ERR_CUDA;
    }
    cudaFreeAsync(base, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) st = QK_ERR_CUDA;
    return st;
}
