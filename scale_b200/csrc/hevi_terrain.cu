// The HEVI stage with terrain-following metrics (GSQRT, J13G, J23G) and map
// factors (MAPF): ATMOS_DYN_Tstep_short_fvm_hevi
// (scale_atmos_dyn_tstep_short_fvm_hevi.F90:128-1089) with every metric term. Line
// numbers refer to that file unless a flux file is named (ud3.F90 is
// scale_atmos_dyn_fvm_flux_ud3.F90; the other schemes' files have the same routines).
// FP64, one domain.
//
// Six launches, a warp per column with its lanes along k:
//   k_t_prep    DPRES (:343-361) and POTT (:586-598), the latter over the halo too
//   k_t_mass    mass fluxes (:365-438), Sr (:443-479), theta fluxes (:603-622), St
//               (:625-661), PT (valueW_Z)
//   k_t_w       w fluxes (:485-525), Sw (:528-578), the coefficients and right-hand
//               side of the column problem (:696-722)
//   k_t_column  solve_direct (:1092-1127) and the back-update (:728-790)
//   k_t_mom     rho*u (:814-928) and rho*v (:934-1048): their fluxes and updates
// A cell forms the fluxes of its own faces, the z flux below a level by warp
// shuffle, so no flux array but the vertical ones of the column problem goes through
// HBM. One launch per loop nest of the reference (26 launches) wrote and read back
// 15 such arrays: 256x256x64, CD4, a short step of four stages 10.36 ms, with this
// form 7.40 ms.
// Quotients are straight-line code (rn_div.cuh). The outputs go through
// put_state/put_flux, so the RK folds of the flat stage apply unchanged.
#include "hevi_epilogue.cuh"
#include "hevi_kernels.cuh"
#include "rn_div.cuh"
#include "tma_util.cuh"

namespace hevi {

namespace {

// staggering ids (scale_atmos_grid_cartesC_index.F90:90-101), variable ids and directions
enum : int { I_XYZ = 1, I_XYW, I_UYW, I_XVW, I_UYZ, I_XVZ, I_UVZ };
enum : int { I_XY = 1, I_UY, I_XV, I_UV };
enum : int { V_DENS = 1, V_MOMZ, V_MOMX, V_MOMY, V_RHOT };
enum : int { DZIR = 1, DXIR, DYIR };

constexpr int TW = 4; // columns (warps) per CTA
using Gd = rn::Guard<double>;
#define TDIV rn::div<FAST>

// keeps the compiler from carrying values of the fast path into the rare exact one
__device__ __forceinline__ void cold() { asm volatile("" ::: "memory"); }

// face value between p[0] and p[s] along a horizontal direction of stride s
template <int S>
__device__ __forceinline__ double hface(double vel, const double *p, int s)
{
    if constexpr (wide_scheme(S)) return ip6<S>(vel, ld(p - 2 * s), ld(p - s), ld(p), ld(p + s), ld(p + 2 * s), ld(p + 3 * s));
    else return ip4<S>(vel, ld(p - s), ld(p), ld(p + s), ld(p + 2 * s));
}

struct Terrain {
    Grid g;
    StageArgsT<double> a;
    Metrics M;
    TerrainWork W;
    size_t N3;
    __device__ double G(int idx, int c) const { return ld(M.GSQRT + (size_t)(idx - 1) * N3 + c); }
    __device__ double J13(int idx, int c) const { return ld(M.J13G + (size_t)(idx - 1) * N3 + c); }
    __device__ double J23(int idx, int c) const { return ld(M.J23G + (size_t)(idx - 1) * N3 + c); }
    __device__ double mapf(int i, int j, int aa, int bb) const
    {
        return ld(M.MAPF + ((size_t)(i - 1) + (size_t)g.IA * ((size_t)(j - 1) + (size_t)g.JA * ((size_t)(aa - 1) + 2 * (size_t)(bb - 1)))));
    }
    __device__ double nd(int v, int dir, int c) const { return ld(a.num_diff + N3 * (size_t)((v - 1) + 5 * (dir - 1)) + c); }
    // F2H(k,1) and F2H(k,2) of a GSQRT slice (ud3.F90:75, :62)
    template <bool FAST>
    __device__ void f2h(Gd &gd, int idx, int c, int k, double &f1, double &f2) const
    {
        const double p = ld(g.CDZ + k - 1) * G(idx, c), q = ld(g.CDZ + k) * G(idx, c + 1), den = p + q;
        const double y = rn::recip<FAST>(gd, den);
        f1 = TDIV(gd, p, den, y);
        f2 = TDIV(gd, q, den, y);
    }
};

// this warp's column
struct Col {
    int i, j, lane;
    bool ok;
};
__device__ __forceinline__ Col column(int i0, int ni, int j0, int ncol)
{
    const int n = (int)blockIdx.x * TW + (int)threadIdx.y;
    return Col{i0 + n % ni, j0 + n / ni, (int)threadIdx.x, n < ncol};
}
// the lane below's value; lane 0 takes the previous pass's lane 31's (carry)
__device__ __forceinline__ double below(double v, double &carry)
{
    const int lane = threadIdx.x;
    const double r = __shfl_sync(0xffffffffu, v, (lane + 31) & 31);
    const double x = lane == 0 ? carry : r;
    carry = r;
    return x;
}

__global__ void __launch_bounds__(32 * TW) k_t_prep(const __grid_constant__ Terrain T)
{
    const Grid &g = T.g;
    const auto &a = T.a;
    const Col q = column(1, g.IA, 1, g.IA * g.JA);
    if (!q.ok) return; // warp-uniform
    const int col = (int)idx3(g, 1, q.i, q.j), KS = g.KS, KE = g.KE;
    const bool dp = q.i >= g.IS && q.i <= g.IE + 1 && q.j >= g.JS && q.j <= g.JE + 1;
    for (int k = KS + q.lane; k <= KE; k += 32) {
        const int c = col + k - 1;
        const double rt = ld(a.RHOT + c);
        T.W.POTT[c] = rt / ld(a.DENS + c);
        if (dp) T.W.DPRES[c] = ld(a.DPRES0 + c) + ld(a.RT2P + c) * (rt - ld(a.REF_rhot + c));
    }
    if (dp && q.lane == 0) {
        const int b = col + KS - 2, t = col + KE; // levels KS-1 and KE+1
        T.W.DPRES[b] = ld(a.DPRES0 + b) - ld(a.DENS + b + 1) * (ld(T.M.PHI + b) - ld(T.M.PHI + b + 2));
        T.W.DPRES[t] = ld(a.DPRES0 + t) - ld(a.DENS + t - 1) * (ld(T.M.PHI + t) - ld(T.M.PHI + t - 2));
    }
}

// Launch bounds of the three flux kernels: 6 CTAs of 4 warps per SM.
#ifndef HEVI_T_MINB
#define HEVI_T_MINB 6
#endif

template <int S>
__global__ void __launch_bounds__(32 * TW, HEVI_T_MINB) k_t_mass(const __grid_constant__ Terrain T)
{
    const Grid &g = T.g;
    const auto &a = T.a;
    const Col q = column(g.IS, g.IMAX, g.JS, g.IMAX * g.JMAX);
    if (!q.ok) return; // warp-uniform
    const int i = q.i, j = q.j, lane = q.lane, KS = g.KS, KE = g.KE, sI = g.KA, sJ = g.KA * g.IA;
    const int col = (int)idx3(g, 1, i, j);
    const double *const MX = a.MOMX, *const MY = a.MOMY;
    const double m1 = T.mapf(i, j, 1, I_XY), m2 = T.mapf(i, j, 2, I_XY), m12 = m1 * m2;
    const double mE = T.mapf(i, j, 2, I_UY), mW = T.mapf(i - 1, j, 2, I_UY);
    const double mN = T.mapf(i, j, 1, I_XV), mS = T.mapf(i, j - 1, 1, I_XV);
    const double rcdx = ld(g.RCDX + i - 1), rcdy = ld(g.RCDY + j - 1);
    // hevi_mflx_z :365-397 at the face above the level of c
    auto mflx_z = [&](auto fast, Gd &gd, int c, double n1, double n2, double n12) {
        constexpr bool FAST = decltype(fast)::value;
        return TDIV(gd, T.J13(I_XYW, c) * 0.25, n2) * (ld(MX + c + 1) + ld(MX + c + 1 - sI) + ld(MX + c) + ld(MX + c - sI))
               + TDIV(gd, T.J23(I_XYW, c) * 0.25, n1) * (ld(MY + c + 1) + ld(MY + c + 1 - sJ) + ld(MY + c) + ld(MY + c - sJ))
               + TDIV(gd, T.G(I_XYW, c), n12) * T.nd(V_DENS, DZIR, c);
    };
    double cm = 0.0, ct = 0.0; // the fluxes below, zero below KS
    for (int k0 = KS; k0 <= KE; k0 += 32) {
        const int k = min(k0 + lane, KE), c = col + k - 1;
        const bool valid = k0 + lane <= KE;
        double mZ, tZ, PT, Xe, Xw, Yn, Ys;
        const double *const P = T.W.POTT + col - 1; // 1-based level index
        auto faces = [&](auto fast) {
            constexpr bool FAST = decltype(fast)::value;
            Gd gd;
            mZ = tZ = PT = 0.0;
            if (k <= KE - 1) {
                mZ = mflx_z(fast, gd, c, m1, m2, m12);
                auto V = [&](int l) { return ld(P + l); };
                tZ = mZ * zface<S>(mZ, k, KS, KE, V) + T.G(I_XYW, c) * T.nd(V_RHOT, DZIR, c);
                PT = zface<S>(ld(a.MOMZ + c), k, KS, KE, V);
            }
            Xe = TDIV(gd, T.G(I_UYZ, c), mE) * (ld(MX + c) + T.nd(V_DENS, DXIR, c));
            Xw = TDIV(gd, T.G(I_UYZ, c - sI), mW) * (ld(MX + c - sI) + T.nd(V_DENS, DXIR, c - sI));
            Yn = TDIV(gd, T.G(I_XVZ, c), mN) * (ld(MY + c) + T.nd(V_DENS, DYIR, c));
            Ys = TDIV(gd, T.G(I_XVZ, c - sJ), mS) * (ld(MY + c - sJ) + T.nd(V_DENS, DYIR, c - sJ));
            return gd.bad();
        };
        if (faces(std::true_type{})) {
            cold();
            faces(std::false_type{});
        }
        const double tXe = Xe * hface<S>(Xe, P + k, sI) + T.G(I_UYZ, c) * T.nd(V_RHOT, DXIR, c);
        const double tXw = Xw * hface<S>(Xw, P + k - sI, sI) + T.G(I_UYZ, c - sI) * T.nd(V_RHOT, DXIR, c - sI);
        const double tYn = Yn * hface<S>(Yn, P + k, sJ) + T.G(I_XVZ, c) * T.nd(V_RHOT, DYIR, c);
        const double tYs = Ys * hface<S>(Ys, P + k - sJ, sJ) + T.G(I_XVZ, c - sJ) * T.nd(V_RHOT, DYIR, c - sJ);
        const double mZm = below(mZ, cm), tZm = below(tZ, ct);
        const double rcdz = ld(g.RCDZ + k - 1);
        const double advr = (-(mZ - mZm) * rcdz + -((Xe - Xw) * rcdx + (Yn - Ys) * rcdy)) * m1 * m2;
        const double advt = (-(tZ - tZm) * rcdz + -((tXe - tXw) * rcdx + (tYn - tYs) * rcdy)) * m1 * m2;
        const double gz = T.G(I_XYZ, c), Dt = ld(a.DENS_t + c), Tt = ld(a.RHOT_t + c);
        double Sr, St;
        auto sources = [&](auto fast) {
            constexpr bool FAST = decltype(fast)::value;
            Gd gd;
            const double y = rn::recip<FAST>(gd, gz);
            Sr = TDIV(gd, advr, gz, y) + Dt;
            St = TDIV(gd, advt, gz, y) + Tt;
            return gd.bad();
        };
        if (sources(std::true_type{})) {
            cold();
            sources(std::false_type{});
        }
        if (valid) {
            T.W.Sr[c] = Sr;
            T.W.St[c] = St;
            T.W.mZ[c] = mZ;
            T.W.tZ[c] = tZ;
            T.W.PT[c] = PT;
            put_flux(a, T.N3, 1, c, Xe, true);
            put_flux(a, T.N3, 2, c, Yn, true);
            put_flux(a, T.N3, 4, c, tXe, true);
            put_flux(a, T.N3, 5, c, tYn, true);
            if (i == g.IS) {
                put_flux(a, T.N3, 1, c - sI, Xw, false);
                put_flux(a, T.N3, 4, c - sI, tXw, false);
                // the halo column IS-1 of the vertical mass flux is an output too (:369-393)
                Gd gd;
                const double n1 = T.mapf(i - 1, j, 1, I_XY), n2 = T.mapf(i - 1, j, 2, I_XY);
                put_flux(a, T.N3, 0, c - sI, k <= KE - 1 ? mflx_z(std::false_type{}, gd, c - sI, n1, n2, n1 * n2) : 0.0, false);
                if (k == KS) put_flux(a, T.N3, 0, c - sI - 1, 0.0, false);
            }
            if (j == g.JS) {
                put_flux(a, T.N3, 2, c - sJ, Ys, false);
                put_flux(a, T.N3, 5, c - sJ, tYs, false);
            }
        }
    }
}

template <int S>
__global__ void __launch_bounds__(32 * TW, HEVI_T_MINB) k_t_w(const __grid_constant__ Terrain T)
{
    constexpr bool wide = wide_scheme(S);
    const Grid &g = T.g;
    const auto &a = T.a;
    const Col q = column(g.IS, g.IMAX, g.JS, g.IMAX * g.JMAX);
    if (!q.ok) return; // warp-uniform
    const int i = q.i, j = q.j, lane = q.lane, KS = g.KS, KE = g.KE, sI = g.KA, sJ = g.KA * g.IA;
    const int col = (int)idx3(g, 1, i, j);
    const double dt = a.dtrk, J33G = a.J33G;
    const bool use_div = a.divdmp_coef != 0.0;
    const double *const MX = a.MOMX, *const MY = a.MOMY, *const MZ = a.MOMZ, *const DN = a.DENS;
    const double *const Z = MZ + col - 1; // 1-based level index
    const double m1 = T.mapf(i, j, 1, I_XY), m2 = T.mapf(i, j, 2, I_XY);
    const double mE = T.mapf(i, j, 2, I_UY), mW = T.mapf(i - 1, j, 2, I_UY);
    const double mN = T.mapf(i, j, 1, I_XV), mS = T.mapf(i, j - 1, 1, I_XV);
    const double rcdx = ld(g.RCDX + i - 1), rcdy = ld(g.RCDY + j - 1);
    double cz = 0.0, c1 = 0.0, c2 = 0.0; // the fluxes below
    for (int k0 = KS; k0 <= KE - 1; k0 += 32) {
        const int k = min(k0 + lane, KE - 1), c = col + k - 1;
        const bool valid = k0 + lane <= KE - 1;
        double qZ, q1, q2, qXe, qXw, qYn, qYs;
        auto faces = [&](auto fast) {
            constexpr bool FAST = decltype(fast)::value;
            Gd gd;
            qZ = q1 = q2 = 0.0; // zero at KE-1
            if (k <= KE - 2) {
                const double dn = ld(DN + c + 1), y = rn::recip<FAST>(gd, dn);
                // fluxZ_XYW (ud3.F90:358-452)
                const double vel = TDIV(gd, 0.5 * (ld(MZ + c) + ld(MZ + c + 1)), dn, y);
                qZ = J33G * vel * zface<S>(vel, k, KS, KE, [&](int l) { return ld(Z + l); })
                     + T.G(I_XYZ, c + 1) * T.nd(V_MOMZ, DZIR, c + 1);
                // fluxJ13_XYW (:457-523) and fluxJ23_XYW (:527-593)
                double v1 = TDIV(gd, 0.5 * (ld(MX + c + 1) + ld(MX + c + 1 - sI)), dn, y);
                double v2 = TDIV(gd, 0.5 * (ld(MY + c + 1) + ld(MY + c + 1 - sJ)), dn, y);
                if (k == KS) {
                    const double d0 = ld(DN + c);
                    v1 = (v1 + TDIV(gd, 0.5 * (ld(MX + c) + ld(MX + c - sI)), d0)) * 0.5;
                    v2 = (v2 + TDIV(gd, 0.5 * (ld(MY + c) + ld(MY + c - sJ)), d0)) * 0.5;
                }
                v1 = v1 * T.J13(I_XYZ, c + 1);
                v2 = v2 * T.J23(I_XYZ, c + 1);
                auto face = [&](double v) {
                    if (k == KS) return ipL<S>(v, ld(Z + KS), ld(Z + KS + 1), ld(Z + KS + 2));
                    if constexpr (wide) {
                        // the 3-point form one level below the KE-1 face (ud5.F90:604-657)
                        if (k == KE - 2) return ipH<S>(v, ld(Z + KE - 1), ld(Z + KE - 2), ld(Z + KE - 3));
                        return ip6<S>(v, ld(Z + k - 2), ld(Z + k - 1), ld(Z + k), ld(Z + k + 1), ld(Z + k + 2), ld(Z + k + 3));
                    } else {
                        return ip4<S>(v, ld(Z + k - 1), ld(Z + k), ld(Z + k + 1), ld(Z + k + 2));
                    }
                };
                q1 = TDIV(gd, v1, m2) * face(v1);
                q2 = TDIV(gd, v2, m1) * face(v2);
            }
            // fluxX_XYW (ud3.F90:598-671) and fluxY_XYW (:675-748)
            auto flux = [&](int idx, const double *mom, int dir, int cf, int s, double mp) {
                double f1, f2;
                T.f2h<FAST>(gd, idx, cf, k, f1, f2);
                const double vel = TDIV(gd, f1 * ld(mom + cf + 1) + f2 * ld(mom + cf),
                                        f1 * 0.5 * (ld(DN + cf + 1) + ld(DN + cf + 1 + s)) + f2 * 0.5 * (ld(DN + cf) + ld(DN + cf + s)));
                const double Gs = T.G(idx, cf);
                return TDIV(gd, Gs, mp) * vel * hface<S>(vel, MZ + cf, s) + Gs * T.nd(V_MOMZ, dir, cf);
            };
            qXe = flux(I_UYW, MX, DXIR, c, sI, mE);
            qXw = flux(I_UYW, MX, DXIR, c - sI, sI, mW);
            qYn = flux(I_XVW, MY, DYIR, c, sJ, mN);
            qYs = flux(I_XVW, MY, DYIR, c - sJ, sJ, mS);
            return gd.bad();
        };
        if (faces(std::true_type{})) {
            cold();
            faces(std::false_type{});
        }
        const double qZm = below(qZ, cz), q1m = below(q1, c1), q2m = below(q2, c2);
        const double rfdz = ld(g.RFDZ + k - 1), gw = T.G(I_XYW, c), gz0 = T.G(I_XYZ, c), gz1 = T.G(I_XYZ, c + 1);
        const double advcv = -(qZ - qZm + q1 - q1m + q2 - q2m) * rfdz;
        const double advch = -((qXe - qXw) * rcdx + (qYn - qYs) * rcdy) * m1 * m2;
        const double wdmp = -ld(a.wdamp + g.z0 + k - 1) * ld(a.MOMZ0 + c);
        const double div = use_div ? a.divdmp_coef / dt * (ld(a.DDIV + c + 1) - ld(a.DDIV + c)) * ld(g.FDZ + k - 1) : 0.0;
        const double cd0 = ld(g.CDZ + k - 1), cd1 = ld(g.CDZ + k);
        const double rt0 = ld(a.RT2P + c), rt1 = ld(a.RT2P + c + 1), Wt = ld(a.MOMZ_t + c);
        const double P0 = T.W.PT[c], Pp = T.W.PT[c + 1], Pm = T.W.PT[c - 1]; // PT(k), PT(k+1), PT(k-1)
        const double b1 = ld(DN + c + 1) - ld(a.REF_dens + c + 1) + T.W.Sr[c + 1] * dt;
        const double b0 = ld(DN + c) - ld(a.REF_dens + c) + T.W.Sr[c] * dt;
        const double dp = -(T.W.DPRES[c + 1] + rt1 * dt * T.W.St[c + 1] - T.W.DPRES[c] - rt0 * dt * T.W.St[c]);
        double F1, F2, F3, C;
        auto coefs = [&](auto fast) {
            constexpr bool FAST = decltype(fast)::value;
            Gd gd;
            const double y = rn::recip<FAST>(gd, gw);
            const double Sw = TDIV(gd, advcv + advch, gw, y) + wdmp + div + Wt;
            const double A0 = TDIV(gd, dt * dt * J33G * ld(g.RCDZ + k - 1) * rt0 * J33G, gz0);
            const double A1 = TDIV(gd, dt * dt * J33G * ld(g.RCDZ + k) * rt1 * J33G, gz1);
            const double B = TDIV(gd, GRAV * (dt * dt) * J33G, cd1 + cd0);
            F1 = k <= KE - 2 ? TDIV(gd, -(Pp * rfdz * A1 + B), gw, y) : 0.0;
            F2 = 1.0 + TDIV(gd, P0 * rfdz * (A1 + A0), gw, y);
            F3 = k >= KS + 1 ? TDIV(gd, -(Pm * rfdz * A0 - B), gw, y) : 0.0;
            double f1, f2;
            T.f2h<FAST>(gd, I_XYZ, c, k, f1, f2);
            const double pg = TDIV(gd, dp * rfdz * J33G, gw, y) - GRAV * (f1 * b1 + f2 * b0);
            C = ld(MZ + c) + dt * (pg + Sw);
            return gd.bad();
        };
        if (coefs(std::true_type{})) {
            cold();
            coefs(std::false_type{});
        }
        if (valid) {
            T.W.F1[c] = F1;
            T.W.F2[c] = F2;
            T.W.F3[c] = F3;
            T.W.C[c] = C;
        }
    }
}

// solve_direct (:1092-1127) and the back-update (:728-790) of SC consecutive columns:
// the coefficients in shared memory (cp.async), one lane per column in the
// recurrence, all warps in the update
constexpr int SC = 16, SW = 8;
inline size_t t_column_smem(int KA) { return (size_t)4 * SC * (KA | 1) * sizeof(double); }
__global__ void __launch_bounds__(32 * SW, 3) k_t_column(const __grid_constant__ Terrain T)
{
    extern __shared__ double sh[];
    const Grid &g = T.g;
    const auto &a = T.a;
    const int KS = g.KS, KE = g.KE, KP = g.KA | 1, lane = threadIdx.x, w = threadIdx.y;
    const int nbx = (g.IMAX + SC - 1) / SC;
    const int i0 = g.IS + ((int)blockIdx.x % nbx) * SC, j = g.JS + (int)blockIdx.x / nbx, ncol = min(SC, g.IE - i0 + 1);
    const int col0 = (int)idx3(g, 1, i0, j);
    const double dt = a.dtrk, J33G = a.J33G;
    double *F1 = sh, *F2 = sh + SC * KP, *F3 = F2 + SC * KP, *C = F3 + SC * KP; // level k of column q at q*KP + k-1
    for (int q = w; q < ncol; q += SW)
        for (int k = KS + lane; k <= KE - 1; k += 32) {
            const int c = col0 + q * g.KA + k - 1, s = q * KP + k - 1;
            tma::copy_async(F1 + s, (const double *)T.W.F1 + c);
            tma::copy_async(F2 + s, (const double *)T.W.F2 + c);
            tma::copy_async(F3 + s, (const double *)T.W.F3 + c);
            tma::copy_async(C + s, (const double *)T.W.C + c);
        }
    tma::copy_wait();
    __syncthreads();
    if (w == (int)blockIdx.x % SW && lane < ncol) {
        // e goes into F1, f into C; the operands of the next level are read before the
        // reciprocal of this one
        double *f1 = F1 + lane * KP, *f2 = F2 + lane * KP, *f3 = F3 + lane * KP, *cc = C + lane * KP;
        double r = 1.0 / f2[KS - 1], e = -f1[KS - 1] * r, f = cc[KS - 1] * r;
        f1[KS - 1] = e;
        cc[KS - 1] = f;
        double n1 = f1[KS], n2 = f2[KS], n3 = f3[KS], nc = cc[KS];
        for (int k = KS + 1; k <= KE - 2; ++k) {
            const double x1 = n1, x3 = n3, xc = nc, den = n2 + n3 * e;
            n1 = f1[k]; n2 = f2[k]; n3 = f3[k]; nc = cc[k];
            r = 1.0 / den;
            e = -x1 * r;
            f = (xc - x3 * f) * r;
            f1[k - 1] = e;
            cc[k - 1] = f;
        }
        f = (nc - n3 * f) / (n2 + n3 * e);
        cc[KE - 2] = f;
#pragma unroll 4
        for (int k = KE - 2; k >= KS; --k) {
            f = f1[k - 1] * f + cc[k - 1];
            cc[k - 1] = f;
        }
    }
    __syncthreads();
    const int NP = (g.KMAX + 31) / 32;
    for (int item = w; item < SC * NP; item += SW) {
        const int q = item % SC, i = i0 + q, k = KS + (item / SC) * 32 + lane;
        if (q >= ncol || k > KE) continue;
        const int c = col0 + q * g.KA + k - 1;
        const double *Cq = C + q * KP - 1; // 1-based level index
        const double mm = T.mapf(i, j, 1, I_XY) * T.mapf(i, j, 2, I_XY);
        const double rcdz = ld(g.RCDZ + k - 1), gz = T.G(I_XYZ, c);
        const double P0 = k <= KE - 1 ? T.W.PT[c] : 0.0, Pm = k >= KS + 1 ? T.W.PT[c - 1] : 0.0;
        const double C0 = k <= KE - 1 ? Cq[k] : 0.0, Cm = k >= KS + 1 ? Cq[k - 1] : 0.0;
        const double D0 = ld(a.DENS0 + c), T0 = ld(a.RHOT0 + c), Sr = T.W.Sr[c], St = T.W.St[c];
        const double W0 = ld(a.MOMZ0 + c), Wz = ld(a.MOMZ + c), mZ = T.W.mZ[c], tZ = T.W.tZ[c];
        double nr, nt; // numerators of the divergences
        if (k == KS) {
            nr = -C0 * J33G * rcdz;
            nt = -C0 * P0 * J33G * rcdz;
        } else if (k == KE) {
            nr = Cm * J33G * rcdz;
            nt = Cm * Pm * J33G * rcdz;
        } else {
            nr = -(C0 - Cm) * J33G * rcdz;
            nt = -(C0 * P0 - Cm * Pm) * J33G * rcdz;
        }
        double adr, adt, fm, ft;
        auto quot = [&](auto fast) {
            constexpr bool FAST = decltype(fast)::value;
            Gd gd;
            const double y = rn::recip<FAST>(gd, gz), ym = rn::recip<FAST>(gd, mm);
            adr = TDIV(gd, nr, gz, y);
            adt = TDIV(gd, nt, gz, y);
            fm = TDIV(gd, J33G * C0, mm, ym);
            ft = TDIV(gd, J33G * C0 * P0, mm, ym);
            return gd.bad();
        };
        if (quot(std::true_type{})) {
            cold();
            quot(std::false_type{});
        }
        put_state(a, T.N3, 0, a.DENS_RK, a.DENS0, c, D0 + dt * (adr + Sr), true);
        put_state(a, T.N3, 4, a.RHOT_RK, a.RHOT0, c, T0 + dt * (adt + St), true);
        if (k <= KE - 1) {
            put_flux(a, T.N3, 0, c, mZ + fm, true);
            put_flux(a, T.N3, 3, c, tZ + ft, true);
            put_state(a, T.N3, 1, a.MOMZ_RK, a.MOMZ0, c, W0 + (C0 - Wz), true);
        } else {
            put_flux(a, T.N3, 0, c, 0.0, true);
            put_flux(a, T.N3, 3, c, 0.0, true);
            put_state(a, T.N3, 1, a.MOMZ_RK, a.MOMZ0, c, 0.0, false);
        }
        if (k == KS) {
            put_state(a, T.N3, 1, a.MOMZ_RK, a.MOMZ0, c - 1, 0.0, false);
            put_flux(a, T.N3, 0, c - 1, 0.0, false);
            put_flux(a, T.N3, 3, c - 1, 0.0, false);
        }
    }
}

// rho*u (DIR = 0) or rho*v (DIR = 1)
template <int S, int DIR>
__global__ void __launch_bounds__(32 * TW, HEVI_T_MINB) k_t_mom(const __grid_constant__ Terrain T)
{
    constexpr bool U = DIR == 0;
    constexpr int V_Q = U ? V_MOMX : V_MOMY, I_W = U ? I_UYW : I_XVW, I_Z = U ? I_UYZ : I_XVZ, I_M = U ? I_UY : I_XV;
    const Grid &g = T.g;
    const auto &a = T.a;
    const Col q = column(g.IS, g.IMAX, g.JS, g.IMAX * g.JMAX);
    if (!q.ok) return; // warp-uniform
    const int i = q.i, j = q.j, lane = q.lane, KS = g.KS, KE = g.KE, sI = g.KA, sJ = g.KA * g.IA;
    const int s = U ? sI : sJ, so = U ? sJ : sI; // strides of the momentum's own and of the other direction
    const int col = (int)idx3(g, 1, i, j);
    const double dt = a.dtrk, J33G = a.J33G;
    const bool use_div = a.divdmp_coef != 0.0;
    const double *const Q = U ? a.MOMX : a.MOMY, *const O = U ? a.MOMY : a.MOMX, *const MZ = a.MOMZ, *const DN = a.DENS;
    const double *const DP = T.W.DPRES, *const Q0 = U ? a.MOMX0 : a.MOMY0, *const Qt = U ? a.MOMX_t : a.MOMY_t;
    const double m1 = T.mapf(i, j, 1, I_M), m2 = T.mapf(i, j, 2, I_M);
    const int ie = U ? i + 1 : i, je = U ? j : j + 1; // the next column along the momentum
    // map factors of the own-direction faces (cell centres) and of the cross faces
    const double mo1 = T.mapf(ie, je, U ? 2 : 1, I_XY), mo0 = T.mapf(i, j, U ? 2 : 1, I_XY);
    const double mc1 = T.mapf(i, j, U ? 1 : 2, I_UV), mc0 = U ? T.mapf(i, j - 1, 1, I_UV) : T.mapf(i - 1, j, 2, I_UV);
    const double rf = U ? ld(g.RFDX + i - 1) : ld(g.RFDY + j - 1), rc = U ? ld(g.RCDY + j - 1) : ld(g.RCDX + i - 1);
    const double co1 = ld(a.CORIOLI + g.c2 + (size_t)(ie - 1) + (size_t)g.IA * (je - 1));
    const double co0 = ld(a.CORIOLI + g.c2 + (size_t)(i - 1) + (size_t)g.IA * (j - 1));
    // the map-factor differences of the curvature term, per column
    double k1, k2;
    if constexpr (U) {
        k1 = 1.0 / T.mapf(i + 1, j, 2, I_XY) - 1.0 / T.mapf(i, j, 2, I_XY);
        k2 = 1.0 / T.mapf(i, j, 1, I_UV) - 1.0 / T.mapf(i, j - 1, 1, I_UV);
    } else {
        k1 = 1.0 / T.mapf(i, j + 1, 1, I_XY) - 1.0 / T.mapf(i, j, 1, I_XY);
        k2 = 1.0 / T.mapf(i, j, 2, I_UV) - 1.0 / T.mapf(i - 1, j, 2, I_UV);
    }
    double cz = 0.0, c1 = 0.0, c2 = 0.0; // the fluxes below
    for (int k0 = KS; k0 <= KE; k0 += 32) {
        const int k = min(k0 + lane, KE), c = col + k - 1;
        const bool valid = k0 + lane <= KE;
        double qZ, q1, q2, qa1, qa0, qb1, qb0;
        auto faces = [&](auto fast) {
            constexpr bool FAST = decltype(fast)::value;
            Gd gd;
            qZ = q1 = q2 = 0.0;
            if (k <= KE - 1) {
                // fluxZ, fluxJ13 and fluxJ23 of UYZ (ud3.F90:753-1049) or XVZ (:1173-1469)
                auto V = [&](int l) { return ld(Q + col - 1 + l); };
                const double dn1 = ld(DN + c + 1) + ld(DN + c + 1 + s), dn0 = ld(DN + c) + ld(DN + c + s);
                double f1, f2;
                T.f2h<FAST>(gd, I_W, c, k, f1, f2);
                const double vel = TDIV(gd, 0.5 * (ld(MZ + c) + ld(MZ + c + s)), f1 * 0.5 * dn1 + f2 * 0.5 * dn0);
                qZ = J33G * vel * zface<S>(vel, k, KS, KE, V) + T.G(I_W, c) * T.nd(V_Q, DZIR, c);
                T.f2h<FAST>(gd, I_Z, c, k, f1, f2);
                const double den = f1 * 0.5 * dn1 + f2 * 0.5 * dn0, y = rn::recip<FAST>(gd, den);
                // the other momentum averaged onto this point
                auto avg = [&](int p) {
                    return U ? 0.25 * (ld(O + p) + ld(O + p + s) + ld(O + p - so) + ld(O + p + s - so))
                             : 0.25 * (ld(O + p) + ld(O + p - so) + ld(O + p + s) + ld(O + p - so + s));
                };
                const double own = TDIV(gd, f1 * ld(Q + c + 1) + f2 * ld(Q + c), den, y);
                const double oth = TDIV(gd, f1 * avg(c + 1) + f2 * avg(c), den, y);
                const double v1 = (U ? own : oth) * T.J13(I_W, c), v2 = (U ? oth : own) * T.J23(I_W, c);
                q1 = TDIV(gd, v1, m2) * zface<S>(v1, k, KS, KE, V);
                q2 = TDIV(gd, v2, m1) * zface<S>(v2, k, KS, KE, V);
            }
            // along the momentum, with the index shift of fluxX_UYZ (:1053-1109) / fluxY_XVZ (:1531-1587)
            auto along = [&](int cf, double mp) {
                const double vel = TDIV(gd, 0.5 * (ld(Q + cf) + ld(Q + cf - s)), ld(DN + cf)), Gs = T.G(I_XYZ, cf);
                return TDIV(gd, Gs, mp) * vel * hface<S>(vel, Q + cf - s, s) + Gs * T.nd(V_Q, U ? DXIR : DYIR, cf);
            };
            // across, fluxY_UYZ (:1113-1167) / fluxX_XVZ (:1473-1527)
            auto across = [&](int cf, double mp) {
                const double vel = TDIV(gd, 0.5 * (ld(O + cf) + ld(O + cf + s)),
                                        0.25 * (ld(DN + cf) + ld(DN + cf + sI) + ld(DN + cf + sJ) + ld(DN + cf + sI + sJ)));
                const double Gs = T.G(I_UVZ, cf);
                return TDIV(gd, Gs, mp) * vel * hface<S>(vel, Q + cf, so) + Gs * T.nd(V_Q, U ? DYIR : DXIR, cf);
            };
            qa1 = along(c + s, mo1);
            qa0 = along(c, mo0);
            qb1 = across(c, mc1);
            qb0 = across(c - so, mc0);
            return gd.bad();
        };
        if (faces(std::true_type{})) {
            cold();
            faces(std::false_type{});
        }
        const double qZm = below(qZ, cz), q1m = below(q1, c1), q2m = below(q2, c2);
        const double rcdz = ld(g.RCDZ + k - 1);
        const double advcv = -(qZ - qZm + q1 - q1m + q2 - q2m) * rcdz;
        const double advch = (U ? -((qa1 - qa0) * rf + (qb1 - qb0) * rc) : -((qb1 - qb0) * rc + (qa1 - qa0) * rf)) * m1 * m2;
        const double dpc = ld(DP + c), dpe = ld(DP + c + s), dpt = ld(DP + c + 1), dpte = ld(DP + c + 1 + s);
        const double dpb = ld(DP + c - 1), dpbe = ld(DP + c - 1 + s);
        const double J0 = U ? T.J13(I_W, c) : T.J23(I_W, c), Jm = U ? T.J13(I_W, c - 1) : T.J23(I_W, c - 1);
        const double g1 = T.G(I_XYZ, c + s), g0 = T.G(I_XYZ, c), gq = T.G(I_Z, c);
        const double o0 = ld(O + c), o1 = ld(O + c + s), o2 = ld(O + c - so), o3 = ld(O + c + s - so);
        const double sum = o0 + o2 + o1 + o3;
        const double dn = U ? ld(DN + c + s) + ld(DN + c) : ld(DN + c) + ld(DN + c + s);
        const double q0 = ld(Q0 + c), qt = ld(Qt + c), qc = ld(Q + c);
        double val;
        auto update = [&](auto fast) {
            constexpr bool FAST = decltype(fast)::value;
            Gd gd;
            double f1, f2, b1, b2; // F2H at k, and at k (u) or k-1 (v) for the lower term
            T.f2h<FAST>(gd, I_Z, c, k, f1, f2);
            if constexpr (U) {
                b1 = f1;
                b2 = f2;
            } else {
                T.f2h<FAST>(gd, I_Z, c - 1, k - 1, b1, b2);
            }
            const double pg = ((g1 * dpe - g0 * dpc) * rf
                               + (J0 * 0.5 * (f1 * (dpte + dpt) + f2 * (dpe + dpc))
                                  - Jm * 0.5 * (b1 * (dpe + dpc) + b2 * (dpbe + dpb)))
                                     * rcdz)
                              * (U ? m1 : m2);
            double cf;
            if constexpr (U)
                cf = 0.125 * (co1 + co0) * (o1 + o0 + o3 + o2)
                     + TDIV(gd, 0.25 * m1 * m2 * sum * (sum * 0.25 * k1 * rf - qc * k2 * rc) * 2.0, dn);
            else
                cf = -0.125 * (co1 + co0) * (o1 + o0 + o3 + o2)
                     - TDIV(gd, 0.25 * m1 * m2 * sum * (qc * k2 * rc - 0.25 * sum * k1 * rf) * 2.0, dn);
            const double div = use_div ? a.divdmp_coef / dt * (ld(a.DDIV + c + s) / mo1 - ld(a.DDIV + c) / T.mapf(i, j, 1, I_XY))
                                             * m1 * m2 * (U ? ld(g.FDX + i - 1) : ld(g.FDY + j - 1))
                                       : 0.0;
            val = q0 + dt * (TDIV(gd, advcv + advch - pg, gq) + cf + div + qt);
            return gd.bad();
        };
        if (update(std::true_type{})) {
            cold();
            update(std::false_type{});
        }
        if (valid && (U ? i <= g.IEH : j <= g.JEH))
            put_state(a, T.N3, U ? 2 : 3, U ? a.MOMX_RK : a.MOMY_RK, Q0, c, val, true);
    }
}
#undef TDIV

template <int S>
cudaError_t terrain_stage(const Terrain &T, cudaStream_t st)
{
    const Grid &g = T.g;
    const int ncol = g.IMAX * g.JMAX, nb = (ncol + TW - 1) / TW;
    const dim3 b(32, TW);
    k_t_prep<<<(g.IA * g.JA + TW - 1) / TW, b, 0, st>>>(T);
    k_t_mass<S><<<nb, b, 0, st>>>(T);
    k_t_w<S><<<nb, b, 0, st>>>(T);
    const cudaError_t e = tma::open_smem(k_t_column, t_column_smem(260));
    if (e != cudaSuccess) return e;
    k_t_column<<<((g.IMAX + SC - 1) / SC) * g.JMAX, dim3(32, SW), t_column_smem(g.KA), st>>>(T);
    k_t_mom<S, 0><<<nb, b, 0, st>>>(T);
    k_t_mom<S, 1><<<nb, b, 0, st>>>(T);
    return cudaGetLastError();
}

} // namespace

cudaError_t launch_terrain_stage(const Grid &g, const StageArgsT<double> &a, const Metrics &M, const TerrainWork &W,
                                 int scheme, cudaStream_t st)
{
    const Terrain T{g, a, M, W, n3(g)};
    switch (scheme) {
    case UD3: return terrain_stage<UD3>(T, st);
    case CD4: return terrain_stage<CD4>(T, st);
    case KOREN: return terrain_stage<KOREN>(T, st);
    case CD2: return terrain_stage<CD2>(T, st);
    case UD5: return terrain_stage<UD5>(T, st);
    case CD6: return terrain_stage<CD6>(T, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace hevi
