// The HEVI stage (ATMOS_DYN_Tstep_short_fvm_hevi,
// scalelib/src/atmos-rm/dynamics/scale_atmos_dyn_tstep_short_fvm_hevi.F90:128-1089)
// as two kernels: k_hevi_explicit, which stages its tiles in shared memory with
// the tensor memory accelerator (TMA), and k_hevi_column, the implicit column
// problem. Line numbers refer to that file unless a flux file is named.
//
// A CTA owns a 4 x 4 tile of columns, one warp per column with its lanes along
// k. It marches up the columns in chunks of 32 levels. For each chunk one
// thread issues cp.async.bulk.tensor copies of the five state fields (DENS,
// MOMZ, MOMX, MOMY, RHOT) over the tile, its lateral halo (2 points; 3 for the
// 6-point schemes) and the levels from 4 below to 2-3 above the chunk into
// shared memory, completing on an mbarrier; the tensor maps cover this GPU's
// own memory and the copies have no cluster multicast. Every stencil then
// reads shared memory at compile-time offsets. Per chunk:
//   a. the pressure deviation DPRES (hevi_pres :343-361) of the tile and of its
//      +x/+y neighbour columns; RHOT -> POTT in place (:586-600)
//   b. x/y mass fluxes (:399-438), Sr (:443-479), PT and the vertical theta
//      flux (valueW_Z, fluxZ_XYZ), the x/y theta fluxes and St (:603-661)
//   c. one level lower: Sw (:528-578) and the right-hand side C (:698-722)
//   d. rho*u and rho*v (hevi_momx :814-928, hevi_momy :934-1048)
// The z flux through the face below a level is the previous lane's flux above it,
// by a warp shuffle; lane 0 takes the previous chunk's lane 31's. Chunks clear of
// the near-wall face forms run without level dispatch. The fluxes and momenta
// leave through the RK folds; Sr, St, tZ, PT and C go to the column scratch.
//
// What bounds the march is the latency of its global loads, at 32 warps per SM
// (the staged boxes fill the shared memory). So each step reads all its global
// operands before it computes, and nothing splits it into blocks that loads
// cannot move across: the quotients are straight-line code (rn_div.cuh), the RK
// fold is a template parameter, and columns and levels beyond the domain run along
// at clamped addresses and only their stores are masked. 512x512x128, CD4, FP64:
// 5.70 -> 4.29 ms per launch, the mean of a step's four (on 256x256x128 405 instead of
// 640 million warp instructions, and 44% instead of 33% of DRAM peak).
//
// Every value keeps the operation order of the fused kernel k_hevi_stage
// (hevi_stage.cu) and of the reference, so the two forms give identical bits.
// Flat terrain.
#include "hevi_epilogue.cuh"
#include "hevi_kernels.cuh"
#include "rn_div.cuh"
#include "tma_util.cuh"

namespace hevi {
namespace tma {

constexpr int TX = 4, TY = 4, NCOL = TX * TY; // tile columns; one warp each
constexpr int KC = 32;                        // levels per chunk (one per lane)
constexpr int KLO = 4;                        // box levels below the chunk's first level
template <int S> __host__ __device__ constexpr int reach() { return wide_scheme(S) ? 3 : 2; }
// box levels: L0-4 .. L0+33 (4-point schemes) or L0-4 .. L0+35 (6-point), L0
// the chunk's first level; 38 and 40 keep the inner box a multiple of 16 bytes
template <int S> __host__ __device__ constexpr int box_k() { return wide_scheme(S) ? 40 : 38; }
template <int S> __host__ __device__ constexpr int box_w() { return TX + 2 * reach<S>(); }
template <int S> __host__ __device__ constexpr int box_h() { return TY + 2 * reach<S>(); }
template <int S> __host__ __device__ constexpr int plane() { return box_k<S>() * box_w<S>() * box_h<S>(); }
// Split march: a CTA takes one chunk instead of the whole column. The lowest two lanes
// of a chunk above the first are then levels of the chunk below, run along for the
// z fluxes, Sr and St that the chunk's first level needs, so a chunk advances 30 levels.
constexpr int NGHOST = 2;
__host__ __device__ constexpr int chunks(int KMAX, bool split)
{
    return !split ? (KMAX + KC - 1) / KC : KMAX <= KC ? 1 : 1 + (KMAX - KC + KC - NGHOST - 1) / (KC - NGHOST);
}
constexpr int NF = 5;                         // staged fields
enum StagedField : int { F_DN = 0, F_MZ = 1, F_MX = 2, F_MY = 3, F_RT = 4 };
constexpr int NDP = 33;                       // levels of a chunk's level tables: L0-1 .. L0+31
constexpr int DP_COLS = NCOL + TX + TY;       // DPRES columns: the tile's, then its +x and its +y side
constexpr int NCARRY = 7;                     // values a column carries into the next chunk
constexpr int NLT = 6;                        // level tables per chunk: RCDZ, RFDZ, F2H1, F2H2, FDZ, wdamp

template <int S> constexpr size_t smem_bytes()
{
    return (size_t)NF * plane<S>() * sizeof(double) + (size_t)((DP_COLS + NCOL + NLT) * NDP + NCOL * NCARRY) * sizeof(double) + 16;
}

struct StateMaps {
    CUtensorMap m[NF]; // DENS, MOMZ, MOMX, MOMY, RHOT as (KA, IA, JA) FP64 tensors
};

// =============================================================================
// k_hevi_explicit
// =============================================================================
// the face value at w-level m in a chunk that lies clear of the near-wall
// forms: zface<S> without its level dispatch
template <int S, typename R, typename V>
__device__ __forceinline__ R zface_in(R vel, int m, const V &v)
{
    if constexpr (wide_scheme(S)) return ip6<S>(vel, v(m - 2), v(m - 1), v(m), v(m + 1), v(m + 2), v(m + 3));
    else return ip4<S>(vel, v(m - 1), v(m), v(m + 1), v(m + 2));
}

// -(dq r) - (A a + B b), a momentum's vertical and horizontal flux divergence. FP64
// code never fuses. FP32 code fuses A a into the horizontal sum and nothing else; left to
// the compiler, what fuses depends on the code around it, and a mixed step's momenta
// move by 1e-8 with it.
__device__ __forceinline__ double advection(double dq, double r, double A, double a, double B, double b)
{
    return -dq * r + -(A * a + B * b);
}
__device__ __forceinline__ float advection(float dq, float r, float A, float a, float B, float b)
{
    return __fadd_rn(__fmul_rn(-dq, r), -__fmaf_rn(A, a, __fmul_rn(B, b)));
}

// keeps the compiler from carrying values of the fast path into the rare exact one
__device__ __forceinline__ void cold() { asm volatile("" ::: "memory"); }

// Where the outputs of a stage go, fixed at compile time so that the marching
// kernel has no dispatch in its loop: the RkMode itself, with RK_STAGE2 standing
// for RK_STAGE3 too and FOLD_ANY for the run-time dispatch of put_state/put_flux
// (Heun's modes).
constexpr int FOLD_ANY = -1;
__host__ __device__ constexpr bool fold_reads(int m) { return m == RK_STAGE2 || m == RK_FINAL; }

// The arrays that a thread addresses at its cell, by component: formed on the
// host, so that an access is one multiply-add on a constant-bank pointer.
template <typename R>
struct StagePtrs {
    const double *in[NF]; // the staged fields
    const R *nd[15]; // num_diff components q + 5*dir
    const double *rk1[5], *rk2[5]; // the first two stage buffers
    R *facc[6], *flx[6]; // mflx z, x, y then tflx z, x, y
    R *Sr, *St, *tZ, *PT;
};

template <typename R>
struct StageMaps { // what the host prepares for one launch
    StagePtrs<R> ptr;
    StateMaps maps;
};

template <int M, typename R>
__device__ __forceinline__ void fold_state(const StageArgsT<R> &a, const StagePtrs<R> &p, size_t N3, int v, double *out,
                                           const double *x0p, int c, double val, double x0, double acc)
{
    if constexpr (M == RK_PLAIN) {
        sts(out + c, val);
        flag_nonfinite(a.status, val);
    } else if constexpr (M == RK_STAGE1 || M == RK_STAGE2) {
        sts(out + c, val);
    } else if constexpr (M == RK_FINAL) {
        const double r = rn::sixth((acc + val) - x0 * 3.0);
        sts(out + c, r);
        flag_nonfinite(a.status, r);
    } else {
        put_state(a, N3, v, out, x0p, (size_t)c, val, true);
    }
}
template <int M, typename R>
__device__ __forceinline__ void fold_flux(const StageArgsT<R> &a, const StagePtrs<R> &p, size_t N3, int f, int c, R val,
                                          R acc)
{
    if constexpr (M == RK_PLAIN) sts(p.flx[f] + c, val);
    else if constexpr (M == RK_STAGE1) sts(p.facc[f] + c, val);
    else if constexpr (M == RK_STAGE2) sts(p.facc[f] + c, acc + val * R(2.0));
    else if constexpr (M == RK_FINAL) sts(p.flx[f] + c, rn::sixth(acc + val));
    else put_flux(a, N3, f, (size_t)c, val, true);
}
// RK1*2 + RK2*4 + RK3*2 of the combine, rk3 being the last stage's input
template <int M, typename R>
__device__ __forceinline__ double rk_sum(const StagePtrs<R> &p, int v, int c, double rk3)
{
    if constexpr (M == RK_FINAL) return (lds(p.rk1[v] + c) * 2.0 + lds(p.rk2[v] + c) * 4.0) + rk3 * 2.0;
    else return 0.0;
}
// a flux through the domain's west or south rim, which the combines leave as the last stage's
template <int M, typename R>
__device__ __forceinline__ void rim_flux(const StageArgsT<R> &a, const StagePtrs<R> &p, size_t N3, int f, int c, R val)
{
    if constexpr (M == RK_PLAIN || M == RK_FINAL) sts(p.flx[f] + c, val);
    else if constexpr (M == FOLD_ANY) put_flux(a, N3, f, (size_t)c, val, false);
}

template <int S, typename R, int M, int LD, int NM>
__global__ void __launch_bounds__(32 * NCOL, wide_scheme(S) ? 1 : 2)
    k_hevi_explicit(const Grid gt, const StageArgsT<R> a, const BatchT<NM> B, const __grid_constant__ StagePtrs<R> ptr,
                    const bool split, const __grid_constant__ StateMaps maps)
{
    constexpr int H = reach<S>(), BW = box_w<S>(), BK = box_k<S>(), PL = plane<S>();
    constexpr int KX = BK, KY = BW * BK; // shared-memory strides of one column step in i and in j
    constexpr bool W6 = wide_scheme(S), ACC = fold_reads(M);
    extern __shared__ __align__(1024) double sm[];
    double *stg = sm;                    // NF staged fields, [j][i][k] each
    double *sdp = sm + NF * PL;          // DPRES, [DP_COLS][NDP]: levels L0-1 .. L0+31
    double *srp = sdp + DP_COLS * NDP;   // RT2P of the tile's own columns, [NCOL][NDP]
    double *slt = srp + NCOL * NDP;      // the chunk's level tables, [NLT][NDP]
    R *scy = reinterpret_cast<R *>(slt + NLT * NDP); // [NCOL][NCARRY]
    uint64_t *bar = reinterpret_cast<uint64_t *>(slt + NLT * NDP + NCOL * NCARRY);
    __shared__ int s_ok;
    __shared__ R s_rc[2][NCOL]; // RCDX, RCDY of the columns

    int b;
    const Grid g = block_domain(gt, B, b);
    const int lane = threadIdx.x, w = threadIdx.y, tid = w * 32 + lane;
    const int tx = w % TX, ty = w / TX;
    // the chunks of this CTA: all of the column's, or one of the split march's
    const int KST = split ? KC - NGHOST : KC, ns = chunks(g.KMAX, split);
    const int ch0 = split ? b % ns : 0, ch1 = split ? ch0 + 1 : ns;
    if (split) b /= ns;
    const int ghosts = ch0 > 0 ? NGHOST : 0; // lanes below the chunk's own levels
    int ti, tj;
    {
        // raster: consecutive CTAs walk down a.raster rows of tiles, then step in i
        const int nti = (g.IMAX + TX - 1) / TX, ntj = (g.JMAX + TY - 1) / TY, RJ = a.raster;
        const int grp = b / (nti * RJ), rem = b - grp * (nti * RJ);
        const int rows = min(RJ, ntj - grp * RJ);
        tj = grp * RJ + rem % rows;
        ti = rem / rows;
    }
    const int i0 = g.IS + ti * TX, j0 = g.JS + tj * TY;
    const bool col_ok = i0 + tx <= g.IE && j0 + ty <= g.JE;
    // warps beyond the domain's edge run along and store nothing; the first halo column's
    // forms the DPRES that the last column needs
    const int i = min(i0 + tx, g.IE + 1), j = min(j0 + ty, g.JE + 1);
    const size_t N3 = n3(g);
    const int sI = g.KA, sJ = g.KA * g.IA;
    const int KS = g.KS, KE = g.KE;
    const int col = (int)idx3(g, 1, i, j); // offset of level 1 of this warp's column
    const double dt = a.dtrk, J33G = a.J33G;
    const bool use_div = a.divdmp_coef != 0.0;
    const R ddc = use_div ? R(a.divdmp_coef / dt) : R(0.0);
    const R h = R(0.5), qr = R(0.25), J33R = R(J33G);
    const unsigned FULL = 0xffffffffu;

    // the chunk's box: levels L0-4 .., columns i0-H .., rows j0-H .. of every staged field
    auto issue = [&](int ch) {
        if constexpr (LD == LD_TMA) {
            if (tid != 0) return;
            // box origin (0-based): level L0-4 = KST*ch - 2 (even, so its byte offset is a
            // multiple of 16), column i0-H, row j0-H
            const int x = KST * ch + (KS - 1) - KLO, y = i0 - H - 1, z = j0 - H - 1;
            fence_proxy_async();
            mbar_expect_tx(bar, (unsigned)(NF * PL * sizeof(double)));
            for (int f = 0; f < NF; ++f) tma_load_3d(stg + f * PL, &maps.m[f], x, y, z, bar);
        } else {
            const int l0 = KS + KST * ch - KLO; // the level of box element 0
            constexpr int TAIL = BK - 32;      // levels of a column beyond one per lane
            for (int q = w; q < BW * BW; q += NCOL) {
                const int ii = i0 - H + q % BW, jj = j0 - H + q / BW;
                if (ii > g.IA || jj > g.JA) continue; // the box of the last tiles reaches beyond the array
                const int at = (int)idx3(g, 1, ii, jj) + l0 - 1;
                double *const dst = stg + q * BK;
                if (l0 + lane >= 1 && l0 + lane <= g.KA)
#pragma unroll
                    for (int f = 0; f < NF; ++f) copy_async(dst + f * PL + lane, ptr.in[f] + at + lane);
                for (int e = lane; e < NF * TAIL; e += 32) {
                    const int f = e / TAIL, lv = 32 + e % TAIL;
                    if (l0 + lv <= g.KA) copy_async(dst + f * PL + lv, ptr.in[f] + at + lv);
                }
            }
        }
    };
    static_assert(TX == TY, "a square box");
    if (LD == LD_TMA && tid == 0) {
        s_ok = 1;
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    issue(ch0);
    __syncthreads();

    // this warp's column in the staged box, at the lane's level of the chunk
    const int cbox = ((ty + H) * BW + (tx + H)) * BK + KLO + lane;
    // the column it computes on: a warp beyond the domain's edge takes the edge's, as its
    // own may have neighbours beyond the array, where nothing (cp.async) or zero (TMA) is
    // staged. On those its quotients left the range of the straight-line form, the Koren
    // limiter took its general form, and the CTA waited for it: a step at 61x53x40, UD3,
    // 281 -> 255 us, at 61x53x41, Koren, 537 -> 409 us with the levels below. FP32 without
    // the limiter keeps its own column, 0.5% faster at 256x256x96.
    constexpr bool EDGE_COL = sizeof(R) == 8 || S == KOREN;
    const int crun = !EDGE_COL ? cbox
                               : ((min(ty, g.JE - j0) + H) * BW + (min(tx, g.IE - i0) + H)) * BK + KLO + lane;
    // this column's DPRES and RT2P at level k = L-1 ([1]: at level L), and DPRES at level L
    // of its +x and +y neighbours: the tile's columns, then the +x and the +y side
    double *const dpc = sdp + w * NDP + lane, *const rtc = srp + w * NDP + lane;
    const int dpE = (tx < TX - 1 ? w + 1 : NCOL + ty) * NDP + lane + 1, dpN = (ty < TY - 1 ? w + TX : NCOL + TY + tx) * NDP + lane + 1;
    // the +x (warps 0..TY-1) or +y (the next TX) side column whose DPRES this warp forms
    const int ex = w < TY ? TX : w - TY, ey = w < TY ? w : TY;
    const bool side = w < TX + TY;
    const int cside = side ? (int)idx3(g, 1, min(i0 + ex, g.IE + 1), min(j0 + ey, g.JE + 1)) : col;
    // The fluxes through the face below a level (mass, theta, w, u, v), and Sr and St
    // one level down, are the lane below's: the values are rotated around the warp, and
    // lane 0, which receives lane 31's, leaves that for the next chunk and takes the
    // previous chunk's. Zero below KS, where every flux is zero. (In shared memory: as
    // registers they would spill.)
    R *const carry = scy + w * NCARRY;
    if (lane < NCARRY) carry[lane] = R(0.0);
    if (lane == 0) {
        s_rc[0][w] = R(ld(g.RCDX + i - 1));
        s_rc[1][w] = R(ld(g.RCDY + j - 1));
    }
    __syncwarp();
    auto below = [&](R v, int q) {
        R r = __shfl_sync(FULL, v, (lane + 31) & 31);
        if (lane == 0) {
            const R x = carry[q];
            carry[q] = r;
            r = x;
        }
        return r;
    };
    enum { C_MZ, C_TZ, C_SR, C_ST, C_QW, C_QU, C_QV };

    for (int ch = ch0; ch < ch1; ++ch) {
        const int L0 = KS + KST * ch, L = L0 + lane;
        const int lev = min(L, KE) - 1;  // lanes above KE run along on the last level
        const int c = col + lev, cs = cside + lev;
        const bool vl = col_ok && L <= KE; // a level of the domain, ghosts included
        const bool vb = vl && lane >= ghosts;

        // ---- a. DPRES (:355) at the chunk's levels of this warp's column and of its side
        // column, the level tables (levels L0-1..L0+31, clamped to KE), RHOT -> POTT.
        // The global operands are on their way before the wait for the copies.
        const double rt_L = ld(a.RT2P + c), dp0 = ld(a.DPRES0 + c), rr0 = ld(a.REF_rhot + c);
        double rt_s = 0.0, dp0_s = 0.0, rr_s = 0.0;
        if (side) { rt_s = ld(a.RT2P + cs); dp0_s = ld(a.DPRES0 + cs); rr_s = ld(a.REF_rhot + cs); }
        if constexpr (LD == LD_TMA) {
            if (!mbar_wait(bar, (ch - ch0) & 1)) { // bounded; the block leaves at the barrier below
                s_ok = 0;
                (void)mbar_wait(bar, (ch - ch0) & 1); // bounded: the copies still in flight
            }
        } else {
            copy_wait();
            __syncthreads();
        }
        double *const sRT = stg + F_RT * PL + cbox;
        if (lane == 31) { // the previous chunk's last level
            dpc[-31] = dpc[1];
            rtc[-31] = rtc[1];
        }
        dpc[1] = dp0 + rt_L * (sRT[0] - rr0);
        rtc[1] = rt_L;
        if (side) {
            const double rt = stg[F_RT * PL + ((ey + H) * BW + (ex + H)) * BK + KLO + lane];
            sdp[(NCOL + w) * NDP + lane + 1] = dp0_s + rt_s * (rt - rr_s);
        }
        if (w == NCOL - 1) {
            for (int lv = lane; lv < NDP; lv += 32) {
                const int Lq = min(L0 - 1 + lv, KE);
                slt[0 * NDP + lv] = ld(g.RCDZ + Lq - 1);
                slt[1 * NDP + lv] = ld(g.RFDZ + Lq - 1);
                slt[2 * NDP + lv] = ld(g.F2H1 + Lq - 1);
                slt[3 * NDP + lv] = ld(g.F2H2 + Lq - 1);
                slt[4 * NDP + lv] = ld(g.FDZ + Lq - 1);
                slt[5 * NDP + lv] = ld(a.wdamp + g.z0 + Lq - 1);
            }
        }
        {
            // RHOT -> POTT = RHOT/DENS (:586-600) in place, at the levels KS..KE: the tile's own
            // columns over the whole box height (the vertical stencils), the x/y arms of the
            // halo at the chunk's levels (the horizontal theta fluxes). A column of the box is
            // converted by the warp that read its RHOT above.
            constexpr int NARM = 2 * H * (TX + TY), NPW = NARM / NCOL; // arm columns; per warp
            static_assert(NARM % NCOL == 0 && TX == TY && TX + TY <= NCOL, "arms per warp");
            int at[2 + NPW];
            bool in[2 + NPW];
            at[0] = cbox - lane - KLO + lane;
            in[0] = L - KLO >= KS && L - KLO <= KE;
            at[1] = min(at[0] + 32, cbox - lane - KLO + BK - 1);
            in[1] = lane < BK - 32 && L - KLO + 32 <= KE;
#pragma unroll
            for (int q = 0; q < NPW; ++q) {
                // arm n: the side column of warp n (n < TX + TY) comes first, so that this warp converts it
                int bx, by;
                const int n = q * NCOL + w;
                if (n < TX + TY) {
                    bx = ex + H;
                    by = ey + H;
                } else {
                    const int m = n - (TX + TY), d = m / (TX + TY), r = m % (TX + TY); // d: which of the other rings
                    const int off = d < H ? d : TX + 1 + d;                           // 0..H-1, then TX+H+1..
                    bx = r < TY ? off : r - TY + H;
                    by = r < TY ? r + H : off;
                }
                at[2 + q] = (by * BW + bx) * BK + KLO + lane;
                in[2 + q] = L <= KE;
            }
            rn::Guard<R> gd;
            R x[2 + NPW], y[2 + NPW];
#pragma unroll
            for (int q = 0; q < 2 + NPW; ++q) {
                x[q] = in[q] ? R(stg[F_RT * PL + at[q]]) : R(0.0);
                y[q] = in[q] ? R(stg[F_DN * PL + at[q]]) : R(1.0);
                x[q] = rn::div<true>(gd, x[q], y[q]);
            }
            if (gd.bad()) {
#pragma unroll
                for (int q = 0; q < 2 + NPW; ++q)
                    if (in[q]) x[q] = R(stg[F_RT * PL + at[q]]) / R(stg[F_DN * PL + at[q]]);
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 2 + NPW; ++q)
                if (in[q]) stg[F_RT * PL + at[q]] = (double)x[q];
        }
        __syncthreads();
        if (LD == LD_TMA && !s_ok) {
            if (tid == 0) atomicOr(a.status, ST_TMA_TIMEOUT);
            return; // block-uniform
        }

        // Chunks clear of the near-wall face forms (every face of the chunk, from
        // the one below L0-1 to the one above L0+31, in the interior range, and
        // every level of the chunk at or below KE) run without level dispatch or
        // range checks: EDGE = false.
        const bool interior = L0 - 1 >= KS + (W6 ? 2 : 1) && L0 + 31 <= KE - (W6 ? 3 : 2);
        // the level tables at this lane's level L (slot lane+1) and at k = L-1 (slot lane)
        const double *lt = slt + lane;
#define rcdx s_rc[0][w]
#define rcdy s_rc[1][w]
#define rcdz_L lt[0 * NDP + 1]
#define rfdz_k lt[1 * NDP]
#define f1_L lt[2 * NDP + 1]
#define f1_k lt[2 * NDP]
#define f2_L lt[3 * NDP + 1]
#define f2_k lt[3 * NDP]
#define fdz_k lt[4 * NDP]
#define wd_k lt[5 * NDP]
        auto chunk = [&](auto edge) {
            constexpr bool EDGE = decltype(edge)::value;
            // without tensor maps, lanes above KE have levels where nothing is staged either;
            // only the limiter minds
            const int here = crun + (S == KOREN && LD == LD_COPY ? lev + 1 - L : 0);
            const double *const sDN = stg + F_DN * PL + here, *const sMZ = stg + F_MZ * PL + here;
            const double *const sMX = stg + F_MX * PL + here, *const sMY = stg + F_MY * PL + here;
            const double *const sPO = stg + F_RT * PL + here; // POTT
            auto zf = [&](R vel, int m, const auto &v) -> R {
                if constexpr (EDGE) return zface<S>(vel, m, KS, KE, v);
                else return zface_in<S>(vel, m, v);
            };
            // a value of a column operand at level l, near level m (EDGE: lanes whose
            // level is out of range evaluate the wall forms at clamped levels, unused)
            const bool zok = !EDGE || L <= KE - 1; // the face above L carries a flux
            // ---- b. level L: mass and theta fluxes, Sr, St, PT, tZ ----
            R Sr = R(0.0), St = R(0.0);
            {
                const R dz = ld(ptr.nd[0] + c), nTZ = lds(ptr.nd[4] + c);
                const R nXe = ld(ptr.nd[5] + c), nXw = ld(ptr.nd[5] + c - sI), nYn = ld(ptr.nd[10] + c), nYs = ld(ptr.nd[10] + c - sJ);
                const R nTXe = ld(ptr.nd[9] + c), nTXw = ld(ptr.nd[9] + c - sI), nTYn = ld(ptr.nd[14] + c), nTYs = ld(ptr.nd[14] + c - sJ);
                const R tD = lds(a.DENS_t + c), tT = lds(a.RHOT_t + c);
                // the vertical mass flux through the face above L (hevi_mflx_z :383-391);
                // the face below is the previous lane's
                const R mZ = zok ? dz : R(0.0);
                const R mZm1 = below(mZ, C_MZ);
                auto P = [&](int l) { return R(sPO[l - L]); };
                R PT = R(0.0), tZ = R(0.0);
                if (zok) {
                    // PT: valueW_Z (ud3.F90:98-153); tZ: fluxZ_XYZ (ud3.F90:157-247)
                    PT = zf(R(sMZ[0]), L, P);
                    tZ = mZ * zf(mZ, L, P) + nTZ;
                }
                const R tZm = below(tZ, C_TZ);
                const R Xe = R(sMX[0]) + nXe, Xw = R(sMX[-KX]) + nXw;
                const R Yn = R(sMY[0]) + nYn, Ys = R(sMY[-KY]) + nYs;
                const R adv_r = -((Xe - Xw) * rcdx + (Yn - Ys) * rcdy);
                const R rcdz = R(rcdz_L);
                Sr = (-(mZ - mZm1) * rcdz + adv_r) + tD;
                const R aX = ACC ? lds(ptr.facc[1] + c) : R(0.0), aY = ACC ? lds(ptr.facc[2] + c) : R(0.0);
                const R aTX = ACC ? lds(ptr.facc[4] + c) : R(0.0), aTY = ACC ? lds(ptr.facc[5] + c) : R(0.0);
                // fluxX/Y_XYZ (ud3.F90:251-353)
                const R P00 = R(sPO[0]);
                const R Pm2 = R(sPO[-2 * KX]), Pm1 = R(sPO[-KX]), Pp1 = R(sPO[KX]), Pp2 = R(sPO[2 * KX]);
                const R Qm2 = R(sPO[-2 * KY]), Qm1 = R(sPO[-KY]), Qp1 = R(sPO[KY]), Qp2 = R(sPO[2 * KY]);
                const R Pm3 = W6 ? R(sPO[-3 * KX]) : R(0.0), Pp3 = W6 ? R(sPO[3 * KX]) : R(0.0);
                const R Qm3 = W6 ? R(sPO[-3 * KY]) : R(0.0), Qp3 = W6 ? R(sPO[3 * KY]) : R(0.0);
                const R tXe = Xe * ip6<S>(Xe, Pm2, Pm1, P00, Pp1, Pp2, Pp3) + nTXe;
                const R tXw = Xw * ip6<S>(Xw, Pm3, Pm2, Pm1, P00, Pp1, Pp2) + nTXw;
                const R tYn = Yn * ip6<S>(Yn, Qm2, Qm1, P00, Qp1, Qp2, Qp3) + nTYn;
                const R tYs = Ys * ip6<S>(Ys, Qm3, Qm2, Qm1, P00, Qp1, Qp2) + nTYs;
                const R adv_t = -((tXe - tXw) * rcdx + (tYn - tYs) * rcdy); // hevi_st :646-648
                St = (-(tZ - tZm) * rcdz + adv_t) + tT;                     // hevi_st :646-649
                if (vb) {
                    fold_flux<M>(a, ptr, N3, 1, c, Xe, aX);
                    fold_flux<M>(a, ptr, N3, 2, c, Yn, aY);
                    fold_flux<M>(a, ptr, N3, 4, c, tXe, aTX);
                    fold_flux<M>(a, ptr, N3, 5, c, tYn, aTY);
                    if constexpr (M == RK_PLAIN || M == RK_FINAL || M == FOLD_ANY) {
                        if (i == g.IS) { rim_flux<M>(a, ptr, N3, 1, c - sI, Xw); rim_flux<M>(a, ptr, N3, 4, c - sI, tXw); }
                        if (j == g.JS) { rim_flux<M>(a, ptr, N3, 2, c - sJ, Ys); rim_flux<M>(a, ptr, N3, 5, c - sJ, tYs); }
                    }
                    ptr.Sr[c] = Sr;
                    ptr.St[c] = St;
                    ptr.tZ[c] = tZ;
                    ptr.PT[c] = PT;
                }
            }

            // ---- c. level k = L-1: Sw (hevi_sw :528-578) and C(k) (:698-722) ----
            {
                const int ck = c - 1;
                const R nZ = lds(ptr.nd[1] + c);
                const double rd1 = ld(a.REF_dens + c), rd0 = ld(a.REF_dens + ck); // REF_dens(k+1), (k)
                const R nXe = ld(ptr.nd[6] + ck), nXw = ld(ptr.nd[6] + ck - sI), nYn = ld(ptr.nd[11] + ck), nYs = ld(ptr.nd[11] + ck - sJ);
                const double W0 = ld(a.MOMZ0 + ck);
                const R tW = lds(a.MOMZ_t + ck);
                const R Sr_k = below(Sr, C_SR), St_k = below(St, C_ST);
                const int k = L - 1;
                const bool vc = col_ok && lane >= ghosts && (!EDGE || (k >= KS && k <= KE - 1));
                const double *cMZ = sMZ - 1, *cDN = sDN - 1, *cMX = sMX - 1, *cMY = sMY - 1; // level k
                R q_k, dX = R(0.0), dY = R(0.0);
                auto fluxes = [&](auto fast) {
                    constexpr bool FAST = decltype(fast)::value;
                    rn::Guard<R> gd;
                    auto vMZ = [&](int l) { return R(cMZ[l - k]); };
                    // vertical w-momentum flux above level k, fluxZ_XYW (ud3.F90:358-452),
                    // zero outside KS..KE-2; the one below is the previous lane's
                    q_k = R(0.0);
                    if (!EDGE || (k >= KS && k <= KE - 2)) {
                        const R vel = rn::div<FAST>(gd, R(0.5) * (vMZ(k) + vMZ(k + 1)), R(cDN[1]));
                        q_k = J33R * vel * zf(vel, k, vMZ) + nZ;
                    }
                    if (!EDGE || (k >= KS && k <= KE - 1)) {
                        // horizontal w-momentum flux divergence, fluxX/Y_XYW (ud3.F90:598-748)
                        const R f1 = R(f1_k), f2 = R(f2_k);
                        const R vXe = rn::div<FAST>(gd, f1 * R(cMX[1]) + f2 * R(cMX[0]),
                                                    f1 * h * (R(cDN[1]) + R(cDN[1 + KX])) + f2 * h * (R(cDN[0]) + R(cDN[KX])));
                        const R vXw = rn::div<FAST>(gd, f1 * R(cMX[1 - KX]) + f2 * R(cMX[-KX]),
                                                    f1 * h * (R(cDN[1 - KX]) + R(cDN[1])) + f2 * h * (R(cDN[-KX]) + R(cDN[0])));
                        const R vYn = rn::div<FAST>(gd, f1 * R(cMY[1]) + f2 * R(cMY[0]),
                                                    f1 * h * (R(cDN[1]) + R(cDN[1 + KY])) + f2 * h * (R(cDN[0]) + R(cDN[KY])));
                        const R vYs = rn::div<FAST>(gd, f1 * R(cMY[1 - KY]) + f2 * R(cMY[-KY]),
                                                    f1 * h * (R(cDN[1 - KY]) + R(cDN[1])) + f2 * h * (R(cDN[-KY]) + R(cDN[0])));
                        const R W_m2 = R(cMZ[-2 * KX]), W_m1 = R(cMZ[-KX]), W_00 = R(cMZ[0]);
                        const R W_p1 = R(cMZ[KX]), W_p2 = R(cMZ[2 * KX]);
                        const R V_m2 = R(cMZ[-2 * KY]), V_m1 = R(cMZ[-KY]), V_p1 = R(cMZ[KY]), V_p2 = R(cMZ[2 * KY]);
                        const R W_m3 = W6 ? R(cMZ[-3 * KX]) : R(0.0), W_p3 = W6 ? R(cMZ[3 * KX]) : R(0.0);
                        const R V_m3 = W6 ? R(cMZ[-3 * KY]) : R(0.0), V_p3 = W6 ? R(cMZ[3 * KY]) : R(0.0);
                        const R qXe = vXe * ip6<S>(vXe, W_m2, W_m1, W_00, W_p1, W_p2, W_p3) + nXe;
                        const R qXw = vXw * ip6<S>(vXw, W_m3, W_m2, W_m1, W_00, W_p1, W_p2) + nXw;
                        const R qYn = vYn * ip6<S>(vYn, V_m2, V_m1, W_00, V_p1, V_p2, V_p3) + nYn;
                        const R qYs = vYs * ip6<S>(vYs, V_m3, V_m2, V_m1, W_00, V_p1, V_p2) + nYs;
                        dX = qXe - qXw;
                        dY = qYn - qYs;
                    }
                    return gd.bad();
                };
                if (fluxes(std::true_type{})) {
                    cold();
                    fluxes(std::false_type{});
                }
                const R q_km = below(q_k, C_QW);
                if (vc) {
                    const R adv = advection(q_k - q_km, R(rfdz_k), dX, rcdx, dY, rcdy);
                    const R wdmp = -R(wd_k) * R(W0);
                    const R div = use_div ? ddc * (ld(a.DDIV + ck + 1) - ld(a.DDIV + ck)) * R(fdz_k) : R(0.0);
                    const R Sw = adv + wdmp + div + tW;
                    const double rfdz = rfdz_k;
                    const double pg = -(dpc[1] + rtc[1] * dt * (double)St - dpc[0] - rtc[0] * dt * (double)St_k) * rfdz * J33G
                                      - GRAV * (f1_k * (cDN[1] - rd1 + (double)Sr * dt)
                                                + f2_k * (cDN[0] - rd0 + (double)Sr_k * dt));
                    if (!EDGE || L <= KE) a.colC[ck] = cMZ[0] + dt * (pg + (double)Sw);
                }
            }

            // ---- d. rho*u (hevi_momx :814-928) and rho*v (hevi_momy :934-1048) at level L ----
            // u
            {
                const R nZ = lds(ptr.nd[2] + c), nXe = ld(ptr.nd[7] + c + sI), nXw = ld(ptr.nd[7] + c);
                const R nYn = ld(ptr.nd[12] + c), nYs = ld(ptr.nd[12] + c - sJ), tU = lds(a.MOMX_t + c);
                const double U0 = lds(a.MOMX0 + c), aU = rk_sum<M>(ptr, 2, c, sMX[0]);
                const R fdx = R(ld(g.FDX + i - 1));
                const double rfdx = ld(g.RFDX + i - 1);
                const R cor_u = R(0.125) * (R(ld(a.CORIOLI + g.c2 + (i) + (size_t)g.IA * (j - 1)))
                                            + R(ld(a.CORIOLI + g.c2 + (i - 1) + (size_t)g.IA * (j - 1))));
                const double dpe = sdp[dpE]; // DPRES at (i+1, j)
                R q_k, dX, dY;
                auto fluxes = [&](auto fast) {
                    constexpr bool FAST = decltype(fast)::value;
                    rn::Guard<R> gd;
                    auto vMX = [&](int l) { return R(sMX[l - L]); };
                    // the z flux at (u,y,w) above L, fluxZ_UYZ (ud3.F90:753-859)
                    q_k = R(0.0);
                    if (zok) {
                        const R den = R(f1_L) * h * (R(sDN[1]) + R(sDN[1 + KX]))
                                      + R(f2_L) * h * (R(sDN[0]) + R(sDN[KX]));
                        const R vel = rn::div<FAST>(gd, h * (R(sMZ[0]) + R(sMZ[KX])), den);
                        q_k = J33R * vel * zf(vel, L, vMX) + nZ;
                    }
                    const R U_m2 = R(sMX[-2 * KX]), U_m1 = R(sMX[-KX]), U_00 = R(sMX[0]);
                    const R U_p1 = R(sMX[KX]), U_p2 = R(sMX[2 * KX]);
                    // x flux at (x,y,z) with the index shift of fluxX_UYZ (ud3.F90:1053-1109)
                    const R vE = rn::div<FAST>(gd, h * (U_p1 + U_00), R(sDN[KX]));
                    const R vW = rn::div<FAST>(gd, h * (U_00 + U_m1), R(sDN[0]));
                    // y flux at (u,v,z), fluxY_UYZ (ud3.F90:1113-1167)
                    const R vN = rn::div<FAST>(gd, h * (R(sMY[0]) + R(sMY[KX])),
                                               qr * (R(sDN[0]) + R(sDN[KX]) + R(sDN[KY]) + R(sDN[KX + KY])));
                    const R vS = rn::div<FAST>(gd, h * (R(sMY[-KY]) + R(sMY[KX - KY])),
                                               qr * (R(sDN[-KY]) + R(sDN[KX - KY]) + R(sDN[0]) + R(sDN[KX])));
                    const R U_m3 = W6 ? R(sMX[-3 * KX]) : R(0.0), U_p3 = W6 ? R(sMX[3 * KX]) : R(0.0);
                    const R qXe = vE * ip6<S>(vE, U_m2, U_m1, U_00, U_p1, U_p2, U_p3) + nXe;
                    const R qXw = vW * ip6<S>(vW, U_m3, U_m2, U_m1, U_00, U_p1, U_p2) + nXw;
                    const R qYn = vN * ip6<S>(vN, W6 ? R(sMX[-2 * KY]) : R(0.0), R(sMX[-KY]), U_00, R(sMX[KY]),
                                              R(sMX[2 * KY]), W6 ? R(sMX[3 * KY]) : R(0.0)) + nYn;
                    const R qYs = vS * ip6<S>(vS, W6 ? R(sMX[-3 * KY]) : R(0.0), R(sMX[-2 * KY]), R(sMX[-KY]), U_00,
                                              R(sMX[KY]), W6 ? R(sMX[2 * KY]) : R(0.0)) + nYs;
                    dX = qXe - qXw;
                    dY = qYn - qYs;
                    return gd.bad() && vl; // a ghost lane hands its q_k on
                };
                if (fluxes(std::true_type{})) {
                    cold();
                    fluxes(std::false_type{});
                }
                const R q_km = below(q_k, C_QU);
                if (vb && i <= g.IEH) {
                    const R adv = advection(q_k - q_km, R(rcdz_L), dX, R(rfdx), dY, rcdy);
                    const double pg = (dpe - dpc[1]) * rfdx;
                    const R cf = cor_u * (R(sMY[KX]) + R(sMY[0]) + R(sMY[KX - KY]) + R(sMY[-KY]));
                    const R div = !use_div ? R(0.0) : ddc * (ld(a.DDIV + c + sI) - ld(a.DDIV + c)) * fdx;
                    const double val = U0 + dt * (((((double)adv) - pg) + (double)cf) + (double)div + (double)tU);
                    fold_state<M>(a, ptr, N3, 2, a.MOMX_RK, a.MOMX0, c, val, U0, aU);
                }
            }
            // v
            {
                const R nZ = lds(ptr.nd[3] + c), nXe = ld(ptr.nd[8] + c), nXw = ld(ptr.nd[8] + c - sI);
                const R nYn = ld(ptr.nd[13] + c + sJ), nYs = ld(ptr.nd[13] + c), tV = lds(a.MOMY_t + c);
                const double V0 = lds(a.MOMY0 + c), aV = rk_sum<M>(ptr, 3, c, sMY[0]);
                const R fdy = R(ld(g.FDY + j - 1));
                const double rfdy = ld(g.RFDY + j - 1);
                const R cor_v = R(-0.125) * (R(ld(a.CORIOLI + g.c2 + (i - 1) + (size_t)g.IA * (j)))
                                             + R(ld(a.CORIOLI + g.c2 + (i - 1) + (size_t)g.IA * (j - 1))));
                const double dpn = sdp[dpN]; // DPRES at (i, j+1)
                R q_k, dX, dY;
                auto fluxes = [&](auto fast) {
                    constexpr bool FAST = decltype(fast)::value;
                    rn::Guard<R> gd;
                    auto vMY = [&](int l) { return R(sMY[l - L]); };
                    // the z flux at (x,v,w), fluxZ_XVZ (ud3.F90:1173-1279)
                    q_k = R(0.0);
                    if (zok) {
                        const R den = R(f1_L) * h * (R(sDN[1]) + R(sDN[1 + KY]))
                                      + R(f2_L) * h * (R(sDN[0]) + R(sDN[KY]));
                        const R vel = rn::div<FAST>(gd, h * (R(sMZ[0]) + R(sMZ[KY])), den);
                        q_k = J33R * vel * zf(vel, L, vMY) + nZ;
                    }
                    const R Y_m2 = R(sMY[-2 * KY]), Y_m1 = R(sMY[-KY]), Y_00 = R(sMY[0]);
                    const R Y_p1 = R(sMY[KY]), Y_p2 = R(sMY[2 * KY]);
                    // x flux at (u,v,z), fluxX_XVZ (ud3.F90:1473-1527)
                    const R vE = rn::div<FAST>(gd, h * (R(sMX[0]) + R(sMX[KY])),
                                               qr * (R(sDN[0]) + R(sDN[KX]) + R(sDN[KY]) + R(sDN[KX + KY])));
                    const R vW = rn::div<FAST>(gd, h * (R(sMX[-KX]) + R(sMX[KY - KX])),
                                               qr * (R(sDN[-KX]) + R(sDN[0]) + R(sDN[KY - KX]) + R(sDN[KY])));
                    // y flux with the index shift of fluxY_XVZ (ud3.F90:1531-1587)
                    const R vN = rn::div<FAST>(gd, h * (Y_p1 + Y_00), R(sDN[KY]));
                    const R vS = rn::div<FAST>(gd, h * (Y_00 + Y_m1), R(sDN[0]));
                    const R qXe = vE * ip6<S>(vE, W6 ? R(sMY[-2 * KX]) : R(0.0), R(sMY[-KX]), Y_00, R(sMY[KX]),
                                              R(sMY[2 * KX]), W6 ? R(sMY[3 * KX]) : R(0.0)) + nXe;
                    const R qXw = vW * ip6<S>(vW, W6 ? R(sMY[-3 * KX]) : R(0.0), R(sMY[-2 * KX]), R(sMY[-KX]), Y_00,
                                              R(sMY[KX]), W6 ? R(sMY[2 * KX]) : R(0.0)) + nXw;
                    const R Y_m3 = W6 ? R(sMY[-3 * KY]) : R(0.0), Y_p3 = W6 ? R(sMY[3 * KY]) : R(0.0);
                    const R qYn = vN * ip6<S>(vN, Y_m2, Y_m1, Y_00, Y_p1, Y_p2, Y_p3) + nYn;
                    const R qYs = vS * ip6<S>(vS, Y_m3, Y_m2, Y_m1, Y_00, Y_p1, Y_p2) + nYs;
                    dX = qXe - qXw;
                    dY = qYn - qYs;
                    return gd.bad() && vl; // a ghost lane hands its q_k on
                };
                if (fluxes(std::true_type{})) {
                    cold();
                    fluxes(std::false_type{});
                }
                const R q_km = below(q_k, C_QV);
                if (vb && j <= g.JEH) {
                    const R adv = advection(q_k - q_km, R(rcdz_L), dX, rcdx, dY, R(rfdy));
                    const double pg = (dpn - dpc[1]) * rfdy;
                    const R cf = cor_v * (R(sMX[KY]) + R(sMX[0]) + R(sMX[KY - KX]) + R(sMX[-KX]));
                    const R div = !use_div ? R(0.0) : ddc * (ld(a.DDIV + c + sJ) - ld(a.DDIV + c)) * fdy;
                    const double val = V0 + dt * (((((double)adv) - pg) + (double)cf) + (double)div + (double)tV);
                    fold_state<M>(a, ptr, N3, 3, a.MOMY_RK, a.MOMY0, c, val, V0, aV);
                }
            }
        };
        if (interior) chunk(std::false_type{});
        else chunk(std::true_type{});
#undef rcdx
#undef rcdy
#undef rcdz_L
#undef rfdz_k
#undef f1_L
#undef f1_k
#undef f2_L
#undef f2_k
#undef fdz_k
#undef wd_k
        __syncthreads(); // every read of the staged box and of DPRES is done
        if (ch + 1 < ch1) issue(ch + 1);
    }
}

// =============================================================================
// k_hevi_column: the column problem of CCOLS columns per CTA
// =============================================================================
// The CTA copies C, PT and RT2P of its columns into shared memory with
// cp.async, every copy in flight at once, and forms the per-level factors of the
// coefficients once for all columns. One warp runs the Thomas solve
// (solve_direct :1092-1127) one lane per column: the operands of level k+2 are
// read and the coefficients of level k+1 formed while the reciprocal of level k
// runs, so that only e(k-1) and f(k-1) chain the levels. The other warps meanwhile load the operands of their first
// part of the back-update of rho, rho*w, rho*theta and the vertical fluxes
// (:728-790), which all warps then run, a column's 32 levels at a time.
//
// The solve's serial chain and the update's 13 to 18 streams bound it in turn: of
// about 115 thousand cycles of a CTA at 128 levels the solve took 57 and the update 45
// (a level 400 cycles, most of it waiting for its operands' shared-memory reads).
// 512x512x128, CD4, FP64: 2.00 -> 1.52 ms per launch, the mean of a step's four, with the
// operands read ahead and the combine's state sums formed from the stage buffers
// instead of accumulated.
constexpr int CCOLS = 16;  // columns per CTA (consecutive in i)
constexpr int CWARPS = 8;
__host__ __device__ inline int col_pitch_c(int KA) { return KA | 1; }
__host__ __device__ inline size_t column_smem(int KA) { return ((size_t)3 * CCOLS * col_pitch_c(KA) + 3 * (size_t)KA) * sizeof(double); }

template <typename R, int M, int NM>
__global__ void __launch_bounds__(32 * CWARPS, 4)
    k_hevi_column(const Grid gt, const StageArgsT<R> a, const BatchT<NM> B, const __grid_constant__ StagePtrs<R> ptr)
{
    constexpr bool ACC = fold_reads(M);
    extern __shared__ double csm[];
    __shared__ int s_solver;
    int b;
    const Grid g = block_domain(gt, B, b);
    const int nbx = (g.IMAX + CCOLS - 1) / CCOLS;
    const int i0 = g.IS + (b % nbx) * CCOLS, j = g.JS + b / nbx;
    const int ncol = min(CCOLS, g.IE - i0 + 1);
    const int lane = threadIdx.x, w = threadIdx.y;
    const size_t N3 = n3(g);
    const int KS = g.KS, KE = g.KE, KP = col_pitch_c(g.KA), NP = (g.KMAX + 31) / 32;
    const double dt = a.dtrk, J33G = a.J33G, dt2 = dt * dt;
    const int col0 = (int)idx3(g, 1, i0, j);
    // per-level arrays of the tile's columns: [array][column][level], odd pitch;
    // then dt^2 J33G RCDZ, B and RFDZ by level
    double *sC = csm, *sA = csm + (size_t)CCOLS * KP;
    R *sP = reinterpret_cast<R *>(csm + (size_t)2 * CCOLS * KP);
    double *sD = csm + (size_t)3 * CCOLS * KP, *sB = sD + g.KA, *sR = sB + g.KA;
#define CA(arr, cc, L) arr[(cc) * KP + (L) - 1]

    // ---- C, PT and RT2P of the columns; the level factors of A(k) (:696), B(k) (:697), RFDZ(k) ----
    for (int cc = w; cc < ncol; cc += CWARPS) {
        const int col = col0 + cc * g.KA;
        for (int L = KS + lane; L <= KE; L += 32) {
            const int c = col + L - 1;
            if (L <= KE - 1) {
                copy_async(&CA(sC, cc, L), (const double *)a.colC + c);
                copy_async(&CA(sP, cc, L), (const R *)ptr.PT + c);
            }
            copy_async(&CA(sA, cc, L), a.RT2P + c);
        }
    }
    for (int k = KS + w * 32 + lane; k <= KE; k += 32 * CWARPS) {
        sD[k - 1] = dt2 * J33G * ld(g.RCDZ + k - 1);
        if (k <= KE - 1) {
            sB[k - 1] = GRAV * dt2 * J33G / (ld(g.CDZ + k) + ld(g.CDZ + k - 1));
            sR[k - 1] = ld(g.RFDZ + k - 1);
        }
    }

    // operands of the back-update of one column's 32 levels
    struct Ops {
        double D0, T0, W0, W, aD, aT, aW;
        R Sr, St, tZ, nDZ, aM, aQ;
    };
    auto load_ops = [&](int item, Ops &o) {
        const int m = min(KS + (item / CCOLS) * 32 + lane, KE), cc = min(item % CCOLS, ncol - 1);
        const int c = col0 + cc * g.KA + m - 1;
        o.Sr = __ldcg(ptr.Sr + c); o.St = __ldcg(ptr.St + c); o.tZ = __ldcg(ptr.tZ + c);
        o.nDZ = ld(ptr.nd[0] + c);
        o.D0 = lds(a.DENS0 + c); o.T0 = lds(a.RHOT0 + c); o.W0 = ld(a.MOMZ0 + c); o.W = ld(a.MOMZ + c);
        if constexpr (M == RK_FINAL) {
            o.aD = rk_sum<M>(ptr, 0, c, ld(a.DENS + c));
            o.aT = rk_sum<M>(ptr, 4, c, ld(a.RHOT + c));
            o.aW = rk_sum<M>(ptr, 1, c, o.W);
        }
        if constexpr (ACC) {
            o.aM = lds(ptr.facc[0] + c); o.aQ = lds(ptr.facc[3] + c);
        }
    };
    // The solver warp differs between the CTAs of an SM, so that the solves spread over
    // its four schedulers and their FP64 lanes: a CTA has a multiple of four warps, so
    // warp 0 everywhere would put them all on one.
    if (threadIdx.x == 0 && w == 0) {
        unsigned slot;
        asm volatile("mov.u32 %0, %%warpid;" : "=r"(slot));
        s_solver = (int)(slot / CWARPS) % CWARPS;
    }
    copy_wait();
    __syncthreads();

    // ---- Thomas solve, one lane per column (F1..F3 of :699-709) ----
    auto solve = [&](auto fast) -> bool {
        constexpr bool FAST = decltype(fast)::value;
        const int cc = lane;
        bool bad = false;
        auto inverse = [&](double x) -> double {
            if constexpr (FAST) {
                // a divisor outside (2^-1000, 2^1000): the solve runs again with `/`
                bad |= (unsigned)__double2hiint(x) - 0x01700000u >= 0x7d000000u;
                return rn::rcp(x);
            } else {
                return 1.0 / x;
            }
        };
        // what level k adds to the operands: PT and the factors of A(k) = dt^2 J33G^2 RCDZ RT2P
        // (:696) one level up, C, RFDZ and B; read a level before they are used
        struct Level { double P, D, T, C, R, B; };
        auto level = [&](int k) {
            const int kp = min(k + 1, KE), kq = min(k + 1, KE - 1), kc = min(k, KE - 1);
            return Level{(double)CA(sP, cc, kq), sD[kp - 1], CA(sA, cc, kp), CA(sC, cc, kc), sR[kc - 1], sB[kc - 1]};
        };
        double Pm = 0.0, P0 = (double)CA(sP, cc, KS), A0 = sD[KS - 1] * CA(sA, cc, KS) * J33G; // PT(k-1), PT(k), A(k)
        double F1, F2, F3, Ck;
        // F1, F2, F3 and C of the level x belongs to (F1 is not used at KE-1, F3 not at KS)
        auto coef = [&](const Level &x) {
            const double A1 = x.D * x.T * J33G;
            F2 = 1.0 + (P0 * x.R * (A1 + A0));
            F1 = -(x.P * x.R * A1 + x.B);
            F3 = -(Pm * x.R * A0 - x.B);
            Ck = x.C;
            Pm = P0;
            P0 = x.P;
            A0 = A1;
        };
        Level x = level(KS), y = level(KS + 1);
        coef(x);
        double r = inverse(F2), e = -F1 * r, f = Ck * r;
        x = level(KS + 2);
        CA(sA, cc, KS) = e;
        CA(sC, cc, KS) = f;
        coef(y);
        // levels KS+1..KE-2: one straight block per level, in which the next level's
        // coefficients fill the latency of this level's reciprocal, so that only e and
        // f chain the levels
#pragma unroll 1
        for (int k = KS + 1; k <= KE - 2; ++k) {
            const double G1 = F1, G3 = F3, Gk = Ck, den = F2 + F3 * e;
            y = level(k + 2); // reads RT2P(k+3) and C(k+2): not yet overwritten
            r = inverse(den);
            coef(x);
            e = -G1 * r;
            f = (Gk - G3 * f) * r;
            CA(sA, cc, k) = e;
            CA(sC, cc, k) = f;
            x = y;
        }
        f = (Ck - F3 * f) / (F2 + F3 * e); // the solution at KE-1
        CA(sC, cc, KE - 1) = f;
        // back substitution, C(k) = e(k) C(k+1) + f(k)
#pragma unroll 4
        for (int k = KE - 2; k >= KS; --k) {
            f = CA(sA, cc, k) * f + CA(sC, cc, k);
            CA(sC, cc, k) = f;
        }
        return bad;
    };
    // the solver warp and the others meet at a barrier of their own: the others
    // arrive with the operands of their first item on the way
    auto meet = [] { asm volatile("bar.sync 1, %0;" ::"n"(32 * CWARPS) : "memory"); };
    Ops o;
    if (w == s_solver) {
        if (lane < ncol && solve(std::true_type{})) {
            const int col = col0 + lane * g.KA;
            for (int L = KS; L <= KE; ++L) { // the solve wrote over its operands
                if (L <= KE - 1) CA(sC, lane, L) = a.colC[col + L - 1];
                CA(sA, lane, L) = a.RT2P[col + L - 1];
            }
            solve(std::false_type{});
        }
        __syncwarp();
        meet();
        load_ops(w, o);
    } else {
        load_ops(w, o);
        meet();
    }

    // ---- back-update (:728-790) ----
    for (int item = w; item < CCOLS * NP; item += CWARPS) {
        if (item != w) load_ops(item, o);
        const int cc = item % CCOLS, i = i0 + cc;
        const int m = KS + (item / CCOLS) * 32 + lane;
        const int c = col0 + cc * g.KA + m - 1;
        if (cc >= ncol) continue;
        if (m <= KE) {
            const double rcdz = ld(g.RCDZ + m - 1);
            const double Cm = m <= KE - 1 ? CA(sC, cc, m) : 0.0, Cm1 = m >= KS + 1 ? CA(sC, cc, m - 1) : 0.0;
            const double Pm = m <= KE - 1 ? (double)CA(sP, cc, m) : 0.0, Pm1 = m >= KS + 1 ? (double)CA(sP, cc, m - 1) : 0.0;
            double adr, adt;
            if (m == KE) {
                adr = Cm1 * J33G * rcdz;
                adt = Cm1 * Pm1 * J33G * rcdz;
            } else if (m == KS) {
                adr = -Cm * J33G * rcdz;
                adt = -Cm * Pm * J33G * rcdz;
            } else {
                adr = -(Cm - Cm1) * J33G * rcdz;
                adt = -(Cm * Pm - Cm1 * Pm1) * J33G * rcdz;
            }
            fold_state<M>(a, ptr, N3, 0, a.DENS_RK, a.DENS0, c, o.D0 + dt * (adr + (double)o.Sr), o.D0, o.aD);
            fold_state<M>(a, ptr, N3, 4, a.RHOT_RK, a.RHOT0, c, o.T0 + dt * (adt + (double)o.St), o.T0, o.aT);
            if (m <= KE - 1) {
                fold_state<M>(a, ptr, N3, 1, a.MOMZ_RK, a.MOMZ0, c, o.W0 + (Cm - o.W), o.W0, o.aW);
                fold_flux<M>(a, ptr, N3, 0, c, R((double)o.nDZ + J33G * Cm), o.aM);
                fold_flux<M>(a, ptr, N3, 3, c, R((double)o.tZ + J33G * Cm * Pm), o.aQ);
            } else {
                put_state(a, N3, 1, a.MOMZ_RK, a.MOMZ0, c, 0.0, false);
                fold_flux<M>(a, ptr, N3, 0, c, R(0.0), o.aM);
                fold_flux<M>(a, ptr, N3, 3, c, R(0.0), o.aQ);
            }
        }
        if (m == KS) {
            // rigid-lid and surface values (:753-754) and the zero fluxes at KS-1 (:371, ud3.F90:222)
            put_state(a, N3, 1, a.MOMZ_RK, a.MOMZ0, c - 1, 0.0, false);
            put_flux(a, N3, 0, c - 1, R(0.0), false);
            put_flux(a, N3, 3, c - 1, R(0.0), false);
        }
        // hevi_mflx_z :369-393 also fills the halo column i = IS-1 with the explicit
        // part of the vertical mass flux; the solver never updates it
        if (i == g.IS && item < CCOLS && (a.rk_mode == RK_PLAIN || a.rk_mode == RK_FINAL || a.rk_mode == RK_HEUN3)) {
            const size_t chl = idx3(g, 1, g.IS - 1, j);
            for (int k = KS - 1 + lane; k <= KE; k += 32)
                a.mflx[chl + k - 1] = (k >= KS && k <= KE - 1) ? ld(ptr.nd[0] + chl + k - 1) : R(0.0);
        }
    }
#undef CA
}

// =============================================================================
// host side
// =============================================================================
inline long long tiles(const Grid &m) { return (long long)((m.IMAX + TX - 1) / TX) * ((m.JMAX + TY - 1) / TY); }

// Whether the explicit kernel splits the march: where that shortens the time of the
// last CTA, counted in chunks, with 148 SMs of `per_sm` CTAs. A CTA that marches takes
// its chunks one after another, so a domain of few tiles leaves most of the chip idle
// (40x40x80: 100 CTAs of 3 chunks against 300 of one), and one of a few waves ends in a
// nearly empty one; the split takes more chunks in deep columns, for the ghost levels.
// Marching against split: 40x40x80, UD3 (3 chunk times against 2), 40 and 31 us per launch,
// a short step 290 and 256 us; 253x187x57, UD3 (22 against 21), a step 2773 and 2700 us;
// 512x512x128, CD4 (224 against 277), 25.9 and 26.8 ms; a stage at 200x136x64, UD5
// (24 against 35), 360 and 476 us. FP64 only: the split moves levels between the code
// with and without wall forms, whose FP32 sums the compiler may fuse differently.
inline bool split_march(const Grid &g, const Members &mem, int per_sm)
{
    long long whole = 0, parts = 0, longest = 0;
    for (int q = 0; q < (mem.n > 1 ? mem.n : 1); ++q) {
        const Grid m = mem.n > 1 ? member_grid(g, mem.m[q]) : g;
        whole += tiles(m) * chunks(m.KMAX, false);
        parts += tiles(m) * chunks(m.KMAX, true);
        longest = chunks(m.KMAX, false) > longest ? chunks(m.KMAX, false) : longest;
    }
    const long long slots = 148LL * per_sm;
    const long long marched = (whole + longest * slots - 1) / (longest * slots) * longest;
    return (parts + slots - 1) / slots < marched;
}

// the two kernels over the blocks of every member
template <int S, int M, int LD, int NM, typename R>
cudaError_t launch_pair(const Grid &g, const Members &mem, const StageArgsT<R> &a, const StageMaps<R> &h, cudaStream_t st)
{
    BatchT<NM> B{};
    B.n = mem.n > 1 ? mem.n : 1;
    int maxKA = g.KA;
    for (int q = 0; q < B.n && mem.n > 0; ++q) {
        B.m[q] = mem.m[q];
        maxKA = mem.m[q].KMAX + 4 > maxKA ? mem.m[q].KMAX + 4 : maxKA;
    }
    // first block of each member; false where they do not fit an int
    auto ranges = [&](auto blocks_of) {
        long long n = 0;
        for (int q = 0; q < B.n; ++q) {
            B.first[q] = (int)n;
            n += blocks_of(mem.n > 1 ? member_grid(g, mem.m[q]) : g);
        }
        B.first[B.n] = (int)n;
        return n > 0 && n < (1LL << 31);
    };
    auto kx = k_hevi_explicit<S, R, M, LD, NM>;
    cudaError_t e = open_smem(kx, smem_bytes<S>());
    if (e != cudaSuccess) return e;
    const bool split = sizeof(R) == 8 && split_march(g, mem, wide_scheme(S) ? 1 : 2);
    if (!ranges([&](const Grid &m) { return tiles(m) * (split ? chunks(m.KMAX, true) : 1); })) return cudaErrorInvalidValue;
    kx<<<B.first[B.n], dim3(32, NCOL), smem_bytes<S>(), st>>>(g, a, B, h.ptr, split, h.maps);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    auto kc = k_hevi_column<R, M, NM>;
    // the attribute is set once per device, so it opens the largest size (KA = 260)
    if ((e = open_smem(kc, column_smem(260))) != cudaSuccess) return e;
    if (!ranges([](const Grid &m) { return ((m.IMAX + CCOLS - 1) / CCOLS) * m.JMAX; })) return cudaErrorInvalidValue;
    kc<<<B.first[B.n], dim3(32, CWARPS), column_smem(maxKA), st>>>(g, a, B, h.ptr);
    return cudaGetLastError();
}

template <int S, int LD, int NM, typename R>
cudaError_t launch_s(const Grid &g, const Members &mem, StageArgsT<R> a, int raster, cudaStream_t st)
{
    StageMaps<R> h{};
    const double *f[NF] = {a.DENS, a.MOMZ, a.MOMX, a.MOMY, a.RHOT};
    const size_t N3 = n3(g);
    for (int q = 0; q < NF; ++q) {
        if (LD == LD_TMA && !encode(&h.maps.m[q], f[q], g, box_k<S>(), box_w<S>(), box_h<S>())) return cudaErrorNotSupported;
        h.ptr.in[q] = f[q];
        h.ptr.rk1[q] = a.rk1 + q * N3;
        h.ptr.rk2[q] = a.rk2 + q * N3;
    }
    for (int q = 0; q < 15; ++q) h.ptr.nd[q] = a.num_diff + q * N3;
    for (int q = 0; q < 6; ++q) {
        h.ptr.facc[q] = a.facc + q * N3;
        h.ptr.flx[q] = (q < 3 ? a.mflx : a.tflx) + (q % 3) * N3;
    }
    h.ptr.Sr = a.colscr; h.ptr.St = a.colscr + N3; h.ptr.tZ = a.colscr + 2 * N3; h.ptr.PT = a.colscr + 3 * N3;
    a.raster = raster > 0 ? raster : STAGE_RASTER_DEFAULT;
    switch (a.rk_mode) {
    case RK_PLAIN: return launch_pair<S, RK_PLAIN, LD, NM>(g, mem, a, h, st);
    case RK_STAGE1: return launch_pair<S, RK_STAGE1, LD, NM>(g, mem, a, h, st);
    case RK_STAGE2:
    case RK_STAGE3: return launch_pair<S, RK_STAGE2, LD, NM>(g, mem, a, h, st);
    case RK_FINAL: return launch_pair<S, RK_FINAL, LD, NM>(g, mem, a, h, st);
    default: return launch_pair<S, FOLD_ANY, LD, NM>(g, mem, a, h, st);
    }
}

template <int LD, int NM, typename R>
cudaError_t launch_scheme(const Grid &g, const Members &mem, const StageArgsT<R> &a, int scheme, int raster, cudaStream_t st)
{
    switch (scheme) {
    case UD3: return launch_s<UD3, LD, NM, R>(g, mem, a, raster, st);
    case CD4: return launch_s<CD4, LD, NM, R>(g, mem, a, raster, st);
    case KOREN: return launch_s<KOREN, LD, NM, R>(g, mem, a, raster, st);
    case CD2: return launch_s<CD2, LD, NM, R>(g, mem, a, raster, st);
    case UD5: return launch_s<UD5, LD, NM, R>(g, mem, a, raster, st);
    case CD6: return launch_s<CD6, LD, NM, R>(g, mem, a, raster, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace tma

#ifndef HEVI_COPY_TU
// The tiled stage where it applies: one domain or, in FP64, an ensemble, KA <= 260 and
// the column scratch of the tiled kernels present. cudaErrorNotSupported otherwise
// (the caller then runs the fused kernel). One domain of even KA whose fields lie on
// 16-byte boundaries stages them by bulk tensor copies, everything else with
// cp.async. Before, ensembles and odd KA ran the fused kernel: 253x187x57, UD3,
// FP64, a short step 3.58 ms; 24 members of 32x32x64 to 128x128x96, UD3, 19.5 ms;
// with it 2.81 ms and 15.9 ms.
template <typename R>
cudaError_t launch_hevi_stage_tiled(const Grid &g, const Members &mem, const StageArgsT<R> &a, int scheme, int raster,
                                    cudaStream_t st)
{
    if (g.KA > 260 || !a.colC || (mem.n > 1 && sizeof(R) != sizeof(double))) return cudaErrorNotSupported;
    if (mem.n <= 1 && (g.KA & 1) == 0) { // 16-byte strides for the tensor maps
        const cudaError_t e = tma::launch_scheme<tma::LD_TMA, 1, R>(g, mem, a, scheme, raster, st);
        if (e != cudaErrorNotSupported) return e;
    }
    return mem.n > 0 ? launch_hevi_stage_copied(g, mem, a, scheme, raster, st) : cudaErrorNotSupported;
}
#ifndef HEVI_FLOAT_TU
template cudaError_t launch_hevi_stage_tiled<double>(const Grid &, const Members &, const StageArgsT<double> &, int,
                                                     int, cudaStream_t);
#else
template cudaError_t launch_hevi_stage_tiled<float>(const Grid &, const Members &, const StageArgsT<float> &, int, int,
                                                    cudaStream_t);
#endif
#else // HEVI_COPY_TU: the instantiations without tensor maps, in their own translation unit
template <typename R>
cudaError_t launch_hevi_stage_copied(const Grid &g, const Members &mem, const StageArgsT<R> &a, int scheme, int raster,
                                     cudaStream_t st)
{
    return tma::launch_scheme<tma::LD_COPY, HEVI_MAX_MEMBERS, R>(g, mem, a, scheme, raster, st);
}
#ifndef HEVI_FLOAT_TU
template cudaError_t launch_hevi_stage_copied<double>(const Grid &, const Members &, const StageArgsT<double> &, int,
                                                      int, cudaStream_t);
#else
template cudaError_t launch_hevi_stage_copied<float>(const Grid &, const Members &, const StageArgsT<float> &, int, int,
                                                     cudaStream_t);
#endif
#endif

}  // namespace hevi
