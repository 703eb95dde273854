// The 15 num_diff components (ATMOS_DYN_numfilter_coef, scale_atmos_dyn_common.F90:
// 385-985, ND_ORDER = 1, with the third differences of calc_diff3 :1600-1760) of a
// 4 x 4 tile of columns from shared memory, after k_phi has formed the five
// filtered quantities. One warp per column, lanes along k, chunks of 32 levels.
// Per chunk the quantities and DENS come into shared memory over the tile, a
// lateral halo of 2 and the levels L0-2..L0+33 (six bulk tensor copies completing on
// an mbarrier with a bounded wait, or cp.async where the arrays admit no tensor map
// and for ensembles). The vertical halo levels of each column follow with global
// loads.
//
// The arithmetic of every component is that of numfilter_cell, operation for
// operation, and gives identical bits; the near-wall rows of the z differences are
// the interior formula with mirrored operands (and, at KE, the negated row KE-1), so
// that no lane takes a branch of its own. A direction's coefficients are read once for
// its five components: read at every component, as numfilter_cell does, they
// were 60 loads per cell, and the kernel waited for them. 512x512x128, FP64: a short
// step 26.77 -> 26.19 ms; odd KA and ensembles took the column kernel before.
#include "numfilter_body.cuh"
#include "tma_util.cuh"

namespace hevi {
namespace tma {

constexpr int NTX = 4, NTY = 4, NWARPS = NTX * NTY; // tile columns; one warp each
constexpr int NKC = 32;                             // levels per chunk
constexpr int NKLO = 2;                             // box levels below the chunk's first
constexpr int NBK = NKC + 4;                        // box levels: L0-2 .. L0+33
constexpr int NBW = NTX + 4, NBH = NTY + 4;         // lateral halo of 2
constexpr int NPL = NBK * NBW * NBH;                // one staged field
template <typename R> constexpr size_t nd_smem_bytes() { return (size_t)NPL * (5 * sizeof(R) + sizeof(double)) + 16; }

struct NdMaps {
    CUtensorMap m[6]; // phi q = 0..4 (type R), DENS (FP64), as (KA, IA, JA) tensors
};
template <typename R>
struct NdPtrs {
    R *nd[15];        // components q + 5*dir
    const R *phi[5];
};

template <typename R, int LD, int NM>
__global__ void __launch_bounds__(32 * NWARPS, 2)
    k_numfilter_tiled(const Grid gt, const NdCoef ct, const NdArgsT<R> a, const BatchT<NM> B,
                      const __grid_constant__ NdPtrs<R> ptr, unsigned *status, const __grid_constant__ NdMaps maps)
{
    extern __shared__ __align__(1024) double sm[];
    R *sphi = reinterpret_cast<R *>(sm); // 5 fields, [j][i][k] each
    double *sdn = reinterpret_cast<double *>(reinterpret_cast<char *>(sm) + (size_t)5 * NPL * sizeof(R));
    uint64_t *bar = reinterpret_cast<uint64_t *>(sdn + NPL);
    __shared__ int s_ok;
    __shared__ R s_x[NTX][10], s_y[NTY][10]; // coefficients of the tile's columns and rows
    int b;
    const Grid g = block_domain(gt, B, b);
    const NdCoef c = NM == 1 ? ct : member_nd(ct, g);
    const int lane = threadIdx.x, w = threadIdx.y, tid = w * 32 + lane;
    const int tx = w % NTX, ty = w / NTX;
    const int nti = (g.IMAX + NTX - 1) / NTX;
    const int i0 = g.IS + (b % nti) * NTX, j0 = g.JS + (b / nti) * NTY;
    const int i = i0 + tx, j = j0 + ty;
    const bool col_ok = i <= g.IE && j <= g.JE;
    const size_t N3 = n3(g);
    const int KS = g.KS, KE = g.KE;
    const int NC = (g.KMAX + NKC - 1) / NKC;

    auto issue = [&](int ch) {
        const int l0 = KS + NKC * ch - NKLO; // the level of box element 0
        if constexpr (LD == LD_TMA) {
            if (tid != 0) return;
            // box origin (0-based): level L0-2 = 32*ch (KS = 3), column i0-2, row j0-2
            const int x = l0 - 1, y = i0 - 2 - 1, z = j0 - 2 - 1;
            fence_proxy_async();
            mbar_expect_tx(bar, (unsigned)(NPL * (5 * sizeof(R) + sizeof(double))));
            for (int q = 0; q < 5; ++q) tma_load_3d(sphi + (size_t)q * NPL, &maps.m[q], x, y, z, bar);
            tma_load_3d(sdn, &maps.m[5], x, y, z, bar);
        } else {
            constexpr int TAIL = NBK - 32;
            static_assert(6 * TAIL <= 32, "one pass for the tail levels");
            for (int q = w; q < NBW * NBH; q += NWARPS) {
                const int ii = i0 - 2 + q % NBW, jj = j0 - 2 + q / NBW;
                if (ii > g.IA || jj > g.JA) continue; // the box of the last tiles reaches beyond the array
                const int at = (int)idx3(g, 1, ii, jj) + l0 - 1, to = q * NBK;
                if (l0 + lane <= g.KA) {
#pragma unroll
                    for (int f = 0; f < 5; ++f) copy_async(sphi + f * NPL + to + lane, ptr.phi[f] + at + lane);
                    copy_async(sdn + to + lane, a.DENS + at + lane);
                }
                const int f = lane / TAIL, lv = 32 + lane % TAIL;
                if (l0 + lv <= g.KA) {
                    if (f < 5) copy_async(sphi + f * NPL + to + lv, ptr.phi[f] + at + lv);
                    else if (f == 5) copy_async(sdn + to + lv, a.DENS + at + lv);
                }
            }
        }
    };
    if (tid == 0) {
        s_ok = 1;
        if constexpr (LD == LD_TMA) {
            mbar_init(bar, 1);
            fence_mbar_init();
        }
    }
    issue(0);
    // x and y coefficients: the four of the differences at a face (the density, w, theta and
    // the other horizontal momentum), the four of its own momentum, and the two filter factors
    for (int e = tid; e < 10 * (NTX + NTY); e += 32 * NWARPS) {
        const bool isx = e < 10 * NTX;
        const int n = e % 10, q = (isx ? e : e - 10 * NTX) / 10;
        const int p = isx ? min(i0 + q, g.IE) : min(j0 + q, g.JE), PA = isx ? g.IA : g.JA;
        const double *C3 = isx ? c.CNX3 : c.CNY3;
        auto c3 = [&](int m, int at, int s) { return ld(C3 + (m - 1) + 3 * ((size_t)(at - 1) + (size_t)PA * (s - 1))); };
        double v;
        switch (n) {
        case 0: v = c3(1, p + 1, 1); break;
        case 1: v = c3(2, p + 1, 1); break;
        case 2: v = c3(3, p + 1, 1); break;
        case 3: v = c3(1, p, 1); break;
        case 4: v = c3(1, p, 2); break;
        case 5: v = c3(2, p, 2); break;
        case 6: v = c3(3, p, 2); break;
        case 7: v = c3(1, p - 1, 2); break;
        case 8: v = ld((isx ? c.cdx : c.cdy) + p - 1); break;
        default: v = ld((isx ? c.fdx : c.fdy) + p - 1);
        }
        (isx ? s_x[q] : s_y[q])[n] = R(v);
    }
    __syncthreads();

    const R sfc = R(c.sfc), qr = R(0.25), h = R(0.5);
    constexpr int KX = NBK, KY = NBK * NBW;
    for (int ch = 0; ch < NC; ++ch) {
        const int L0 = KS + NKC * ch, k = min(L0 + lane, KE); // lanes above KE run along on KE
        const bool valid = col_ok && L0 + lane <= KE;
        // z coefficients: of the row m that the level's difference is formed at (KE takes the
        // negated row KE-1), and of w
        const int m = min(k, KE - 1);
        const R z1 = CZ3(1, m + 1, 1), z2 = CZ3(2, m + 1, 1), z3 = CZ3(3, m + 1, 1), z4 = CZ3(1, m, 1);
        const R w1 = CZ3(1, k, 2), w2 = CZ3(2, k, 2), w3 = CZ3(3, k, 2), w4 = CZ3(1, k - 1, 2);
        const R ncz = R(ld(c.cdz + k - 1)), nfz = R(ld(c.fdz + k - 1));
        if constexpr (LD == LD_TMA) {
            if (!mbar_wait(bar, ch & 1)) { // bounded; the block leaves after the chunk
                s_ok = 0;
                (void)mbar_wait(bar, ch & 1); // bounded: the copies still in flight
            }
        } else {
            copy_wait();
            __syncthreads();
        }
        const int at = ((ty + 2) * NBW + (tx + 2)) * NBK + (k - (L0 - NKLO));
        const R *const P = sphi + at;
        const double *const D = sdn + at;
        const size_t o = idx3(g, k, min(i, g.IE), min(j, g.JE));
        const bool kz = k <= KE - 1, top = k == KE;
        // surface-factor tail of every x/y component (:581-585 and the analogous blocks)
        auto sfct = [&](R v) {
            if (k == KS) return v * sfc;
            if (k == KS + 1) return v * (R(1.0) + sfc) * h;
            return v;
        };
        auto put = [&](int q, R v) {
            if (valid) ptr.nd[q][o] = v;
        };
        const R d000 = R(D[0]), d100 = R(D[1]), d010 = R(D[KX]), d001 = R(D[KY]);
        const R d110 = R(D[1 + KX]), d101 = R(D[1 + KY]), d011 = R(D[KX + KY]);
        const R sxz = d110 + d100 + d010 + d000, syz = d101 + d100 + d001 + d000;
        {
            // z: phi(KS-1) mirrors phi(KS+1), phi(KE+1) mirrors phi(KE-1)
            const int p0 = m - k, p1 = p0 + 1, p2 = m == KE - 1 ? p0 : p0 + 2, pm = m == KS ? p1 : p0 - 1;
            auto dz = [&](int q) {
                const R *F = P + q * NPL;
                const R v = (+z1 * F[p2] - z2 * F[p1] + z3 * F[p0] - z4 * F[pm]);
                return top ? -v : v;
            };
            put(0, dz(0) * ncz);
            put(2, kz ? dz(2) * ncz * qr * sxz : R(0.0));
            put(3, kz ? dz(3) * ncz * qr * syz : R(0.0));
            const R v = dz(4) * ncz;
            put(4, kz ? v * h * (d100 + d000) : v * d000);
            // w on KS+1..KE-1: phi(KS-1) mirrors phi(KS+1), phi(KE) is zero
            const R *F = P + NPL;
            const R up = k >= KE - 1 ? R(0.0) : F[1];
            const R t = (+w1 * up - w2 * F[0] + w3 * F[-1] - w4 * F[k <= KS + 1 ? 0 : -2]);
            put(1, k >= KS + 1 && kz ? t * nfz * d000 : R(0.0));
        }
        // a horizontal difference of quantity q along a stride; own: the momentum along it
        auto dh = [&](const R (&C)[10], int q, int s, bool own) {
            const R *F = P + q * NPL;
            if (own) return (+C[4] * F[s] - C[5] * F[0] + C[6] * F[-s] - C[7] * F[-2 * s]);
            return (+C[0] * F[2 * s] - C[1] * F[s] + C[2] * F[0] - C[3] * F[-s]);
        };
        {
            const R (&X)[10] = s_x[tx];
            const R nc = X[8], nf = X[9];
            put(5, sfct(dh(X, 0, KX, false) * nc));
            put(6, kz ? sfct(dh(X, 1, KX, false) * nc * qr * sxz) : R(0.0));
            put(7, sfct(dh(X, 2, KX, true) * nf * d000));
            put(8, sfct(dh(X, 3, KX, false) * nc * qr * (d011 + d001 + d010 + d000)));
            put(9, sfct(dh(X, 4, KX, false) * nc * h * (d010 + d000)));
        }
        {
            const R (&Y)[10] = s_y[ty];
            const R nc = Y[8], nf = Y[9];
            put(10, sfct(dh(Y, 0, KY, false) * nc));
            put(11, kz ? sfct(dh(Y, 1, KY, false) * nc * qr * syz) : R(0.0));
            put(12, sfct(dh(Y, 2, KY, false) * nc * qr * (d011 + d010 + d001 + d000)));
            put(13, sfct(dh(Y, 3, KY, true) * nf * d000));
            put(14, sfct(dh(Y, 4, KY, false) * nc * h * (d001 + d000)));
        }
        __syncthreads(); // every read of the staged box is done
        if (LD == LD_TMA && !s_ok) {
            if (tid == 0) atomicOr(status, ST_TMA_TIMEOUT);
            return; // block-uniform
        }
        if (ch + 1 < NC) issue(ch + 1);
    }
    if (col_ok) numfilter_halo_levels<false>(g, c, Phi<R>{g, a}, nullptr, a.num_diff, N3, a.DENS, i, j, lane);
}

template <typename R, int LD, int NM>
cudaError_t launch_nd(const Grid &g, const Members &mem, const NdCoef &c, const NdArgsT<R> &a, unsigned *status,
                      cudaStream_t st)
{
    NdMaps maps{};
    NdPtrs<R> ptr;
    for (int q = 0; q < 5; ++q) ptr.phi[q] = a.phi + (size_t)q * n3(g);
    for (int q = 0; q < 15; ++q) ptr.nd[q] = a.num_diff + (size_t)q * n3(g);
    if (LD == LD_TMA) {
        for (int q = 0; q < 5; ++q)
            if (!encode(&maps.m[q], ptr.phi[q], g, NBK, NBW, NBH)) return cudaErrorNotSupported;
        if (!encode(&maps.m[5], a.DENS, g, NBK, NBW, NBH)) return cudaErrorNotSupported;
    }
    BatchT<NM> B{};
    B.n = mem.n > 1 ? mem.n : 1;
    long long nb = 0;
    for (int q = 0; q < B.n; ++q) {
        const Grid m = mem.n > 1 ? member_grid(g, mem.m[q]) : g;
        if (mem.n > 0) B.m[q] = mem.m[q];
        B.first[q] = (int)nb;
        nb += ((m.IMAX + NTX - 1) / NTX) * ((m.JMAX + NTY - 1) / NTY);
    }
    if (nb >= (1LL << 31)) return cudaErrorInvalidValue;
    B.first[B.n] = (int)nb;
    auto k = k_numfilter_tiled<R, LD, NM>;
    const cudaError_t e = open_smem(k, nd_smem_bytes<R>());
    if (e != cudaSuccess) return e;
    k<<<(unsigned)nb, dim3(32, NWARPS), nd_smem_bytes<R>(), st>>>(g, c, a, B, ptr, status, maps);
    return cudaGetLastError();
}

}  // namespace tma

// The filter's components from staged tiles: one domain or an ensemble of KHALO = 2
// at ND_ORDER = 1. Bulk tensor copies where one domain's arrays admit tensor maps
// (16-byte aligned bases and strides), cp.async otherwise. cudaErrorNotSupported
// where neither applies.
template <typename R>
cudaError_t launch_numfilter_tiled(const Grid &g, const Members &mem, const NdCoef &c, const NdArgsT<R> &a,
                                   unsigned *status, cudaStream_t st)
{
    if (g.KS != 3 || c.order != 1 || !status) return cudaErrorNotSupported;
    if (mem.n <= 1) {
        const cudaError_t e = tma::launch_nd<R, tma::LD_TMA, 1>(g, mem, c, a, status, st);
        if (e != cudaErrorNotSupported) return e;
    }
    return mem.n > 0 ? tma::launch_nd<R, tma::LD_COPY, HEVI_MAX_MEMBERS>(g, mem, c, a, status, st) : cudaErrorNotSupported;
}
#ifndef HEVI_FLOAT_TU
template cudaError_t launch_numfilter_tiled<double>(const Grid &, const Members &, const NdCoef &,
                                                    const NdArgsT<double> &, unsigned *, cudaStream_t);
#else
template cudaError_t launch_numfilter_tiled<float>(const Grid &, const Members &, const NdCoef &,
                                                   const NdArgsT<float> &, unsigned *, cudaStream_t);
#endif

}  // namespace hevi
