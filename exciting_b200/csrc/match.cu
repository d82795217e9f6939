// APW matching coefficients on the device (src/match.f90:83-191).
//
// A(l, m, io; G) = c_{l,io}(|G+k|) 4 pi / sqrt(Omega) i^l e^{i(G+k).tau_a} conj(Y_lm(G+k)),
// c = D_l^-1 (|G+k|^{io} j_l^{(io)}(|G+k| R)): only the real c and the phase
// depend on the atom.  A block takes 32 G+k (one per lane) of one k-point and
// a run of atoms: its warps first share out the spherical angles, the l of
// the Y_lm recursion (genylm), e^{i m phi} and the Bessel derivatives
// (sbesseldm), then, atom by atom, the D_l solves (the steps of zgesv on the
// real system) and the (l, m) rows.  Everything is FP64.
//
// Two output layouts:
//   * planes   -- A split into real/imaginary planes [f][G], f = stacked
//                 APW rows (atom, l, m, io), G contiguous (coalesced writes);
//                 the operand layout of the contraction kernels.
//   * apwalm   -- the reference's apwalm(ngkmax, apwordmax, lmmaxapw, natmtot).
#include <algorithm>
#include <type_traits>

#include "exs_internal.cuh"

namespace exs {

// D_l for atom ias (match.f90:136-148) factorised in place; returns info.
__device__ inline int match_dmat(const DevParams &p, int ias, int is, int l, int n, double *d, int *ipiv)
{
    const double *xa = p.spr_tail + (size_t)p.np_tail * is;
    const double rmt = p.rmt[is];
    for (int io2 = 0; io2 < n; io2++) {
        const double *ya = p.apwfr_tail +
            (size_t)p.np_tail * (io2 + (size_t)p.apwordmax * (l + (size_t)(p.lmaxapw + 1) * ias));
        for (int io1 = 0; io1 < n; io1++) d[io1 + n * io2] = polynom(io1, p.np_tail, xa, ya, rmt);
    }
    return lu_factor(n, d, ipiv);
}

constexpr int MA_WARPS = 8, MA_ATOMS = 4;      // warps of a block; atoms whose solves are staged together

// Shared memory of a block, in columns of 32 doubles (one per lane).
struct MatchLayout {
    int xm, cm, dj, tmp, c, sf, pt, red, total;
    __host__ __device__ MatchLayout(int lmaxapw, int lmax_out, int omax)
    {
        int o = 0;
        xm = o;  o += (lmax_out + 1) * (lmax_out + 2) / 2;      // Y_lm without e^{i m phi}, m >= 0
        cm = o;  o += 2 * (lmax_out + 1);                       // cos, sin of m phi
        dj = o;  o += omax * (lmaxapw + 1);                     // |G+k|^io j_l^(io)
        tmp = o; o += (omax - 1) * (lmaxapw + 2);               // j_l for the derivatives
        c = o;   o += MA_ATOMS * omax * (lmax_out + 1);         // D_l^-1 dj
        sf = o;  o += 2 * MA_ATOMS;                             // e^{i(G+k).tau}
        pt = o;  o += 4;                                        // |G+k|, sin(theta), cos(theta), phi
        red = o; o += MA_WARPS;                                 // column partial results of the warps
        total = o;
    }
};

// PLANES: k-point descriptors ks; else the reference's match inputs gpc,
// tpgpc, sfacgp of one k-point.  Blocks: x 32 G+k, y a run of `run` atoms, z
// the k-point.  Latency, then HBM: the outputs of 27 k-points of the
// eight-atom cell (0.86 GB) take 295 us (one thread per (G+k, atom) with
// its recursions in local memory: 790), one k-point of the two-atom cell
// 20 us (132), 64 atoms 0.46 ms (1.2).
template <bool PLANES>
__global__ void __launch_bounds__(32 * MA_WARPS, 3) match_kernel(DevParams p, const KDesc *ks, int omax, int run,
                                                              int maxima, int ngp_ref, const double *gpc,
                                                              const double *tpgpc, const exs_complex *sfacgp,
                                                              exs_complex *apwalm)
{
    extern __shared__ __align__(16) double ma_smem[];
    const int lmax_out = PLANES ? p.lmaxmat : p.lmaxapw;
    const MatchLayout L(p.lmaxapw, lmax_out, omax);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = blockIdx.x * 32 + lane;
    KDesc k{};
    if (PLANES) k = ks[blockIdx.z];
    const int ngp = PLANES ? k.ngp : ngp_ref;
    const bool on = g < ngp;
    auto col = [&](int c) -> double & { return ma_smem[c * 32 + lane]; };
    auto cols = [&](int c) { return Strided{ma_smem + c * 32 + lane, 32}; };

    double v[3] = {0.0, 0.0, 0.0};
    if (PLANES && on)
        for (int x = 0; x < 3; x++) v[x] = k.vgpc[3 * g + x];
    if (warp == 0) {
        double r = 1.0, theta = 0.0, phi = 0.0, sn, cs;     // lanes past ngp: any point
        if (PLANES) {
            if (on) sphcrd(v, &r, &theta, &phi);
        } else if (on) {
            r = gpc[g];
            theta = tpgpc[2 * g];
            phi = tpgpc[2 * g + 1];
        }
        sincos(theta, &sn, &cs);
        col(L.pt) = r;
        col(L.pt + 1) = sn;
        col(L.pt + 2) = cs;
        col(L.pt + 3) = phi;
    }
    __syncthreads();
    const double r = col(L.pt);
    int species = -1;
    const int a_end = min(p.natmtot, (int)(blockIdx.y + 1) * run);
    for (int a0 = blockIdx.y * run; a0 < a_end;) {
        const int is = p.atoms[a0].species;
        const int *apw = p.apword + (size_t)(p.lmaxapw + 1) * is;
        int na = 1;                                          // atoms a0 .. a0 + na - 1 of one species
        while (na < MA_ATOMS && a0 + na < a_end && p.atoms[a0 + na].species == is) na++;
        if (is != species) {
            // the Bessel derivatives of this species and, the first time, the angular factors: one task per warp
            const int ny = species < 0 ? lmax_out + 1 : 0, nm = species < 0 ? lmax_out : 0;
            const int ns = (omax - 1) * (p.lmaxapw + 1);
            const double x = r * p.rmt[is];
            for (int t = warp; t < omax + ny + nm + ns; t += MA_WARPS) {
                int q = t;
                if (q < omax) {                              // recurrences, the longest first
                    const int io = omax - 1 - q;
                    if (io == 0) {
                        sbessel(p.lmaxapw, x, cols(L.dj));
                    } else {
                        const Strided jl = cols(L.tmp + (io - 1) * (p.lmaxapw + 2)), d = cols(L.dj + io * (p.lmaxapw + 1));
                        if (x > 1.0) {
                            sbessel(p.lmaxapw + 1, x, jl);
                            sbesseldm_large(io, p.lmaxapw, x, jl, d);
                        }
                    }
                    double t1 = 1.0;
                    for (int i = 0; i < io; i++) t1 *= r;
                    if (io > 0 && x > 1.0)
                        for (int l = 0; l <= p.lmaxapw; l++) col(L.dj + io * (p.lmaxapw + 1) + l) *= t1;
                } else if ((q -= omax) < ny) {
                    const int l = lmax_out - q;
                    ylm_l(l, col(L.pt + 1), col(L.pt + 2), cols(L.xm + l * (l + 1) / 2));
                } else if ((q -= ny) < nm) {
                    double sn, cs;
                    sincos((double)(q + 1) * col(L.pt + 3), &sn, &cs);
                    col(L.cm + 2 * (q + 1)) = cs;
                    col(L.cm + 2 * (q + 1) + 1) = sn;
                } else {                                     // power series of the derivatives, lanes with x <= 1
                    q -= nm;
                    const int io = 1 + q / (p.lmaxapw + 1), l = q % (p.lmaxapw + 1);
                    if (x <= 1.0) {
                        double t1 = 1.0;
                        for (int i = 0; i < io; i++) t1 *= r;
                        col(L.dj + io * (p.lmaxapw + 1) + l) = sbesseldm_small(io, l, x) * t1;
                    }
                }
            }
            species = is;
            __syncthreads();
        }
        // phases and D_l solves of the na atoms
        for (int t = warp; t < na * (lmax_out + 2); t += MA_WARPS) {
            const int ia = t / (lmax_out + 2), l = t % (lmax_out + 2) - 1, ias = a0 + ia;
            if (l < 0) {
                double sn = 0.0, cs = 0.0;
                if (PLANES) {
                    const AtomDesc &at = p.atoms[ias];
                    sincos(v[0] * at.pos[0] + v[1] * at.pos[1] + v[2] * at.pos[2], &sn, &cs);
                } else if (on) {
                    const exs_complex z = sfacgp[g + (size_t)p.ngkmax * ias];
                    cs = z.re;
                    sn = z.im;
                }
                col(L.sf + 2 * ia) = cs;
                col(L.sf + 2 * ia + 1) = sn;
                continue;
            }
            // D_l of this atom, factorised once per set of SCF inputs (match_dlu_kernel)
            const int n = apw[l];
            const double *lu = p.dlu + ((size_t)ias * (p.lmaxapw + 1) + l) * DLU_STRIDE;
            const int from = L.dj + l, to = L.c + (ia * (lmax_out + 1) + l) * omax;
            const bool ok = (int)lu[12] == 0;                // else the right-hand sides stay (match.f90:166-175)
            if (!ok && lane == 0) atomicOr(p.err, DEV_WARN_SINGULAR);
            auto solve = [&](auto tag) {
                constexpr int N = decltype(tag)::value;
                double b[N];
#pragma unroll
                for (int i = 0; i < N; i++) b[i] = col(from + i * (p.lmaxapw + 1));
                if (ok) lu_solve<N>(lu, lu + 9, b);
#pragma unroll
                for (int i = 0; i < N; i++) col(to + i) = b[i];
            };
            if (n == 1)
                solve(std::integral_constant<int, 1>{});
            else if (n == 2)
                solve(std::integral_constant<int, 2>{});
            else
                solve(std::integral_constant<int, 3>{});
        }
        __syncthreads();
        const double fpso = 12.566370614359172954 / sqrt(p.omega);
        for (int ia = 0; ia < na; ia++) {
            const int ias = a0 + ia;
            const AtomDesc &at = p.atoms[ias];
            const double cr = fpso * col(L.sf + 2 * ia), ci = fpso * col(L.sf + 2 * ia + 1);
            double acc = 0.0;                                // maximum, or sum of squares
            int l = 0, f0 = 0;                               // f0: first row of l
            for (int lm = warp; lm < (lmax_out + 1) * (lmax_out + 1); lm += MA_WARPS) {
                while (lm >= (l + 1) * (l + 1)) {
                    f0 += (2 * l + 1) * apw[l];
                    l++;
                }
                const int n = apw[l], m = lm - l * (l + 1), mm = m < 0 ? -m : m;
                // z2 = fpso i^l e^{i(G+k).tau}; Y_lm as genylm builds it: m > 0: x(m) e^{i m phi};
                // m < 0: (-1)^|m| conj(Y_{l,|m|})
                const double z2r = (l & 3) == 0 ? cr : ((l & 3) == 1 ? -ci : ((l & 3) == 2 ? -cr : ci));
                const double z2i = (l & 3) == 0 ? ci : ((l & 3) == 1 ? cr : ((l & 3) == 2 ? -ci : -cr));
                double yr = col(L.xm + l * (l + 1) / 2 + mm), yi = 0.0;
                if (mm > 0) {
                    yi = yr * col(L.cm + 2 * mm + 1);
                    yr = yr * col(L.cm + 2 * mm);
                    if (m < 0) {
                        if (mm & 1) yr = -yr;
                        else yi = -yi;
                    }
                }
                const double wr = z2r * yr + z2i * yi, wi = z2i * yr - z2r * yi;
                const int f = f0 + (m + l) * n;
#pragma unroll 2
                for (int io = 0; io < n; io++) {
                    const double c = col(L.c + (ia * (lmax_out + 1) + l) * omax + io);
                    const double re = on ? c * wr : 0.0, im = on ? c * wi : 0.0;
                    if (PLANES) {
                        const size_t o = (size_t)(at.apw_off + f + io) * p.npad + g;   // npad: a multiple of 32
                        k.ar[o] = re;
                        k.ai[o] = im;
                        acc = maxima ? fmax(acc, fmax(fabs(re), fabs(im))) : fma(re, re, fma(im, im, acc));
                    } else if (on) {
                        exs_complex z;
                        z.re = re;
                        z.im = im;
                        apwalm[g + (size_t)p.ngkmax * (io + (size_t)p.apwordmax * (lm + (size_t)p.lmmaxapw * ias))] = z;
                    }
                }
                if (!PLANES && on)   // orders beyond apword(l) are not set by match: zero them
                    for (int io = n; io < p.apwordmax; io++)
                        apwalm[g + (size_t)p.ngkmax * (io + (size_t)p.apwordmax * (lm + (size_t)p.lmmaxapw * ias))] =
                            exs_complex{0.0, 0.0};
            }
            if (PLANES && k.oz_scale) {
                // split precision: this atom's part of the column bound, the warps' parts in order
                col(L.red + warp) = acc;
                __syncthreads();
                if (warp == ia % MA_WARPS) {
                    double t = 0.0;
                    for (int w = 0; w < MA_WARPS; w++) t = maxima ? fmax(t, col(L.red + w)) : t + col(L.red + w);
                    if (maxima)
                        atomic_max_nonneg(k.oz_scale + g, t);
                    else
                        k.oz_part[(size_t)ias * p.npad + g] = t;
                }
                __syncthreads();
            }
        }
        a0 += na;
        __syncthreads();                                     // c and sf are rewritten
    }
}

// apwalm (reference layout) -> A planes of one k-point, with this atom's part
// of the column bounds: the maxima raised in amax_out, or the sums of squares
// in part_out (either may be null).
__global__ void apwalm_to_planes_kernel(DevParams p, int ngp, const exs_complex *apwalm, double *ar, double *ai,
                                        double *amax_out, double *part_out)
{
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int ias = blockIdx.y;
    if (g >= p.npad) return;
    const AtomDesc at = p.atoms[ias];
    const int *apw = p.apword + (size_t)(p.lmaxapw + 1) * at.species;
    int f = at.apw_off;
    double amax = 0.0, sum = 0.0;
    for (int l = 0; l <= p.lmaxmat; l++)
        for (int m = -l; m <= l; m++) {
            const int lm = l * (l + 1) + m;
            for (int io = 0; io < apw[l]; io++, f++) {
                double re = 0.0, im = 0.0;
                if (g < ngp) {
                    const exs_complex z = apwalm[g + (size_t)p.ngkmax * (io + (size_t)p.apwordmax * (lm + (size_t)p.lmmaxapw * ias))];
                    re = z.re; im = z.im;
                }
                ar[(size_t)f * p.npad + g] = re;
                ai[(size_t)f * p.npad + g] = im;
                amax = fmax(amax, fmax(fabs(re), fabs(im)));
                sum = fma(re, re, fma(im, im, sum));
            }
        }
    if (amax_out) atomic_max_nonneg(amax_out + g, amax);
    if (part_out) part_out[(size_t)ias * p.npad + g] = sum;
}

// (I + h1aa) A for the IORA overlap (overlapsetup.f90:72-87):
// C(f2) = A(f2) + sum_io1 h1aa(io1, io2, l, ias) A(f1), f = (l, m, io).  Blocks
// per (atom, l) (one per atom walks 162 rows in a thread: 80 us for nine
// k-points of the eight-atom cell, 47 us with l apart): the l beside the G in
// the grid's x, which alone goes past 65,535, the atoms in y.
__global__ void iora_planes_kernel(DevParams p, const KDesc *ks)
{
    const KDesc k = ks[blockIdx.z];
    const int l = blockIdx.x % (p.lmaxmat + 1), ias = blockIdx.y;
    const int g = blockIdx.x / (p.lmaxmat + 1) * blockDim.x + threadIdx.x;
    if (g >= p.npad) return;
    const AtomDesc &at = p.atoms[ias];
    const int *apw = p.apword + (size_t)(p.lmaxapw + 1) * at.species;
    int f = at.apw_off;
    for (int q = 0; q < l; q++) f += (2 * q + 1) * apw[q];
    const int n = apw[l];
    const double *h1 = p.h1aa + (size_t)p.apwordmax * p.apwordmax * (l + (size_t)(p.lmaxapw + 1) * ias);
#pragma unroll 2
    for (int m = -l; m <= l; m++, f += n) {
        double ar[EXS_APWORD_MAX], ai[EXS_APWORD_MAX];
#pragma unroll
        for (int io = 0; io < EXS_APWORD_MAX; io++)
            if (io < n) {
                ar[io] = k.ar[(size_t)(f + io) * p.npad + g];
                ai[io] = k.ai[(size_t)(f + io) * p.npad + g];
            }
#pragma unroll
        for (int io2 = 0; io2 < EXS_APWORD_MAX; io2++) {
            if (io2 >= n) break;
            double re = ar[io2], im = ai[io2];
#pragma unroll
            for (int io1 = 0; io1 < EXS_APWORD_MAX; io1++)
                if (io1 < n) {
                    const double w = h1[io1 + (size_t)p.apwordmax * io2];
                    re += w * ar[io1];
                    im += w * ai[io1];
                }
            k.cr[(size_t)(f + io2) * p.npad + g] = re;
            k.ci[(size_t)(f + io2) * p.npad + g] = im;
        }
    }
}

// LU factors of D_l for every (atom, l <= lmaxapw) (match.f90:136-163):
// one thread per l, one block per atom.
__global__ void match_dlu_kernel(DevParams p, double *dlu)
{
    const int ias = blockIdx.x, l = threadIdx.x;
    if (l > p.lmaxapw) return;
    const int is = p.atoms[ias].species;
    const int n = p.apword[l + (size_t)(p.lmaxapw + 1) * is];
    double d[EXS_APWORD_MAX * EXS_APWORD_MAX];
    int ipiv[EXS_APWORD_MAX];
    const int info = match_dmat(p, ias, is, l, n, d, ipiv);
    double *out = dlu + ((size_t)ias * (p.lmaxapw + 1) + l) * DLU_STRIDE;
    for (int i = 0; i < 9; i++) out[i] = i < n * n ? d[i] : 0.0;
    for (int i = 0; i < 3; i++) out[9 + i] = i < n ? (double)ipiv[i] : 0.0;
    out[12] = (double)info;
}

cudaError_t launch_match_dlu(const DevParams &p, double *dlu, cudaStream_t s)
{
    match_dlu_kernel<<<p.natmtot, 32 * ((p.lmaxapw + 32) / 32), 0, s>>>(p, dlu);
    return cudaGetLastError();
}

// The angular factors and Bessel functions are computed once per block, so a
// block takes as many atoms as still leave about eight blocks per SM.
template <bool PLANES>
static cudaError_t launch_match(const DevParams &p, const KDesc *d_k, int nk, int maxima, int ngp, const double *gpc,
                                const double *tpgpc, const exs_complex *sfacgp, exs_complex *apwalm, cudaStream_t s)
{
    static std::atomic<unsigned long long> attr{0};
    cudaError_t e = once_per_device(attr, [] {
        return cudaFuncSetAttribute(match_kernel<PLANES>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    MatchLayout(EXS_LMAX_APW, EXS_LMAX_APW, EXS_APWORD_MAX).total * 32 *
                                        (int)sizeof(double));
    });
    if (e != cudaSuccess) return e;
    const int gx = PLANES ? p.npad / 32 : (ngp + 31) / 32;
    const int groups = (int)std::min<long long>(p.natmtot, (148 * 8 + (long long)gx * nk - 1) / ((long long)gx * nk));
    const int run = (p.natmtot + groups - 1) / groups;
    const MatchLayout L(p.lmaxapw, PLANES ? p.lmaxmat : p.lmaxapw, p.apwordmax);
    match_kernel<PLANES><<<dim3(gx, (p.natmtot + run - 1) / run, nk), 32 * MA_WARPS, L.total * 32 * sizeof(double), s>>>(
        p, d_k, p.apwordmax, run, maxima, ngp, gpc, tpgpc, sfacgp, apwalm);
    return cudaGetLastError();
}

cudaError_t launch_match_planes(const DevParams &p, const KDesc *d_k, int nk, int maxima, cudaStream_t s)
{
    return launch_match<true>(p, d_k, nk, maxima, 0, nullptr, nullptr, nullptr, nullptr, s);
}

cudaError_t launch_match_ref(const DevParams &p, int ngp, const double *gpc, const double *tpgpc,
                             const exs_complex *sfacgp, exs_complex *apwalm, cudaStream_t s)
{
    if (ngp <= 0) return cudaSuccess;
    return launch_match<false>(p, nullptr, 1, 0, ngp, gpc, tpgpc, sfacgp, apwalm, s);
}

cudaError_t launch_apwalm_to_planes(const DevParams &p, int ngp, const exs_complex *apwalm, double *ar,
                                    double *ai, double *amax, double *part, cudaStream_t s)
{
    dim3 grid((p.npad + 127) / 128, p.natmtot, 1);
    apwalm_to_planes_kernel<<<grid, 128, 0, s>>>(p, ngp, apwalm, ar, ai, amax, part);
    return cudaGetLastError();
}

cudaError_t launch_iora_planes(const DevParams &p, const KDesc *d_k, int nk, int ngp_max, cudaStream_t s)
{
    (void)ngp_max;
    dim3 grid((p.npad + 127) / 128 * (p.lmaxmat + 1), p.natmtot, nk);
    iora_planes_kernel<<<grid, 128, 0, s>>>(p, d_k);
    return cudaGetLastError();
}

}  // namespace exs
