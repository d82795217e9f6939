// The modular split-precision contraction (EXS_PREC_OZAKI_MOD) on the 5th-gen
// tensor cores: the complex integer products as int8 products in rings where
// -1 is a square.
//
// Operands.  Every column G of A, of B = blockdiag(h_a) A and (iora*) of
// C = (I + h1aa) A is scaled by sigma = a power of two above its 2-norm and
// rounded to b-bit integers x' = rint(x 2^b / sigma) (exact in FP64; the
// scaled column has norm <= 2^b (1 + eps)); the rows of h_a and loa likewise
// to bx bits.  By the Cauchy-Schwarz inequality the integer products obey
// |X| <= 2^(2b) (1 + eps)^2 (H, O) and 2^(b+bx) (1 + eps)^2 (h_a A, loa A),
// whatever K.  b and bx are the plan's (oz_mod_plan, exs_ozaki_moduli).
//
// Products.  The moduli p_m of the table below are pairwise coprime and all
// their prime factors are 1 mod 4, so an integer i_m with i_m^2 = -1 (mod p_m)
// exists and Z_p[i] is a product of two copies of Z_p: a complex number
// z = x + iy has the two images z+ = x + i_m y and z- = x - i_m y, and complex
// multiplication acts on each image alone.  A complex product therefore costs
// TWO integer products per modulus (with real and imaginary planes it costs
// four, or three by Karatsuba's identity, which would need a third plane of
// every operand):
//   H = A^H B:   (A-)^T (B+) = Re H + i_m Im H,   (A+)^T (B-) = Re H - i_m Im H
//   O = A^H A:   (A-)^T (A+) = Re O + i_m Im O,   (A+)^T (A-) = Re O - i_m Im O
//   h A:         (h+)   (A+) = Re + i_m Im,       (h-)   (A-) = Re - i_m Im
// Plane P = 2m + q holds, as int8 residues in [-127, 127], A-, B+, C+ and h-
// for q = 0 and A+, B-, C-, h+ for q = 1: product P of the H/O tiles is
// A_P^T [B_P | A_(P^1)] (with iora* [B_P | C_P]), product P of the per-atom
// tiles is A_P^T h_P.  n moduli make 2n products of two operands each: 14
// moduli (104.4 bits) and 28 products at b = 49, where 13 larger moduli
// (101.8 bits) with real and imaginary planes take 52.
//
// oz_plane_kernel forms the products tile by tile and stores the residues
// z = v mod p in [0, p) of the int32 sums as bytes; oz_crt_kernel (H, O) and
// oz_bcrt_kernel (h_a A, loa A) recombine them: 2 Re X = z+ + z-,
// 2 i_m Im X = z+ - z- (mod p_m), then the Chinese remainder theorem.
//
// Storage of a slot: [plane P][array: B, A, (C)][G (npad rows)][kp8] bytes, K
// contiguous and zero-padded to kp8 (a multiple of 128); of the per-atom
// operands [atom][plane P][row (h_a rows, then lo rows, padded)][lw], a
// window of lw K bytes starting at the atom's oz_x0 (apw_off rounded down to
// 16), zero outside the atom's own rows.
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "exs_internal.cuh"
#include "interstitial.cuh"
#include "tcgen05.cuh"

namespace exs {

constexpr int RG_CHUNK = 128;                    // bytes of K in one swizzle row
constexpr int RG_BOX = 128 * RG_CHUNK;           // 16 KB: one K chunk of 128 operand rows
constexpr int RG_KCH = 2;                        // K chunks per stage
constexpr int RG_STAGE = 2 * RG_KCH * RG_BOX;    // 64 KB: this CTA's A rows, then its half of B
constexpr int RG_NST = 3;
constexpr int RG_SMEM = RG_NST * RG_STAGE + 1024;
constexpr int RG_THREADS = 384;                  // 12 warps: see the roles below
constexpr int RG_BM = 256, RG_BJ = 128;          // H/O tile of a CTA pair: 256 G_i x 128 G_j
constexpr int RG_ACC = 256;                      // tensor-memory columns of one accumulator

// ------------------------------------------------------------ residues
// int8 x int8 dot products with unsigned bytes in a and signed ones in b.
__device__ __forceinline__ int dp4a_us(uint32_t a, int b, int c)
{
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// The bytes (in the low 8 bits) of the residues of s = x + i_m y and of
// d = x - i_m y for the integers x, y given as the 56-bit unsigned values
// x + 2^55 in two words.  x = sum_k (byte k) 2^(8k) - 2^55, so x mod p is two
// dot products of four bytes with the symmetric residues of 2^(8k) (and of
// i_m 2^(8k) for y): |sum| <= 7 * 255 * 120 + p < 2^18.  base starts the sum
// at the bits of an FP32 integer near 1.5 * 2^23 (a multiple of p, plus
// -2^55 mod p), so s and d are FP32 integers without a conversion: q = round(s / p)
// is one FMA with 1.5 * 2^23 (|s / p| < 2^18; 1/p in FP32 moves it by under
// 2^-6), and s - q p, |.| <= p / 2 + 4 <= 127, is exact in the low byte.
__device__ __forceinline__ void ring_pair(const OzRing &rg, int m, uint2 x, uint2 y, uint32_t &s, uint32_t &d)
{
    constexpr float MAGIC = 12582912.0f;           // 1.5 * 2^23
    const int vr = dp4a_us(x.x, rg.clo[m], dp4a_us(x.y, rg.chi[m], rg.base[m]));
    const int vi = dp4a_us(y.x, rg.ilo[m], dp4a_us(y.y, rg.ihi[m], rg.icorr[m]));
    const int vs = vr + vi, vd = vr - vi;
    const int qs = __float_as_int(fmaf(__int_as_float(vs), rg.inv[m], MAGIC));
    const int qd = __float_as_int(fmaf(__int_as_float(vd), rg.inv[m], MAGIC));
    s = (uint32_t)(vs - qs * rg.p[m]);
    d = (uint32_t)(vd - qd * rg.p[m]);
}

__device__ __forceinline__ uint32_t pack4(uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}

__device__ __forceinline__ uint2 ring_digits(double x, double sc)
{
    const unsigned long long u = (unsigned long long)(__double2ll_rn(x * sc) + (1ll << 55));
    return make_uint2((uint32_t)u, (uint32_t)(u >> 32));
}

// Column 2-norms of the A, B or C planes (which = 0, 1, 2) into oz_scale
// block `which`.  One column per thread column of a 32 x 32 block, the rows
// of threads covering interleaved rows f (stride 32), the partial sums
// combined in a fixed order, so that the scales, and every result, are the
// same from run to run.  The factor 1 + 2^-30 covers the rounding of a sum of
// squares.  HBM bound (one read of the planes); 32 row threads instead of
// eight keep enough loads in flight when few columns are left per SM: 64
// atoms (254 blocks) 555 -> 201 us, 8 k-points of the two-atom cell 21 -> 7 us.
__global__ void __launch_bounds__(1024) oz_norm_kernel(DevParams p, const KDesc *ks, int which)
{
    __shared__ double part[32][33];
    const KDesc k = ks[blockIdx.y];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int g = blockIdx.x * 32 + tx;
    const double *pr, *pi;
    oz_operand(k, which, pr, pi);
    double s = 0.0;
    if (g < k.ngp) {
#pragma unroll 4
        for (int f = ty; f < p.K; f += 32) {
            const size_t i = (size_t)f * p.npad + g;
            const double xr = pr[i], xi = pi[i];
            s = fma(xr, xr, fma(xi, xi, s));
        }
    }
    part[ty][tx] = s;
    __syncthreads();
    // 32 partial sums per column: one column per warp, fixed tree
    double t = part[tx][ty];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    const int gc = blockIdx.x * 32 + ty;
    if (tx == 0 && gc < p.npad) k.oz_scale[(size_t)which * p.npad + gc] = sqrt(t) * (1.0 + 0x1p-30);
}

// The 2n residue planes of one operand (which = 0: A, 1: B, 2: C).  A
// 128(f) x 32(G) tile per block, transposed through shared memory: reads
// G-contiguous planes (a warp reads 32 consecutive G), writes K-contiguous
// int8 rows 16 bytes per thread (8 threads cover a whole 128-byte line of one
// G row).  The padding of two doubles per 16 rows of the tile spreads the
// transposed reads over the banks.
constexpr int RS_F = 128;
constexpr int RS_LD = RS_F * 33 + 2 * (RS_F / 16);
__device__ __forceinline__ int rs_at(int f, int g) { return f * 33 + 2 * (f >> 4) + g; }

__global__ void __launch_bounds__(256, 2) oz_ring_split_kernel(DevParams p, const KDesc *ks,
                                                               const __grid_constant__ OzRing rg, int kp8, int which)
{
    extern __shared__ __align__(16) double rs_t[];       // [re, im][RS_LD]
    const KDesc k = ks[blockIdx.z];
    const int f0 = blockIdx.x * RS_F, g0 = blockIdx.y * 32;
    if (g0 >= k.ngp) return;                             // columns that no output reads
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;      // 32 x 8
    const double *pr, *pi;
    oz_operand(k, which, pr, pi);
    {
        const int g = g0 + tx;
        double vr[RS_F / 8], vi[RS_F / 8];
#pragma unroll
        for (int q = 0; q < RS_F / 8; q++) {
            const int f = f0 + ty + 8 * q;
            const bool v = f < p.K && g < k.ngp;
            const size_t i = (size_t)f * p.npad + g;
            vr[q] = v ? pr[i] : 0.0;
            vi[q] = v ? pi[i] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < RS_F / 8; q++) {
            rs_t[rs_at(ty + 8 * q, tx)] = vr[q];
            rs_t[RS_LD + rs_at(ty + 8 * q, tx)] = vi[q];
        }
    }
    __syncthreads();
    const int gl = threadIdx.x >> 3, fl = (threadIdx.x & 7) * 16;
    const int g = g0 + gl, f = f0 + fl;
    if (g >= p.npad) return;
    // 1/sigma is a power of two: the scaling is exact
    const double sc = ldexp(1.0 / oz_sigma(k.oz_scale[(size_t)which * p.npad + g]), rg.b);
    uint2 x[16], y[16];
#pragma unroll
    for (int e = 0; e < 16; e++) {
        x[e] = ring_digits(rs_t[rs_at(fl + e, gl)], sc);
        y[e] = ring_digits(rs_t[RS_LD + rs_at(fl + e, gl)], sc);
    }
    const int narr = ring_narr(p.relativity), arr = which == 0 ? 1 : (which == 1 ? 0 : 2);
    const size_t plane = (size_t)narr * p.npad * kp8;
    int8_t *out = k.oz_slices + ((size_t)arr * p.npad + g) * kp8 + f;
#pragma unroll 1
    for (int m = 0; m < rg.n; m++, out += 2 * plane) {
        uint32_t ws[4], wd[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            uint32_t s[4], d[4];
#pragma unroll
            for (int e = 0; e < 4; e++) ring_pair(rg, m, x[4 * q + e], y[4 * q + e], s[e], d[e]);
            ws[q] = pack4(s[0], s[1], s[2], s[3]);
            wd[q] = pack4(d[0], d[1], d[2], d[3]);
        }
        // plane 2m: A-, B+, C+; plane 2m + 1: A+, B-, C-
        *reinterpret_cast<uint4 *>(out + (which == 0 ? plane : 0)) = make_uint4(ws[0], ws[1], ws[2], ws[3]);
        *reinterpret_cast<uint4 *>(out + (which == 0 ? 0 : plane)) = make_uint4(wd[0], wd[1], wd[2], wd[3]);
    }
}

// ------------------------------------------------------------ per-atom operands
// X(n, f'): row n < napw of h_a (hamiltonsetup.f90:75-88), then the lo rows of
// loa (hamiltonsetup.f90:131-145); zero past them.
__device__ __forceinline__ void ring_x_value(const OzAtomArgs &xa, const AtomDesc &at, int ias, int n, int fp,
                                             double &re, double &im)
{
    re = im = 0.0;
    if (fp < 0 || fp >= at.napw || n >= at.napw + at.losize) return;
    if (n < at.napw) {
        const size_t i = ((size_t)ias * xa.ldh + fp) * xa.ldh + n;                  // h(f, f') at [ias][f'][f]
        re = xa.hr[i];
        im = xa.hi[i];
    } else {
        const size_t i = ((size_t)ias * xa.maxaa + fp) * xa.ldlo + (n - at.napw);   // loa(r, f) at [ias][f][r]
        re = xa.lr[i];
        im = xa.li[i];
    }
}

// Row 2-norms (their powers of two into xsig) and residue planes of 32 rows
// of one atom's X: the norms first (interleaved f', fixed order), then the
// window in steps of 64 bytes transposed through shared memory.
__global__ void __launch_bounds__(256) oz_ring_x_kernel(DevParams p, OzAtomArgs xa, const __grid_constant__ OzRing rg)
{
    __shared__ double t[2][64][33];
    __shared__ double part[8][33];
    const int ias = blockIdx.y, n0 = blockIdx.x * 32;
    const AtomDesc at = p.atoms[ias];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    double s = 0.0;
#pragma unroll 4
    for (int fp = ty; fp < at.napw; fp += 8) {
        double re, im;
        ring_x_value(xa, at, ias, n0 + tx, fp, re, im);
        s = fma(re, re, fma(im, im, s));
    }
    part[ty][tx] = s;
    __syncthreads();
    if (ty == 0) {
        double v = 0.0;
        for (int q = 0; q < 8; q++) v += part[q][tx];
        v = oz_sigma(sqrt(v) * (1.0 + 0x1p-30));
        part[0][tx] = v;
        xa.xsig[(size_t)ias * xa.nrows + n0 + tx] = v;
    }
    __syncthreads();
    const int delta = at.apw_off - at.oz_x0;
    const int nl = threadIdx.x >> 3, kl = (threadIdx.x & 7) * 8;
    const double sc = ldexp(1.0 / part[0][nl], rg.bx);
    for (int k0 = 0; k0 < xa.lw; k0 += 64) {
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int k = ty + 8 * q;
            ring_x_value(xa, at, ias, n0 + tx, k0 + k - delta, t[0][k][tx], t[1][k][tx]);
        }
        __syncthreads();
        uint2 x[8], y[8];
#pragma unroll
        for (int e = 0; e < 8; e++) {
            x[e] = ring_digits(t[0][kl + e][nl], sc);
            y[e] = ring_digits(t[1][kl + e][nl], sc);
        }
        int8_t *out = xa.xs + ((size_t)ias * 2 * rg.n * xa.nrows + n0 + nl) * xa.lw + k0 + kl;
        const size_t plane = (size_t)xa.nrows * xa.lw;
#pragma unroll 1
        for (int m = 0; m < rg.n; m++, out += 2 * plane) {
            uint32_t ws[2], wd[2];
#pragma unroll
            for (int q = 0; q < 2; q++) {
                uint32_t sr[4], dr[4];
#pragma unroll
                for (int e = 0; e < 4; e++) ring_pair(rg, m, x[4 * q + e], y[4 * q + e], sr[e], dr[e]);
                ws[q] = pack4(sr[0], sr[1], sr[2], sr[3]);
                wd[q] = pack4(dr[0], dr[1], dr[2], dr[3]);
            }
            *reinterpret_cast<uint2 *>(out) = make_uint2(wd[0], wd[1]);              // h-
            *reinterpret_cast<uint2 *>(out + plane) = make_uint2(ws[0], ws[1]);      // h+
        }
    }
}

// ------------------------------------------------------------ the products
// A cluster of two CTAs forms tiles of 256 rows with tcgen05.mma.cta_group::2
// (M = 256): each CTA holds its own 128 rows of the A operand and half of the
// B operand's N rows.
//   RG_HO    tiles {k, ib, jb}: 256 G_i x 128 G_j, N = 256: CTA 0 holds B_P,
//            CTA 1 A_(P^1) (C_P with iora*) of the G_j; columns 0..127 of the
//            sums are H, 128..255 O
//   RG_ATOM  tiles {k, atom, ib, xb}: 256 G x nb rows of h_a and loa of one
//            atom (N = nb, a multiple of 32), over the atom's K window
// The work list is flat in (tile, plane): while full rounds of one tile per
// cluster last, a cluster takes a tile and walks its 2n planes; the (tile,
// plane) pairs of the remaining tiles are dealt out one by one, so that a
// handful of tiles (two for a k-point of the two-atom cell) still occupies
// every SM pair and the last round is never short of more than one product.
// Two accumulators in tensor memory: the MMAs of one product run while the
// epilogue reduces the previous one.
//
// Roles (384 threads): warp 0 / 1 TMA producers of the A / B operand, warp 3
// MMA issuer (CTA 0) and tensor-memory owner, warps 4-11 epilogue: two per
// tensor-memory lane quadrant, half the columns each; residues of 16 columns
// leave as 16 bytes per row, 512 contiguous bytes per warp.
// CTA 0's full barriers count the bytes of both CTAs' copies; MMA completion
// is committed to both CTAs; both epilogues report to CTA 0's barrier.
// Every wait is bounded and gives up when another role of the CTA gave up;
// the kernel then lets its copies and MMAs drain, records DEV_ERR_TIMEOUT,
// frees tensor memory and returns.
//
// What bounds it: the L2 -> SM operand stream (32 KB per K chunk and CTA
// against 512 cycles of MMAs) while K is long.  Measured, H/O: 64 atoms (N =
// 8075, K = 10,368) 14.4 ms, 27 k-points of the eight-atom cell 1.50 ms; the
// real-and-imaginary form with 13 moduli, 256 x 64 tiles and one accumulator
// set took 23.1 and 2.65 ms.  Per-atom products with their recombination: 3.6
// and 2.5 ms, against 4.07 and 2.21 ms for 128 x 64 tiles with 64-bit sums in
// tensor memory (L2 -> SM stream of 25.8 GB in the eight-atom batch).
enum : int { RG_HO = 0, RG_ATOM = 1 };

// Pacing of large H/O launches (pace != null): every cluster publishes, every
// RG_PACE_STAGES stages it issues, its step count in pace[cluster] and waits
// until the slowest cluster is at most RG_PACE_LAG steps behind, so that the
// tiles running at one time read the same row and column blocks within a few
// MB of each other's position and the L2 serves the repeats.  The wait is a
// hint, not a dependency: it gives up after RG_PACE_CYCLES (a cluster that is
// not resident, or a slow one, delays the others by that much per step at
// most) and never raises an error.  A finished cluster publishes INT_MAX.
constexpr int RG_PACE_STAGES = 16;                // 32 K chunks
constexpr int RG_PACE_LAG = 1;
constexpr long long RG_PACE_CYCLES = 40000;
constexpr int RG_PACE_MAX = 1024;                 // clusters (ints of the pace array)

__device__ __forceinline__ int ld_relaxed_gpu(const int *p)
{
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_relaxed_gpu(int *p, int v)
{
    asm volatile("st.relaxed.gpu.global.s32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ void ring_pace(int *pace, int me, int ncl, int step)
{
    const long long t0 = clock64();
    while (true) {
        int mn = 0x7fffffff;
        for (int c = 0; c < ncl; c++) mn = min(mn, ld_relaxed_gpu(pace + c));
        if (mn >= step - RG_PACE_LAG || clock64() - t0 > RG_PACE_CYCLES) break;
    }
    st_relaxed_gpu(pace + me, step);
}

__device__ __forceinline__ void tma_load_4d_2sm(uint32_t dst, const CUtensorMap *map, int c0, int c1, int c2, int c3,
                                                uint32_t bar)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
        "%3, %4, %5}], [%6];\n" ::"r"(dst),
        "l"((uint64_t)map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar & OZ_PEER_BIT_MASK)
        : "memory");
}

// The flat work list of cluster c: count() products, at(i) the i-th.
struct RingUnits {
    int ncl, np, full, rest;         // full rounds of one tile per cluster, remaining tiles
    __device__ RingUnits(int ntiles, int ncl_, int np_) : ncl(ncl_), np(np_), full(ntiles / ncl_), rest(ntiles % ncl_) {}
    __device__ int count(int c) const { return full * np + (rest * np - c + ncl - 1) / ncl; }
    __device__ void at(int i, int c, int &tile, int &P) const
    {
        if (i < full * np) {
            tile = (i / np) * ncl + c;
            P = i % np;
        } else {
            const int v = (i - full * np) * ncl + c;
            tile = full * ncl + v % rest;
            P = v / rest;
        }
    }
};

// Residue of an int32 sum in [0, p): q = floor(v mg / 2^32), mg = round(2^32 / p),
// leaves v - q p in [-p/4, 5p/4]; the unsigned minima add or take p.
__device__ __forceinline__ uint32_t ring_mod(int v, int p, int mg)
{
    uint32_t x = (uint32_t)(v - __mulhi(v, mg) * p);
    x = min(x, x + (uint32_t)p);
    return min(x, x - (uint32_t)p);
}

template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(RG_THREADS, 1)
oz_plane_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, DevParams p,
                const KDesc *ks, const int *tiles, int ntiles, const __grid_constant__ OzRing rg, OzAtomArgs xa,
                uint8_t *res, int *pace)
{
    extern __shared__ __align__(1024) uint8_t rg_smem[];
    __shared__ uint64_t full[RG_NST], empty[RG_NST], accf[2], acce[2];
    __shared__ uint32_t tmem_sh;
    __shared__ int abort_sh;
    volatile int *abort = &abort_sh;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_ctarank();
    const uint32_t sbase = (smem_u32(rg_smem) + 1023u) & ~1023u;
    const int cl = (int)(blockIdx.x >> 1), NP = 2 * rg.n;
    const RingUnits units(ntiles, (int)(gridDim.x >> 1), NP);
    const int nu = units.count(cl);
    const int N = MODE == RG_HO ? 2 * RG_BJ : xa.nb;
    const int b_rows = N / 2;                            // operand rows of B in this CTA

    if (warp == 3) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_sh)),
                     "r"(OZ_TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::);
    }
    if (tid == 0) {
        for (int q = 0; q < RG_NST; q++) {
            mbar_init(&full[q], 1);      // CTA 0: one arrive (with the bytes of both CTAs)
            mbar_init(&empty[q], 1);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(&accf[a], 1);
            mbar_init(&acce[a], 16);     // CTA 0: eight epilogue warps in each CTA
        }
        abort_sh = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                  // the peer's barriers are initialised before anyone signals them
    tc_fence_after();
    const uint32_t tbase = tmem_sh;

    if (warp < 2) {
        // ------------------------------------------------ TMA producers (both CTAs)
        if (lane == 0) {
            const int role = warp;       // 0: this CTA's A rows, 1: this CTA's half of B
            uint32_t fills[RG_NST];
#pragma unroll
            for (int q = 0; q < RG_NST; q++) fills[q] = 0;
            int st = 0, issued = 0;
            bool bad = false;
            const bool pacer = pace != nullptr && rank == 0 && role == 0;
            for (int u = 0; u < nu && !bad; u++) {
                int tile, P;
                units.at(u, cl, tile, P);
                int slot, row, arr, plane, x0 = 0, nch;
                if (MODE == RG_HO) {
                    slot = ks[tiles[3 * tile]].oz_slot;
                    nch = (p.K + RG_CHUNK - 1) / RG_CHUNK;
                    if (role == 0) {
                        row = tiles[3 * tile + 1] * RG_BM + (int)rank * 128;
                        arr = 1;
                        plane = P;
                    } else {             // H: B_P; O: A_(P^1), or C_P with iora*
                        row = tiles[3 * tile + 2] * RG_BJ;
                        arr = rank == 0 ? 0 : (p.relativity == EXS_REL_IORA ? 2 : 1);
                        plane = (rank == 0 || arr == 2) ? P : (P ^ 1);
                    }
                } else {
                    const int ias = tiles[4 * tile + 1];
                    const AtomDesc &at = p.atoms[ias];
                    nch = at.oz_nch;
                    if (role == 0) {
                        slot = ks[tiles[4 * tile]].oz_slot;
                        row = tiles[4 * tile + 2] * RG_BM + (int)rank * 128;
                        x0 = at.oz_x0;
                    } else {
                        slot = ias;
                        row = tiles[4 * tile + 3] * xa.nb + (int)rank * b_rows;
                    }
                    arr = 1;
                    plane = P;
                }
                for (int kb = 0; kb < nch; kb += RG_KCH, issued++) {
                    if (pacer && issued % RG_PACE_STAGES == 0) ring_pace(pace, cl, units.ncl, issued / RG_PACE_STAGES);
                    if (fills[st] > 0 && !mbar_wait_ab(&empty[st], (fills[st] - 1) & 1, abort, rg.wait)) {
                        bad = true;
                        break;
                    }
                    const int nc = min(RG_KCH, nch - kb);
                    const uint32_t bar = smem_u32(&full[st]);
                    const uint32_t dst = sbase + st * RG_STAGE + role * RG_KCH * RG_BOX;
                    if (MODE == RG_HO) {                 // one box of two K chunks (zeros past the last one)
                        if (rank == 0 && role == 0) mbar_expect_tx(&full[st], 2 * RG_STAGE);
                        tma_load_5d_2sm(dst, &mapA, 0, row, arr, kb, slot * NP + plane, bar);
                    } else {
                        if (rank == 0 && role == 0)
                            mbar_expect_tx(&full[st], 2 * nc * (RG_BOX + b_rows * RG_CHUNK));
                        for (int c = 0; c < nc; c++) {
                            if (role == 0)
                                tma_load_4d_2sm(dst + c * RG_BOX, &mapA, x0 + (kb + c) * RG_CHUNK, row, arr,
                                                slot * NP + plane, bar);
                            else
                                tma_load_4d_2sm(dst + c * RG_BOX, &mapB, 0, row, slot * NP + plane, kb + c, bar);
                        }
                    }
                    fills[st]++;
                    st = (st + 1 == RG_NST) ? 0 : st + 1;
                }
            }
            if (pacer) st_relaxed_gpu(pace + cl, 0x7fffffff);     // done: nobody waits for this cluster
            // copies already issued (both CTAs') must land before the pair goes away: CTA 0 waits on its full
            // barriers, CTA 1, whose copies signal CTA 0's barriers, lets far more than their time pass
            if (bad && rank == 0)
                for (int q = 0; q < RG_NST; q++)
                    if (fills[q] > 0) mbar_drain(&full[q], (fills[q] - 1) & 1);
            if (bad && rank == 1)
                for (const long long t0 = clock64(); clock64() - t0 < 1000000;) {
                }
        }
    } else if (warp == 3) {
        // ------------------------------------------------ MMA issuer (CTA 0)
        if (lane == 0 && rank == 0) {
            const uint32_t idesc = umma_idesc_i8(256, N);
            uint32_t uses[RG_NST];
#pragma unroll
            for (int q = 0; q < RG_NST; q++) uses[q] = 0;
            int st = 0;
            bool bad = false;
            for (int u = 0; u < nu && !bad; u++) {
                const int buf = u & 1, use = u >> 1;
                int steps;                                // K steps of 32 bytes
                if (MODE == RG_HO) {
                    steps = (p.K + 31) / 32;
                } else {
                    int tile, P;
                    units.at(u, cl, tile, P);
                    const AtomDesc &at = p.atoms[tiles[4 * tile + 1]];
                    steps = (at.apw_off - at.oz_x0 + at.napw + 31) / 32;
                }
                // the epilogues of both CTAs must have read this accumulator's previous product
                if (use > 0 && !mbar_wait_ab(&acce[buf], (use - 1) & 1, abort, rg.wait)) {
                    bad = true;
                    break;
                }
                tc_fence_after();
                const uint32_t tacc = tbase + (uint32_t)(buf * RG_ACC);
                for (int k0 = 0; k0 < steps; k0 += RG_KCH * 4) {
                    if (!mbar_wait_ab(&full[st], uses[st] & 1, abort, rg.wait)) {
                        bad = true;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sa = sbase + st * RG_STAGE, sb = sa + RG_KCH * RG_BOX;
#pragma unroll
                    for (int q = 0; q < RG_KCH * 4; q++)
                        if (k0 + q < steps) {
                            const uint32_t o = (q >> 2) * RG_BOX + (q & 3) * 32;
                            umma_i8_2sm(tacc, umma_desc_sw128(sa + o), umma_desc_sw128(sb + o), idesc,
                                        k0 + q > 0 ? 1u : 0u);
                        }
                    umma_commit_2sm(&empty[st]);
                    uses[st]++;
                    st = (st + 1 == RG_NST) ? 0 : st + 1;
                }
                if (!bad) umma_commit_2sm(&accf[buf]);
            }
            if (bad)
                for (int q = 0; q < RG_NST; q++)
                    if (uses[q] > 0) mbar_drain(&empty[q], (uses[q] - 1) & 1);
        }
    } else if (warp >= 4) {
        // ------------------------------------------------ epilogue (both CTAs, warps 4..11)
        const int qd = warp & 3, half = (warp - 4) >> 2;
        const int row = qd * 32 + lane;
        const int nq = b_rows / 16;                                 // 16-column chunks of this half
        const uint32_t acce0[2] = {mapa_shared(smem_u32(&acce[0]), 0), mapa_shared(smem_u32(&acce[1]), 0)};
        const size_t plane_bytes = (size_t)N * 128;                 // residues of one product, this CTA's 128 rows
        for (int u = 0; u < nu; u++) {
            const int buf = u & 1, use = u >> 1;
            int tile, P;
            units.at(u, cl, tile, P);
            if (!__all_sync(0xffffffffu, mbar_wait_ab(&accf[buf], use & 1, abort, rg.wait))) break;
            tc_fence_after();
            const int pm = rg.p[P >> 1], mg = rg.mg[P >> 1];
            const uint32_t tacc = tbase + ((uint32_t)(qd * 32) << 16) + (uint32_t)(buf * RG_ACC + half * b_rows);
            uint8_t *out = res + ((size_t)(2 * tile + (int)rank) * NP + P) * plane_bytes +
                           ((size_t)half * nq * 128 + row) * 16;
            for (int c = 0; c < nq; c++) {
                uint32_t v[16];
                tm_ld16(tacc + c * 16, v);
                tm_wait_ld();
                uint32_t w[4];
#pragma unroll
                for (int q = 0; q < 4; q++)
                    w[q] = pack4(ring_mod((int)v[4 * q], pm, mg), ring_mod((int)v[4 * q + 1], pm, mg),
                                 ring_mod((int)v[4 * q + 2], pm, mg), ring_mod((int)v[4 * q + 3], pm, mg));
                *reinterpret_cast<uint4 *>(out + (size_t)c * 128 * 16) = make_uint4(w[0], w[1], w[2], w[3]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(acce0[buf]);          // CTA 0's barrier (also from CTA 0)
        }
    }
    if (tid == 0 && *abort) atomicOr(p.err, DEV_ERR_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                  // neither CTA leaves while the pair still uses its memory
    if (warp == 3) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tbase), "r"(OZ_TMEM_COLS));
    }
}

// ------------------------------------------------------------ recombination
// Eight real or imaginary parts from the residues of both images (wp[m] of
// z+, wm[m] of z-: 8 bytes each).  With s_m = z+ + z- (real parts) or
// z+ - z- + p_m (imaginary parts), s_m < 2 p_m, X / M = sum_m s_m e_m / p_m
// (mod 1), e_m = y_m / 2 or y_m / (2 i_m) mod p_m, y_m = (M / p_m)^-1.  Two
// moduli at a time: w = s_m (e_m p_m') + s_m' (e_m' p_m) < 2^26, and
// t += w D (mod 2^96), D = round(2^96 / (p_m p_m')), three 32 x 32 -> 64-bit
// multiply-adds per PAIR of moduli, carries propagated once at the end.  The
// signed 64-bit window sh bits below the top of t is 2^(64+sh) X / M up to
// the rounding of D (below 2^29 units of 2^-96).
__device__ __forceinline__ void ring_crt8(const OzRing &rg, const uint2 (&wp)[OZ_RING_MAX],
                                          const uint2 (&wm)[OZ_RING_MAX], bool im, int sh, double fin, double (&v)[8])
{
    unsigned long long a[8][3];
#pragma unroll
    for (int e = 0; e < 8; e++) a[e][0] = a[e][1] = a[e][2] = 0ull;
#pragma unroll
    for (int q = 0; q < OZ_RING_MAX / 2; q++) {
        if (2 * q >= rg.n) break;
        uint32_t w[8];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int m = 2 * q + j;
            // an odd count leaves the last pair half empty: weight 0
            const uint32_t f = im ? rg.fim[m] : rg.fre[m], pp = (uint32_t)rg.p[m] * 0x10001u;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint32_t zp = h ? wp[m].y : wp[m].x, zm = h ? wm[m].y : wm[m].x;
                uint32_t s[2];                          // 16-bit lanes: bytes 0, 2 and 1, 3
                const uint32_t p0 = zp & 0xff00ffu, p1 = (zp >> 8) & 0xff00ffu;
                const uint32_t m0 = zm & 0xff00ffu, m1 = (zm >> 8) & 0xff00ffu;
                s[0] = im ? p0 + pp - m0 : p0 + m0;
                s[1] = im ? p1 + pp - m1 : p1 + m1;
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const uint32_t x = (e & 2) ? s[e & 1] >> 16 : s[e & 1] & 0xffffu;
                    w[4 * h + e] = (j ? w[4 * h + e] : 0u) + x * f;
                }
            }
        }
        const unsigned long long d0 = rg.d96[0][q], d1 = rg.d96[1][q], d2 = rg.d96[2][q];
#pragma unroll
        for (int e = 0; e < 8; e++) {
            a[e][0] += w[e] * d0;
            a[e][1] += w[e] * d1;
            a[e][2] += w[e] * d2;
        }
    }
#pragma unroll
    for (int e = 0; e < 8; e++) {
        const unsigned long long a1 = a[e][1] + (a[e][0] >> 32);
        const unsigned long long a2 = a[e][2] + (a1 >> 32);
        const unsigned long long top = (((a2 << 32) | (a1 & 0xffffffffull)) << sh) |
                                       ((a[e][0] & 0xffffffffull) >> (32 - sh));
        v[e] = (double)(long long)top * fin;
    }
}

// The residue bytes of 8 columns of one row: z+ of modulus m in plane 2m + first.
__device__ __forceinline__ void ring_load8(const uint8_t *tres, size_t plane, int n, int first,
                                           uint2 (&wp)[OZ_RING_MAX], uint2 (&wm)[OZ_RING_MAX])
{
#pragma unroll
    for (int m = 0; m < OZ_RING_MAX; m++) {
        wp[m] = wm[m] = make_uint2(0u, 0u);
        if (m < n) {
            wp[m] = *reinterpret_cast<const uint2 *>(tres + (size_t)(2 * m + first) * plane);
            wm[m] = *reinterpret_cast<const uint2 *>(tres + (size_t)(2 * m + 1 - first) * plane);
        }
    }
}

// Recombination, scaling, interstitial term and store of the H/O tiles: one
// thread per (row of a 128-row tile, 8-column group, matrix: 0 = H, 1 = O):
// blocks of 128 threads (the rows), blockIdx.y = (matrix, column group).
// Every thread first issues the loads of its residue bytes, then recombines:
// the loads of a warp cover 32 rows of 16 bytes of which the group uses half.
__global__ void __launch_bounds__(128) oz_crt_kernel(DevParams p, const KDesc *ks, const int *tiles,
                                                     const __grid_constant__ OzRing rg, const uint8_t *res)
{
    constexpr int NG = RG_BJ / 8;                                // 8-column groups
    const int tile = blockIdx.x >> 1, row = threadIdx.x;
    const int cg = blockIdx.y % NG, half = blockIdx.y / NG;
    const KDesc kd = ks[tiles[3 * tile]];
    const int i = tiles[3 * tile + 1] * RG_BM + (blockIdx.x & 1) * 128 + row;
    const int jb = tiles[3 * tile + 2] * RG_BJ + cg * 8;
    if (i >= kd.ngp || jb >= kd.ngp || jb + 7 < i) return;     // no element i <= j < ngp here
    constexpr size_t plane = 2 * RG_BJ * 128;
    const uint8_t *tres = res + (size_t)blockIdx.x * 2 * rg.n * plane +
                          ((size_t)(half * (RG_BJ / 16) + (cg >> 1)) * 128 + row) * 16 + (cg & 1) * 8;
    uint2 wp[OZ_RING_MAX], wm[OZ_RING_MAX];
    ring_load8(tres, plane, rg.n, 0, wp, wm);
    // row data
    int gi = kd.igpig[i] - 1;
    if (gi < 0 || gi >= p.ngrtot) {
        atomicOr(p.err, DEV_ERR_INDEX);
        gi = 0;
    }
    const int ivi[3] = {p.ivg[3 * gi], p.ivg[3 * gi + 1], p.ivg[3 * gi + 2]};
    const double vi[3] = {kd.vgpc[3 * i], kd.vgpc[3 * i + 1], kd.vgpc[3 * i + 2]};
    const double sai = oz_sigma(kd.oz_scale[i]);
    // H: sigma_B(j); O: sigma_A(j), or sigma_C(j) with iora* (O = A^H C)
    const double *scol = kd.oz_scale + (half == 0 ? p.npad : (p.relativity == EXS_REL_IORA ? 2 * p.npad : 0));
    const int kind = half == 0 ? EPI_HAM : EPI_OVL;
    exs_complex *out = half == 0 ? kd.h : kd.o;
    double vre[8], vim[8];
    ring_crt8(rg, wp, wm, false, rg.sh, rg.fin, vre);
    ring_crt8(rg, wp, wm, true, rg.sh, rg.fin, vim);
#pragma unroll
    for (int e = 0; e < 8; e++) {
        const int j = jb + e;
        if (j >= kd.ngp || j < i) continue;
        int gj = kd.igpig[j] - 1;
        if (gj < 0 || gj >= p.ngrtot) {
            atomicOr(p.err, DEV_ERR_INDEX);
            gj = 0;
        }
        const int ivj[3] = {p.ivg[3 * gj], p.ivg[3 * gj + 1], p.ivg[3 * gj + 2]};
        const double vj[3] = {kd.vgpc[3 * j], kd.vgpc[3 * j + 1], kd.vgpc[3 * j + 2]};
        const double sc = sai * oz_sigma(scol[j]);
        double re = vre[e] * sc, im = vim[e] * sc;
        double ar, ai;
        if (interstitial(p, kind, ivi, ivj, vi, vj, ar, ai)) {
            re += ar;
            im += ai;
        }
        exs_complex v;
        v.re = re;
        v.im = im;
        out[(size_t)i + (size_t)kd.nmat * j] = v;
        if (i < j) {
            v.im = -im;
            out[(size_t)j + (size_t)kd.nmat * i] = v;
        }
    }
}

// Recombination of the per-atom tiles: the B planes and the APW-lo rows of H
// with their mirror.  One thread per (G of a 128-row tile, 8 rows of X),
// blockIdx.y = the 8-row group: a warp writes 32 consecutive G of one plane row.
__global__ void __launch_bounds__(128) oz_bcrt_kernel(DevParams p, const KDesc *ks, const int *tiles,
                                                      const __grid_constant__ OzRing rg, OzAtomArgs xa,
                                                      const uint8_t *res)
{
    const int tile = blockIdx.x >> 1, row = threadIdx.x, cg = blockIdx.y;
    const KDesc kd = ks[tiles[4 * tile]];
    const int ias = tiles[4 * tile + 1];
    const int g = tiles[4 * tile + 2] * RG_BM + (blockIdx.x & 1) * 128 + row;
    const int n0 = tiles[4 * tile + 3] * xa.nb + cg * 8;
    const AtomDesc at = p.atoms[ias];
    if (g >= kd.ngp || n0 >= at.napw + at.losize) return;
    const size_t plane = (size_t)xa.nb * 128;
    const uint8_t *tres = res + (size_t)blockIdx.x * 2 * rg.n * plane + ((size_t)(cg >> 1) * 128 + row) * 16 + (cg & 1) * 8;
    uint2 wp[OZ_RING_MAX], wm[OZ_RING_MAX];
    ring_load8(tres, plane, rg.n, 1, wp, wm);
    const double sa = oz_sigma(kd.oz_scale[g]);
    const double *sig = xa.xsig + (size_t)ias * xa.nrows + n0;
    double vre[8], vim[8];
    ring_crt8(rg, wp, wm, false, rg.shx, rg.finx, vre);
    ring_crt8(rg, wp, wm, true, rg.shx, rg.finx, vim);
    const size_t row0 = (size_t)kd.ngp + at.lo_off;
#pragma unroll
    for (int e = 0; e < 8; e++) {
        const int n = n0 + e;
        const double sc = sa * sig[e];
        const double re = vre[e] * sc, im = vim[e] * sc;
        if (n < at.napw) {
            const size_t off = (size_t)(at.apw_off + n) * p.npad + g;
            kd.br[off] = re;
            kd.bi[off] = im;
        } else if (n < at.napw + at.losize) {
            const int r = n - at.napw;
            exs_complex v;
            v.re = re;
            v.im = im;
            kd.h[(row0 + r) + (size_t)kd.nmat * g] = v;
            v.im = -im;
            kd.h[(size_t)g + (size_t)kd.nmat * (row0 + r)] = v;
        }
    }
}

// ------------------------------------------------------------ host side
// The plan's moduli, the precision contract of exs_set_precision and
// exs_ozaki_moduli: pairwise coprime odd, largest first (253 = 11 * 23,
// 247 = 13 * 19, 217 = 7 * 31, 185 = 5 * 37; the others are primes).
static const int OZ_MODULI[OZ_MAX_MODULI] = {253, 251, 247, 241, 239, 233, 229, 227,
                                             223, 217, 211, 199, 197, 193, 191, 185};

// log2 M for the first n moduli (a sum of logarithms: the plan keeps a
// margin of one bit beyond it).
static double oz_log2_modulus(int n)
{
    double lm = 0.0;
    for (int m = 0; m < n; m++) lm += std::log2((double)OZ_MODULI[m]);
    return lm;
}

static int oz_inverse_mod(long long a, long long p)
{
    // extended Euclid on (a mod p, p); gcd is 1 for coprime moduli
    long long r0 = p, r1 = ((a % p) + p) % p, t0 = 0, t1 = 1;
    while (r1 != 0) {
        const long long q = r0 / r1, r2 = r0 - q * r1, t2 = t0 - q * t1;
        r0 = r1; r1 = r2; t0 = t1; t1 = t2;
    }
    return r0 == 1 ? (int)(((t0 % p) + p) % p) : -1;
}

// The plan for n moduli, contraction length K (H/O tiles) and per-atom
// window kx: the bits b of the A and B columns and bx of the h_a / loa rows,
// b = min(52, floor((log2 M - 2) / 2)) keeping one bit of margin beyond
// 2|X| < M, bx = min(52, floor(log2 M - 7 - b)), and the headroom
// h = floor(log2 M - 2 - b - bx) of a 64-bit recombination of the per-atom
// products.  The quantisation error of the operands grows like
// 2^-b sqrt(K), so n = 0 takes the fewest moduli in 6..16 with
// b >= 41 + log2(K) / 2 and bx >= 44 (13 moduli, b = 49 and bx = 45, at both
// K = 1936 and K = 34,992).  Returns 0, or -1 if no valid plan exists (n out
// of range, b or bx below 8, or K past the exact int32 range of one product:
// 2 K 127^2 < 2^31).  The device forms the same integer products X exactly
// in the rings of oz_ring_plan.
static void oz_mod_bits(int n, int *b, int *h, int *bx)
{
    const double lm = oz_log2_modulus(n) - 1e-9;
    *b = std::min(52, (int)std::floor((lm - 2.0) / 2.0));
    *bx = std::min(52, (int)std::floor(lm - 7.0 - *b));
    *h = (int)std::floor(lm - 2.0 - *b - *bx);
}

int oz_mod_plan(int n, int K, int kx, OzScheme *sch)
{
    if (K < 1 || kx < 1 || K > 65536 || kx > 65536) return -1;
    int b = 0, h = 0, bx = 0;
    if (n == 0) {
        const int want = (int)std::ceil(41.0 + 0.5 * std::log2((double)K) - 1e-9);
        n = OZ_MAX_MODULI;
        for (int q = 6; q <= OZ_MAX_MODULI; q++) {
            oz_mod_bits(q, &b, &h, &bx);
            if (b >= want && bx >= 44) {
                n = q;
                break;
            }
        }
    }
    if (n < 6 || n > OZ_MAX_MODULI) return -1;
    oz_mod_bits(n, &b, &h, &bx);
    if (b < 8 || bx < 8 || h < 5) return -1;
    OzScheme s{};
    s.mod = 1;
    s.n = n;
    s.seg = s.segx = 1;
    s.b = b;
    s.bx = bx;
    s.h = h;
    *sch = s;
    return 0;
}

// The rings: pairwise coprime moduli whose prime factors are all 1 mod 4
// (221 = 13 * 17, 205 = 5 * 41; the others are primes), largest first, at
// most 254 so that a rounded residue fits int8.
static const int OZ_RINGS[OZ_RING_MAX] = {241, 233, 229, 221, 205, 197, 193, 181, 173,
                                          157, 149, 137, 113, 109, 101, 97};

// Device constants for operands of b and bx bits: the fewest moduli whose
// product M holds the integer products with one bit of margin,
// log2 M >= max(2b, b + bx) + 2.
int oz_ring_plan(int b, int bx, OzRing *out)
{
    OzRing r{};
    const int bits = std::max(2 * b, b + bx) + 2;
    double lm = 0.0;
    while (r.n < OZ_RING_MAX && lm - 1e-9 < bits) lm += std::log2((double)OZ_RINGS[r.n++]);
    if (lm - 1e-9 < bits) return -1;
    r.b = b;
    r.bx = bx;
    double M = 1.0;
    for (int m = 0; m < r.n; m++) M *= (double)OZ_RINGS[m];
    // |X| / M < 2^-(sh + 2): the window's top bit is still the sign
    r.sh = std::max(0, std::min(20, (int)std::floor(lm - 1e-9 - 2.0 * b - 3.0)));
    r.shx = std::max(0, std::min(20, (int)std::floor(lm - 1e-9 - (double)(b + bx) - 3.0)));
    r.fin = std::ldexp(M, -64 - r.sh - 2 * b);
    r.finx = std::ldexp(M, -64 - r.shx - b - bx);
    for (int m = 0; m < r.n; m++) {
        const int p = OZ_RINGS[m];
        int im = 0;
        while (im < p && (im * im + 1) % p != 0) im++;
        long long mm = 1;   // (M / p) mod p
        for (int q = 0; q < r.n; q++)
            if (q != m) mm = mm * OZ_RINGS[q] % p;
        const int y = oz_inverse_mod(mm, p), half = oz_inverse_mod(2, p), iinv = oz_inverse_mod(im, p);
        if (im >= p || y < 0 || half < 0 || iinv < 0) return -1;
        r.p[m] = p;
        r.mg[m] = (int)((((long long)1 << 32) + p / 2) / p);
        r.inv[m] = 1.0f / (float)p;
        // symmetric residues of 2^(8k) and of i_m 2^(8k), k = 0..6, packed as signed bytes
        auto sym = [p](long long v) { v = ((v % p) + p) % p; return (int)(v > p / 2 ? v - p : v); };
        unsigned c[2] = {0, 0}, ci[2] = {0, 0};
        for (int k = 0; k < 7; k++) {
            const long long w = (1LL << (8 * k)) % p;
            c[k >> 2] |= (unsigned)(uint8_t)(int8_t)sym(w) << (8 * (k & 3));
            ci[k >> 2] |= (unsigned)(uint8_t)(int8_t)sym(w * im) << (8 * (k & 3));
        }
        r.clo[m] = (int)c[0];
        r.chi[m] = (int)c[1];
        r.ilo[m] = (int)ci[0];
        r.ihi[m] = (int)ci[1];
        // -2^55 removes the digits' offset; the sums start at the FP32 bits of a multiple of p near 1.5 2^23
        const int start = 12582912 / p * p;
        r.base[m] = 0x4B000000 - (1 << 23) + start + sym(-((1LL << 55) % p));
        r.icorr[m] = sym(-((1LL << 55) % p) * im);
        // recombination: e_m times the other modulus of the pair (2q, 2q + 1)
        const int other = (m ^ 1) < r.n ? OZ_RINGS[m ^ 1] : 1;
        r.fre[m] = (unsigned)((long long)y * half % p) * (unsigned)other;
        r.fim[m] = (unsigned)((long long)y * half % p * iinv % p) * (unsigned)other;
        if ((m & 1) == 0) {
            const unsigned pq = (unsigned)(p * other);
            const unsigned __int128 d = (((unsigned __int128)1 << 96) + pq / 2) / pq;
            for (int w = 0; w < 3; w++) r.d96[w][m / 2] = (unsigned)(d >> (32 * w));
        }
    }
    *out = r;
    return 0;
}

int ring_kpad(int K) { return (K + RG_CHUNK - 1) / RG_CHUNK * RG_CHUNK; }

size_t ring_slot_bytes(const OzRing &rg, int npad, int kp8, int relativity)
{
    return (size_t)2 * rg.n * ring_narr(relativity) * npad * (size_t)kp8;
}

size_t ring_ho_tile_bytes(const OzRing &rg) { return (size_t)2 * rg.n * RG_BM * 2 * RG_BJ; }

size_t ring_atom_tile_bytes(const OzRing &rg, int nb) { return (size_t)2 * rg.n * RG_BM * nb; }

size_t ring_pace_bytes() { return sizeof(int) * RG_PACE_MAX; }

// Row blocks of the per-atom tiles: rows (h_a rows and lo rows of the largest
// species) in equal blocks of nb <= 256, a multiple of 32 (the MMA's N).
void ring_row_blocks(int rows, int *nb, int *nrows)
{
    const int blocks = (rows + 255) / 256;
    *nb = ((rows + blocks - 1) / blocks + 31) / 32 * 32;
    *nrows = blocks * *nb;
}

cudaError_t launch_oz_norm(const DevParams &p, const KDesc *d_k, int nk, int which, cudaStream_t s)
{
    oz_norm_kernel<<<dim3(p.npad / 32, nk), dim3(32, 32), 0, s>>>(p, d_k, which);
    return cudaGetLastError();
}

cudaError_t launch_ring_split(const DevParams &p, const KDesc *d_k, int nk, const OzRing &rg, int kp8, int which,
                              cudaStream_t s)
{
    constexpr int smem = 2 * RS_LD * (int)sizeof(double);
    static std::atomic<unsigned long long> attr{0};
    cudaError_t e = once_per_device(attr, [] {
        return cudaFuncSetAttribute(oz_ring_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    });
    if (e != cudaSuccess) return e;
    oz_ring_split_kernel<<<dim3(kp8 / RS_F, p.npad / 32, nk), 256, smem, s>>>(p, d_k, rg, kp8, which);
    return cudaGetLastError();
}

cudaError_t launch_ring_x(const DevParams &p, const OzAtomArgs &xa, const OzRing &rg, cudaStream_t s)
{
    oz_ring_x_kernel<<<dim3(xa.nrows / 32, p.natmtot), 256, 0, s>>>(p, xa, rg);
    return cudaGetLastError();
}

// Clusters that can be resident at once (one per SM pair), at most one per
// product of the list.
template <int MODE>
static cudaError_t plane_grid(int ntiles, int np, cudaStream_t s, int *ncl)
{
    static std::atomic<unsigned long long> attr{0};
    cudaError_t e = once_per_device(attr, [] {
        return cudaFuncSetAttribute(oz_plane_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, RG_SMEM);
    });
    if (e != cudaSuccess) return e;
    static std::atomic<int> resident{0};         // the same for every device of this build's architecture
    int act = resident.load(std::memory_order_relaxed);
    if (act == 0) {
        cudaLaunchConfig_t lc = {};
        lc.gridDim = dim3(2 * RG_PACE_MAX);
        lc.blockDim = dim3(RG_THREADS);
        lc.dynamicSmemBytes = RG_SMEM;
        lc.stream = s;
        if (cudaOccupancyMaxActiveClusters(&act, (void *)oz_plane_kernel<MODE>, &lc) != cudaSuccess || act < 1) {
            (void)cudaGetLastError();
            int dev = 0, nsm = 148;
            cudaGetDevice(&dev);
            cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
            act = nsm / 2;
        }
        resident.store(act, std::memory_order_relaxed);
    }
    *ncl = (int)std::min<long long>((long long)ntiles * np, std::min(act, RG_PACE_MAX));
    return cudaSuccess;
}

// H/O: the products of all tiles, then their recombination.  Large problems
// are paced: when the operand planes of one product (three arrays of npad x
// kp8 bytes) exceed RG_PACE_BYTES, clusters that drift apart stream them from
// HBM again and again.
constexpr size_t RG_PACE_BYTES = (size_t)100 << 20;

cudaError_t launch_ring_ho(const CUtensorMap *map, const DevParams &p, const KDesc *d_k, const void *d_tiles,
                           int ntiles, const OzRing &rg, int kp8, uint8_t *res, int *pace, cudaStream_t s)
{
    if (ntiles <= 0) return cudaSuccess;
    int ncl = 0;
    cudaError_t e = plane_grid<RG_HO>(ntiles, 2 * rg.n, s, &ncl);
    if (e != cudaSuccess) return e;
    const bool paced = (size_t)3 * p.npad * kp8 > RG_PACE_BYTES;
    if (paced) {
        e = cudaMemsetAsync(pace, 0, sizeof(int) * ncl, s);
        if (e != cudaSuccess) return e;
    }
    oz_plane_kernel<RG_HO><<<2 * ncl, RG_THREADS, RG_SMEM, s>>>(*map, *map, p, d_k, (const int *)d_tiles, ntiles, rg,
                                                                OzAtomArgs{}, res, paced ? pace : nullptr);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    oz_crt_kernel<<<dim3(2 * ntiles, 2 * (RG_BJ / 8)), 128, 0, s>>>(p, d_k, (const int *)d_tiles, rg, res);
    return cudaGetLastError();
}

// Per-atom products in chunks of tiles whose residues fit the residue buffer.
cudaError_t launch_ring_atom(const CUtensorMap *mapA, const CUtensorMap *mapX, const DevParams &p, const KDesc *d_k,
                             const void *d_tiles, int ntiles, const OzRing &rg, const OzAtomArgs &xa, uint8_t *res,
                             size_t res_bytes, cudaStream_t s)
{
    const int cap = (int)std::min<size_t>(res_bytes / ring_atom_tile_bytes(rg, xa.nb), 1 << 24);
    if (cap < 1) return cudaErrorInvalidValue;
    for (int t0 = 0; t0 < ntiles; t0 += cap) {
        const int nt = std::min(cap, ntiles - t0);
        const int *tiles = (const int *)d_tiles + 4 * (size_t)t0;
        int ncl = 0;
        cudaError_t e = plane_grid<RG_ATOM>(nt, 2 * rg.n, s, &ncl);
        if (e != cudaSuccess) return e;
        oz_plane_kernel<RG_ATOM><<<2 * ncl, RG_THREADS, RG_SMEM, s>>>(*mapA, *mapX, p, d_k, tiles, nt, rg, xa, res,
                                                                      nullptr);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        oz_bcrt_kernel<<<dim3(2 * nt, xa.nb / 8), 128, 0, s>>>(p, d_k, tiles, rg, xa, res);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// TMA views (int8):
//   ho    the planes of all slots as 5D (K byte in a 128-byte chunk, G,
//         array, K chunk, slot x plane), box {128, 128, 1, 2, 1}: 128 G rows of
//         one array, two K chunks, each chunk contiguous in shared memory
//   arow  the same bytes as 4D (K byte, G, array, slot x plane), box {128,
//         128, 1, 1}: a K chunk starting at any multiple of 16 bytes (the atom
//         windows are not chunk aligned)
//   x     the per-atom operands as 4D (K byte in a chunk, row, atom x plane,
//         K chunk), box {128, nb / 2, 1, 1}
// Rows past npad (or past the rows of X) and K chunks past kp8 arrive as zeros.
bool make_ring_maps(void *base, size_t nsp, int npad, int kp8, int narr, void *xbase, size_t xgroups, int nrows,
                    int nb, int lw, CUtensorMap *ho, CUtensorMap *arow, CUtensorMap *x)
{
    typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn)
        return false;
    EncodeFn encode = (EncodeFn)fn;
    if (kp8 % RG_CHUNK != 0 || lw % RG_CHUNK != 0 || nb % 32 != 0) return false;
    const cuuint32_t es[5] = {1, 1, 1, 1, 1};
    auto make = [&](CUtensorMap *m, int rank, void *b, const cuuint64_t *dims, const cuuint64_t *strides,
                    const cuuint32_t *box) {
        return encode(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, rank, b, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                      CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    const cuuint64_t K = kp8, G = npad, A = narr;
    const cuuint64_t dho[5] = {RG_CHUNK, G, A, K / RG_CHUNK, nsp}, sho[4] = {K, G * K, RG_CHUNK, A * G * K};
    const cuuint32_t bho[5] = {RG_CHUNK, 128, 1, RG_KCH, 1};
    const cuuint64_t dar[4] = {K, G, A, nsp}, sar[3] = {K, G * K, A * G * K};
    const cuuint32_t bar[4] = {RG_CHUNK, 128, 1, 1};
    const cuuint64_t L = lw, R = nrows;
    const cuuint64_t dx[4] = {RG_CHUNK, R, xgroups, L / RG_CHUNK}, sx[3] = {L, R * L, RG_CHUNK};
    const cuuint32_t bx[4] = {RG_CHUNK, (cuuint32_t)(nb / 2), 1, 1};
    return make(ho, 5, base, dho, sho, bho) && make(arow, 4, base, dar, sar, bar) && make(x, 4, xbase, dx, sx, bx);
}

}  // namespace exs

extern "C" int exs_ozaki_moduli(int n, int K, int kx, int *n_out, int *p, unsigned long long *c, int *b, int *bx,
                                int *h)
{
    exs::OzScheme s{};
    if (exs::oz_mod_plan(n, K, kx, &s) != 0) return EXS_ERR_ARG;
    if (n_out) *n_out = s.n;
    for (int m = 0; m < s.n; m++) {
        const int pm = exs::OZ_MODULI[m];
        long long mm = 1;   // (M / p) mod p
        for (int q = 0; q < s.n; q++)
            if (q != m) mm = mm * exs::OZ_MODULI[q] % pm;
        const int y = exs::oz_inverse_mod(mm, pm);
        if (y < 0) return EXS_ERR_ARG;
        // round(2^(64+h) y / p) mod 2^64 (y < p < 2^8 and h <= 18: the numerator fits 128 bits)
        const unsigned __int128 num = ((unsigned __int128)y << (64 + s.h)) + (unsigned)(pm / 2);
        if (p) p[m] = pm;
        if (c) c[m] = (unsigned long long)(num / (unsigned)pm);
    }
    if (b) *b = s.b;
    if (bx) *bx = s.bx;
    if (h) *h = s.h;
    return EXS_OK;
}
