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
// whatever K.  b and bx are the plan's (oz_mod_plan, exs_ozaki_moduli), the
// moduli below exs_ozaki_rings'.
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
// tiles is A_P^T h_P.  n moduli make 2n products of two operands each: at
// b = 49, bx = 45 14 moduli (104.4 bits) and 28 products for H and O, 13 and 26
// for the per-atom products, where 13 larger moduli (101.8 bits) with real and
// imaginary planes take 52.
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
constexpr int RG_EPI = 16;                       // epilogue warps of a CTA
constexpr int RG_THREADS = 128 + 32 * RG_EPI;    // see the roles below
constexpr int RG_BM = 256;                       // tile rows of a CTA pair
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

// The residue bytes of E (8 or 16) elements to os (x + i_m y) and od (x - i_m y).
template <int E>
__device__ __forceinline__ void ring_emit(const OzRing &rg, int m, const uint2 (&x)[E], const uint2 (&y)[E], int8_t *os,
                                          int8_t *od)
{
    uint32_t ws[E / 4], wd[E / 4];
#pragma unroll
    for (int q = 0; q < E / 4; q++) {
        uint32_t s[4], d[4];
#pragma unroll
        for (int e = 0; e < 4; e++) ring_pair(rg, m, x[4 * q + e], y[4 * q + e], s[e], d[e]);
        ws[q] = pack4(s[0], s[1], s[2], s[3]);
        wd[q] = pack4(d[0], d[1], d[2], d[3]);
    }
    if constexpr (E == 16) {
        *reinterpret_cast<uint4 *>(os) = make_uint4(ws[0], ws[1], ws[2], ws[3]);
        *reinterpret_cast<uint4 *>(od) = make_uint4(wd[0], wd[1], wd[2], wd[3]);
    } else {
        *reinterpret_cast<uint2 *>(os) = make_uint2(ws[0], ws[1]);
        *reinterpret_cast<uint2 *>(od) = make_uint2(wd[0], wd[1]);
    }
}

__device__ __forceinline__ uint2 ring_digits(double x, double sc)
{
    const unsigned long long u = (unsigned long long)(__double2ll_rn(x * sc) + (1ll << 55));
    return make_uint2((uint32_t)u, (uint32_t)(u >> 32));
}

// Column 2-norms of one operand (which = 0: A, 1: B, 2: C) into its oz_scale
// block.  One column per thread column of a 32 x 32 block, the rows of threads
// covering interleaved rows (stride 32), the partial sums combined in a fixed
// order, so that the scales, and every result, are the same from run to run.
// The factor 1 + 2^-30 covers the rounding of a sum of squares.
// PARTS: the rows are the sums of squares that the operand's producer left in
// oz_part (A: one per atom; B: one per 16 rows of an atom, `per` of them);
// else the planes themselves are read again (C, and B when it comes from the
// FP64 products): 64 atoms 201 us, from the parts 7 and 16 us.
template <bool PARTS>
__global__ void __launch_bounds__(1024) oz_norm_kernel(DevParams p, const KDesc *ks, int which, int per)
{
    __shared__ double part[32][33];
    const KDesc k = ks[blockIdx.y];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int g = blockIdx.x * 32 + tx;
    double s = 0.0;
    if (g < k.ngp) {
        if (PARTS) {
#pragma unroll 4
            for (int r = ty; r < p.natmtot * per; r += 32)
                if (per == 1 || r % per * 16 < p.atoms[r / per].napw) s += k.oz_part[(size_t)r * p.npad + g];
        } else {
            const double *pr, *pi;
            oz_operand(k, which, pr, pi);
#pragma unroll 4
            for (int f = ty; f < p.K; f += 32) {
                const size_t i = (size_t)f * p.npad + g;
                const double xr = pr[i], xi = pi[i];
                s = fma(xr, xr, fma(xi, xi, s));
            }
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
// transposed reads over the banks.  Bound by HBM and the residue arithmetic
// (14 moduli: about 230 instructions per complex element): 27 k-points of the
// eight-atom cell 0.55 ms, 0.40 of it without the arithmetic; eight elements per
// thread and twice the warps: 0.74 ms.
constexpr int RS_F = 128, RS_E = 16;             // tile rows f; elements per thread
constexpr int RS_THREADS = 32 * RS_F / RS_E;
constexpr int RS_LD = RS_F * 33 + 2 * (RS_F / RS_E);
__device__ __forceinline__ int rs_at(int f, int g) { return f * 33 + 2 * (f / RS_E) + g; }

__global__ void __launch_bounds__(RS_THREADS, 2) oz_ring_split_kernel(DevParams p, const KDesc *ks,
                                                                      const __grid_constant__ OzRing rg, int kp8,
                                                                      int which)
{
    extern __shared__ __align__(16) double rs_t[];       // [re, im][RS_LD]
    const KDesc k = ks[blockIdx.z];
    const int f0 = blockIdx.x * RS_F, g0 = blockIdx.y * 32;
    if (g0 >= k.ngp) return;                             // columns that no output reads
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;      // 32 x 8
    const double *pr, *pi;
    oz_operand(k, which, pr, pi);
    {
        constexpr int R = RS_THREADS / 32, NQ = RS_F / R;
        const int g = g0 + tx;
        double vr[NQ], vi[NQ];
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const int f = f0 + ty + R * q;
            const bool v = f < p.K && g < k.ngp;
            const size_t i = (size_t)f * p.npad + g;
            vr[q] = v ? pr[i] : 0.0;
            vi[q] = v ? pi[i] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            rs_t[rs_at(ty + R * q, tx)] = vr[q];
            rs_t[RS_LD + rs_at(ty + R * q, tx)] = vi[q];
        }
    }
    __syncthreads();
    const int gl = threadIdx.x / (RS_F / RS_E), fl = threadIdx.x % (RS_F / RS_E) * RS_E;
    const int g = g0 + gl, f = f0 + fl;
    // 1/sigma is a power of two: the scaling is exact
    const double sc = ldexp(1.0 / oz_sigma(k.oz_scale[(size_t)which * p.npad + g]), rg.b);
    uint2 x[RS_E], y[RS_E];
#pragma unroll
    for (int e = 0; e < RS_E; e++) {
        x[e] = ring_digits(rs_t[rs_at(fl + e, gl)], sc);
        y[e] = ring_digits(rs_t[RS_LD + rs_at(fl + e, gl)], sc);
    }
    const int narr = ring_narr(p.relativity), arr = which == 0 ? 1 : (which == 1 ? 0 : 2);
    const size_t plane = (size_t)narr * p.npad * kp8;
    // plane 2m: A-, B+, C+; plane 2m + 1: A+, B-, C-
    int8_t *os = k.oz_slices + ((size_t)arr * p.npad + g) * kp8 + f + (which == 0 ? plane : 0);
    int8_t *od = k.oz_slices + ((size_t)arr * p.npad + g) * kp8 + f + (which == 0 ? 0 : plane);
#pragma unroll 1
    for (int m = 0; m < rg.n; m++, os += 2 * plane, od += 2 * plane) ring_emit(rg, m, x, y, os, od);
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
// of one atom's X, 64 window bytes per block (blockIdx.y): every block forms
// the norms again (interleaved f', fixed order; the operands are in the L2), then
// transposes its step through shared memory.  Latency: eight atoms 34 us (50
// with one block walking the whole window).
__global__ void __launch_bounds__(256) oz_ring_x_kernel(DevParams p, OzAtomArgs xa, const __grid_constant__ OzRing rg)
{
    __shared__ double t[2][64][33];
    __shared__ double part[8][33];
    const int ias = blockIdx.z, n0 = blockIdx.x * 32, k0 = blockIdx.y * 64;
    const AtomDesc &at = p.atoms[ias];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int napw = at.napw, delta = at.apw_off - at.oz_x0;
    double s = 0.0;
#pragma unroll 8
    for (int fp = ty; fp < napw; fp += 8) {
        double re, im;
        ring_x_value(xa, at, ias, n0 + tx, fp, re, im);
        s = fma(re, re, fma(im, im, s));
    }
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const int k = ty + 8 * q;
        ring_x_value(xa, at, ias, n0 + tx, k0 + k - delta, t[0][k][tx], t[1][k][tx]);
    }
    part[ty][tx] = s;
    __syncthreads();
    const int nl = threadIdx.x >> 3, kl = (threadIdx.x & 7) * 8;
    double v = 0.0;
    for (int q = 0; q < 8; q++) v += part[q][nl];
    v = oz_sigma(sqrt(v) * (1.0 + 0x1p-30));
    if (k0 == 0 && kl == 0) xa.xsig[(size_t)ias * xa.nrows + n0 + nl] = v;
    const double sc = ldexp(1.0 / v, rg.bx);
    uint2 x[8], y[8];
#pragma unroll
    for (int e = 0; e < 8; e++) {
        x[e] = ring_digits(t[0][kl + e][nl], sc);
        y[e] = ring_digits(t[1][kl + e][nl], sc);
    }
    const size_t plane = (size_t)xa.nrows * xa.lw;
    int8_t *out = xa.xs + ((size_t)ias * 2 * rg.at.n * xa.nrows + n0 + nl) * xa.lw + k0 + kl;
#pragma unroll 1
    for (int m = 0; m < rg.at.n; m++, out += 2 * plane) ring_emit(rg, m, x, y, out + plane, out);   // h+, h-
}

// ------------------------------------------------------------ the products
// A cluster of two CTAs forms tiles of 256 rows with tcgen05.mma.cta_group::2
// (M = 256): each CTA holds its own 128 rows of the A operand and half of the
// N rows of each B operand.
//   RG_HO    tiles {k, ib, jb}: 256 G_i x 128 G_j, one MMA of N = 256: CTA 0
//            holds B_P, CTA 1 A_(P^1) (C_P with iora*) of the G_j; columns
//            0..127 of the sums are H, 128..255 O
//   RG_WIDE  tiles {k, ib, jb}: 256 G_i x 256 G_j, two MMAs of N = 256 on the
//            same A operand, one for H and one for O
//   RG_ATOM  tiles {k, atom, ib, xb}: 256 G x nb rows of h_a and loa of one
//            atom (N = nb rounded up to 32; the rows past nb belong to the next
//            tile), over the atom's K window
// The work list is flat in (tile, plane): while full rounds of one tile per
// cluster last, a cluster takes a tile and walks its 2n planes; the (tile,
// plane) pairs of the remaining tiles are dealt out in equal shares, so that a
// handful of tiles (two for a k-point of the two-atom cell) still occupies
// every SM pair and the last round is never short of more than one product.
// Two accumulators in tensor memory.  RG_HO, RG_ATOM: products take them in
// turn, the MMAs of one run while the epilogue reduces the previous one.
// RG_WIDE: every product fills both, and the epilogue frees H while O waits.
//
// Roles (640 threads): warps 0, 1 (and 2) TMA producers of the A and B (O)
// operands, warp 3 MMA issuer (CTA 0) and tensor-memory owner, warps 4-19
// epilogue: four per tensor-memory lane quadrant, every fourth chunk of 16
// columns each, whose residues leave as 16 bytes per row, 512 contiguous
// bytes per warp.  (Eight warps: 4 % slower on the per-atom products,
// where the reduction of a short product is a chain of latencies.)
// CTA 0's full barriers count the bytes of both CTAs' copies; MMA completion
// is committed to both CTAs; both epilogues report to CTA 0's barrier.
// Every wait is bounded and gives up when another role of the CTA gave up.
// The issuer always waits for its last MMAs; once all roles are out, a CTA in
// which one gave up records DEV_ERR_TIMEOUT and lets its copies land, then
// tensor memory is freed.
//
// What bounds it: the power cap while K is long (64 atoms, N = 8075, K =
// 10,368: 13.9 - 14.6 ms from box to box, 2.8 POP/s, the SM clock down to
// 1.5 GHz; the form with real and imaginary planes, 13 moduli and 256 x 64
// tiles took 23.1 ms); HBM for the per-atom products (64 atoms 1.25 ms, the 27
// k-points of the eight-atom cell 0.89 ms at about 4 TB/s of residues out
// and operands in).  H/O of the 27 k-points 1.5 - 1.6 ms (was 2.65).
enum : int { RG_HO = 0, RG_ATOM = 1, RG_WIDE = 2 };

template <int MODE>
struct RingCfg {
    static constexpr bool WIDE = MODE == RG_WIDE;
    static constexpr int KCH = WIDE ? 1 : 2;             // K chunks per stage
    static constexpr int NB = WIDE ? 2 : 1;              // B operands (accumulators per product)
    static constexpr int OPER = KCH * RG_BOX;            // one operand of a stage
    static constexpr int STAGE = (1 + NB) * OPER;        // this CTA's A rows, then its half of each B
    static constexpr int NST = WIDE ? 4 : 3;             // 192 KB in all
    static constexpr int SMEM = NST * STAGE + 1024;
    static constexpr int BJ = WIDE ? 256 : 128;          // H/O tile columns
};

// Pacing of large H/O launches (pace != null): every cluster publishes, every
// RG_PACE_CHUNKS K chunks it issues, its step count in pace[cluster] and waits
// until the slowest cluster is at most RG_PACE_LAG steps behind, so that the
// tiles running at one time read the same row and column blocks within a few
// MB of each other's position and the L2 serves the repeats.  The wait is a
// hint, not a dependency: it gives up after RG_PACE_CYCLES (a cluster that is
// not resident, or a slow one, delays the others by that much per step at
// most) and never raises an error.  A finished cluster publishes INT_MAX.
constexpr int RG_PACE_CHUNKS = 32;
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

// An arrival that orders nothing but the tensor-memory reads before it.  Those
// need no release: the warp waits for its loads (tcgen05.wait::ld), every lane
// fences them (tcgen05.fence::before_thread_sync), and an mbarrier arrival and a
// wait, both relaxed at cluster scope, with the issuer's after_thread_sync order
// them before its MMAs (the pattern that PTX gives for tcgen05.ld and MMAs in
// different threads).  A release would make the warp wait until its residue
// stores are performed (per-atom products of 64 atoms: 2.19 ms with release, 1.36 ms
// without; with a release ahead of the product's own stores, all columns
// loaded first, 27 k-points of the eight-atom cell still 6.06 against 5.62 ms).
__device__ __forceinline__ void mbar_arrive_relaxed(uint32_t cluster_addr)
{
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(cluster_addr) : "memory");
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

// The flat work list of cluster c, walked by every role: np products of each
// of its full-round tiles, then its share of the (tile, plane) pairs of the
// remaining tiles: by planes (H/O), so that the clusters work on the same plane
// of all these tiles at a time and share its operands in the L2 (dealt out in
// runs, every cluster on another plane, each streams its own from HBM:
// three k-points of 16 atoms 836 us, by planes 766), or in one run of planes per cluster (per-atom
// tiles, which share little and whose producers then look a tile up once).
template <bool RUNS>
struct RingUnits {
    int ncl, np, count, tile, P, full_end, rest, rest_tile, rest_P;
    __host__ __device__ RingUnits(int ntiles, int ncl_, int np_, int c) : ncl(ncl_), np(np_)
    {
        const int full = ntiles / ncl;
        full_end = full * ncl;
        rest = ntiles - full_end;
        const int pairs = rest * np;                       // rest < ncl
        const int first = RUNS ? (int)((long long)pairs * c / ncl) : c;
        const int mine = RUNS ? (int)((long long)pairs * (c + 1) / ncl) - first : (pairs - c + ncl - 1) / ncl;
        const int div = rest > 0 ? rest : 1;
        count = full * np + mine;
        rest_tile = full_end + (RUNS ? first / np : first % div);
        rest_P = RUNS ? first % np : first / div;
        tile = full > 0 ? c : rest_tile;
        P = full > 0 ? 0 : rest_P;
    }
    __host__ __device__ void next()
    {
        if (tile >= full_end) {                            // among the remaining tiles
            if (RUNS) {
                if (++P < np) return;
                P = 0;
                tile++;
            } else {
                const int v = tile - full_end + ncl;       // ncl pairs on
                P += v / rest;
                tile = full_end + v % rest;
            }
            return;
        }
        if (++P < np) return;
        P = 0;
        tile += ncl;
        if (tile >= full_end) {
            tile = rest_tile;
            P = rest_P;
        }
    }
};

// Residue bytes of an int32 sum |v| < 2^30: q = floor(v mg / 2^32), mg =
// round(2^32 / p), leaves v - q p in [-p/4, 5p/4]; the unsigned minima add or
// take p.
__device__ __forceinline__ uint32_t ring_mod(int v, int p, int mg)
{
    uint32_t x = (uint32_t)(v - __mulhi(v, mg) * p);
    x = min(x, x + (uint32_t)p);
    return min(x, x - (uint32_t)p);
}

// The same for |v| < 2^27 (K <= RG_SHORT_K, |residue| <= 123) in half the
// instructions: with x = v + up, up = the multiple of p just above 2^27, and
// mf = floor(2^32 / p), q = floor(x mf / 2^32) is at most floor(x / p), and
// x - q p <= p + p f / 16, f = frac(2^32 / p): at most 246 for every modulus
// of the table, a byte, though not always below p (the recombination takes
// any representative below 2 p).
constexpr int RG_SHORT_K = 8192;
__device__ __forceinline__ uint32_t ring_mod_short(int v, int p, uint32_t mf, int up)
{
    const uint32_t x = (uint32_t)(v + up);
    return x - __umulhi(x, mf) * (uint32_t)p;
}

template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(RG_THREADS, 1)
oz_plane_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, DevParams p,
                int slot0, const int *tiles, int ntiles, const __grid_constant__ OzRing rg, OzAtomArgs xa,
                uint8_t *res, int *pace)
{
    using C = RingCfg<MODE>;
    constexpr int NST = C::NST, KCH = C::KCH;
    extern __shared__ __align__(1024) uint8_t rg_smem[];
    __shared__ uint64_t full[NST], empty[NST], accf[2], acce[2];
    __shared__ uint32_t tmem_sh;
    __shared__ int abort_sh;
    volatile int *abort = &abort_sh;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_ctarank();
    const uint32_t sbase = (smem_u32(rg_smem) + 1023u) & ~1023u;
    const int cl = (int)(blockIdx.x >> 1), NP = 2 * (MODE == RG_ATOM ? rg.at.n : rg.n);
    RingUnits<MODE == RG_ATOM> units(ntiles, (int)(gridDim.x >> 1), NP, cl);
    const int N = MODE == RG_ATOM ? (xa.nb + 31) / 32 * 32 : 256;         // MMA N
    const int b_rows = N / 2;                            // operand rows of a B operand in this CTA

    if (warp == 3) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_sh)),
                     "r"(OZ_TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::);
    }
    if (tid == 0) {
        for (int q = 0; q < NST; q++) {
            mbar_init(&full[q], 1);      // CTA 0: one arrive (with the bytes of both CTAs)
            mbar_init(&empty[q], 1);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(&accf[a], 1);
            mbar_init(&acce[a], 2 * RG_EPI);     // CTA 0: the epilogue warps of both CTAs
        }
        abort_sh = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                  // the peer's barriers are initialised before anyone signals them
    tc_fence_after();
    const uint32_t tbase = tmem_sh;

    if (warp < 1 + C::NB) {
        // ------------------------------------------------ TMA producers (both CTAs)
        if (lane == 0) {
            const int role = warp;       // 0: this CTA's A rows, 1 (2): this CTA's half of B (of O's operand)
            uint32_t fills[NST];
#pragma unroll
            for (int q = 0; q < NST; q++) fills[q] = 0;
            int st = 0, chunks = 0, last = -1;
            bool bad = false;
            const bool pacer = pace != nullptr && rank == 0 && role == 0;
            int slot = 0, row = 0, arr = 1, flip = 0, x0 = 0, nch = (p.K + RG_CHUNK - 1) / RG_CHUNK;
            if (MODE != RG_ATOM && role > 0) {           // H: B_P; O: A_(P^1), or C_P with iora*
                const bool o = C::WIDE ? role == 2 : rank == 1;
                arr = !o ? 0 : (p.relativity == EXS_REL_IORA ? 2 : 1);
                flip = o && arr == 1 ? 1 : 0;
            }
            // H/O: the next product's tile entries are loaded during the current one (among the remaining
            // tiles every product has another tile)
            auto entry = [&](int tile, int q) { return units.count > 0 ? tiles[3 * tile + q] : 0; };
            int k_next = 0, b_next = 0;
            if (MODE != RG_ATOM) {
                k_next = entry(units.tile, 0);
                b_next = entry(units.tile, role == 0 ? 1 : 2);
            }
            auto ahead = units;
            for (int u = 0; u < units.count && !bad; u++, units.next()) {
                const int tile = units.tile, P = units.P;
                if (MODE != RG_ATOM) {
                    slot = slot0 + k_next;
                    row = role == 0 ? b_next * RG_BM + (int)rank * 128 : b_next * C::BJ + (C::WIDE ? (int)rank * 128 : 0);
                    if (u + 1 < units.count) {
                        ahead.next();
                        k_next = entry(ahead.tile, 0);
                        b_next = entry(ahead.tile, role == 0 ? 1 : 2);
                    }
                } else if (tile != last) {      // dependent loads, once per tile
                    last = tile;
                    const int ias = tiles[4 * tile + 1];
                    const AtomDesc &at = p.atoms[ias];
                    nch = at.oz_nch;
                    if (role == 0) {
                        slot = slot0 + tiles[4 * tile];
                        row = tiles[4 * tile + 2] * RG_BM + (int)rank * 128;
                        x0 = at.oz_x0;
                    } else {
                        slot = ias;
                        row = tiles[4 * tile + 3] * xa.nb + (int)rank * b_rows;
                    }
                }
                // planes per slot of the split operands, per atom of h_a and loa
                const int plane = slot * (MODE == RG_ATOM && role > 0 ? NP : 2 * rg.n) + (P ^ flip);
                for (int kb = 0; kb < nch; kb += KCH, chunks += KCH) {
                    if (pacer && chunks % RG_PACE_CHUNKS == 0) ring_pace(pace, cl, units.ncl, chunks / RG_PACE_CHUNKS);
                    if (fills[st] > 0 && !mbar_wait_ab(&empty[st], (fills[st] - 1) & 1, abort, rg.wait)) {
                        bad = true;
                        break;
                    }
                    const int nc = min(KCH, nch - kb);
                    const uint32_t bar = smem_u32(&full[st]);
                    const uint32_t dst = sbase + st * C::STAGE + role * C::OPER;
                    if (MODE != RG_ATOM) {               // one box of KCH chunks (zeros past the last one)
                        if (rank == 0 && role == 0) mbar_expect_tx(&full[st], 2 * C::STAGE);
                        tma_load_5d_2sm(dst, &mapA, 0, row, arr, kb, plane, bar);
                    } else {
                        if (rank == 0 && role == 0)
                            mbar_expect_tx(&full[st], 2 * nc * (RG_BOX + b_rows * RG_CHUNK));
                        for (int c = 0; c < nc; c++) {
                            if (role == 0)
                                tma_load_4d_2sm(dst + c * RG_BOX, &mapA, x0 + (kb + c) * RG_CHUNK, row, 1, plane, bar);
                            else
                                tma_load_4d_2sm(dst + c * RG_BOX, &mapB, 0, row, plane, kb + c, bar);
                        }
                    }
                    fills[st]++;
                    st = (st + 1 == NST) ? 0 : st + 1;
                }
            }
            if (pacer) st_relaxed_gpu(pace + cl, 0x7fffffff);     // done: nobody waits for this cluster
        }
    } else if (warp == 3) {
        // ------------------------------------------------ MMA issuer (CTA 0)
        if (lane == 0 && rank == 0) {
            const uint32_t idesc = umma_idesc_i8(256, N);
            uint32_t uses[NST];
#pragma unroll
            for (int q = 0; q < NST; q++) uses[q] = 0;
            int st = 0, last = -1;
            int steps = (p.K + 31) / 32;                  // K steps of 32 bytes
            bool bad = false;
            for (int u = 0; u < units.count && !bad; u++, units.next()) {
                const int buf = C::WIDE ? 0 : u & 1, use = C::WIDE ? u : u >> 1;
                if (MODE == RG_ATOM) {
                    const int tile = units.tile;
                    if (tile != last) {
                        last = tile;
                        const AtomDesc &at = p.atoms[tiles[4 * tile + 1]];
                        steps = (at.apw_off - at.oz_x0 + at.napw + 31) / 32;
                    }
                }
                for (int k0 = 0; k0 < steps; k0 += KCH * 4) {
                    if (!mbar_wait_ab(&full[st], uses[st] & 1, abort, rg.wait)) {
                        bad = true;
                        break;
                    }
#pragma unroll
                    for (int o = 0; o < C::NB; o++) {
                        // the epilogues of both CTAs must have read this accumulator's previous product
                        if (k0 == 0 && use > 0 && !mbar_wait_ab<true>(&acce[buf + o], (use - 1) & 1, abort, rg.wait)) {
                            bad = true;
                            if (o > 0) {             // H's MMAs of this stage are under way: commit them too
                                umma_commit_2sm(&empty[st]);
                                uses[st]++;
                            }
                            break;
                        }
                        tc_fence_after();
                        const uint32_t sa = sbase + st * C::STAGE, sb = sa + (1 + o) * C::OPER;
#pragma unroll
                        for (int q = 0; q < KCH * 4; q++)
                            if (k0 + q < steps) {
                                const uint32_t off = (q >> 2) * RG_BOX + (q & 3) * 32;
                                umma_i8_2sm(tbase + (uint32_t)((buf + o) * RG_ACC), umma_desc_sw128(sa + off),
                                            umma_desc_sw128(sb + off), idesc, k0 + q > 0 ? 1u : 0u);
                            }
                        if (C::WIDE && k0 + KCH * 4 >= steps) umma_commit_2sm(&accf[o]);   // H first, then O
                    }
                    if (bad) break;
                    umma_commit_2sm(&empty[st]);
                    uses[st]++;
                    st = (st + 1 == NST) ? 0 : st + 1;
                }
                if (!C::WIDE && !bad) umma_commit_2sm(&accf[buf]);
            }
            // every MMA is done before the pair may go away, also when only an epilogue gave up
            for (int q = 0; q < NST; q++)
                if (uses[q] > 0) mbar_drain(&empty[q], (uses[q] - 1) & 1);
        }
    } else if (warp >= 4) {
        // ------------------------------------------------ epilogue (both CTAs, warps 4..19)
        const int qd = warp & 3, part = (warp - 4) >> 2;
        const int row = qd * 32 + lane;
        int nq = N / 16, last = -1;                                 // 16-column chunks of an accumulator
        const uint32_t acce0[2] = {mapa_shared(smem_u32(&acce[0]), 0), mapa_shared(smem_u32(&acce[1]), 0)};
        // residues of one product, this CTA's 128 rows
        const size_t plane_bytes = (size_t)(MODE == RG_ATOM ? xa.nb : C::NB * N) * 128;
        bool bad = false;
        for (int u = 0; u < units.count && !bad; u++, units.next()) {
            const int P = units.P, m = P >> 1;
            if (MODE == RG_ATOM && units.tile != last) {            // only the chunks that hold rows of the atom
                last = units.tile;
                const AtomDesc &at = p.atoms[tiles[4 * last + 1]];
                nq = min(xa.nb, at.napw + at.losize - tiles[4 * last + 3] * xa.nb + 15) / 16;
            }
            const int pm = rg.p[m], mg = rg.mg[m], up = rg.up[m];
            const uint32_t mf = rg.mf[m];
            uint8_t *out = res + ((size_t)(2 * units.tile + (int)rank) * NP + P) * plane_bytes + (size_t)row * 16;
#pragma unroll
            for (int o = 0; o < C::NB; o++) {
                const int buf = C::WIDE ? o : u & 1, use = C::WIDE ? u : u >> 1;
                if (!__all_sync(0xffffffffu, mbar_wait_ab(&accf[buf], use & 1, abort, rg.wait))) {
                    bad = true;
                    break;
                }
                tc_fence_after();
                const uint32_t tacc = tbase + ((uint32_t)(qd * 32) << 16) + (uint32_t)(buf * RG_ACC);
                uint8_t *po = out + (size_t)o * N * 128;
                // 16 columns at a time, the next 16 on their way while these are reduced
                auto put = [&](const uint32_t (&v)[16], int c) {
                    uint32_t w[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        uint32_t x[4];
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            x[e] = C::WIDE ? ring_mod((int)v[4 * q + e], pm, mg)
                                           : ring_mod_short((int)v[4 * q + e], pm, mf, up);
                        w[q] = pack4(x[0], x[1], x[2], x[3]);
                    }
                    *reinterpret_cast<uint4 *>(po + (size_t)c * 128 * 16) = make_uint4(w[0], w[1], w[2], w[3]);
                };
                uint32_t v0[16], v1[16];
                if (part < nq) tm_ld16(tacc + part * 16, v0);
                for (int c = part; c < nq; c += 8) {
                    tm_wait_ld();
                    if (c + 4 < nq) tm_ld16(tacc + (c + 4) * 16, v1);
                    put(v0, c);
                    if (c + 4 < nq) {
                        tm_wait_ld();
                        if (c + 8 < nq) tm_ld16(tacc + (c + 8) * 16, v0);
                        put(v1, c + 4);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_relaxed(acce0[buf]);     // CTA 0's barrier (also from CTA 0)
            }
        }
    }
    tc_fence_before();
    __syncthreads();                     // every role is out: the flag is final
    if (*abort) {                        // if CTA 0's issuer gave up, CTA 1's epilogue misses a product and does too
        if (tid == 0) atomicOr(p.err, DEV_ERR_TIMEOUT);
        abort_settle();
    }
    cluster_sync_all();                  // neither CTA leaves while the pair still uses its memory
    if (warp == 3) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tbase), "r"(OZ_TMEM_COLS));
    }
}

// ------------------------------------------------------------ recombination
// The residue words of four columns of one row: z+ of modulus m in plane
// 2m + first, z- in the other.
struct RingWords {
    uint32_t p[OZ_RING_MAX], m[OZ_RING_MAX];
};

__device__ __forceinline__ void ring_load4(const uint8_t *tres, size_t plane, int n, int first, RingWords &w)
{
#pragma unroll
    for (int m = 0; m < OZ_RING_MAX; m++) {
        w.p[m] = w.m[m] = 0u;
        if (m < n) {
            w.p[m] = *reinterpret_cast<const uint32_t *>(tres + (size_t)(2 * m + first) * plane);
            w.m[m] = *reinterpret_cast<const uint32_t *>(tres + (size_t)(2 * m + 1 - first) * plane);
        }
    }
}

// Real and imaginary parts of four values from their residues z+, z- (any
// representatives in [0, 255]).  X / M = sum_m s_m e_m / p_m (mod 1) with
// s_m = z+ + z-, e_m = y_m / 2 mod p_m for the real parts, s_m = z+ - z-,
// e_m = y_m / (2 i_m) mod p_m for the imaginary parts, y_m = (M / p_m)^-1.
// Two moduli p, p' at a time: w = s_m (e_m p') + s_m' (e_m' p) with both
// weights reduced to symmetric residues mod p p' (|.| < 2^15), in two signed
// bytes: two dot products with the bytes z+, z-, z+', z-' of the value, the
// low one started at a multiple of p p' that keeps 0 <= w < 2^27.  Then
// t += w D (mod 2^96), D = round(2^(96+sh) / (p p')) mod 2^96: three 32 x
// 32-bit multiply-adds (the top one needs 32 bits only) per PAIR of moduli,
// carries propagated once at the end.  The top sh bits of 2^96 X / M are copies
// of its sign, so the top 64 bits of t as a signed integer are 2^(64+sh) X / M
// up to the rounding of D (below 2^29 units of 2^-96).
__device__ __forceinline__ void ring_crt4(const OzCrt &rg, const RingWords &z, double (&re)[4], double (&im)[4])
{
    unsigned long long a0[8], a1[8];                    // re 0..3, im 0..3
    uint32_t a2[8];
#pragma unroll
    for (int e = 0; e < 8; e++) {
        a0[e] = a1[e] = 0ull;
        a2[e] = 0u;
    }
#pragma unroll
    for (int q = 0; q < OZ_RING_MAX / 2; q++) {
        if (2 * q >= rg.n) break;
        // bytes (z+, z-, z+', z-') of each value: a 4 x 4 byte transpose
        const uint32_t t0 = __byte_perm(z.p[2 * q], z.m[2 * q], 0x5140), t1 = __byte_perm(z.p[2 * q], z.m[2 * q], 0x7362);
        const uint32_t u0 = __byte_perm(z.p[2 * q + 1], z.m[2 * q + 1], 0x5140),
                       u1 = __byte_perm(z.p[2 * q + 1], z.m[2 * q + 1], 0x7362);
        const uint32_t b[4] = {__byte_perm(t0, u0, 0x5410), __byte_perm(t0, u0, 0x7632), __byte_perm(t1, u1, 0x5410),
                               __byte_perm(t1, u1, 0x7632)};
        const uint32_t d0 = rg.d96[0][q], d1 = rg.d96[1][q], d2 = rg.d96[2][q];
#pragma unroll
        for (int e = 0; e < 8; e++) {
            const int c = e >> 2;                       // 0: real part, 1: imaginary part
            const uint32_t w = (uint32_t)(dp4a_us(b[e & 3], rg.wlo[c][q], rg.woff[q]) +
                                          256 * dp4a_us(b[e & 3], rg.whi[c][q], 0));
            a0[e] += (unsigned long long)w * d0;
            a1[e] += (unsigned long long)w * d1;
            a2[e] += w * d2;
        }
    }
#pragma unroll
    for (int e = 0; e < 8; e++) {
        const unsigned long long c1 = a1[e] + (a0[e] >> 32);
        const unsigned long long top = ((unsigned long long)(a2[e] + (uint32_t)(c1 >> 32)) << 32) | (uint32_t)c1;
        const double v = (double)(long long)top * rg.fin;
        if (e < 4)
            re[e] = v;
        else
            im[e - 4] = v;
    }
}

// Recombination, scaling, interstitial term and store of the H/O tiles: a
// block of four warps takes 32 rows x 16 columns of both matrices.  First lane
// l of a warp recombines row l / 4 of its eight, columns 4 (l % 4) .. + 3, so a
// warp reads 128 contiguous residue bytes per plane, and stages the values in
// shared memory.  Then a lane takes a row and every fourth column: the index of
// G_i - G_j, looked up once for H and O before the recombination, and the table
// entries, all in flight together; the values leave as whole column segments,
// 512 bytes of the upper triangle, 256 bytes of the mirror.  The blocks of a
// tile follow each other, so that the pieces of a column meet in the L2 before
// they go to HBM.  Bound by the residue reads and the H/O writes: 27 k-points of
// the eight-atom cell 0.48 ms, 64 atoms 1.19 ms (0.52 and 1.31 with the column
// groups launched apart, 0.88 and 2.18 with one thread per row and eight
// columns and the mirror stored from registers).
constexpr int RC_R = 32, RC_C = 16;

template <int BJ>
__global__ void __launch_bounds__(128) oz_crt_kernel(DevParams p, const KDesc *ks, const int *tiles,
                                                     const __grid_constant__ OzRing rg, const uint8_t *res)
{
    __shared__ exs_complex T[2][RC_R][RC_C + 1];
    __shared__ double sv[RC_R + RC_C][3], ssig[RC_R + 2 * RC_C];
    __shared__ int siv[RC_R + RC_C][3];
    constexpr int NR = RG_BM / RC_R, NC = RC_C / 4;              // row groups of a tile; columns of a lane
    constexpr int NB = BJ / RC_C;                                // column groups, fastest: see above
    const int cgrp = blockIdx.x % NB, rgrp = blockIdx.x / NB % NR, tile = blockIdx.x / (NB * NR);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const KDesc kd = ks[tiles[3 * tile]];
    const int i0 = tiles[3 * tile + 1] * RG_BM + rgrp * RC_R;
    const int j0 = tiles[3 * tile + 2] * BJ + cgrp * RC_C;
    if (i0 >= kd.ngp || j0 >= kd.ngp || j0 + RC_C - 1 < i0) return;    // no element i <= j < ngp here
    constexpr size_t plane = 2 * BJ * 128;
    const int r = warp * 8 + (lane >> 2), cq = lane & 3;
    const int row = (rgrp * RC_R & 127) + r;                     // of the 128-row tile
    const uint8_t *tres = res + (size_t)(2 * tile + rgrp * RC_R / 128) * 2 * rg.n * plane +
                          ((size_t)cgrp * 128 + row) * 16 + cq * 4;
    RingWords z;
    ring_load4(tres, plane, rg.n, 0, z);                         // H
    if (tid < RC_R + RC_C) {                                     // G vectors and scales of the rows and columns
        const int g = tid < RC_R ? i0 + tid : j0 + tid - RC_R;
        if (g < kd.ngp) {
            int ig = kd.igpig[g] - 1;
            if (ig < 0 || ig >= p.ngrtot) {
                atomicOr(p.err, DEV_ERR_INDEX);
                ig = 0;
            }
            for (int x = 0; x < 3; x++) {
                siv[tid][x] = p.ivg[3 * ig + x];
                sv[tid][x] = kd.vgpc[3 * g + x];
            }
            if (tid < RC_R) {
                ssig[tid] = oz_sigma(kd.oz_scale[g]);
            } else {   // H: sigma_B(j); O: sigma_A(j), or sigma_C(j) with iora* (O = A^H C)
                ssig[tid] = oz_sigma(kd.oz_scale[p.npad + g]);
                ssig[tid + RC_C] = oz_sigma(kd.oz_scale[(p.relativity == EXS_REL_IORA ? 2 * p.npad : 0) + g]);
            }
        }
    }
    __syncthreads();
    const int i = i0 + lane;                                     // this lane's row of the second part
    int ig[NC];
#pragma unroll
    for (int q = 0; q < NC; q++) {
        const int c = warp + 4 * q, j = j0 + c;
        ig[q] = i <= j && j < kd.ngp ? interstitial_index(p, siv[lane], siv[RC_R + c]) : 0;
    }
#pragma unroll
    for (int w = 0; w < 2; w++) {
        double re[4], im[4];
        ring_crt4(rg.ho, z, re, im);
        if (w == 0) ring_load4(tres + (size_t)BJ * 128, plane, rg.n, 0, z);      // O
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const double sc = ssig[r] * ssig[RC_R + w * RC_C + cq * 4 + e];
            exs_complex v;
            v.re = re[e] * sc;
            v.im = im[e] * sc;
            T[w][r][cq * 4 + e] = v;
        }
    }
    // the interstitial terms of this lane's elements
    double2 hi[NC], oi[NC];
#pragma unroll
    for (int q = 0; q < NC; q++) {
        hi[q] = oi[q] = make_double2(0.0, 0.0);
        if (ig[q] > 0) {
            const int c = RC_R + warp + 4 * q;
            interstitial_value(p, EPI_HAM, ig[q], sv[lane], sv[c], hi[q].x, hi[q].y);
            interstitial_value(p, EPI_OVL, ig[q], sv[lane], sv[c], oi[q].x, oi[q].y);
        }
    }
    __syncthreads();
    const size_t nm = (size_t)kd.nmat;
#pragma unroll
    for (int q = 0; q < NC; q++) {                               // upper: lane = row
        const int c = warp + 4 * q, j = j0 + c;
        if (j < kd.ngp && i <= j) {
            exs_complex h = T[0][lane][c], o = T[1][lane][c];
            if (ig[q] > 0) {
                h.re += hi[q].x;
                h.im += hi[q].y;
                o.re += oi[q].x;
                o.im += oi[q].y;
                T[0][lane][c] = h;
                T[1][lane][c] = o;
            }
            kd.h[(size_t)i + nm * j] = h;
            kd.o[(size_t)i + nm * j] = o;
        }
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 2; w++) {
        exs_complex *out = w == 0 ? kd.h : kd.o;
#pragma unroll
        for (int q = 0; q < RC_R / 8; q++) {                     // mirror: lanes = two rows of 16 columns
            const int rr = warp * 8 + 2 * q + (lane >> 4), ii = i0 + rr, j = j0 + (lane & 15);
            if (j < kd.ngp && ii < j) {
                exs_complex v = T[w][rr][lane & 15];
                v.im = -v.im;
                out[(size_t)j + nm * ii] = v;
            }
        }
    }
}

// Recombination of the per-atom tiles, organised like oz_crt_kernel (32 G x
// 16 rows of X per block): the B planes, 256 contiguous bytes per row, and the
// APW-lo rows of H with their mirror.  64 atoms 1.04 ms (one thread per G and
// eight rows: 1.36 ms); 27 k-points of the eight-atom cell 0.71 ms, 0.47 of it
// without the arithmetic.
__global__ void __launch_bounds__(128, 6) oz_bcrt_kernel(DevParams p, const KDesc *ks, const int *tiles,
                                                      const __grid_constant__ OzRing rg, OzAtomArgs xa,
                                                      const uint8_t *res)
{
    __shared__ double T[2][RC_R][RC_C + 1], ssq[4][32];
    constexpr int NR = RG_BM / RC_R;
    const int tile = blockIdx.x / NR, rgrp = blockIdx.x % NR;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const KDesc kd = ks[tiles[4 * tile]];
    const int ias = tiles[4 * tile + 1];
    const int g0 = tiles[4 * tile + 2] * RG_BM + rgrp * RC_R;
    const int n0 = tiles[4 * tile + 3] * xa.nb + blockIdx.y * RC_C;
    const AtomDesc &at = p.atoms[ias];
    const int napw = at.napw, nrow = at.napw + at.losize;
    if (g0 >= kd.ngp || n0 >= nrow) return;
    const size_t plane = (size_t)xa.nb * 128;
    const int r = warp * 8 + (lane >> 2), cq = lane & 3;
    const int row = (rgrp * RC_R & 127) + r;
    RingWords z;
    ring_load4(res + (size_t)(2 * tile + rgrp * RC_R / 128) * 2 * rg.at.n * plane +
                   ((size_t)blockIdx.y * 128 + row) * 16 + cq * 4,
               plane, rg.at.n, 1, z);
    const double sa = g0 + r < kd.ngp ? oz_sigma(kd.oz_scale[g0 + r]) : 0.0;
    const double *sig = xa.xsig + (size_t)ias * xa.nrows + n0 + cq * 4;
    double re[4], im[4];
    ring_crt4(rg.at, z, re, im);
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const double sc = sa * sig[e];
        T[0][r][cq * 4 + e] = re[e] * sc;
        T[1][r][cq * 4 + e] = im[e] * sc;
    }
    __syncthreads();
    const int g = g0 + lane;
    const size_t row0 = (size_t)kd.ngp + at.lo_off, nm = (size_t)kd.nmat;
#pragma unroll
    for (int q = 0; q < RC_C / 4; q++) {                         // lane = G
        const int c = warp + 4 * q, n = n0 + c;
        if (g >= kd.ngp) continue;
        if (n < napw) {
            const size_t off = (size_t)(at.apw_off + n) * p.npad + g;
            kd.br[off] = T[0][lane][c];
            kd.bi[off] = T[1][lane][c];
        } else if (n < nrow) {
            exs_complex v;
            v.re = T[0][lane][c];
            v.im = -T[1][lane][c];
            kd.h[(size_t)g + nm * (row0 + n - napw)] = v;
        }
    }
    // sums of squares of the B columns over this block's rows: the warps' parts in order
    if (n0 < napw) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < RC_C / 4; q++) {
            const int c = warp + 4 * q;
            if (n0 + c < napw) s = fma(T[0][lane][c], T[0][lane][c], fma(T[1][lane][c], T[1][lane][c], s));
        }
        ssq[warp][lane] = s;
        __syncthreads();
        if (warp == 0 && g < kd.ngp)
            kd.oz_part[((size_t)ias * (xa.nrows / RC_C) + n0 / RC_C) * p.npad + g] =
                ((ssq[0][lane] + ssq[1][lane]) + ssq[2][lane]) + ssq[3][lane];
    }
    if (n0 + RC_C > napw) {                                      // lo rows: lanes = two G of 16 rows
#pragma unroll
        for (int q = 0; q < RC_R / 8; q++) {
            const int rr = warp * 8 + 2 * q + (lane >> 4), n = n0 + (lane & 15), gg = g0 + rr;
            if (gg < kd.ngp && n >= napw && n < nrow) {
                exs_complex v;
                v.re = T[0][rr][lane & 15];
                v.im = T[1][rr][lane & 15];
                kd.h[(row0 + n - napw) + nm * gg] = v;
            }
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

// The recombination constants of products of `bits` bits: the fewest moduli
// whose product M holds them with one bit of margin, log2 M >= bits + 2.
static int oz_crt_plan(int bits, OzCrt *out)
{
    OzCrt r{};
    double lm = 0.0, M = 1.0;
    while (r.n < OZ_RING_MAX && lm - 1e-9 < bits + 2) {
        lm += std::log2((double)OZ_RINGS[r.n]);
        M *= (double)OZ_RINGS[r.n++];
    }
    if (lm - 1e-9 < bits + 2) return -1;
    // |X| / M < 2^-(sh + 2): the window's top bit is still the sign
    r.sh = std::max(0, std::min(20, (int)std::floor(lm - 1e-9 - (double)bits - 3.0)));
    r.fin = std::ldexp(M, -64 - r.sh - bits);
    for (int m = 0; m < r.n; m++) {
        const int p = OZ_RINGS[m];
        int im = 0;
        while (im < p && (im * im + 1) % p != 0) im++;
        long long mm = 1;   // (M / p) mod p
        for (int q = 0; q < r.n; q++)
            if (q != m) mm = mm * OZ_RINGS[q] % p;
        const int y = oz_inverse_mod(mm, p), half = oz_inverse_mod(2, p), iinv = oz_inverse_mod(im, p);
        if (im >= p || y < 0 || half < 0 || iinv < 0) return -1;
        // e_m times the other modulus of the pair (2q, 2q + 1), symmetric mod their product, as signed bytes
        // 256 h + l for z+ (and, negated for the imaginary parts, z-); an odd count leaves the last pair half
        // empty: weight 0
        const int other = (m ^ 1) < r.n ? OZ_RINGS[m ^ 1] : 1, pq = p * other, q = m / 2, sft = 16 * (m & 1);
        for (int c = 0; c < 2; c++) {
            long long f = (long long)y * half % p * (c ? iinv : 1) % p * other;
            if (f > pq / 2) f -= pq;
            for (int w = 0; w < 2; w++) {                // z+, z-
                const int v = (int)(c && w ? -f : f);
                const int l = (int)(int8_t)(uint8_t)(v & 255), h = (v - l) / 256;
                if (h < -128 || h > 127) return -1;
                r.wlo[c][q] |= (int)((unsigned)(uint8_t)(int8_t)l << (sft + 8 * w));
                r.whi[c][q] |= (int)((unsigned)(uint8_t)(int8_t)h << (sft + 8 * w));
            }
        }
        if ((m & 1) == 0) {
            r.woff[q] = (((1 << 26) + pq - 1) / pq) * pq;   // |w| <= 4 * 255 * 2^15 < 2^26 before the offset
            const unsigned __int128 d = (((unsigned __int128)1 << (96 + r.sh)) + pq / 2) / pq;
            for (int w = 0; w < 3; w++) r.d96[w][q] = (unsigned)(d >> (32 * w));       // mod 2^96
        }
    }
    *out = r;
    return 0;
}

// Device constants for operands of b and bx bits: the moduli of the H/O
// products (2b bits) and of the per-atom products (b + bx bits; 13 of the 14 at
// b = 49, bx = 45: 7 % fewer products and residues than with all of them).
int oz_ring_plan(int b, int bx, OzRing *out)
{
    OzRing r{};
    if (oz_crt_plan(2 * b, &r.ho) != 0 || oz_crt_plan(b + bx, &r.at) != 0) return -1;
    r.n = std::max(r.ho.n, r.at.n);
    r.b = b;
    r.bx = bx;
    for (int m = 0; m < r.n; m++) {
        const int p = OZ_RINGS[m];
        int im = 0;
        while (im < p && (im * im + 1) % p != 0) im++;
        if (im >= p) return -1;
        r.p[m] = p;
        r.mg[m] = (int)((((long long)1 << 32) + p / 2) / p);
        r.mf[m] = (unsigned)((1LL << 32) / p);
        r.up[m] = ((1 << 27) / p + 1) * p;
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
    }
    *out = r;
    return 0;
}

// Columns of the H/O tiles.  256-column tiles read three quarters of the
// operand bytes per product, but their epilogue stops the MMAs once per
// product: 0.85 against 0.81 ms at K = 2592 (16 atoms, 3 k), 1.68 against
// 1.49 ms at K = 1936, 13.9 against 14.3 ms at K = 10,368.  Up to RG_SHORT_K
// the 128-column tiles also have the short residue reduction.
int ring_ho_cols(int K) { return K > RG_SHORT_K ? 256 : 128; }

int ring_kpad(int K) { return (K + RG_CHUNK - 1) / RG_CHUNK * RG_CHUNK; }

size_t ring_slot_bytes(const OzRing &rg, int npad, int kp8, int relativity)
{
    return (size_t)2 * rg.n * ring_narr(relativity) * npad * (size_t)kp8;
}

size_t ring_ho_tile_bytes(const OzRing &rg, int cols) { return (size_t)2 * rg.n * RG_BM * 2 * cols; }

size_t ring_atom_tile_bytes(const OzRing &rg, int nb) { return (size_t)2 * rg.at.n * RG_BM * nb; }

size_t ring_pace_bytes() { return sizeof(int) * RG_PACE_MAX; }

// Row blocks of the per-atom tiles: rows (h_a rows and lo rows of the largest
// species) in as few blocks of nb <= 256 rows as hold them, nb a multiple of 16.
// (In multiples of the MMA's 32 the 269 rows of the eight-atom cell went 160 + 109:
// every other cluster had the long tiles, and the two that share A drifted apart.)
void ring_row_blocks(int rows, int *nb, int *nrows)
{
    const int blocks = (rows + 255) / 256;
    *nb = ((rows + blocks - 1) / blocks + 15) / 16 * 16;
    *nrows = (blocks * *nb + 31) / 32 * 32;
}

size_t ring_part_rows(int natmtot, int nrows) { return (size_t)natmtot * (nrows / RC_C); }

cudaError_t launch_oz_norm(const DevParams &p, const KDesc *d_k, int nk, int which, int per, cudaStream_t s)
{
    const dim3 grid(p.npad / 32, nk), block(32, 32);
    if (per > 0)
        oz_norm_kernel<true><<<grid, block, 0, s>>>(p, d_k, which, per);
    else
        oz_norm_kernel<false><<<grid, block, 0, s>>>(p, d_k, which, 0);
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
    oz_ring_split_kernel<<<dim3(kp8 / RS_F, p.npad / 32, nk), RS_THREADS, smem, s>>>(p, d_k, rg, kp8, which);
    return cudaGetLastError();
}

cudaError_t launch_ring_x(const DevParams &p, const OzAtomArgs &xa, const OzRing &rg, cudaStream_t s)
{
    oz_ring_x_kernel<<<dim3(xa.nrows / 32, xa.lw / 64, p.natmtot), 256, 0, s>>>(p, xa, rg);
    return cudaGetLastError();
}

// Clusters that can be resident at once (one per SM pair), at most one per
// product of the list.
template <int MODE>
static cudaError_t plane_grid(int ntiles, int np, cudaStream_t s, int *ncl)
{
    static std::atomic<unsigned long long> attr{0};
    cudaError_t e = once_per_device(attr, [] {
        return cudaFuncSetAttribute(oz_plane_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, RingCfg<MODE>::SMEM);
    });
    if (e != cudaSuccess) return e;
    static std::atomic<int> resident{0};         // the same for every device of this build's architecture
    int act = resident.load(std::memory_order_relaxed);
    if (act == 0) {
        cudaLaunchConfig_t lc = {};
        lc.gridDim = dim3(2 * RG_PACE_MAX);
        lc.blockDim = dim3(RG_THREADS);
        lc.dynamicSmemBytes = RingCfg<MODE>::SMEM;
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

// H/O: the products, then their recombination, in equal chunks of tiles whose
// residues fit the residue buffer (one chunk up to 4 GB of them).  Large problems
// are paced: when the operand planes of one product (three arrays of npad x
// kp8 bytes) exceed RG_PACE_BYTES, clusters that drift apart stream them from
// HBM again and again.
constexpr size_t RG_PACE_BYTES = (size_t)100 << 20;

template <int MODE>
static cudaError_t launch_ho(const CUtensorMap *map, const DevParams &p, const KDesc *d_k, int slot0,
                             const int *d_tiles, int ntiles, const OzRing &rg, int kp8, uint8_t *res, size_t res_bytes,
                             int *pace, cudaStream_t s)
{
    using C = RingCfg<MODE>;
    const int cap = (int)std::min<size_t>(res_bytes / ring_ho_tile_bytes(rg, C::BJ), 1 << 24);
    if (cap < 1) return cudaErrorInvalidValue;
    const int nchunk = (ntiles + cap - 1) / cap, chunk = (ntiles + nchunk - 1) / nchunk;
    const bool paced = (size_t)3 * p.npad * kp8 > RG_PACE_BYTES;
    for (int t0 = 0; t0 < ntiles; t0 += chunk) {
        const int nt = std::min(chunk, ntiles - t0);
        const int *tiles = d_tiles + 3 * (size_t)t0;
        int ncl = 0;
        cudaError_t e = plane_grid<MODE>(nt, 2 * rg.n, s, &ncl);
        if (e == cudaSuccess && paced) e = cudaMemsetAsync(pace, 0, sizeof(int) * ncl, s);
        if (e != cudaSuccess) return e;
        oz_plane_kernel<MODE><<<2 * ncl, RG_THREADS, C::SMEM, s>>>(*map, *map, p, slot0, tiles, nt, rg, OzAtomArgs{}, res,
                                                                   paced ? pace : nullptr);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        oz_crt_kernel<C::BJ><<<(unsigned)nt * (RG_BM / RC_R) * (C::BJ / RC_C), 128, 0, s>>>(p, d_k, tiles, rg, res);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_ring_ho(int cols, const CUtensorMap *map1, const CUtensorMap *map2, const DevParams &p,
                           const KDesc *d_k, int slot0, const void *d_tiles, int ntiles, const OzRing &rg, int kp8,
                           uint8_t *res, size_t res_bytes, int *pace, cudaStream_t s)
{
    if (ntiles <= 0) return cudaSuccess;
    const int *t = (const int *)d_tiles;
    return cols == 256 ? launch_ho<RG_WIDE>(map1, p, d_k, slot0, t, ntiles, rg, kp8, res, res_bytes, pace, s)
                       : launch_ho<RG_HO>(map2, p, d_k, slot0, t, ntiles, rg, kp8, res, res_bytes, pace, s);
}

// Per-atom products in chunks of tiles whose residues fit the residue buffer.
cudaError_t launch_ring_atom(const CUtensorMap *mapA, const CUtensorMap *mapX, const DevParams &p, const KDesc *d_k,
                             int slot0, const void *d_tiles, int ntiles, const OzRing &rg, const OzAtomArgs &xa, uint8_t *res,
                             size_t res_bytes, cudaStream_t s)
{
    const int cap = (int)std::min<size_t>(res_bytes / ring_atom_tile_bytes(rg, xa.nb), 1 << 24);
    if (cap < 1) return cudaErrorInvalidValue;
    for (int t0 = 0; t0 < ntiles; t0 += cap) {
        const int nt = std::min(cap, ntiles - t0);
        const int *tiles = (const int *)d_tiles + 4 * (size_t)t0;
        int ncl = 0;
        cudaError_t e = plane_grid<RG_ATOM>(nt, 2 * rg.at.n, s, &ncl);
        if (e != cudaSuccess) return e;
        oz_plane_kernel<RG_ATOM><<<2 * ncl, RG_THREADS, RingCfg<RG_ATOM>::SMEM, s>>>(*mapA, *mapX, p, slot0, tiles, nt, rg, xa, res,
                                                                      nullptr);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        oz_bcrt_kernel<<<dim3(nt * (RG_BM / RC_R), xa.nb / RC_C), 128, 0, s>>>(p, d_k, tiles, rg, xa, res);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// TMA views (int8):
//   ho1, ho2  the planes of all slots as 5D (K byte in a 128-byte chunk, G,
//         array, K chunk, slot x plane), boxes {128, 128, 1, 1 or 2, 1}: 128 G
//         rows of one array, one or two K chunks, each contiguous in shared memory
//   arow  the same bytes as 4D (K byte, G, array, slot x plane), box {128,
//         128, 1, 1}: a K chunk starting at any multiple of 16 bytes (the atom
//         windows are not chunk aligned)
//   x     the per-atom operands as 4D (K byte in a chunk, row, atom x plane,
//         K chunk), box {128, N / 2, 1, 1}, N = nb rounded up to 32
// Rows past npad (or past the rows of X) and K chunks past kp8 arrive as zeros.
bool make_ring_maps(void *base, size_t nsp, int npad, int kp8, int narr, void *xbase, size_t xgroups, int nrows,
                    int nb, int lw, CUtensorMap *ho1, CUtensorMap *ho2, CUtensorMap *arow, CUtensorMap *x)
{
    typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn)
        return false;
    EncodeFn encode = (EncodeFn)fn;
    if (kp8 % RG_CHUNK != 0 || lw % RG_CHUNK != 0 || nb % 16 != 0) return false;
    const cuuint32_t es[5] = {1, 1, 1, 1, 1};
    auto make = [&](CUtensorMap *m, int rank, void *b, const cuuint64_t *dims, const cuuint64_t *strides,
                    const cuuint32_t *box) {
        return encode(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, rank, b, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                      CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    const cuuint64_t K = kp8, G = npad, A = narr;
    const cuuint64_t dho[5] = {RG_CHUNK, G, A, K / RG_CHUNK, nsp}, sho[4] = {K, G * K, RG_CHUNK, A * G * K};
    const cuuint32_t bho1[5] = {RG_CHUNK, 128, 1, 1, 1}, bho2[5] = {RG_CHUNK, 128, 1, 2, 1};
    const cuuint64_t dar[4] = {K, G, A, nsp}, sar[3] = {K, G * K, A * G * K};
    const cuuint32_t bar[4] = {RG_CHUNK, 128, 1, 1};
    const cuuint64_t L = lw, R = nrows;
    const cuuint64_t dx[4] = {RG_CHUNK, R, xgroups, L / RG_CHUNK}, sx[3] = {L, R * L, RG_CHUNK};
    const cuuint32_t bx[4] = {RG_CHUNK, (cuuint32_t)((nb + 31) / 32 * 16), 1, 1};
    return make(ho1, 5, base, dho, sho, bho1) && make(ho2, 5, base, dho, sho, bho2) &&
           make(arow, 4, base, dar, sar, bar) && make(x, 4, xbase, dx, sx, bx);
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

extern "C" int exs_ozaki_rings(int n, int K, int kx, int *n_ho, int *n_atom, int *p)
{
    exs::OzScheme s{};
    exs::OzRing r{};
    if (exs::oz_mod_plan(n, K, kx, &s) != 0 || exs::oz_ring_plan(s.b, s.bx, &r) != 0) return EXS_ERR_ARG;
    if (n_ho) *n_ho = r.n;
    if (n_atom) *n_atom = r.at.n;
    for (int m = 0; p && m < r.n; m++) p[m] = r.p[m];
    return EXS_OK;
}
