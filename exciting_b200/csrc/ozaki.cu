// Split-precision MT contraction on the 5th-gen tensor cores (tcgen05.mma
// kind::i8, int32 accumulators in tensor memory) from int8 slices (Ozaki
// scheme).  The modular scheme, the default of the benchmark, is in
// oz_ring.cu.
//
// H = A^H B and O = A^H A in real arithmetic: with the real and imaginary
// planes of A and B,
//   Re H = Ar^T Br + Ai^T Bi    Im H = Ar^T Bi - Ai^T Br
//   Re O = Ar^T Ar + Ai^T Ai    Im O = Ar^T Ai - Ai^T Ar
// so one B operand tile [Br | Bi | Ar | Ai] (32 columns G_j each, N = 128)
// against the two A operands Ar and Ai (two int32 accumulators r and i)
// yields all four: Re H = r0 + i1, Im H = r1 - i0, Re O = r2 + i3,
// Im O = r3 - i2 (rq = block q of accumulator r).
//
// Every column G of A (and of B) is scaled by a power of two sigma(G) >
// max|column| and cut into S int8 slices of 7 bits each by truncation,
//   x = sigma * sum_s q_s 2^{-7s} + rest,  |q_s| <= 127,  |rest| < sigma 2^{-7S}
// (exact in FP64).  The product keeps the slice pairs s + t <= S + 1.  Pairs
// are accumulated in int32 in segments short enough to be exact (the pairs of
// one diagonal d = s + t in groups of P with P * K * 127^2 < 2^31), and each
// finished segment is added in FP64 as 2^{-7d} times its int32 sums to an
// FP64 accumulator that also lives in tensor memory.  The final epilogue
// multiplies by sigma_A(i) sigma_B(j), adds the interstitial term and writes
// the upper triangle and its conjugate mirror, as the FP64 path does.
//
// Slice storage (int8, K contiguous, K padded to kp8 = multiple of 256):
//   [slot][slice][array: Br, Bi, Ar, Ai][G (npad rows)][kp8]
// viewed by TMA as 5D (K byte in a 128-byte chunk, G, array, K chunk,
// slot x slice), so that both A operands of a stage (Ar and Ai, 128 G rows
// each) are ONE box and the B operand (32 G rows of all four arrays) is
// another: two boxes per stage.  Rows past npad fall outside the view and
// arrive as zeros.  Boxes are written with 128-byte swizzling; the MMA
// descriptors use the matching SWIZZLE_128B K-major layout (8-row x 128-byte
// atoms, 1024 B between 8-row groups, K advanced 32 bytes per MMA).
//
// Configurations (chosen per problem by the autotuner): KCH K chunks per
// stage x NST stages, 192 KB in all: (2, 2) or (1, 4) for the H/O tiles;
// one CTA per tile or a persistent grid of one CTA per SM, for the H/O tiles
// and the per-atom tiles separately.
//
// Roles (one CTA per 128 x 32 output tile, 384 threads):
//   warps 0-1  one TMA producer thread each (the A box and the B box of a stage)
//   warp 3     MMA issuer (one thread); allocates tensor memory
//   warps 4-11 epilogue: segment folds and the final store, two warps per
//              tensor-memory lane quadrant, each with two of the four value
//              blocks (H/O tiles: half 0 Re H, Im H, half 1 Re O, Im O;
//              per-atom tiles: half h the re and im blocks of rows 32h..32h+31)
// The same kernel (MODE OZ_ATOM) forms the per-atom products B_a = h_a A_a
// and the APW-lo rows loa_a A_a from int8 slices of h_a and loa.
// Tensor memory (512 columns): r at [0,128), i at [128,256), the FP64 running
// sums (two 32-bit columns per value) at [256,512).  With one tile per CTA the H/O tile's conjugate
// mirror is staged in the stage buffers (idle by then) and written as whole
// columns.  Every wait on an mbarrier is
// bounded (about one second) and gives up early once another role has given
// up; the kernel then records an error, lets its own copies and MMAs drain
// (bounded), frees tensor memory and returns.
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "exs_internal.cuh"
#include "interstitial.cuh"
#include "tcgen05.cuh"

namespace exs {

constexpr int OZ_BM = 128;                       // tile rows (G_i)
constexpr int OZ_BJ = 32;                        // tile columns (G_j); MMA N = 4 * OZ_BJ
constexpr int OZ_N = 4 * OZ_BJ;
constexpr int OZ_NARR = 4;                       // Br, Bi, Ar, Ai (the B box: four arrays)
constexpr int OZ_CHUNK = 128;                    // bytes of K in one swizzle row
constexpr int OZ_TILE = 128 * OZ_CHUNK;          // 16 KB: one K chunk of a 128-row operand
constexpr int OZ_THREADS = 384;                  // 12 warps: see the roles below
constexpr int OZ_MAX_KCH = 2;                    // K chunks per stage of the widest configuration
constexpr int OZ_FP64_COL = 256;

// ------------------------------------------------------------ preparation
// Arrays of one slice of a slot: Br, Bi, Ar, Ai, or with iora* (O = A^H C,
// C = (I + h1aa) A) Br, Bi, Cr, Ci, Ar, Ai, so that the B box is always the
// first four arrays and the A operand the last two.
__host__ __device__ __forceinline__ int oz_narr(int relativity) { return relativity == EXS_REL_IORA ? 6 : 4; }

// Byte offset of (slice s, array a, row G, K index f) inside one slot.
__device__ __forceinline__ size_t oz_off(int s, int a, int g, int f, int npad, int kp8, int narr)
{
    return (((size_t)s * narr + a) * npad + g) * (size_t)kp8 + f;
}

__device__ __forceinline__ void oz_put(uint32_t (&o0)[16], uint32_t (&o1)[16], int e, uint32_t w0, uint32_t w1)
{
    if (e < 8) {
        o0[2 * e] = w0;
        o0[2 * e + 1] = w1;
    } else {
        o1[2 * (e - 8)] = w0;
        o1[2 * (e - 8) + 1] = w1;
    }
}

// Fold 16 finished int32 sums of diagonal g (slices) into the FP64 running
// sums (two 32-bit tensor-memory words each, low word first; lo / hi hold
// the previous values unless init): a += 2^{-7(g+2)} (r + sg i), r + sg i
// exact in FP64, one rounding per fold.
__device__ __forceinline__ void oz_fold16(int g, bool init, int sg, const uint32_t (&rv)[16], const uint32_t (&iv)[16],
                                          const uint32_t (&lo)[16], const uint32_t (&hi)[16], uint32_t (&o0)[16],
                                          uint32_t (&o1)[16])
{
    const double scale = ldexp(1.0, -7 * (g + 2));
    const double sgd = (double)sg;
#pragma unroll
    for (int e = 0; e < 16; e++) {
        double a = 0.0;
        if (!init) {
            const uint32_t w0 = e < 8 ? lo[2 * e] : hi[2 * (e - 8)];
            const uint32_t w1 = e < 8 ? lo[2 * e + 1] : hi[2 * (e - 8) + 1];
            a = __hiloint2double((int)w1, (int)w0);
        }
        a += scale * ((double)(int)rv[e] + sgd * (double)(int)iv[e]);
        oz_put(o0, o1, e, (uint32_t)__double2loint(a), (uint32_t)__double2hiint(a));
    }
}

// Value blocks of an epilogue half: H/O tiles {2h, 2h + 1} (Re H, Im H or
// Re O, Im O); per-atom tiles {h, h + 2} (re and im of rows 32h..32h+31).
template <int MODE>
__device__ __forceinline__ int oz_block(int half, int k)
{
    return MODE == OZ_HO ? 2 * half + k : half + 2 * k;
}

// Final store of one row of a 128 x 32 H/O tile by epilogue half `half`:
// half 0 writes H (Re H, Im H scaled by sigma_A(i) sigma_B(j), plus the
// hmlistln term), half 1 writes O (sigma_A(i) sigma_A(j), plus olpistln);
// the upper triangle and its conjugate mirror, like the FP64 path.  With
// T (shared memory, OZ_MIRROR_LD x 64 values) the mirror values go to
// T[(half * 32 + j - j0) * OZ_MIRROR_LD + row] instead, for oz_store_mirror.
constexpr int OZ_MIRROR_LD = 129;                 // 16-byte values; odd stride: no bank conflicts

__device__ __forceinline__ void oz_store_ho(const DevParams &p, const KDesc &kd, int i0, int j0,
                                            uint32_t t_lane, int row, int half, exs_complex *T)
{
    const int i = i0 + row;
    int ivi[3] = {0, 0, 0};
    double vi[3] = {0.0, 0.0, 0.0};
    const bool row_ok = i < kd.ngp;
    if (row_ok) {
        int g = kd.igpig[i] - 1;
        if (g < 0 || g >= p.ngrtot) {
            atomicOr(p.err, DEV_ERR_INDEX);
            g = 0;
        }
        for (int x = 0; x < 3; x++) {
            ivi[x] = p.ivg[3 * g + x];
            vi[x] = kd.vgpc[3 * i + x];
        }
    }
    const double sai = row_ok ? oz_sigma(kd.oz_scale[i]) : 0.0;
    const int kind = half == 0 ? EPI_HAM : EPI_OVL;
    exs_complex *out = half == 0 ? kd.h : kd.o;
    // H: sigma_B(j); O: sigma_A(j), or sigma_C(j) with iora* (O = A^H C)
    const double *scol = kd.oz_scale + (half == 0 ? p.npad : (p.relativity == EXS_REL_IORA ? 2 * p.npad : 0));
#pragma unroll 1
    for (int jc = 0; jc < OZ_BJ; jc += 8) {
        double val[2][8];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            uint32_t w[16];
            tm_ld16(t_lane + OZ_FP64_COL + 2 * ((2 * half + k) * 32 + jc), w);
            tm_wait_ld();
#pragma unroll
            for (int e = 0; e < 8; e++) val[k][e] = __hiloint2double((int)w[2 * e + 1], (int)w[2 * e]);
        }
        if (!row_ok) continue;
#pragma unroll
        for (int e = 0; e < 8; e++) {
            const int j = j0 + jc + e;
            if (j >= kd.ngp || i > j) continue;
            // column data (the same for the whole warp: broadcast loads)
            int gj = kd.igpig[j] - 1;
            if (gj < 0 || gj >= p.ngrtot) {
                atomicOr(p.err, DEV_ERR_INDEX);
                gj = 0;
            }
            const int ivj[3] = {p.ivg[3 * gj], p.ivg[3 * gj + 1], p.ivg[3 * gj + 2]};
            const double vj[3] = {kd.vgpc[3 * j], kd.vgpc[3 * j + 1], kd.vgpc[3 * j + 2]};
            const double sj = oz_sigma(scol[j]);
            double re = val[0][e] * sai * sj, im = val[1][e] * sai * sj;
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
                if (T)
                    T[(half * 32 + jc + e) * OZ_MIRROR_LD + row] = v;
                else
                    out[(size_t)j + (size_t)kd.nmat * i] = v;
            }
        }
    }
}

// The staged mirror of a 128 x 32 H/O tile, written as whole columns: the
// 256 (matrix, row i) pairs are split over the eight epilogue warps (ew =
// 0..7); lane l writes element (j0 + l, i), so each warp store covers 32
// consecutive rows of one column (512 contiguous bytes).
__device__ __forceinline__ void oz_store_mirror(const KDesc &kd, int i0, int j0, const exs_complex *T, int ew, int lane)
{
    const int j = j0 + lane;
#pragma unroll 4
    for (int q = 0; q < 32; q++) {
        const int pr = ew * 32 + q, h = pr >> 7, il = pr & 127;
        const int i = i0 + il;
        if (i < kd.ngp && j < kd.ngp && i < j)
            (h ? kd.o : kd.h)[(size_t)j + (size_t)kd.nmat * i] = T[(h * 32 + lane) * OZ_MIRROR_LD + il];
    }
}

// Column maxima of |re|, |im| of the C planes (iora*), whose producer raises
// none, into oz_scale block 2.  One column per thread column of a 32 x 8
// block, the eight rows of threads covering interleaved rows f (stride 8).
__global__ void __launch_bounds__(256) oz_colmax_kernel(DevParams p, const KDesc *ks)
{
    __shared__ double part[8][33];
    const KDesc k = ks[blockIdx.y];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int g = blockIdx.x * 32 + tx;
    double s = 0.0;
    if (g < k.ngp) {
#pragma unroll 4
        for (int f = ty; f < p.K; f += 8) {
            const size_t i = (size_t)f * p.npad + g;
            s = fmax(s, fmax(fabs(k.cr[i]), fabs(k.ci[i])));
        }
    }
    part[ty][tx] = s;
    __syncthreads();
    if (ty == 0 && g < p.npad) {
        double t = 0.0;
        for (int q = 0; q < 8; q++) t = fmax(t, part[q][tx]);
        k.oz_scale[(size_t)2 * p.npad + g] = t;
    }
}

// The S slices of one operand (which = 0: A into the last two arrays of the
// slot; 1: B into arrays 0, 1; 2: C into arrays 2, 3 (iora*)).
// A 64(f) x 32(G) tile per block, transposed through shared memory: reads
// G-contiguous planes (a warp reads 32 consecutive G; 16 loads per thread in
// flight), writes K-contiguous int8 rows eight bytes per thread (8 threads
// cover the tile's 64 K bytes of one G row).
constexpr int SPLIT_F = 64;

__global__ void __launch_bounds__(256) oz_split_kernel(DevParams p, const KDesc *ks,
                                                       const __grid_constant__ OzScheme sch, int kp8, int which)
{
    const int S = sch.n;
    __shared__ double t[2][SPLIT_F][33];
    const KDesc k = ks[blockIdx.z];
    const int f0 = blockIdx.x * SPLIT_F, g0 = blockIdx.y * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;      // 32 x 8
    const int narr = oz_narr(p.relativity);
    const int a0 = which == 0 ? narr - 2 : (which == 1 ? 0 : 2);
    const double *pr, *pi;
    oz_operand(k, which, pr, pi);
    {
        double vr[SPLIT_F / 8], vi[SPLIT_F / 8];
#pragma unroll
        for (int q = 0; q < SPLIT_F / 8; q++) {
            const int f = f0 + ty + 8 * q, g = g0 + tx;
            const bool v = f < p.K && g < k.ngp;
            const size_t i = (size_t)f * p.npad + g;
            vr[q] = v ? pr[i] : 0.0;
            vi[q] = v ? pi[i] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < SPLIT_F / 8; q++) {
            t[0][ty + 8 * q][tx] = vr[q];
            t[1][ty + 8 * q][tx] = vi[q];
        }
    }
    __syncthreads();
    const int tid = ty * 32 + tx;
    const int gl = tid >> 3, fl = (tid & 7) * 8;
    const int g = g0 + gl, f = f0 + fl;
    if (g >= p.npad || f >= kp8) return;
    // 1/sigma is a power of two: the scaling is exact
    const double rs = 1.0 / oz_sigma(k.oz_scale[(size_t)which * p.npad + g]);
    // The slices are the base-128 digits of |x| 2^(7S) truncated, with the
    // sign of x: the same digits as S steps of (x *= 128, q = trunc(x),
    // x -= q) in exact FP64, taken from one integer (7S <= 63 bits).
    const double two7s = ldexp(1.0, 7 * S);
    unsigned long long mag[2][8];
    uint32_t neg[2] = {0, 0};
#pragma unroll
    for (int e = 0; e < 8; e++)
#pragma unroll
        for (int a = 0; a < 2; a++) {
            const long long X = (long long)(t[a][fl + e][gl] * rs * two7s);   // |.| < 2^63, truncated
            neg[a] |= (X < 0 ? 1u : 0u) << e;
            mag[a][e] = (unsigned long long)(X < 0 ? -X : X);
        }
    for (int s = 0; s < S; s++) {
        const int sh = 7 * (S - 1 - s);
#pragma unroll
        for (int a = 0; a < 2; a++) {
            uint32_t w[2] = {0, 0};
#pragma unroll
            for (int e = 0; e < 8; e++) {
                int q = (int)((mag[a][e] >> sh) & 127u);
                if ((neg[a] >> e) & 1u) q = -q;
                w[e >> 2] |= ((uint32_t)(uint8_t)(int8_t)q) << (8 * (e & 3));
            }
            *reinterpret_cast<uint2 *>(k.oz_slices + oz_off(s, a0 + a, g, f, p.npad, kp8, narr)) = make_uint2(w[0], w[1]);
        }
    }
}

// ------------------------------------------------------------ per-atom operands
// Slices of the per-atom MT integrals that multiply A from the left in the
// per-atom products B_a = h_a A_a (hamiltonsetup.f90:75-88) and
// H_lo,a = loa_a A_a (hamiltonsetup.f90:131-145):
//   X(n, k) for n = output row (f of h_a in blocks of 64, then the lo rows r
//   of loa in blocks of 64 from block nfb on), k = K byte of the atom's window: the window starts
//   at oz_x0 (apw_off rounded down to 16) so that X(n, k) = 0 unless
//   0 <= k - (apw_off - oz_x0) < napw.
// Layout [atom][slice][block xb][array re, im][64 rows][lw bytes], one scale
// sigma per row (power of two above the row maximum).
__device__ __forceinline__ void x_value(const DevParams &p, const OzAtomArgs &xa, int ias, int xb, int n, int fp,
                                        double &re, double &im)
{
    re = im = 0.0;
    const AtomDesc at = p.atoms[ias];
    if (fp < 0 || fp >= at.napw) return;
    if (xb < xa.nfb) {
        const int f = xb * 64 + n;
        if (f >= at.napw) return;
        const size_t i = (size_t)ias * xa.ldh * xa.ldh + (size_t)fp * xa.ldh + f;   // h(f, f') at [ias][f'][f]
        re = xa.hr[i];
        im = xa.hi[i];
    } else {
        const int r = (xb - xa.nfb) * 64 + n;
        if (r >= at.losize) return;
        const size_t i = (size_t)ias * xa.ldlo * xa.maxaa + (size_t)fp * xa.ldlo + r;   // loa(r, f) at [ias][f][r]
        re = xa.lr[i];
        im = xa.li[i];
    }
}

// sigma of every X row: one thread per (atom, block, row), from the row maximum.
__global__ void oz_xsig_kernel(DevParams p, OzAtomArgs xa)
{
    const int n = threadIdx.x, xb = blockIdx.x, ias = blockIdx.y;
    double m = 0.0;
    for (int fp = 0; fp < p.atoms[ias].napw; fp++) {
        double re, im;
        x_value(p, xa, ias, xb, n, fp, re, im);
        m = fmax(m, fmax(fabs(re), fabs(im)));
    }
    xa.xsig[((size_t)ias * xa.nxb + xb) * 64 + n] = oz_sigma(m);
}

// The slices of X: one thread per (atom, block, row, 4 window bytes).
__global__ void oz_xsplit_kernel(DevParams p, OzAtomArgs xa, const __grid_constant__ OzScheme sch)
{
    const int S = sch.n;
    const int ias = blockIdx.z, xb = blockIdx.y;
    const int n = threadIdx.y + blockIdx.x * blockDim.y;        // row 0..63
    const int k4 = threadIdx.x * 4;                             // window byte
    if (n >= 64 || k4 >= xa.lw) return;
    const AtomDesc at = p.atoms[ias];
    const int delta = at.apw_off - at.oz_x0;
    const double r = 1.0 / xa.xsig[((size_t)ias * xa.nxb + xb) * 64 + n];
    double x[2][4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
        double re, im;
        x_value(p, xa, ias, xb, n, k4 + e - delta, re, im);
        x[0][e] = re * r;
        x[1][e] = im * r;
    }
    for (int s = 0; s < S; s++)
#pragma unroll
        for (int a = 0; a < 2; a++) {
            uint32_t w = 0;
#pragma unroll
            for (int e = 0; e < 4; e++) {
                x[a][e] *= 128.0;
                const double tq = trunc(x[a][e]);
                x[a][e] -= tq;
                w |= ((uint32_t)(uint8_t)(int8_t)tq) << (8 * e);
            }
            const size_t row = ((((size_t)ias * S + s) * xa.nxb + xb) * 2 + a) * 64 + n;
            *reinterpret_cast<uint32_t *>(xa.xs + row * xa.lw + k4) = w;
        }
}

// ------------------------------------------------------------ main kernel

// MODE OZ_HO: tiles {k, ib, jb}: H and O, 128 G_i x 32 G_j, B operand
//   [Br | Bi | Ar | Ai] of one G block, contraction over all K.
// MODE OZ_ATOM: tiles {k, atom, ib, xb}: 128 G x 64 output rows n of one
//   atom, B operand [X re | X im] (64 rows each), contraction over the
//   atom's K window; writes B planes (xb < nfb) or the APW-lo rows of H.
struct OzTileInfo {
    int k, i0, j0, ias, xb, nst;
};

template <int MODE, int KCH>
__device__ __forceinline__ OzTileInfo oz_tile(const DevParams &p, const int *tiles, int t, int kp8)
{
    OzTileInfo ti{};
    if (MODE == OZ_HO) {
        ti.k = tiles[3 * t];
        ti.i0 = tiles[3 * t + 1] * OZ_BM;
        ti.j0 = tiles[3 * t + 2] * OZ_BJ;
        ti.nst = kp8 / (KCH * OZ_CHUNK);
    } else {
        ti.k = tiles[4 * t];
        ti.ias = tiles[4 * t + 1];
        ti.i0 = tiles[4 * t + 2] * OZ_BM;
        ti.xb = tiles[4 * t + 3];
        ti.nst = p.atoms[ti.ias].oz_nch / KCH;
    }
    return ti;
}

// Persistent: each CTA walks the tiles blockIdx.x, blockIdx.x + gridDim.x, ...
// and every role walks the same sequence (tile, diagonal d = 2..S+1, left
// slice s = 1..d-1 with t = d - s on the right, K stages), so the mbarrier
// phases simply continue from tile to tile.  The MMAs of a tile's first
// segment overlap the final epilogue of the previous tile (the int32
// accumulators are free once the last fold has read them).
template <int MODE, int KCH, int NST>
__global__ void __launch_bounds__(OZ_THREADS, 1)
oz_mma_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, DevParams p,
              const KDesc *ks, const int *tiles, int ntiles, const __grid_constant__ OzScheme sch, int kp8,
              OzAtomArgs xa)
{
    const int S = sch.n;
    const int seg_pairs = MODE == OZ_HO ? sch.seg : sch.segx;
    constexpr int BOX = KCH * OZ_TILE;          // one operand of a stage
    constexpr int STAGE = 3 * BOX;              // A box [chunk][Ar, Ai][128 rows], B box [chunk][128 rows]
    extern __shared__ __align__(1024) uint8_t oz_smem[];
    __shared__ uint64_t full[NST], empty[NST], accf, acce, stg;
    __shared__ uint32_t tmem_sh;
    __shared__ int abort_sh;
    volatile int *abort = &abort_sh;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t sbase = (smem_u32(oz_smem) + 1023u) & ~1023u;
    // one tile per CTA: at the final store the stage buffers are idle and
    // hold the H/O mirror (2 x 32 x OZ_MIRROR_LD values, below the stages' size)
    static_assert(2 * 32 * OZ_MIRROR_LD * 16 <= NST * 3 * KCH * OZ_TILE, "mirror staging fits the stages");
    const bool staged = MODE == OZ_HO && (int)gridDim.x >= ntiles;
    exs_complex *mirror = reinterpret_cast<exs_complex *>(oz_smem + (sbase - smem_u32(oz_smem)));

    if (warp == 3) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_sh)),
                     "r"(OZ_TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    if (tid == 0) {
        for (int s = 0; s < NST; s++) {
            mbar_init(&full[s], 2);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&accf, 1);
        mbar_init(&acce, 8);                  // the eight epilogue warps
        mbar_init(&stg, 8);                   // the mirror is staged (one tile per CTA only)
        abort_sh = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = tmem_sh;

    if (warp < 3) {
        // ------------------------------------------------ TMA producers: warp 0 the A box, warp 1 the B box
        if (lane == 0 && warp < 2) {
            const int role = warp;
            uint32_t fills[NST];
#pragma unroll
            for (int q = 0; q < NST; q++) fills[q] = 0;
            int st = 0;
            bool bad = false;
            for (int tile = blockIdx.x; tile < ntiles && !bad; tile += gridDim.x) {
                const OzTileInfo ti = oz_tile<MODE, KCH>(p, tiles, tile, kp8);
                const int slot = ks[ti.k].oz_slot;
                const int x0 = (MODE == OZ_ATOM) ? p.atoms[ti.ias].oz_x0 : 0;
                // group g: the pairs (s, t) of diagonal s + t = g + 2
                for (int g = 0; g < S && !bad; g++)
                    for (int j = 0; j < g + 1 && !bad; j++) {
                        const int s = j + 1, t = g + 1 - j;
                        for (int kb = 0; kb < ti.nst; kb++) {
                            if (fills[st] > 0 && !mbar_wait_ab(&empty[st], (fills[st] - 1) & 1, abort, sch.wait)) {
                                bad = true;
                                break;
                            }
                            mbar_expect_tx(&full[st], role == 0 ? 2 * BOX : BOX);
                            const uint32_t dst = sbase + st * STAGE + role * 2 * BOX;
                            if (role == 0) {   // Ar and Ai (the slot's last two arrays) of G rows i0 .. i0+127, slice s
                                if (MODE == OZ_HO)
                                    tma_load_5d(dst, &mapA, 0, ti.i0, oz_narr(p.relativity) - 2, kb * KCH, slot * S + s - 1, &full[st]);
                                else
                                    tma_load_4d(dst, &mapA, x0 + kb * OZ_CHUNK, ti.i0, oz_narr(p.relativity) - 2, slot * S + s - 1,
                                                &full[st]);
                            } else if (MODE == OZ_HO) {   // the four arrays of G rows j0 .. j0+31, slice t
                                tma_load_5d(dst, &mapB, 0, ti.j0, 0, kb * KCH, slot * S + t - 1, &full[st]);
                            } else {                      // X rows of block xb, slice t
                                const int grp = (ti.ias * S + (t - 1)) * xa.nxb + ti.xb;
                                tma_load_4d(dst, &mapB, 0, 0, grp, kb * KCH, &full[st]);
                            }
                            fills[st]++;
                            st = (st + 1 == NST) ? 0 : st + 1;
                        }
                    }
            }
        }
    } else if (warp == 3) {
        // ------------------------------------------------ MMA issuer
        if (lane == 0) {
            const uint32_t idesc = umma_idesc_i8(128, OZ_N);
            uint32_t uses[NST];
#pragma unroll
            for (int q = 0; q < NST; q++) uses[q] = 0;
            int nseg = 0, st = 0;
            bool bad = false;
            for (int tile = blockIdx.x; tile < ntiles && !bad; tile += gridDim.x) {
                const int nst = oz_tile<MODE, KCH>(p, tiles, tile, kp8).nst;
                for (int g = 0; g < S && !bad; g++)
                    for (int s0 = 1; s0 <= g + 1 && !bad; s0 += seg_pairs) {
                        const int s1 = min(g + 1, s0 + seg_pairs - 1);
                        // the epilogue must have folded the previous segment
                        if (nseg > 0 && !mbar_wait_ab(&acce, (nseg - 1) & 1, abort, sch.wait)) {
                            bad = true;
                            break;
                        }
                        tc_fence_after();
                        bool first = true;
                        for (int s = s0; s <= s1 && !bad; s++)
                            for (int kb = 0; kb < nst; kb++) {
                                if (!mbar_wait_ab(&full[st], uses[st] & 1, abort, sch.wait)) {
                                    bad = true;
                                    break;
                                }
                                tc_fence_after();
                                const uint32_t sa = sbase + st * STAGE;
#pragma unroll
                                for (int c = 0; c < KCH; c++)
#pragma unroll
                                    for (int q = 0; q < OZ_CHUNK / 32; q++) {
                                        const uint32_t ao = c * 2 * OZ_TILE + q * 32;   // Ar; Ai one tile on
                                        const uint64_t bd = umma_desc_sw128(sa + 2 * BOX + c * OZ_TILE + q * 32);
                                        const uint32_t acc = (first && c == 0 && q == 0) ? 0u : 1u;
                                        umma_i8(tbase, umma_desc_sw128(sa + ao), bd, idesc, acc);
                                        umma_i8(tbase + 128, umma_desc_sw128(sa + ao + OZ_TILE), bd, idesc, acc);
                                    }
                                first = false;
                                umma_commit(&empty[st]);
                                uses[st]++;
                                st = (st + 1 == NST) ? 0 : st + 1;
                            }
                        if (!bad) {
                            umma_commit(&accf);
                            nseg++;
                        }
                    }
            }
            // every MMA is done before tensor memory is freed, also when only an epilogue gave up
            for (int q = 0; q < NST; q++)
                if (uses[q] > 0) mbar_drain(&empty[q], (uses[q] - 1) & 1);
        }
    } else {
        // ------------------------------------------------ epilogue (warps 4..11)
        const int qd = warp & 3;                                    // tensor-memory lane quadrant
        const int half = (warp - 4) >> 2;                           // which two value blocks
        const uint32_t t_lane = tbase + ((uint32_t)(qd * 32) << 16);
        int nseg = 0;
        bool bad = false;
        for (int tile = blockIdx.x; tile < ntiles && !bad; tile += gridDim.x) {
            const OzTileInfo ti = oz_tile<MODE, KCH>(p, tiles, tile, kp8);
            for (int g = 0; g < S && !bad; g++) {
                for (int s0 = 1; s0 <= g + 1; s0 += seg_pairs) {
                    const bool ok = __all_sync(0xffffffffu, mbar_wait_ab(&accf, nseg & 1, abort, sch.wait));
                    if (!ok) {
                        bad = true;
                        break;
                    }
                    tc_fence_after();
                    const bool init = (g == 0 && s0 == 1);      // first segment of the tile
                    // running-sum block o (32 values) = r block o +- i block (o ^ 1) (HO:
                    // Re H, Im H, Re O, Im O) or (o ^ 2) (ATOM: Re rows 0-63, Im rows 0-63)
#pragma unroll 1
                    for (int k = 0; k < 2; k++) {
                        const int o = oz_block<MODE>(half, k);
                        const int sg = (MODE == OZ_HO) ? ((o & 1) ? -1 : 1) : ((o < 2) ? -1 : 1);
                        const int oi = (MODE == OZ_HO) ? (o ^ 1) : (o ^ 2);
#pragma unroll 1
                        for (int jc = 0; jc < 32; jc += 16) {
                            uint32_t rv[16], iv[16], lo[16], hi[16];
                            const uint32_t fcol = OZ_FP64_COL + 2 * (o * 32 + jc);
                            tm_ld16(t_lane + o * 32 + jc, rv);
                            tm_ld16(t_lane + 128 + oi * 32 + jc, iv);
                            if (!init) {
                                tm_ld16(t_lane + fcol, lo);
                                tm_ld16(t_lane + fcol + 16, hi);
                            }
                            tm_wait_ld();
                            uint32_t o0[16], o1[16];
                            oz_fold16(g, init, sg, rv, iv, lo, hi, o0, o1);
                            tm_st16(t_lane + fcol, o0);
                            tm_st16(t_lane + fcol + 16, o1);
                        }
                    }
                    tm_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acce);
                    nseg++;
                }
            }
            if (!__all_sync(0xffffffffu, !bad && !*abort)) {
                bad = true;
                break;
            }
            const KDesc kd = ks[ti.k];
            if (MODE == OZ_HO) {
                oz_store_ho(p, kd, ti.i0, ti.j0, t_lane, qd * 32 + lane, half, staged ? mirror : nullptr);
                if (staged) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&stg);
                    if (__all_sync(0xffffffffu, mbar_wait_ab(&stg, 0, abort, sch.wait)))
                        oz_store_mirror(kd, ti.i0, ti.j0, mirror, warp - 4, lane);
                }
            } else {
                // row G of the tile; values v = 0..63 real, 64..127 imaginary parts of the 64 output
                // rows, of which this half holds rows 32 half .. 32 half + 31
                const int g = ti.i0 + qd * 32 + lane;
                const bool g_ok = g < p.npad;
                const AtomDesc at = p.atoms[ti.ias];
                const bool lorows = ti.xb >= xa.nfb;
                const double sa = g_ok ? oz_sigma(kd.oz_scale[g]) : 0.0;
                const double *sig = xa.xsig + ((size_t)ti.ias * xa.nxb + ti.xb) * 64;
                const size_t row0 = (size_t)kd.ngp + at.lo_off;
                double bmax = 0.0;
#pragma unroll 1
                for (int jc = 32 * half; jc < 32 * half + 32; jc += 8) {
                    uint32_t wr[16], wi[16];
                    tm_ld16(t_lane + OZ_FP64_COL + 2 * jc, wr);
                    tm_ld16(t_lane + OZ_FP64_COL + 2 * (64 + jc), wi);
                    tm_wait_ld();
                    if (!g_ok) continue;
#pragma unroll
                    for (int e = 0; e < 8; e++) {
                        const int n = jc + e;
                        const double sc = sa * sig[n];
                        const double re = __hiloint2double((int)wr[2 * e + 1], (int)wr[2 * e]) * sc;
                        const double im = __hiloint2double((int)wi[2 * e + 1], (int)wi[2 * e]) * sc;
                        if (!lorows) {
                            const int f = ti.xb * 64 + n;
                            if (f >= at.napw) continue;
                            const size_t off = (size_t)(at.apw_off + f) * p.npad + g;
                            kd.br[off] = re;
                            kd.bi[off] = im;
                            bmax = fmax(bmax, fmax(fabs(re), fabs(im)));
                        } else {
                            const int r = (ti.xb - xa.nfb) * 64 + n;
                            if (r >= at.losize || g >= kd.ngp) continue;
                            exs_complex v;
                            v.re = re;
                            v.im = im;
                            kd.h[(row0 + r) + (size_t)kd.nmat * g] = v;
                            v.im = -im;
                            kd.h[(size_t)g + (size_t)kd.nmat * (row0 + r)] = v;
                        }
                    }
                }
                if (!lorows && g_ok) atomic_max_nonneg(kd.oz_scale + p.npad + g, bmax);
            }
            // the FP64 region is read; the next tile's first fold may overwrite it
            tc_fence_before();
        }
    }
    tc_fence_before();
    __syncthreads();                     // every role is out: the flag is final
    if (*abort) {
        if (tid == 0) atomicOr(p.err, DEV_ERR_TIMEOUT);
        abort_settle();
    }
    if (warp == 3) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tbase), "r"(OZ_TMEM_COLS));
    }
}

// ------------------------------------------------------------ two-SM H/O tiles
// A cluster of two CTAs computes a 256 (G_i) x 32 (G_j) tile with
// tcgen05.mma.cta_group::2 (M = 256): each CTA holds its own 128 rows of the
// A operands (Ar, Ai) and half of the B operand (CTA 0: Br, Bi; CTA 1: Ar,
// Ai of the 32 G_j), so each SM fetches 320 instead of 384 operand rows per
// K byte.  CTA 0 issues the MMAs; its full barriers count the bytes of both
// CTAs' copies (the copies of CTA 1 signal CTA 0's barrier); MMA completion
// is signalled to both CTAs (multicast commit); both CTAs' epilogues fold
// their own 128 rows and report to CTA 0's barrier.  Each CTA loads its own operands.
template <int KCH, int NST>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(OZ_THREADS, 1)
oz_mma2_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB2, DevParams p,
               const KDesc *ks, const int *tiles, const __grid_constant__ OzScheme sch, int kp8)
{
    const int S = sch.n;
    const int seg_pairs = sch.seg;
    constexpr int ABOX = 2 * KCH * OZ_TILE;          // Ar, Ai of this CTA's 128 rows
    constexpr int BBOX = KCH * OZ_TILE / 2;          // this CTA's 64 rows of B
    constexpr int STAGE = ABOX + BBOX;
    extern __shared__ __align__(1024) uint8_t oz_smem[];
    __shared__ uint64_t full[NST], empty[NST], accf, acce, stg;
    __shared__ uint32_t tmem_sh;
    __shared__ int abort_sh;
    volatile int *abort = &abort_sh;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_ctarank();
    static_assert(2 * 32 * OZ_MIRROR_LD * 16 <= NST * STAGE, "mirror staging fits the stages");
    const uint32_t sbase = (smem_u32(oz_smem) + 1023u) & ~1023u;
    const int t3 = 3 * (blockIdx.x >> 1);
    const KDesc kd = ks[tiles[t3]];
    const int i0 = (2 * tiles[t3 + 1] + (int)rank) * OZ_BM, j0 = tiles[t3 + 2] * OZ_BJ;
    const int nst = kp8 / (KCH * OZ_CHUNK);

    if (warp == 3) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_sh)),
                     "r"(OZ_TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::);
    }
    if (tid == 0) {
        for (int s = 0; s < NST; s++) {
            mbar_init(&full[s], 1);      // CTA 0: one arrive (with the bytes of both CTAs)
            mbar_init(&empty[s], 1);
        }
        mbar_init(&accf, 1);
        mbar_init(&acce, 16);            // CTA 0: eight epilogue warps in each CTA
        mbar_init(&stg, 8);              // this CTA's epilogue warps: the mirror is staged
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
            uint32_t fills[NST];
#pragma unroll
            for (int q = 0; q < NST; q++) fills[q] = 0;
            int st = 0;
            bool bad = false;
            const int slot = kd.oz_slot;
            for (int g = 0; g < S && !bad; g++)
                for (int j = 0; j < g + 1 && !bad; j++) {
                    const int s = j + 1, t = g + 1 - j;
                    for (int kb = 0; kb < nst; kb++) {
                        if (fills[st] > 0 && !mbar_wait_ab(&empty[st], (fills[st] - 1) & 1, abort, sch.wait)) {
                            bad = true;
                            break;
                        }
                        if (rank == 0 && role == 0) mbar_expect_tx(&full[st], 2 * STAGE);
                        const uint32_t bar = smem_u32(&full[st]);
                        if (role == 0)
                            tma_load_5d_2sm(sbase + st * STAGE, &mapA, 0, i0, oz_narr(p.relativity) - 2, kb * KCH,
                                            slot * S + s - 1, bar);
                        else
                            tma_load_5d_2sm(sbase + st * STAGE + ABOX, &mapB2, 0, j0, 2 * (int)rank, kb * KCH,
                                            slot * S + t - 1, bar);
                        fills[st]++;
                        st = (st + 1 == NST) ? 0 : st + 1;
                    }
                }
        }
    } else if (warp == 3) {
        // ------------------------------------------------ MMA issuer (CTA 0)
        if (lane == 0 && rank == 0) {
            const uint32_t idesc = umma_idesc_i8(256, OZ_N);
            uint32_t uses[NST];
#pragma unroll
            for (int q = 0; q < NST; q++) uses[q] = 0;
            int nseg = 0, st = 0;
            bool bad = false;
            for (int g = 0; g < S && !bad; g++)
                for (int s0 = 1; s0 <= g + 1 && !bad; s0 += seg_pairs) {
                    const int s1 = min(g + 1, s0 + seg_pairs - 1);
                    if (nseg > 0 && !mbar_wait_ab(&acce, (nseg - 1) & 1, abort, sch.wait)) {
                        bad = true;
                        break;
                    }
                    tc_fence_after();
                    bool first = true;
                    for (int s = s0; s <= s1 && !bad; s++)
                        for (int kb = 0; kb < nst; kb++) {
                            if (!mbar_wait_ab(&full[st], uses[st] & 1, abort, sch.wait)) {
                                bad = true;
                                break;
                            }
                            tc_fence_after();
                            const uint32_t sa = sbase + st * STAGE;
#pragma unroll
                            for (int c = 0; c < KCH; c++)
#pragma unroll
                                for (int q = 0; q < OZ_CHUNK / 32; q++) {
                                    const uint32_t ao = c * 2 * OZ_TILE + q * 32;
                                    const uint64_t bd = umma_desc_sw128(sa + ABOX + c * (OZ_TILE / 2) + q * 32);
                                    const uint32_t acc = (first && c == 0 && q == 0) ? 0u : 1u;
                                    umma_i8_2sm(tbase, umma_desc_sw128(sa + ao), bd, idesc, acc);
                                    umma_i8_2sm(tbase + 128, umma_desc_sw128(sa + ao + OZ_TILE), bd, idesc, acc);
                                }
                            first = false;
                            umma_commit_2sm(&empty[st]);
                            uses[st]++;
                            st = (st + 1 == NST) ? 0 : st + 1;
                        }
                    if (!bad) {
                        umma_commit_2sm(&accf);
                        nseg++;
                    }
                }
            // every MMA is done before the pair may go away, also when only an epilogue gave up
            for (int q = 0; q < NST; q++)
                if (uses[q] > 0) mbar_drain(&empty[q], (uses[q] - 1) & 1);
        }
    } else if (warp >= 4) {
        // ------------------------------------------------ epilogue (both CTAs, warps 4..11)
        const int qd = warp & 3;
        const int half = (warp - 4) >> 2;
        const uint32_t t_lane = tbase + ((uint32_t)(qd * 32) << 16);
        const uint32_t acce0 = mapa_shared(smem_u32(&acce), 0);
        int nseg = 0;
        bool bad = false;
        for (int g = 0; g < S && !bad; g++) {
            for (int s0 = 1; s0 <= g + 1; s0 += seg_pairs) {
                const bool ok = __all_sync(0xffffffffu, mbar_wait_ab(&accf, nseg & 1, abort, sch.wait));
                if (!ok) {
                    bad = true;
                    break;
                }
                tc_fence_after();
                const bool init = (nseg == 0);
#pragma unroll 1
                for (int k = 0; k < 2; k++) {
                    const int o = oz_block<OZ_HO>(half, k);
                    const int sg = (o & 1) ? -1 : 1;
#pragma unroll 1
                    for (int jc = 0; jc < 32; jc += 16) {
                        uint32_t rv[16], iv[16], lo[16], hi[16];
                        const uint32_t fcol = OZ_FP64_COL + 2 * (o * 32 + jc);
                        tm_ld16(t_lane + o * 32 + jc, rv);
                        tm_ld16(t_lane + 128 + (o ^ 1) * 32 + jc, iv);
                        if (!init) {
                            tm_ld16(t_lane + fcol, lo);
                            tm_ld16(t_lane + fcol + 16, hi);
                        }
                        tm_wait_ld();
                        uint32_t o0[16], o1[16];
                        oz_fold16(g, init, sg, rv, iv, lo, hi, o0, o1);
                        tm_st16(t_lane + fcol, o0);
                        tm_st16(t_lane + fcol + 16, o1);
                    }
                }
                tm_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_remote(acce0);      // CTA 0's barrier (also from CTA 0)
                nseg++;
            }
        }
        exs_complex *mirror = reinterpret_cast<exs_complex *>(oz_smem + (sbase - smem_u32(oz_smem)));
        if (__all_sync(0xffffffffu, !bad && !*abort))
            oz_store_ho(p, kd, i0, j0, t_lane, qd * 32 + lane, half, mirror);
        __syncwarp();
        if (lane == 0) mbar_arrive(&stg);
        if (__all_sync(0xffffffffu, mbar_wait_ab(&stg, 0, abort, sch.wait) && !*abort))
            oz_store_mirror(kd, i0, j0, mirror, warp - 4, lane);
    }
    tc_fence_before();
    __syncthreads();                     // every role is out: the flag is final
    if (*abort) {
        if (tid == 0) atomicOr(p.err, DEV_ERR_TIMEOUT);
        abort_settle();
    }
    cluster_sync_all();                  // neither CTA leaves while the pair still uses its memory
    if (warp == 3) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tbase), "r"(OZ_TMEM_COLS));
    }
}

// ------------------------------------------------------------ host side
int oz_kpad(int K) { return (K + OZ_MAX_KCH * OZ_CHUNK - 1) / (OZ_MAX_KCH * OZ_CHUNK) * (OZ_MAX_KCH * OZ_CHUNK); }

size_t oz_slot_bytes(int S, int npad, int kp8, int narr) { return (size_t)S * npad * narr * (size_t)kp8; }

int oz_seg_pairs(int S, int kp8)
{
    // pairs whose int32 sums over K stay exact: pairs * kp8 * 127^2 < 2^31
    const long long per = (long long)kp8 * 127 * 127;
    long long n = (((long long)1 << 31) - 1) / per;
    return (int)(n < 1 ? 0 : (n > S ? S : n));
}

// configuration index: bit 0 = pipeline shape (KCH, NST) of the H/O tiles,
// bit 1 = persistent launch (one CTA per SM) of the H/O tiles, bit 2 =
// persistent launch of the per-atom tiles, bit 3 = two-SM H/O tiles (256 x 32
// per CTA pair; bit 1 unused then)
// bit 0 of a configuration: two 96 KB stages of 2 K chunks, or four 48 KB stages of 1
const int OZ_CFG_KCH[OZ_NCFG] = {2, 1, 2, 1, 2, 1, 2, 1, 2, 1, 2, 1, 2, 1, 2, 1,
                                 2, 1, 2, 1, 2, 1, 2, 1, 2, 1, 2, 1, 2, 1, 2, 1};
const int OZ_CFG_NST[OZ_NCFG] = {2, 4, 2, 4, 2, 4, 2, 4, 2, 4, 2, 4, 2, 4, 2, 4,
                                 2, 4, 2, 4, 2, 4, 2, 4, 2, 4, 2, 4, 2, 4, 2, 4};

cudaError_t launch_oz_split(const DevParams &p, const KDesc *d_k, int nk, const OzScheme &sch, int kp8, int which,
                            cudaStream_t s)
{
    oz_split_kernel<<<dim3(kp8 / SPLIT_F, p.npad / 32, nk), dim3(32, 8), 0, s>>>(p, d_k, sch, kp8, which);
    return cudaGetLastError();
}

cudaError_t launch_oz_colmax(const DevParams &p, const KDesc *d_k, int nk, cudaStream_t s)
{
    oz_colmax_kernel<<<dim3(p.npad / 32, nk), dim3(32, 8), 0, s>>>(p, d_k);
    return cudaGetLastError();
}

cudaError_t launch_oz_x(const DevParams &p, const OzAtomArgs &xa, const OzScheme &sch, cudaStream_t s)
{
    oz_xsig_kernel<<<dim3(xa.nxb, p.natmtot), 64, 0, s>>>(p, xa);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    oz_xsplit_kernel<<<dim3(8, xa.nxb, p.natmtot), dim3(xa.lw / 4, 8), 0, s>>>(p, xa, sch);
    return cudaGetLastError();
}

template <int MODE, int KCH, int NST>
static cudaError_t launch_cfg(const CUtensorMap *mapA, const CUtensorMap *mapB, const DevParams &p, const KDesc *d_k,
                              const void *d_tiles, int ntiles, const OzScheme &sch, int kp8, const OzAtomArgs &xa,
                              bool persistent, cudaStream_t s)
{
    constexpr int smem = NST * 3 * KCH * OZ_TILE + 1024;
    static std::atomic<unsigned long long> attr{0};
    cudaError_t e = once_per_device(attr, [] {
        return cudaFuncSetAttribute(oz_mma_kernel<MODE, KCH, NST>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    });
    if (e != cudaSuccess) return e;
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    // persistent: one CTA per SM walking the tiles; else one CTA per tile
    const int grid = (persistent && nsm < ntiles) ? nsm : ntiles;
    oz_mma_kernel<MODE, KCH, NST><<<grid, OZ_THREADS, smem, s>>>(*mapA, *mapB, p, d_k, (const int *)d_tiles, ntiles,
                                                                 sch, kp8, xa);
    return cudaGetLastError();
}

template <int KCH, int NST>
static cudaError_t launch_2sm(const CUtensorMap *mapA, const CUtensorMap *mapB2, const DevParams &p, const KDesc *d_k,
                              const void *d_tiles, int ntiles, const OzScheme &sch, int kp8, cudaStream_t s)
{
    constexpr int smem = NST * (2 * KCH * OZ_TILE + KCH * OZ_TILE / 2) + 1024;
    static std::atomic<unsigned long long> attr{0};
    cudaError_t e = once_per_device(attr, [] {
        return cudaFuncSetAttribute(oz_mma2_kernel<KCH, NST>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    });
    if (e != cudaSuccess) return e;
    oz_mma2_kernel<KCH, NST><<<2 * ntiles, OZ_THREADS, smem, s>>>(*mapA, *mapB2, p, d_k, (const int *)d_tiles, sch,
                                                                  kp8);
    return cudaGetLastError();
}

cudaError_t launch_oz_mma(int cfg, const CUtensorMap *mapA, const CUtensorMap *mapB, const DevParams &p,
                          const KDesc *d_k, const void *d_tiles, int ntiles, const OzScheme &sch, int kp8,
                          cudaStream_t s)
{
    if (ntiles <= 0) return cudaSuccess;
    if (cfg & 8) {   // two-SM tiles: mapB is the half-B view
        if (cfg & 1) return launch_2sm<1, 4>(mapA, mapB, p, d_k, d_tiles, ntiles, sch, kp8, s);
        return launch_2sm<2, 2>(mapA, mapB, p, d_k, d_tiles, ntiles, sch, kp8, s);
    }
    const OzAtomArgs none{};
    const bool persistent = (cfg & 2) != 0;
    switch (cfg & 1) {
    case 0: return launch_cfg<OZ_HO, 2, 2>(mapA, mapB, p, d_k, d_tiles, ntiles, sch, kp8, none, persistent, s);
    default: return launch_cfg<OZ_HO, 1, 4>(mapA, mapB, p, d_k, d_tiles, ntiles, sch, kp8, none, persistent, s);
    }
}

cudaError_t launch_oz_atom(int cfg, const CUtensorMap *mapArow, const CUtensorMap *mapX, const DevParams &p,
                           const KDesc *d_k, const void *d_tiles, int ntiles, const OzScheme &sch, int kp8,
                           const OzAtomArgs &xa, cudaStream_t s)
{
    if (ntiles <= 0) return cudaSuccess;
    return launch_cfg<OZ_ATOM, 1, 4>(mapArow, mapX, p, d_k, d_tiles, ntiles, sch, kp8, xa, (cfg & 4) != 0, s);
}

// TMA views of the slices of all slots (int8, 5D):
//   d0: K byte within a 128-byte chunk                       stride 1
//   d1: G row (npad)                                         stride kp8
//   d2: array (Br, Bi, Ar, Ai; iora*: Br, Bi, Cr, Ci, Ar, Ai) stride npad kp8
//   d3: K chunk                                              stride 128
//   d4: slot x slice                                         stride narr npad kp8
// A box {128, 128, 2, kch, 1}: Ar and Ai of 128 G rows; B box
// {128, 32, 4, kch, 1}: the four arrays of 32 G rows.  d3 is outside d1, d2
// in the box, so each K chunk lands in shared memory as contiguous
// 128-byte rows (A: 2 x 128 rows, B: 4 x 32 rows).
bool make_oz_tensor_maps(void *base, size_t nss, int npad, int kp8, int kch, int narr, CUtensorMap *mapA,
                         CUtensorMap *mapB, CUtensorMap *mapB2)
{
    typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn)
        return false;
    EncodeFn encode = (EncodeFn)fn;
    if (kch < 1 || kch > OZ_MAX_KCH || kp8 % (OZ_MAX_KCH * OZ_CHUNK) != 0) return false;
    const cuuint64_t dims[5] = {(cuuint64_t)OZ_CHUNK, (cuuint64_t)npad, (cuuint64_t)narr, (cuuint64_t)(kp8 / OZ_CHUNK),
                                (cuuint64_t)nss};
    const cuuint64_t strides[4] = {(cuuint64_t)kp8, (cuuint64_t)npad * kp8, (cuuint64_t)OZ_CHUNK,
                                   (cuuint64_t)narr * npad * kp8};
    const cuuint32_t es[5] = {1, 1, 1, 1, 1};
    const cuuint32_t boxA[5] = {OZ_CHUNK, OZ_BM, 2, (cuuint32_t)kch, 1};
    const cuuint32_t boxB[5] = {OZ_CHUNK, OZ_BJ, OZ_NARR, (cuuint32_t)kch, 1};
    if (encode(mapA, CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, base, dims, strides, boxA, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    if (encode(mapB, CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, base, dims, strides, boxB, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    // half of B (two of the four arrays) for the two-SM tiles
    const cuuint32_t boxB2[5] = {OZ_CHUNK, OZ_BJ, 2, (cuuint32_t)kch, 1};
    if (encode(mapB2, CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, base, dims, strides, boxB2, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    return true;
}

// TMA views for the per-atom products:
//   mapArow: the slices as [slot x slice][array][G][kp8 bytes] (4D), box
//     {128, 128, 2, 1}: Ar and Ai of 128 G rows, one 128-byte K chunk
//     starting at any multiple of 16 bytes (the atom windows are not chunk
//     aligned);
//   mapX: the X slices as [group][128 rows][lw bytes] viewed like the B tiles
//     (4D, K chunked), box {128, 128, 1, 1}.
bool make_oz_atom_maps(void *base, size_t nss, int npad, int kp8, int narr, void *xbase, size_t xgroups, int lw,
                       CUtensorMap *mapArow, CUtensorMap *mapX)
{
    typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn)
        return false;
    EncodeFn encode = (EncodeFn)fn;
    if (kp8 % OZ_CHUNK != 0 || lw % OZ_CHUNK != 0) return false;
    const cuuint32_t es[4] = {1, 1, 1, 1};
    {
        const cuuint64_t dims[4] = {(cuuint64_t)kp8, (cuuint64_t)npad, (cuuint64_t)narr, (cuuint64_t)nss};
        const cuuint64_t strides[3] = {(cuuint64_t)kp8, (cuuint64_t)npad * kp8, (cuuint64_t)narr * npad * kp8};
        const cuuint32_t box[4] = {OZ_CHUNK, OZ_BM, 2, 1};
        if (encode(mapArow, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, base, dims, strides, box, es,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    }
    {
        const cuuint64_t dims[4] = {(cuuint64_t)OZ_CHUNK, 128, (cuuint64_t)xgroups, (cuuint64_t)(lw / OZ_CHUNK)};
        const cuuint64_t strides[3] = {(cuuint64_t)lw, (cuuint64_t)128 * lw, (cuuint64_t)OZ_CHUNK};
        const cuuint32_t box[4] = {OZ_CHUNK, 128, 1, 1};
        if (encode(mapX, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, xbase, dims, strides, box, es,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    }
    return true;
}

}  // namespace exs
