// Native-FP64 path of the H/O setup: grouped complex contractions on the
// FP64 tensor instruction (DMMA m8n8k4), with the epilogues that place the
// results into the reference's za(nmat, nmat) layout.
//
// Stages of one k-point (the reference's per-atom loop of
// src/src_eigensystem/hamiltonsetup.f90:53-168 and overlapsetup.f90:47-154,
// regrouped so that all atoms and k-points of a call share one launch):
//   1. B_a = h_a A_a per atom              (hamiltonsetup.f90:75-88)
//   2. H = A^H B, O = A^H A (or A^H C, iora*), K = all atoms' APW rows at
//      once; upper tiles only; the epilogue adds the interstitial term
//      (hmlistln.f90 / olpistln.f90) and writes the conjugate mirror
//      (hamiltonoverlapocopy_UL.f90)
//   3. APW-lo rows of H (hamiltonsetup.f90:131-149) as a grouped GEMM,
//      APW-lo of O (overlapsetup.f90:111-127) and the lo-lo blocks
//      (hamiltonsetup.f90:154-161, overlapsetup.f90:131-146) elementwise.
//
// Operand layout: real and imaginary parts in separate planes; an operand
// X of an M x K product is stored [k][m] (m contiguous), i.e. X^T, which is
// how both the matching coefficients (G contiguous) and the Fortran MT
// integrals (first index contiguous) already lie in memory.
#include <algorithm>

#include "exs_internal.cuh"
#include "interstitial.cuh"

namespace exs {

// Tiles are EDGE x EDGE (64, 32 or 16), 128 threads: 2 x 2 warps of EDGE/2 x
// EDGE/2, K slabs of 16 in a three-stage cp.async ring.  A 64 x 64 tile of
// K = 316 keeps one SM's FP64 pipe busy for 42 us, so a single k-point of the
// two-atom cell (six tiles) left 142 SMs idle; gemm_edge picks the edge.
// Every element is summed over K in the same order whatever the edge, so the
// results do not depend on the batch that an element's k-point comes in.  Rows
// are padded to 4 (mod 16) doubles: the four K rows and four columns that half
// a warp reads fall into different banks.
constexpr int GB_K = 16, GB_STAGES = 3, GB_THREADS = 128;
template <int EDGE>
struct GemmCfg {
    static constexpr int WT = EDGE / 2;                         // edge of a warp's sub-tile
    static constexpr int MT = WT / 8;                           // 8 x 8 MMA tiles per warp and direction
    static constexpr int LDS = EDGE + 4;
    static constexpr int PLANE = GB_K * LDS;                    // doubles per plane per stage
    static constexpr int STAGE = 4 * PLANE;                     // xr, xi, yr, yi
    static constexpr size_t SMEM = (size_t)GB_STAGES * STAGE * sizeof(double);
};

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, bool valid)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// Load one K-slab (GB_K rows) of the four operand planes into stage buffer st.
template <int EDGE>
__device__ __forceinline__ void load_stage(double *st, const GemmProb &P, int m0, int n0, int k0)
{
    using C = GemmCfg<EDGE>;
    const int tid = threadIdx.x;
#pragma unroll
    for (int it = 0; it < (GB_K * EDGE / 2) / GB_THREADS; it++) {
        const int c = tid + it * GB_THREADS;
        const int row = c / (EDGE / 2);
        const int col = (c % (EDGE / 2)) * 2;
        const int gk = k0 + row;
        {
            const int gm = m0 + col;
            const bool v = gk < P.K && gm < P.M;
            const size_t off = v ? (size_t)gk * P.ldx + gm : 0;
            cp_async16(st + 0 * C::PLANE + row * C::LDS + col, P.xr + off, v);
            cp_async16(st + 1 * C::PLANE + row * C::LDS + col, P.xi + off, v);
        }
        {
            const int gn = n0 + col;
            const bool v = gk < P.K && gn < P.N;
            const size_t off = v ? (size_t)gk * P.ldy + gn : 0;
            cp_async16(st + 2 * C::PLANE + row * C::LDS + col, P.yr + off, v);
            cp_async16(st + 3 * C::PLANE + row * C::LDS + col, P.yi + off, v);
        }
    }
}

// GROUP 0: EPI_PLANAR and EPI_LOROWS problems, GROUP 1: EPI_HAM and EPI_OVL
// (the problem's kind); one launch takes a group's problems together.
template <int GROUP, int EDGE>
__global__ void __launch_bounds__(GB_THREADS, 2)
zgemm_dmma_kernel(DevParams p, const GemmProb *probs, const TileWork *work, const KDesc *ks)
{
    using C = GemmCfg<EDGE>;
    constexpr int MT = C::MT;
    extern __shared__ __align__(16) double smem[];
    const TileWork tw = work[blockIdx.x];
    const GemmProb P = probs[tw.prob];
    const int m0 = tw.tm * EDGE, n0 = tw.tn * EDGE;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wm = warp >> 1, wn = warp & 1;
    const int mw = wm * C::WT, nw = wn * C::WT;            // this warp's sub-tile
    // upper tiles: sub-tiles below the diagonal are not formed
    const bool idle = GROUP == 1 && m0 + mw > n0 + nw + C::WT - 1;

    double cre[MT][MT][2], cim[MT][MT][2];
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int j = 0; j < MT; j++) { cre[i][j][0] = cre[i][j][1] = cim[i][j][0] = cim[i][j][1] = 0.0; }

    const int nkt = (P.K + GB_K - 1) / GB_K;
#pragma unroll
    for (int s = 0; s < GB_STAGES - 1; s++) {
        if (s < nkt) load_stage<EDGE>(smem + s * C::STAGE, P, m0, n0, s * GB_K);
        cp_async_commit();
    }
    const double sgn = P.conjx ? 1.0 : -1.0;
    for (int kt = 0; kt < nkt; kt++) {
        cp_async_wait<GB_STAGES - 2>();
        __syncthreads();
        {
            const int nt = kt + GB_STAGES - 1;
            if (nt < nkt) load_stage<EDGE>(smem + (nt % GB_STAGES) * C::STAGE, P, m0, n0, nt * GB_K);
            cp_async_commit();
        }
        const double *st = smem + (kt % GB_STAGES) * C::STAGE;
        if (idle) continue;
#pragma unroll
        for (int kq = 0; kq < GB_K / 4; kq++) {
            const int kr = kq * 4 + (lane & 3);
            double ar[MT], aim[MT], naim[MT], br[MT], bi[MT];
#pragma unroll
            for (int i = 0; i < MT; i++) {
                const int mm = mw + i * 8 + (lane >> 2);
                ar[i] = st[0 * C::PLANE + kr * C::LDS + mm];
                aim[i] = sgn * st[1 * C::PLANE + kr * C::LDS + mm];   // conj: +ai, plain: -ai
                naim[i] = -aim[i];
            }
#pragma unroll
            for (int j = 0; j < MT; j++) {
                const int nn = nw + j * 8 + (lane >> 2);
                br[j] = st[2 * C::PLANE + kr * C::LDS + nn];
                bi[j] = st[3 * C::PLANE + kr * C::LDS + nn];
            }
            // four passes over the MT x MT sub-tiles so that the two products
            // accumulated into one register pair are MT^2 DMMAs apart
#pragma unroll
            for (int i = 0; i < MT; i++)
#pragma unroll
                for (int j = 0; j < MT; j++) dmma(cre[i][j][0], cre[i][j][1], ar[i], br[j]);
#pragma unroll
            for (int i = 0; i < MT; i++)
#pragma unroll
                for (int j = 0; j < MT; j++) dmma(cim[i][j][0], cim[i][j][1], ar[i], bi[j]);
#pragma unroll
            for (int i = 0; i < MT; i++)
#pragma unroll
                for (int j = 0; j < MT; j++) dmma(cre[i][j][0], cre[i][j][1], aim[i], bi[j]);
#pragma unroll
            for (int i = 0; i < MT; i++)
#pragma unroll
                for (int j = 0; j < MT; j++) dmma(cim[i][j][0], cim[i][j][1], naim[i], br[j]);
        }
    }
    cp_async_wait<0>();
    __syncthreads();

    if (GROUP == 0) {
        if (P.kind == EPI_PLANAR) {
            // split-precision path: column maxima of |B| (rows m of this tile),
            // reduced over the 8 row groups of a warp, then one atomic per column
            double *bmax = P.colmax;
            if (bmax) {
#pragma unroll
                for (int j = 0; j < MT; j++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        double mx = 0.0;
#pragma unroll
                        for (int i = 0; i < MT; i++) mx = fmax(mx, fmax(fabs(cre[i][j][h]), fabs(cim[i][j][h])));
                        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
                        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                        const int n = n0 + nw + j * 8 + 2 * (lane & 3) + h;
                        if (lane < 4 && n < P.N) atomic_max_nonneg(bmax + n, mx);
                    }
            }
#pragma unroll
            for (int i = 0; i < MT; i++)
#pragma unroll
                for (int j = 0; j < MT; j++) {
                    const int m = m0 + mw + i * 8 + (lane >> 2);
                    const int n = n0 + nw + j * 8 + 2 * (lane & 3);
                    if (m >= P.M) continue;
                    if (n + 1 < P.N) {
                        *reinterpret_cast<double2 *>(P.outr + (size_t)m * P.ldo + n) = make_double2(cre[i][j][0], cre[i][j][1]);
                        *reinterpret_cast<double2 *>(P.outi + (size_t)m * P.ldo + n) = make_double2(cim[i][j][0], cim[i][j][1]);
                    } else if (n < P.N) {
                        P.outr[(size_t)m * P.ldo + n] = cre[i][j][0];
                        P.outi[(size_t)m * P.ldo + n] = cim[i][j][0];
                    }
                }
            return;
        }
        // EPI_LOROWS
#pragma unroll
        for (int i = 0; i < MT; i++)
#pragma unroll
            for (int j = 0; j < MT; j++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int r = m0 + mw + i * 8 + (lane >> 2);
                    const int g = n0 + nw + j * 8 + 2 * (lane & 3) + h;
                    if (r >= P.M || g >= P.N) continue;
                    exs_complex v; v.re = cre[i][j][h]; v.im = cim[i][j][h];
                    exs_complex vc; vc.re = v.re; vc.im = -v.im;
                    P.z[(size_t)(P.row0 + r) + (size_t)P.ldz * g] = v;
                    P.z[(size_t)g + (size_t)P.ldz * (P.row0 + r)] = vc;
                }
        return;
    }
    // EPI_HAM / EPI_OVL: APW-APW block, upper tiles, interstitial + mirror.
    int *s_iv = reinterpret_cast<int *>(smem);                 // [2 EDGE][3]
    double *s_v = smem + 3 * EDGE;                             // [2 EDGE][3], after 24 EDGE bytes
    const KDesc kd = ks[P.kidx];
    {
        const int t = threadIdx.x;                             // rows, then columns
        const int idx = (t < EDGE) ? (m0 + t) : (n0 + t - EDGE);
        if (t < 2 * EDGE && idx < kd.ngp) {
            int g = kd.igpig[idx] - 1;
            if (g < 0 || g >= p.ngrtot) {      // caller's index table out of range
                atomicOr(p.err, DEV_ERR_INDEX);
                g = 0;
            }
            s_iv[3 * t + 0] = p.ivg[3 * g + 0];
            s_iv[3 * t + 1] = p.ivg[3 * g + 1];
            s_iv[3 * t + 2] = p.ivg[3 * g + 2];
            s_v[3 * t + 0] = kd.vgpc[3 * idx + 0];
            s_v[3 * t + 1] = kd.vgpc[3 * idx + 1];
            s_v[3 * t + 2] = kd.vgpc[3 * idx + 2];
        }
    }
    __syncthreads();
    if (idle) return;
    const int ngp = kd.ngp;
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int j = 0; j < MT; j++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int li = mw + i * 8 + (lane >> 2);
                const int lj = nw + j * 8 + 2 * (lane & 3) + h;
                const int gi = m0 + li, gj = n0 + lj;
                if (gi >= ngp || gj >= ngp || gi > gj) continue;
                double zr = cre[i][j][h], zi = cim[i][j][h];
                double ar, ai;
                if (interstitial(p, P.kind, s_iv + 3 * li, s_iv + 3 * (EDGE + lj), s_v + 3 * li, s_v + 3 * (EDGE + lj),
                                 ar, ai)) {
                    zr += ar;
                    zi += ai;
                }
                exs_complex v; v.re = zr; v.im = zi;
                P.z[(size_t)gi + (size_t)P.ldz * gj] = v;
                if (gi < gj) {
                    exs_complex vc; vc.re = zr; vc.im = -zi;
                    P.z[(size_t)gj + (size_t)P.ldz * gi] = vc;
                }
            }
}

// ---------------------------------------------------------------- host side
// Tile edge for a set of problems.  A tile's time is its area over the FP64
// pipe of one SM, so a launch of n tiles takes edge^2 max(1, n / 148) units;
// the smaller tiles re-read more of their operands (0.9 and 0.7 of the rate).
// One k-point of the two-atom cell: H and O 156 us in two launches of 64-tiles
// -> 14 us (16), h_a A and the lo rows 62 -> 8 us; APW-lo rows of 27 k-points
// (27 rows) 926 -> 498 us (32); A C of the eight-atom adjoint 178 -> 124 us (32).
int gemm_edge(const long long n[3])
{
    const int edge[3] = {64, 32, 16};
    const double rate[3] = {1.0, 0.9, 0.7};
    int best = 0;
    double tb = 0.0;
    for (int q = 0; q < 3; q++) {
        const double t = (double)edge[q] * edge[q] * std::max(1.0, (double)n[q] / 148.0) / rate[q];
        if (q == 0 || t < tb) {
            tb = t;
            best = q;
        }
    }
    return edge[best];
}

static long long tile_count(const GemmProb &P, int edge)
{
    const long long tm = (P.M + edge - 1) / edge, tn = (P.N + edge - 1) / edge;
    return (P.kind == EPI_HAM || P.kind == EPI_OVL) ? tm * (tm + 1) / 2 : tm * tn;
}

void gemm_tiles(const std::vector<GemmProb> &probs, int first, int last, int edge, std::vector<TileWork> &w)
{
    for (int i = first; i < last; i++) {
        const GemmProb &P = probs[i];
        const bool upper = P.kind == EPI_HAM || P.kind == EPI_OVL;
        for (int tm = 0; tm < (P.M + edge - 1) / edge; tm++)
            for (int tn = upper ? tm : 0; tn < (P.N + edge - 1) / edge; tn++) w.push_back({i, tm, tn});
    }
}

int gemm_edge_of(const std::vector<GemmProb> &probs, int first, int last)
{
    long long n[3] = {0, 0, 0};
    const int edge[3] = {64, 32, 16};
    for (int q = 0; q < 3; q++)
        for (int i = first; i < last; i++) n[q] += tile_count(probs[i], edge[q]);
    return gemm_edge(n);
}

template <int GROUP, int EDGE>
static cudaError_t launch_edge(const DevParams &p, const GemmProb *d_probs, const TileWork *d_work, int nwork,
                               const KDesc *d_k, cudaStream_t s)
{
    static std::atomic<unsigned long long> attr{0};
    cudaError_t e = once_per_device(attr, [] {
        return cudaFuncSetAttribute(zgemm_dmma_kernel<GROUP, EDGE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)GemmCfg<EDGE>::SMEM);
    });
    if (e != cudaSuccess) return e;
    zgemm_dmma_kernel<GROUP, EDGE><<<(unsigned)nwork, GB_THREADS, GemmCfg<EDGE>::SMEM, s>>>(p, d_probs, d_work, d_k);
    return cudaGetLastError();
}

template <int GROUP>
static cudaError_t launch_group(int edge, const DevParams &p, const GemmProb *d_probs, const TileWork *d_work,
                                int nwork, const KDesc *d_k, cudaStream_t s)
{
    if (nwork <= 0) return cudaSuccess;
    if (edge == 16) return launch_edge<GROUP, 16>(p, d_probs, d_work, nwork, d_k, s);
    if (edge == 32) return launch_edge<GROUP, 32>(p, d_probs, d_work, nwork, d_k, s);
    return launch_edge<GROUP, 64>(p, d_probs, d_work, nwork, d_k, s);
}

// Problem and tile tables of the GEMM launches of one batched call: work[0]
// h_a A and work[1] the APW-lo rows of H (in work[0] too when they take the
// same tile edge), work[2] H and O.
void build_gemm_tables(const exs_ctx *c, const std::vector<KDesc> &ks, GemmTables &t)
{
    t.probs.clear();
    for (auto &w : t.work) w.clear();
    for (int kind : {EPI_PLANAR, EPI_LOROWS})
        for (size_t k = 0; k < ks.size(); k++) {
            const int ncols = std::min(c->npad, (ks[k].ngp + 63) / 64 * 64);
            for (int ias = 0; ias < c->natmtot; ias++) {
                const AtomDesc &a = c->atoms[ias];
                GemmProb P{};
                P.kind = (short)kind;
                P.yr = ks[k].ar + (size_t)a.apw_off * c->npad;
                P.yi = ks[k].ai + (size_t)a.apw_off * c->npad;
                P.ldy = c->npad;
                P.K = a.napw;
                P.conjx = 0;
                P.kidx = (int)k;
                if (kind == EPI_PLANAR) {      // B_a = h_a A_a (planar output, all padded columns)
                    P.xr = c->d_haa_r + (size_t)ias * c->ldh * c->ldh;
                    P.xi = c->d_haa_i + (size_t)ias * c->ldh * c->ldh;
                    P.ldx = c->ldh;
                    P.M = a.napw;
                    P.N = ncols;
                    P.outr = ks[k].br + (size_t)a.apw_off * c->npad;
                    P.outi = ks[k].bi + (size_t)a.apw_off * c->npad;
                    P.ldo = c->npad;
                    P.colmax = ks[k].oz_scale && !ks[k].oz_part ? ks[k].oz_scale + c->npad : nullptr;
                } else {                       // APW-lo rows of H
                    if (a.losize == 0) continue;
                    P.xr = c->d_loa_r + (size_t)ias * c->ldlo * c->maxaa;
                    P.xi = c->d_loa_i + (size_t)ias * c->ldlo * c->maxaa;
                    P.ldx = c->ldlo;
                    P.M = a.losize;
                    P.N = ks[k].ngp;
                    P.z = ks[k].h;
                    P.ldz = ks[k].nmat;
                    P.row0 = ks[k].ngp + a.lo_off;
                }
                t.probs.push_back(P);
            }
            if (kind == EPI_PLANAR && k + 1 == ks.size()) t.first_lo = (int)t.probs.size();
        }
    t.first_ho = (int)t.probs.size();
    // H = A^H B and O = A^H A (A^H C for iora*), upper tiles
    for (size_t k = 0; k < ks.size(); k++)
        for (int kind : {EPI_HAM, EPI_OVL}) {
            GemmProb P{};
            P.kind = (short)kind;
            P.xr = ks[k].ar; P.xi = ks[k].ai; P.ldx = c->npad;
            if (kind == EPI_HAM) { P.yr = ks[k].br; P.yi = ks[k].bi; }
            else { P.yr = ks[k].cr; P.yi = ks[k].ci; }
            P.ldy = c->npad;
            P.M = P.N = ks[k].ngp;
            P.K = c->K;
            P.conjx = 1;
            P.z = kind == EPI_HAM ? ks[k].h : ks[k].o;
            P.ldz = ks[k].nmat;
            P.kidx = (int)k;
            t.probs.push_back(P);
        }
    t.edge[0] = gemm_edge_of(t.probs, 0, t.first_lo);
    t.edge[1] = gemm_edge_of(t.probs, t.first_lo, t.first_ho);
    t.edge[2] = gemm_edge_of(t.probs, t.first_ho, (int)t.probs.size());
    gemm_tiles(t.probs, 0, t.first_lo, t.edge[0], t.work[0]);
    gemm_tiles(t.probs, t.first_lo, t.first_ho, t.edge[1], t.work[t.edge[1] == t.edge[0] ? 0 : 1]);
    gemm_tiles(t.probs, t.first_ho, (int)t.probs.size(), t.edge[2], t.work[2]);
}

cudaError_t launch_gemm(int group, int edge, const DevParams &p, const void *d_probs, const void *d_work, int nwork,
                        const KDesc *d_k, cudaStream_t s)
{
    const GemmProb *P = (const GemmProb *)d_probs;
    const TileWork *W = (const TileWork *)d_work;
    return group == 0 ? launch_group<0>(edge, p, P, W, nwork, d_k, s) : launch_group<1>(edge, p, P, W, nwork, d_k, s);
}

// ------------------------------------------- lo blocks that need no product
// Local lo row rl of a species as (ilo, m): l of ilo, and m + l in `ml`.
__device__ __forceinline__ int lo_row(const DevParams &p, int is, int rl, int &l, int &ml)
{
    int ilo = 0, base = 0;
    l = 0;
    for (; ilo < p.nlorb[is]; ilo++) {
        l = p.lorbl[ilo + p.nlomax * is];
        if (rl < base + 2 * l + 1) break;
        base += 2 * l + 1;
    }
    ml = rl - base;
    return ilo;
}

// One atom (blockIdx.y) of one k-point (z).  Blocks x < gx: the APW-lo block
// of O (overlapsetup.f90:111-127) for 32 G: for lo function j = (ilo, m),
// O(G, ngp+idxlo) = sum_io conj(A(G, io, lm) (oalo(io,ilo) + h1loa)), and its
// conjugate, 32 lo rows at a time: the block decodes the rows once, writes
// O(G, j) column by column and O(j, G) from shared memory, j contiguous.  Blocks
// x >= gx: the atom's rows of 64 columns of the lo-lo blocks of H and O, zero
// in the columns of other atoms.  Bound by the writes: 27 k-points of the
// eight-atom cell 65 us (137 with one thread per element and 16-byte pieces of
// O(j, G)), 64 atoms 76 us (215).
constexpr int LO_R = 32, LO_COLS = 64;

__global__ void __launch_bounds__(256) lo_blocks_kernel(DevParams p, const KDesc *ks, int gx)
{
    __shared__ double2 T[LO_R][33];
    __shared__ double sw[LO_R][EXS_APWORD_MAX];
    __shared__ int sf[LO_R], sn[LO_R];
    const KDesc k = ks[blockIdx.z];
    const int ias = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const AtomDesc &at = p.atoms[ias];
    const int is = at.species, losize = at.losize, lo_off = at.lo_off;
    if (losize == 0) return;
    const size_t nm = (size_t)k.nmat;
    if ((int)blockIdx.x < gx) {
        const int g0 = blockIdx.x * 32;
        if (g0 >= k.ngp) return;
        for (int r0 = 0; r0 < losize; r0 += LO_R) {
            const int nr = min(LO_R, losize - r0);
            if (tid < nr) {
                int l, ml;
                const int ilo = lo_row(p, is, r0 + tid, l, ml);
                const int *apw = p.apword + (size_t)(p.lmaxapw + 1) * is;
                int f = at.apw_off;                              // APW row of (l, m, io = 0)
                for (int ll = 0; ll < l; ll++) f += (2 * ll + 1) * apw[ll];
                sf[tid] = f + ml * apw[l];
                sn[tid] = apw[l];
                for (int io = 0; io < apw[l]; io++) {
                    const size_t q = io + (size_t)p.apwordmax * (ilo + (size_t)p.nlomax * ias);
                    sw[tid][io] = p.oalo[q] + (p.h1loa ? p.h1loa[q] : 0.0);
                }
            }
            __syncthreads();
            const int g = g0 + lane;
            for (int r = warp; r < nr; r += 8) {
                double sr = 0.0, si = 0.0;
                if (g < k.ngp) {
                    for (int io = 0; io < sn[r]; io++) {
                        const size_t q = (size_t)(sf[r] + io) * p.npad + g;
                        sr += k.ar[q] * sw[r][io];
                        si -= k.ai[q] * sw[r][io];
                    }
                    exs_complex v;
                    v.re = sr;
                    v.im = si;
                    k.o[(size_t)g + nm * (k.ngp + lo_off + r0 + r)] = v;
                }
                T[r][lane] = make_double2(sr, -si);
            }
            __syncthreads();
            for (int q = warp; q < 32; q += 8)                   // lane = lo row
                if (g0 + q < k.ngp && lane < nr) {
                    const double2 z = T[lane][q];
                    exs_complex v;
                    v.re = z.x;
                    v.im = z.y;
                    k.o[(size_t)(k.ngp + lo_off + r0 + lane) + nm * (g0 + q)] = v;
                }
            __syncthreads();
        }
        return;
    }
    const int c0 = ((int)blockIdx.x - gx) * LO_COLS;
    for (int c = c0 + warp; c < min(p.nlotot, c0 + LO_COLS); c += 8)
        for (int r = lane; r < losize; r += 32) {
            const int cl = c - lo_off;
            exs_complex hv, ov;
            hv.re = hv.im = ov.re = ov.im = 0.0;
            if (cl >= 0 && cl < losize) {
                // H: upper from lolo(r, c); lower = conj(lolo(c, r))   (copy_UL)
                const int ru = min(r, cl), cu = max(r, cl);
                const exs_complex v = p.lolo[ru + (size_t)p.maxnlo * (cu + (size_t)p.maxnlo * ias)];
                hv.re = v.re;
                hv.im = r <= cl ? v.im : -v.im;
                // O: ololo(ilo1, ilo2) + h1lolo on equal l and m (taken from the upper element)
                int l1, m1, l2, m2;
                const int i1 = lo_row(p, is, ru, l1, m1), i2 = lo_row(p, is, cu, l2, m2);
                if (l1 == l2 && m1 == m2) {
                    ov.re = p.ololo[i1 + (size_t)p.nlomax * (i2 + (size_t)p.nlomax * ias)];
                    if (p.h1lolo) ov.re += p.h1lolo[i1 + (size_t)p.nlomax * (i2 + (size_t)p.nlomax * ias)];
                }
            }
            const size_t idx = (size_t)(k.ngp + lo_off + r) + nm * (k.ngp + c);
            k.h[idx] = hv;
            k.o[idx] = ov;
        }
}

cudaError_t launch_lo_blocks(const DevParams &p, const KDesc *d_k, int nk, int ngp_max, cudaStream_t s)
{
    if (p.nlotot == 0) return cudaSuccess;
    const int gx = (ngp_max + 31) / 32;
    lo_blocks_kernel<<<dim3(gx + (p.nlotot + LO_COLS - 1) / LO_COLS, p.natmtot, nk), 256, 0, s>>>(p, d_k, gx);
    return cudaGetLastError();
}

}  // namespace exs
