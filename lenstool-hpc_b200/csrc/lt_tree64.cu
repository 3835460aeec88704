/*
 * lt_tree64.cu -- FP64 closed-form sums of a large grid with the far halos interpolated.
 *
 * Every sum of lt_closed64.cuh is analytic away from its halo, so over a tile of T x T pixels
 * the summed contribution of the halos that are far from the tile is a smooth function: it is
 * evaluated at 16 x 16 Chebyshev nodes of the tile and interpolated to the pixels by the tensor
 * Lagrange polynomial; only the halos near the tile are evaluated at its pixels.  The halos that
 * are far from the square of 2 x 2 tiles around it (its parent) as well are summed at the
 * parent's nodes instead, once for the four tiles, and interpolated to theirs.  A tile then costs
 * 64 (halos far from the parent) + 256 (far from the tile only) + T^2 (near halos) pairs instead
 * of T^2 (halos).  No counterpart in the reference, which evaluates every pair
 * (src/grid_gradient_GPU.cu:77-179).
 *
 * Which halos are far.  Continued to complex x (or y), a halo's sums are singular where
 * psi = sqrt(q^2 (s^2 + u^2) + v^2) vanishes: at an imaginary distance of at least
 * q sqrt(d^2 + s^2) from the real point at distance d.  Degree-15 interpolation converges like
 * rho^-16 with rho the sum of the semi-axes of the largest regular ellipse around the tile, so a
 * halo is far when
 *   q^2 (max(0, d - diagonal/2)^2 + s^2) >= (kFar h)^2,
 * d from the tile's centre, h the larger half width, and lies outside the circle around the tile.
 * kFar is 3.2 for the deflection, 3.0 for the potential, 4.0 for convergence and shear.  The largest
 * truncation of one term at that limit against extended precision (q 0.02 to 1, random
 * orientation, core and cut radii; relative to its largest value over the tile): PIEMD 5e-15,
 * 3e-15, 4e-15; cut dPIE 7e-15, 1.4e-15, 7e-15 up to q = 0.9 and 2.7e-14, 2.5e-15, 2.0e-14 for
 * rounder ones, beyond whose cut core and cut terms cancel; SIS 1.1e-14, 1.1e-15, 4.5e-15 down to
 * q = 0.7 and 7e-14, 6e-15, 9e-15 at 0.02.  It falls by 16 powers of the distance, so that in a map
 * the sums' rounding is the larger: deflection of 200 halos on 1024^2 3.5e-16 (2-norm) of extended
 * precision, every pair in turn in 64 bits 5.4e-16 to 5.8e-16; fields with one dominant halo of
 * any of these kinds 2e-16 to 1.1e-15, at single pixels up to 4e-14 of the RMS.
 *
 * Layout.  One CTA of 256 threads a tile, a cluster of four CTAs a parent (two and eight for a
 * grid of few tiles: half of the tile's far halos and of its passes each).  A CTA sorts the
 * halos into lists, a halo a thread: its share of those far from the parent, those far from its
 * tile only, those near it; the listed records are gathered in shared memory, 128 at a time, and
 * each thread sums them at one node of the parent, then of the tile, two records at a time.  The
 * four shares of the parent's node values are read from the cluster's shared memory and
 * interpolated to the tile's nodes, those along y to the rows of a pass and along x to each pixel
 * (17 FP64 operations a pixel and plane); then each thread walks the near records for two pixels.
 * Bound by the FP64 pipe and, with few tiles, by the dearest tile's chain, so rows of parents
 * start from the middle of the grid outwards, where most halos are.
 * B200, ms, tiles alone (no parent, tiles streamed in order) / middle first and two records at a
 * time / parents: deflection of 200 halos on 1024^2 0.375 / 0.340 / 0.225, of 1000 on 4096^2
 * 6.6 / 5.03 / 3.27; potential of 200 on 512^2 0.24 / 0.25 / 0.18; lens maps of 500 on 1199 x 901
 * 1.69 / 1.56 / 1.01.
 */
#include <algorithm>
#include <cmath>
#include <cuda_runtime.h>

#include "lt_eval.cuh"
#include "lt_internal.h"

namespace lt {

constexpr int kTreeThreads = 256;
constexpr int kNodes = 16;
constexpr int kStage = 128;  /* records staged at once */
constexpr int kRound = 1024; /* halos classified between two walks */
constexpr int kNearBlock = 8;
constexpr int kSplit = 1024;    /* tree_side()'s mark of two CTAs a tile */
constexpr int kNearList = 2048; /* near halos of a tile; a tile with more evaluates every halo */

/* Tile sides, and per side T the Lagrange basis of the nodes: L[i][c] at pixel c of the tile, and
 * B[o][i][k] of the parent's nodes at node k of its child o. */
constexpr int kSides[] = {16, 32, 40, 48, 64, 96, 128};
constexpr int kSideCount = sizeof(kSides) / sizeof(int);
constexpr int kSideTotal = 16 + 32 + 40 + 48 + 64 + 96 + 128;
__device__ double g_nodes[kNodes];
__device__ double g_lagrange[kNodes * kSideTotal];
__device__ double g_parent[kSideCount * 2 * kNodes * kNodes];

/* The Lagrange polynomial of node i at x. */
static double basis(const double *nodes, int i, long double x)
{
    long double l = 1.0L;
    for (int j = 0; j < kNodes; j++)
        if (j != i) l *= (x - nodes[j]) / ((long double)nodes[i] - nodes[j]);
    return (double)l;
}

/* Fill the tables of the current device (identical values every time). */
int tree_tables()
{
    static double nodes[kNodes], lag[kNodes * kSideTotal], par[kSideCount * 2 * kNodes * kNodes];
    const long double pi = acosl(-1.0L);
    for (int k = 0; k < kNodes; k++) nodes[k] = (double)cosl((2 * k + 1) * pi / (2 * kNodes));
    double *l = lag, *p = par;
    for (int T : kSides) {
        for (int i = 0; i < kNodes; i++)
            for (int c = 0; c < T; c++) *l++ = basis(nodes, i, -1.0L + 2.0L * c / (T - 1));
        for (int o = 0; o < 2; o++)
            for (int i = 0; i < kNodes; i++)
                for (int k = 0; k < kNodes; k++) /* pixel o T + (T - 1) (1 + node) / 2 of 2 T */
                    *p++ = basis(nodes, i, -1.0L + 2.0L * (o * T + 0.5L * (T - 1) * (1.0L + nodes[k])) / (2 * T - 1));
    }
    cudaError_t e = cudaMemcpyToSymbol(g_nodes, nodes, sizeof(nodes));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_lagrange, lag, sizeof(lag));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_parent, par, sizeof(par));
    return (int)e;
}

struct TreeArgs {
    GridArgs g;
    const int32_t *types; /* profile type per halo */
    int32_t nhalos;
    int32_t T;            /* tile side */
    int32_t table;        /* its Lagrange table in g_lagrange */
    int32_t parent;       /* and in g_parent */
};

/* The cluster's barrier, and a double of CTA `rank`'s shared memory. */
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ double cluster_load(const double *p, int rank)
{
    uint32_t addr = (uint32_t)__cvta_generic_to_shared(p), at;
    double v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(at) : "memory");
    return v;
}

template <int OP>
struct TreeOp {
    static constexpr int planes = (OP & OP_GRAD ? 2 : 0) + (OP & OP_HESS ? 3 : 0) + (OP & OP_POT ? 1 : 0);
    static constexpr double far = OP & OP_HESS ? 4.0 : OP & OP_GRAD ? 3.2 : 3.0;
};

/* Shared memory: the stage, node values of the tile and of this CTA's share of the parent's, one
 * pass's row values, the Lagrange table, the lists. */
template <int OP>
static size_t tree_smem(int T)
{
    return kStage * sizeof(lt_nie64) +
           sizeof(double) * (TreeOp<OP>::planes * kNodes * (2 * kNodes + 2 * kTreeThreads / T) + kNodes * T) +
           sizeof(int32_t) * (kNearList + kRound + kRound / 4);
}

template <int OP, int TYPE, int P>
__device__ __forceinline__ void tree_pair(const lt_nie64 &r, const double (&px)[P], const double (&py)[P], int kmap,
                                          double (&s)[P][TreeOp<OP>::planes])
{
    constexpr int kh = OP & OP_GRAD ? 2 : 0, kp = kh + (OP & OP_HESS ? 3 : 0);
    const double w = kmap ? r.w : 1.0;
#pragma unroll
    for (int k = 0; k < P; k++) {
        const Nie64 n = nie64<TYPE>(r, px[k], py[k]);
        if (OP & OP_GRAD) grad_nie<TYPE>(r, n, s[k][0], s[k][1 % TreeOp<OP>::planes]);
        if (OP & OP_HESS)
            kg_nie<TYPE>(r, n, w, s[k][kh], s[k][(kh + 1) % TreeOp<OP>::planes], s[k][(kh + 2) % TreeOp<OP>::planes]);
        if (OP & OP_POT) pot_nie<TYPE>(r, n, s[k][kp % TreeOp<OP>::planes]);
    }
}

template <int OP, int P>
__device__ __forceinline__ void tree_any(int type, const lt_nie64 &r, const double (&px)[P], const double (&py)[P],
                                         int kmap, double (&s)[P][TreeOp<OP>::planes])
{
    switch (type) {
    case 81: tree_pair<OP, 81, P>(r, px, py, kmap, s); break;
    case 8: tree_pair<OP, 8, P>(r, px, py, kmap, s); break;
    case 5: tree_pair<OP, 5, P>(r, px, py, kmap, s); break;
    default: break;
    }
}

/* Two records at one point: two chains that interleave, added in their order. */
template <int OP>
__device__ __forceinline__ void tree_two(int type, const lt_nie64 &r0, const lt_nie64 &r1, const double (&px)[1],
                                         const double (&py)[1], int kmap, double (&s)[1][TreeOp<OP>::planes])
{
    double t[2][1][TreeOp<OP>::planes];
#pragma unroll
    for (int q = 0; q < TreeOp<OP>::planes; q++) t[0][0][q] = t[1][0][q] = 0.;
    switch (type) {
    case 81:
        tree_pair<OP, 81, 1>(r0, px, py, kmap, t[0]);
        tree_pair<OP, 81, 1>(r1, px, py, kmap, t[1]);
        break;
    case 8:
        tree_pair<OP, 8, 1>(r0, px, py, kmap, t[0]);
        tree_pair<OP, 8, 1>(r1, px, py, kmap, t[1]);
        break;
    case 5:
        tree_pair<OP, 5, 1>(r0, px, py, kmap, t[0]);
        tree_pair<OP, 5, 1>(r1, px, py, kmap, t[1]);
        break;
    default: break;
    }
#pragma unroll
    for (int q = 0; q < TreeOp<OP>::planes; q++) s[0][q] += t[0][0][q] + t[1][0][q];
}

/* The pixels of a tile: the interpolated far sums and its near halos, two pixels a thread a pass. */
template <int OP, int N>
__device__ __forceinline__ void tree_pixels(const TreeArgs &A, unsigned char *smem, int32_t *s_type,
                                            const int32_t *list, int near, int tx0, int ty0, int part, const double *F,
                                            double *H, const double *L)
{
    constexpr int NQ = TreeOp<OP>::planes;
    const GridArgs &a = A.g;
    lt_nie64 *stage = reinterpret_cast<lt_nie64 *>(smem);
    const int T = A.T, rows = 2 * kTreeThreads / T, tid = threadIdx.x;
    const bool all = near > kNearList; /* more than the list holds: every halo at every pixel */
    if (all) near = A.nhalos;
    auto gather = [&](int i0, int n) { /* near records i0 .. i0 + n - 1 */
        for (int e = tid; e < n * (int)(sizeof(lt_nie64) / 16); e += kTreeThreads) {
            const int i = i0 + e / (int)(sizeof(lt_nie64) / 16);
            const int4 *src = reinterpret_cast<const int4 *>(a.nie + (all ? i : list[i]));
            reinterpret_cast<int4 *>(stage)[e] = src[e % (int)(sizeof(lt_nie64) / 16)];
        }
        for (int e = tid; e < n; e += kTreeThreads) s_type[e] = A.types[all ? i0 + e : list[i0 + e]];
    };
    if (near <= kStage) gather(0, near);

    for (int r0 = part * rows; r0 < T && ty0 + r0 < a.ny; r0 += N * rows) {
        __syncthreads(); /* F and the gathered records; H is free */
        for (int e = tid; e < NQ * rows * kNodes; e += kTreeThreads) {
            const int q = e / (rows * kNodes), r = (e / kNodes) % rows, i = e % kNodes;
            const int row = r0 + r < T ? r0 + r : T - 1;
            double h = 0.;
#pragma unroll
            for (int j = 0; j < kNodes; j++) h = fma(L[j * T + row], F[q * kNodes * kNodes + j * kNodes + i], h);
            H[e] = h;
        }
        double px[2], py[2], s[2][NQ];
        int ix[2], iy[2], rr[2], cc[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int p = tid + k * kTreeThreads;
            rr[k] = p / T;
            cc[k] = p % T;
            ix[k] = tx0 + cc[k];
            iy[k] = rr[k] < rows && r0 + rr[k] < T ? ty0 + r0 + rr[k] : a.ny; /* >= ny: no pixel */
            if (rr[k] >= rows) rr[k] = 0;
            px[k] = pixel_x(a, ix[k] < a.nx ? ix[k] : a.nx - 1);
            py[k] = pixel_y(a, iy[k] < a.ny ? iy[k] : a.ny - 1);
#pragma unroll
            for (int q = 0; q < NQ; q++) s[k][q] = 0.;
        }
        for (int i0 = 0; i0 < near; i0 += kStage) {
            const int n = near - i0 < kStage ? near - i0 : kStage;
            if (near > kStage) {
                __syncthreads();
                gather(i0, n);
                __syncthreads();
            }
#pragma unroll 1
            for (int b = 0; b < n; b += kNearBlock) { /* sums of blocks, as the chunks above */
                double sb[2][NQ];
#pragma unroll
                for (int q = 0; q < NQ; q++) sb[0][q] = sb[1][q] = 0.;
#pragma unroll 1
                for (int i = b; i < n && i < b + kNearBlock; i++)
                    tree_any<OP, 2>(s_type[i], stage[i], px, py, a.kmap, sb);
#pragma unroll
                for (int q = 0; q < NQ; q++) {
                    s[0][q] += sb[0][q];
                    s[1][q] += sb[1][q];
                }
            }
        }
        __syncthreads(); /* H */
#pragma unroll
        for (int k = 0; k < 2; k++) {
            if (all) continue;
            double t[NQ];
#pragma unroll
            for (int q = 0; q < NQ; q++) t[q] = 0.;
#pragma unroll
            for (int i = 0; i < kNodes; i++) {
                const double l = L[i * T + cc[k]];
#pragma unroll
                for (int q = 0; q < NQ; q++) t[q] = fma(l, H[(q * rows + rr[k]) * kNodes + i], t[q]);
            }
#pragma unroll
            for (int q = 0; q < NQ; q++) s[k][q] += t[q];
        }
#pragma unroll
        for (int k = 0; k < 2; k++) {
            if (ix[k] >= a.nx || iy[k] >= a.ny) continue;
            constexpr int kh = OP & OP_GRAD ? 2 : 0, kp = kh + (OP & OP_HESS ? 3 : 0);
            double hxx = 0., hyy = 0., hxy = 0.;
            if (OP & OP_HESS) nie_hessian(s[k][kh], s[k][(kh + 1) % NQ], s[k][(kh + 2) % NQ], hxx, hyy, hxy);
            const long pix = (long)iy[k] * a.nx + ix[k];
            for (int o = 0; o < a.nout; o++)
                a.out[o][pix] = map_value4(a.kinds[o], OP & OP_GRAD ? s[k][0] : 0., OP & OP_GRAD ? s[k][1 % NQ] : 0.,
                                           hxx, hyy, hxy, hxy, OP & OP_POT ? s[k][kp % NQ] : 0., a.D, a.mult, a.scale);
        }
    }
}

/* Records [b, e) of the stage summed at one node a thread, two at a time where they are alike. */
template <int OP>
__device__ __forceinline__ void tree_walk(const lt_nie64 *stage, const int32_t *type, int b, int e,
                                          const double (&px)[1], const double (&py)[1], int kmap, double *out)
{
    constexpr int NQ = TreeOp<OP>::planes;
    if (b >= e) return;
    double fc[1][NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) fc[0][q] = 0.;
#pragma unroll 1
    for (; b < e; b++) {
        if (b + 1 < e && type[b] == type[b + 1]) {
            tree_two<OP>(type[b], stage[b], stage[b + 1], px, py, kmap, fc);
            b++;
        } else
            tree_any<OP, 1>(type[b], stage[b], px, py, kmap, fc);
    }
#pragma unroll
    for (int q = 0; q < NQ; q++) out[q * kNodes * kNodes] += fc[0][q];
}

/* The centre, half widths and reach of a square of tiles. */
struct Square {
    double xc, yc, hx, hy, diag, reach2;
    __device__ __forceinline__ Square(const GridArgs &a, int tx0, int ty0, int T, double far)
    {
        const double x0 = pixel_x(a, tx0), x1 = pixel_x(a, tx0 + T - 1);
        const double y0 = pixel_y(a, ty0), y1 = pixel_y(a, ty0 + T - 1);
        xc = 0.5 * (x0 + x1);
        yc = 0.5 * (y0 + y1);
        hx = 0.5 * (x1 - x0);
        hy = 0.5 * (y1 - y0);
        diag = 1.0001 * sqrt(hx * hx + hy * hy); /* the corners' pixels inside */
        const double r = far * fmax(fabs(hx), fabs(hy));
        reach2 = r * r;
    }
    __device__ __forceinline__ bool is_far(double x, double y, double q2, double s2) const
    {
        const double dx = x - xc, dy = y - yc, d = fmax(sqrt(dx * dx + dy * dy) - diag, 0.);
        /* d = 0: a halo inside is near whatever its core, for at its centre the potential is 0/0 */
        return d > 0. && q2 * (d * d + s2) >= reach2;
    }
};

/* N CTAs a tile, 4 N a cluster. */
template <int OP, int N>
__global__ void __launch_bounds__(kTreeThreads, 2) tree64_kernel(const TreeArgs A)
{
    constexpr int NQ = TreeOp<OP>::planes, NN = kNodes * kNodes;
    const GridArgs &a = A.g;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int32_t s_type[kStage];
    __shared__ int s_cnt[2][3][kTreeThreads / 32];
    lt_nie64 *stage = reinterpret_cast<lt_nie64 *>(smem);
    const int T = A.T, rows = 2 * kTreeThreads / T;
    double *F = reinterpret_cast<double *>(smem + kStage * sizeof(lt_nie64)); /* [plane][j][i] */
    double *S = F + NQ * NN;                                                  /* the share, [plane][j][i] */
    double *H = S + NQ * NN;                                                  /* [plane][row][i] */
    double *L = H + NQ * kNodes * rows;                                       /* [i][column] */
    int32_t *list = reinterpret_cast<int32_t *>(L + kNodes * T);              /* near halos */
    int32_t *own = list + kNearList, *share = own + kRound;                   /* far halos of a round */

    constexpr int size = 4 * N;
    const int tid = threadIdx.x;
    const int rank = blockIdx.x & (size - 1), tile = rank & 3, part = rank >> 2;
    for (int e = tid; e < kNodes * T; e += kTreeThreads) L[e] = g_lagrange[A.table + e];
    const double node_x = g_nodes[tid & 15], node_y = g_nodes[tid >> 4];

    /* rows of clusters from the middle outwards: the halos crowd there, and the dear tiles go first */
    const int ccols = (a.tiles_x + 1) / 2, crows = (int)gridDim.x / (size * ccols), cl = (int)blockIdx.x / size;
    const int r = cl / ccols, crow = (crows - 1) / 2 + ((r & 1) ? (r + 1) / 2 : -(r / 2));
    const int px0 = 2 * T * (cl % ccols), py0 = 2 * T * crow;
    const int tx0 = px0 + (tile & 1) * T, ty0 = py0 + (tile >> 1) * T;
    const bool alive = tx0 < a.nx && ty0 < a.ny; /* a tile beyond the grid does its share only */
    const Square P(a, px0, py0, 2 * T, TreeOp<OP>::far), C(a, tx0, ty0, T, TreeOp<OP>::far);

#pragma unroll
    for (int q = 0; q < NQ; q++) F[q * NN + tid] = S[q * NN + tid] = 0.;
    int near = 0;
    for (int base = 0; base < A.nhalos; base += kRound) {
        /* the round's halos to the lists, in the catalogue's order: far from the parent (this
         * CTA's share of them), far from the tile only (all, or this CTA's half), near */
        int nshare = 0, nown = 0;
        for (int sub = 0; sub < kRound && base + sub < A.nhalos; sub += kTreeThreads) {
            const int i = base + sub + tid;
            int cls = -1;
            if (i < A.nhalos) {
                const lt_nie64 &h = a.nie[i];
                const bool point = A.types[i] == 5;
                const double x = h.x0, y = h.y0, q2 = point ? h.q2 / h.k : h.q2, s = point ? 0. : h.sc;
                if (P.is_far(x, y, q2, s * s))
                    cls = (i & (size - 1)) == rank ? 0 : -1;
                else if (alive)
                    cls = !C.is_far(x, y, q2, s * s) ? 2 : (i & (N - 1)) == part ? 1 : -1;
            }
            int at[3], tot[3];
            int (*cnt)[kTreeThreads / 32] = s_cnt[(sub / kTreeThreads) & 1];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const uint32_t m = __ballot_sync(0xffffffffu, cls == k);
                at[k] = __popc(m & ((1u << (tid & 31)) - 1u));
                if ((tid & 31) == 0) cnt[k][tid >> 5] = __popc(m);
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 3; k++) {
                tot[k] = 0;
#pragma unroll
                for (int w = 0; w < kTreeThreads / 32; w++) {
                    if (w == tid >> 5) at[k] += tot[k];
                    tot[k] += cnt[k][w];
                }
            }
            if (cls == 0) share[nshare + at[0]] = i;
            if (cls == 1) own[nown + at[1]] = i;
            if (cls == 2 && near + at[2] < kNearList) list[near + at[2]] = i;
            nshare += tot[0];
            nown += tot[1];
            near += tot[2];
        }
        /* their sums at this thread's node of the parent and of the tile */
        const int nfar = nshare + nown;
        for (int b = 0; b < nfar; b += kStage) {
            const int n = nfar - b < kStage ? nfar - b : kStage;
            __syncthreads(); /* the lists; the stage is free */
            for (int e = tid; e < n * (int)(sizeof(lt_nie64) / 16); e += kTreeThreads) {
                const int k = b + e / (int)(sizeof(lt_nie64) / 16);
                const int4 *src = reinterpret_cast<const int4 *>(a.nie + (k < nshare ? share[k] : own[k - nshare]));
                reinterpret_cast<int4 *>(stage)[e] = src[e % (int)(sizeof(lt_nie64) / 16)];
            }
            for (int e = tid; e < n; e += kTreeThreads)
                s_type[e] = A.types[b + e < nshare ? share[b + e] : own[b + e - nshare]];
            __syncthreads();
            const int m = nshare - b < 0 ? 0 : nshare - b < n ? nshare - b : n;
#pragma unroll 1
            for (int k = 0; k < 2; k++) {
                const double nx[1] = {k ? fma(C.hx, node_x, C.xc) : fma(P.hx, node_x, P.xc)};
                const double ny[1] = {k ? fma(C.hy, node_y, C.yc) : fma(P.hy, node_y, P.yc)};
                tree_walk<OP>(stage, s_type, k ? m : 0, k ? n : m, nx, ny, a.kmap, (k ? F : S) + tid);
            }
        }
        __syncthreads(); /* the lists are refilled */
    }

    /* the parent's node values, summed over the cluster, interpolated to the tile's nodes */
    cluster_arrive();
    cluster_wait();
    double *PP = reinterpret_cast<double *>(stage), *G = PP + NQ * NN; /* [plane][j][i] */
    double far_sum[NQ]; /* the tile's far halos at this node */
#pragma unroll
    for (int q = 0; q < NQ; q++) {
        double v[size];
#pragma unroll
        for (int k = 0; k < size; k++) v[k] = cluster_load(S + q * NN + tid, k);
        if (N == 2) {
#pragma unroll
            for (int k = 0; k < 4; k++) v[k] += v[(k + 4) % size];
            far_sum[q] = cluster_load(F + q * NN + tid, tile) + cluster_load(F + q * NN + tid, tile + 4);
        }
        PP[q * NN + tid] = (v[0] + v[1]) + (v[2] + v[3]);
    }
    cluster_arrive(); /* the shares are read: waited for before the exit and, N = 2, before F changes */
    if (alive) {
        __syncthreads();
        const double *bx = g_parent + A.parent + (tile & 1) * NN;
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            double g = 0.;
#pragma unroll
            for (int i = 0; i < kNodes; i++)
                g = fma(bx[i * kNodes + (tid & 15)], PP[q * NN + (tid & ~15) + i], g);
            G[q * NN + tid] = g;
        }
    }
    if (N == 2) cluster_wait();
    if (alive) {
        __syncthreads();
        const double *by = g_parent + A.parent + (tile >> 1) * NN;
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            double g = 0.;
#pragma unroll
            for (int j = 0; j < kNodes; j++)
                g = fma(by[j * kNodes + (tid >> 4)], G[q * NN + j * kNodes + (tid & 15)], g);
            F[q * NN + tid] = (N == 2 ? far_sum[q] : F[q * NN + tid]) + g;
        }
        __syncthreads(); /* F; the stage is free */
        tree_pixels<OP, N>(A, smem, s_type, list, near, tx0, ty0, part, F, H, L);
    }
    if (N == 1) cluster_wait();
}

template <int OP, int N>
static int launch_tree_op(TreeArgs &A, cudaStream_t s)
{
    const int clusters = ((A.g.tiles_x + 1) / 2) * ((A.g.ntiles / A.g.tiles_x + 1) / 2);
    cudaLaunchAttribute cluster = {};
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim.x = 4 * N;
    cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(4 * N * clusters);
    c.blockDim = dim3(kTreeThreads);
    c.dynamicSmemBytes = tree_smem<OP>(A.T);
    c.stream = s;
    c.attrs = &cluster;
    c.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&c, tree64_kernel<OP, N>, (const TreeArgs)A);
    count_launch(1);
    return (int)(e != cudaSuccess ? e : cudaGetLastError());
}

int launch_tree64(const lt_catalog *cat, int op, const GridArgs &args, int side, void *stream)
{
    TreeArgs A;
    A.g = args;
    A.types = reinterpret_cast<const Fp32cCatalog *>(&cat->aux_desc)->types;
    A.nhalos = cat->nhalos;
    A.T = side & (kSplit - 1);
    const bool two = side & kSplit;
    side = A.T;
    A.table = A.parent = 0;
    for (int T : kSides) {
        if (T == side) break;
        A.table += kNodes * T;
        A.parent += 2 * kNodes * kNodes;
    }
    A.g.tiles_x = (args.nx + side - 1) / side;
    A.g.ntiles = A.g.tiles_x * ((args.ny + side - 1) / side);
    cudaStream_t s = (cudaStream_t)stream;
    switch (op) {
    case OP_GRAD: return two ? launch_tree_op<OP_GRAD, 2>(A, s) : launch_tree_op<OP_GRAD, 1>(A, s);
    case OP_POT: return two ? launch_tree_op<OP_POT, 2>(A, s) : launch_tree_op<OP_POT, 1>(A, s);
    case OP_HESS: return two ? launch_tree_op<OP_HESS, 2>(A, s) : launch_tree_op<OP_HESS, 1>(A, s);
    case OP_HESS | OP_POT: return two ? launch_tree_op<OP_HESS | OP_POT, 2>(A, s) : launch_tree_op<OP_HESS | OP_POT, 1>(A, s);
    default: return (int)cudaErrorInvalidValue;
    }
}

/* Rows of a cluster of tiles. */
int tree_rows(int side) { return 2 * (side & (kSplit - 1)); }

/* The tile side for sums `op` of a grid, or 0 where the direct kernels are the faster: costs in
 * pairs per resident CTA (two an SM), fitted to 54 measured combinations of sum, grid (96^2 to
 * 4096^2) and halos (10 to 1000).  A tile costs its lists and quarter of the parent's nodes (57 a
 * halo: 64 pairs, cheaper for the halos that are not far), its own nodes for the halos that are
 * near the parent only, its passes of 512 pixels with the near halos and the interpolation; the
 * halos count as spread over their bounding box, tiles inside it being the dearest, and such a
 * tile alone on its SM runs at twice the rate.  The direct kernels cost their waves and the chain
 * of one record after another.  B200, ms, every pair / sides 16, 32, 40, 48, 64, 128, the pick in
 * brackets: deflection of 200 halos on 256^2 0.14 / [0.07] 0.14 0.28 0.43; of 1000 on 500^2
 * 2.00 / - [0.53] 1.00 1.43 3.2 23; of 200 on 1024^2 1.41 / - [0.22] 0.23 0.24 0.35 2.5; of 350 on
 * 1501 x 777 2.14 / - 0.32 [0.30] 0.33 0.42 2.7; of 1000 on 4096^2 110 / - 8.7 6.3 4.7 [3.3] 4.5;
 * lens maps of 300 on 96^2 [0.12] / 0.32 0.72. */
int tree_side(const lt_catalog *cat, int op, int nx, int ny, double dx, double dy, int num_sms)
{
    const double n = cat->nhalos, slots = 2. * num_sms;
    if (op & ~(OP_GRAD | OP_HESS | OP_POT)) return 0;
    const double far = op & OP_HESS ? 4.0 : op & OP_GRAD ? 3.2 : 3.0, d = std::sqrt(2.);
    const double spread = M_PI * (far * far * cat->sum_iq2 + 2. * d * far * cat->sum_iq + 2. * n);
    const double grid = std::fabs(nx * dx * ny * dy), box = cat->box;
    const double pixels = (double)nx * ny;
    double best = 512. * n * (0.265 + pixels / (512. * slots));
    int side = 0;
    for (int T : kSides) {
        const double h = 0.5 * T * std::fmax(std::fabs(dx), std::fabs(dy));
        const double tiles = 4. * std::ceil(nx / (2. * T)) * std::ceil(ny / (2. * T));
        const int rows = 2 * kTreeThreads / T, passes = (T + rows - 1) / rows;
        auto cost = [&](double area) {
            const double near = area > 0. ? std::fmin(n, h * h * spread / area) : n;
            const double parent = std::fmin(n, 4. * near);
            return 57. * n + 310. * (parent - near) + 512. * passes * (1.22 * near + 4.9) + 3250.;
        };
        const double t = std::fmax(tiles * cost(std::fmax(grid, box)) / slots, 0.5 * cost(std::fmin(grid, box)));
        if (t < best) {
            best = t;
            side = T;
        }
    }
    /* Two CTAs a tile where the tiles are fewer than the resident CTAs and dear enough for the
     * second's lists and interpolation.  B200, us, one / two: potential of 200 halos on 512^2 (256
     * tiles of 32) 179 / 162, of 400 on 400^2 340 / 313; deflection of 1000 on 500^2 538 / 501, on
     * 256^2 (256 tiles of 16, whose one pass is not shared) 538 / 455, but of 200 on 256^2 74 / 94,
     * of 10 on 400^2 21 / 32, of 300 on 800^2 (676 tiles) 246 / 273. */
    const double tiles = side ? 4. * std::ceil(nx / (2. * side)) * std::ceil(ny / (2. * side)) : 0.;
    return side && tiles <= slots && n >= (side > 16 ? 40 : 500) ? side | kSplit : side;
}

template <int OP>
static cudaError_t allow_smem()
{
    size_t most = 0;
    for (int T : kSides) most = std::max(most, tree_smem<OP>(T));
    const cudaError_t e = cudaFuncSetAttribute(tree64_kernel<OP, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(tree64_kernel<OP, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
}

/* Once per context: the kernels' shared memory on the current device. */
int configure_tree64()
{
    for (cudaError_t e : {allow_smem<OP_GRAD>(), allow_smem<OP_POT>(), allow_smem<OP_HESS>(), allow_smem<OP_HESS | OP_POT>()})
        if (e != cudaSuccess) return (int)e;
    return (int)cudaSuccess;
}

} // namespace lt
