/*
 * lt_tree64.cu -- FP64 closed-form sums of a large grid with the far halos interpolated.
 *
 * Every sum of lt_closed64.cuh is analytic away from its halo, so over a tile of T x T pixels
 * the summed contribution of the halos that are far from the tile is a smooth function: it is
 * evaluated at 16 x 16 Chebyshev nodes of the tile and interpolated to the pixels by the tensor
 * Lagrange polynomial.  Only the halos near the tile are evaluated at its pixels.  A tile then
 * costs 256 (halos) + T^2 (near halos) pairs instead of T^2 (halos).  No counterpart in the
 * reference, which evaluates every pair (src/grid_gradient_GPU.cu:77-179).
 *
 * Which halos are far.  Continued to complex x (or y), a halo's sums are singular where
 * psi = sqrt(q^2 (s^2 + u^2) + v^2) vanishes: at an imaginary distance of at least
 * q sqrt(d^2 + s^2) from the real point at distance d.  Degree-15 interpolation converges like
 * rho^-16 with rho the sum of the semi-axes of the largest regular ellipse around the tile, so a
 * halo is far when
 *   q^2 (max(0, d - diagonal/2)^2 + s^2) >= (kFar h)^2,
 * d from the tile's centre, h the larger half width.  kFar is taken per sum from the measured
 * error of one term against extended precision (q 0.4 to 0.9, random orientation, core and cut
 * radii; relative to the term): deflection 5e-15 at 3.2, potential 2e-16 at 3.0, convergence and
 * shear 3e-15 at 4.0.  A far term is ~1% of its sum, so the truncation stays below the sum's own
 * rounding.
 *
 * Layout.  One CTA of 256 threads a tile: each thread owns one node while the catalogue streams
 * through shared memory (cp.async.bulk, two 64-record stages), then two pixels a pass while the
 * near records, gathered in shared memory, are walked.  Between them the node values are
 * contracted along y for the rows of a pass and along x for each pixel: 17 FP64 operations a
 * pixel and plane.  A tile's time is a latency chain (8 warps, one node a thread), so far records
 * go two at a time: 410 -> 360 us for the deflection of 200 halos on 1024^2 with the rows of
 * tiles launched from the middle outwards, where most halos are, one CTA each (tiles strided over
 * resident CTAs left SMs idle for 26% of the time).
 */
#include <cmath>
#include <cuda_runtime.h>

#include "lt_bulk.cuh"
#include "lt_eval.cuh"
#include "lt_internal.h"

namespace lt {

constexpr int kTreeThreads = 256;
constexpr int kNodes = 16;
constexpr int kNearStage = 128; /* near records staged at once: both stages of the walk */
constexpr int kNearBlock = 8;
constexpr int kNearList = 2048; /* near halos of a tile; a tile with more evaluates every halo */

/* Tile sides, and per side the Lagrange basis L[i][c] of the nodes at pixel c of T. */
constexpr int kSides[] = {32, 48, 64, 128};
constexpr int kSideTotal = 32 + 48 + 64 + 128;
__device__ double g_nodes[kNodes];
__device__ double g_lagrange[kNodes * kSideTotal];

/* Fill the tables of the current device (identical values every time). */
int tree_tables()
{
    static double nodes[kNodes], lag[kNodes * kSideTotal];
    const long double pi = acosl(-1.0L);
    for (int k = 0; k < kNodes; k++) nodes[k] = (double)cosl((2 * k + 1) * pi / (2 * kNodes));
    int off = 0;
    for (int T : kSides) {
        for (int c = 0; c < T; c++) {
            const long double x = -1.0L + 2.0L * c / (T - 1);
            for (int i = 0; i < kNodes; i++) {
                long double l = 1.0L;
                for (int j = 0; j < kNodes; j++)
                    if (j != i) l *= (x - nodes[j]) / ((long double)nodes[i] - nodes[j]);
                lag[off + i * T + c] = (double)l;
            }
        }
        off += kNodes * T;
    }
    cudaError_t e = cudaMemcpyToSymbol(g_nodes, nodes, sizeof(nodes));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_lagrange, lag, sizeof(lag));
    return (int)e;
}

struct TreeArgs {
    GridArgs g;
    const int32_t *types; /* profile type per halo */
    int32_t nhalos;
    int32_t T;            /* tile side */
    int32_t table;        /* its Lagrange table in g_lagrange */
};

template <int OP>
struct TreeOp {
    static constexpr int planes = (OP & OP_GRAD ? 2 : 0) + (OP & OP_HESS ? 3 : 0) + (OP & OP_POT ? 1 : 0);
    static constexpr double far = OP & OP_HESS ? 4.0 : OP & OP_GRAD ? 3.2 : 3.0;
};

/* Shared memory: the two stages, node values, one pass's row values, the Lagrange table. */
template <int OP>
static size_t tree_smem(int T)
{
    return 2 * LT_CHUNK * sizeof(lt_nie64) +
           sizeof(double) * (TreeOp<OP>::planes * kNodes * (kNodes + 2 * kTreeThreads / T) + kNodes * T) +
           sizeof(int32_t) * kNearList;
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

template <int OP>
__global__ void __launch_bounds__(kTreeThreads, 2) tree64_kernel(const TreeArgs A)
{
    constexpr int NQ = TreeOp<OP>::planes;
    const GridArgs &a = A.g;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ uint32_t s_far[2];
    __shared__ int32_t s_type[kNearStage];
    __shared__ int s_near;
    lt_nie64 *stage = reinterpret_cast<lt_nie64 *>(smem);
    const int T = A.T, rows = 2 * kTreeThreads / T;
    double *F = reinterpret_cast<double *>(smem + 2 * LT_CHUNK * sizeof(lt_nie64)); /* [plane][j][i] */
    double *H = F + NQ * kNodes * kNodes;                                           /* [plane][row][i] */
    double *L = H + NQ * kNodes * rows;                                             /* [i][column] */
    int32_t *list = reinterpret_cast<int32_t *>(L + kNodes * T);

    const int tid = threadIdx.x;
    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        mbar_fence_init();
    }
    for (int e = tid; e < kNodes * T; e += kTreeThreads) L[e] = g_lagrange[A.table + e];
    const double node_x = g_nodes[tid & 15], node_y = g_nodes[tid >> 4];
    uint32_t phase[2] = {0, 0};
    __syncthreads();

    auto issue = [&](int ci) {
        const lt_chunk c = a.chunks[ci];
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(&bars[ci & 1], (uint32_t)c.count * (uint32_t)sizeof(lt_nie64));
        bulk_g2s(stage + (ci & 1) * LT_CHUNK, a.nie + c.start, (uint32_t)c.count * (uint32_t)sizeof(lt_nie64),
                 &bars[ci & 1]);
    };

    /* rows of tiles from the middle outwards: the halos crowd there, and the dear tiles go first */
    const int trows = a.ntiles / a.tiles_x, mid = (trows - 1) / 2;
    const int r = (int)blockIdx.x / a.tiles_x, row = mid + ((r & 1) ? (r + 1) / 2 : -(r / 2));
    const int tx0 = ((int)blockIdx.x % a.tiles_x) * T, ty0 = row * T;
    const double x0 = pixel_x(a, tx0), x1 = pixel_x(a, tx0 + T - 1);
    const double y0 = pixel_y(a, ty0), y1 = pixel_y(a, ty0 + T - 1);
    const double xc = 0.5 * (x0 + x1), yc = 0.5 * (y0 + y1), hx = 0.5 * (x1 - x0), hy = 0.5 * (y1 - y0);
    const double diag = sqrt(hx * hx + hy * hy), reach = TreeOp<OP>::far * fmax(fabs(hx), fabs(hy));

    /* the walk: near halos to the list, far ones summed at this thread's node */
    double f[1][NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) f[0][q] = 0.;
    const double nx[1] = {fma(hx, node_x, xc)}, ny[1] = {fma(hy, node_y, yc)};
    int nlist = 0; /* warp 0's count of near halos */
    if (tid == 0) issue(0);
    for (int ci = 0; ci < a.nchunks; ci++) {
        const int b = ci & 1;
        if (tid == 0 && ci + 1 < a.nchunks) issue(ci + 1);
        if (!wait_tile(&bars[b], phase[b], a.status)) {
            if (tid == 0 && ci + 1 < a.nchunks) drain_tile(&bars[b ^ 1], phase[b ^ 1]);
            return;
        }
        phase[b] ^= 1;
        const lt_chunk c = a.chunks[ci];
        const lt_nie64 *recs = stage + b * LT_CHUNK;
        if (tid < 32) { /* one warp, so that the list keeps the catalogue's order */
#pragma unroll
            for (int w = 0; w < 2; w++) {
                const int i = 32 * w + tid;
                bool far = false;
                if (i < c.count) {
                    const lt_nie64 &r = recs[i];
                    const double dx = r.x0 - xc, dy = r.y0 - yc;
                    const double d = fmax(sqrt(dx * dx + dy * dy) - diag, 0.);
                    const double s = c.type == 5 ? 0. : r.sc;
                    far = (c.type == 5 ? r.q2 / r.k : r.q2) * (d * d + s * s) >= reach * reach;
                }
                const uint32_t m = __ballot_sync(0xffffffffu, far);
                const uint32_t near = __ballot_sync(0xffffffffu, i < c.count && !far);
                const int at = nlist + __popc(near & ((1u << tid) - 1u));
                if (i < c.count && !far && at < kNearList) list[at] = c.start + i;
                nlist += __popc(near);
                if (tid == 0) s_far[w] = m;
            }
        }
        __syncthreads();
        double fc[1][NQ]; /* the chunk's own sum: fewer roundings of the large total */
#pragma unroll
        for (int q = 0; q < NQ; q++) fc[0][q] = 0.;
#pragma unroll 1
        for (uint64_t m = (uint64_t)s_far[1] << 32 | s_far[0]; m;) { /* two records at a time */
            const int i = __ffsll(m) - 1;
            m &= m - 1;
            const int j = m ? __ffsll(m) - 1 : -1;
            m &= m - 1;
            if (j >= 0)
                tree_two<OP>(c.type, recs[i], recs[j], nx, ny, a.kmap, fc);
            else
                tree_any<OP, 1>(c.type, recs[i], nx, ny, a.kmap, fc);
        }
#pragma unroll
        for (int q = 0; q < NQ; q++) f[0][q] += fc[0][q];
        __syncthreads(); /* the stage and s_far are refilled */
    }
#pragma unroll
    for (int q = 0; q < NQ; q++) F[q * kNodes * kNodes + tid] = f[0][q];
    if (tid == 0) s_near = nlist;
    __syncthreads();
    int near = s_near;
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
    if (near <= kNearStage) gather(0, near);

    for (int r0 = 0; r0 < T && ty0 + r0 < a.ny; r0 += rows) {
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
        for (int i0 = 0; i0 < near; i0 += kNearStage) {
            const int n = near - i0 < kNearStage ? near - i0 : kNearStage;
            if (near > kNearStage) {
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

template <int OP>
static int launch_tree_op(TreeArgs &A, cudaStream_t s)
{
    const size_t smem = tree_smem<OP>(A.T);
    tree64_kernel<OP><<<A.g.ntiles, kTreeThreads, smem, s>>>(A);
    count_launch(1);
    return (int)cudaGetLastError();
}

int launch_tree64(const lt_catalog *cat, int op, const GridArgs &args, int side, void *stream)
{
    TreeArgs A;
    A.g = args;
    A.types = reinterpret_cast<const Fp32cCatalog *>(&cat->aux_desc)->types;
    A.nhalos = cat->nhalos;
    A.T = side;
    A.table = 0;
    for (int T : kSides) {
        if (T == side) break;
        A.table += kNodes * T;
    }
    A.g.tiles_x = (args.nx + side - 1) / side;
    A.g.ntiles = A.g.tiles_x * ((args.ny + side - 1) / side);
    cudaStream_t s = (cudaStream_t)stream;
    switch (op) {
    case OP_GRAD: return launch_tree_op<OP_GRAD>(A, s);
    case OP_POT: return launch_tree_op<OP_POT>(A, s);
    case OP_HESS: return launch_tree_op<OP_HESS>(A, s);
    case OP_HESS | OP_POT: return launch_tree_op<OP_HESS | OP_POT>(A, s);
    default: return (int)cudaErrorInvalidValue;
    }
}

/* The tile side for sums `op` of a grid, or 0 where the direct kernels are the faster: costs in
 * pairs per resident CTA (two an SM).  A tile costs 256 halos at the nodes (one pair a thread
 * in flight there instead of two, and the walk's barriers: x 1.25) and its near halos at T^2
 * pixels; the halos count as spread over their bounding box, tiles inside it being the dearest.
 * B200, ms, every pair / sides 32, 48, 64, 128: deflection of 200 halos on 1024^2 1.41 / 0.51,
 * 0.40, 0.38, 2.58; of 1000 on 4096^2 110 / 31.3, 14.7, 8.8, 6.6; of 1000 on 500^2 2.00 / 0.77,
 * 1.37, 3.14, 23; potential of 1000 on 2048^2 45.3 / 11.6, 6.0, 4.3, 10.2; lens maps of 500 on
 * 1199 x 901 7.11 / 2.18, 1.72, 1.74, 13.2.  The rule takes 0.41, 6.8, 0.78, 4.3 and 1.69
 * (block sums included). */
int tree_side(const lt_catalog *cat, int op, int nx, int ny, double dx, double dy, int num_sms)
{
    const double n = cat->nhalos, slots = 2. * num_sms;
    if (op & ~(OP_GRAD | OP_HESS | OP_POT)) return 0;
    const double far = op & OP_HESS ? 4.0 : op & OP_GRAD ? 3.2 : 3.0, d = std::sqrt(2.);
    const double spread = M_PI * (far * far * cat->sum_iq2 + 2. * d * far * cat->sum_iq + 2. * n);
    const double grid = std::fabs(nx * dx * ny * dy), box = cat->box;
    const double pixels = (double)nx * ny;
    double best = 0.8 * n * 512. * std::ceil(pixels / (512. * slots));
    int side = 0;
    for (int T : kSides) {
        const double h = 0.5 * T * std::fmax(std::fabs(dx), std::fabs(dy));
        const double tiles = std::ceil(nx / (double)T) * std::ceil(ny / (double)T);
        auto cost = [&](double area) {
            const double near = area > 0. ? std::fmin(n, h * h * spread / area) : n;
            return 320. * n + (double)T * T * (1.1 * near + 1.5) + 4000.;
        };
        const double t = std::fmax(tiles * cost(std::fmax(grid, box)) / slots, cost(std::fmin(grid, box)));
        if (t < best) {
            best = t;
            side = T;
        }
    }
    return side;
}

template <int OP>
static cudaError_t allow_smem()
{
    return cudaFuncSetAttribute(tree64_kernel<OP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tree_smem<OP>(128) + 4096);
}

/* Once per context: the kernels' shared memory on the current device. */
int configure_tree64()
{
    for (cudaError_t e : {allow_smem<OP_GRAD>(), allow_smem<OP_POT>(), allow_smem<OP_HESS>(), allow_smem<OP_HESS | OP_POT>()})
        if (e != cudaSuccess) return (int)e;
    return (int)cudaSuccess;
}

} // namespace lt
