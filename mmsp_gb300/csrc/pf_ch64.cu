// pf_ch64.cu -- FP64 Cahn-Hilliard step in two passes, as the reference runs it.
//
// The reference's update() (cahn-hilliard.cpp:69-79) makes two node loops per
// step: temp = mu(c) over every node, then c' = c + dt*M*lap(temp).  On GB300
// the FP64 pipe issues about two operations per clock per SM, a 64th of the
// FP32 rate, so the FP64 form is bound by its count of FP64 instructions,
// not by memory: HBM traffic is nearly free beside it.  A fused kernel has
// to recompute mu on the halo of every tile (1.2x the mu work on 256^3);
// these two kernels keep the reference's temp grid in HBM instead, so each
// mu is computed exactly once and each pass does the minimum FP64 work:
//
//   exact form       23 operations per cell (13 for mu, 10 for the update),
//                    the reference's order, every operation rounded on its
//                    own: bit-identical to the reference
//   contracted form  15 operations per cell on unit spacing (14.3 with shared
//                    pair sums, below; one more where kappa is not 1): the
//                    six-neighbour sum once,
//                    the centre term folded into the chemical potential's
//                    polynomial and into the update's multiply-add.  Within
//                    a few ulps per step of the exact form; held to 1e-12
//                    relative against the reference after the full runs.
//
// A thread owns one (y, z) column and walks a run of X planes, carrying
// c(x-1), c(x), c(x+1) in registers; the four in-plane neighbours come
// through L1 with periodic wraps precomputed per thread.  Blocks are small,
// so the block scheduler balances the FP64 work across SMs.
// Multiplies by 2 and the 0.0 + t of the Laplacian's first axis are done on
// the integer pipe (pf_device.cuh), and every decision about parameters
// (unit weights, kappa == 1, noise) is a template argument, so no FP64
// compare runs per cell.
#include <algorithm>

#include "pf_async.cuh"
#include "pf_device.cuh"
#include "pf_internal.h"

namespace pf {

constexpr int kC64Z = 32;        // block width along Z (one warp)
constexpr int kC64Y = 4;         // rows per block: 128 threads
// X planes per block (3D): short runs, so that small grids fill the SMs and
// no SM is left with a long last block.  us per step at 16 / 2 planes, exact
// form: 40^3 23.3 / 8.4, 100^3 72.3 / 59.7, 33x200x150 59.1 / 50.4, 256^3
// 742 / 739 (a run of 1 measured as 2).  Grids of so many planes that the
// launch's 65535 blocks along X would not do take longer runs, up to 16 planes.
constexpr int kC64Planes = 2, kC64MostPlanes = 16;
// The stochastic FP32 kernels (below) are bound by the deviates' arithmetic and
// by HBM, not by the FP64 pipe: short runs, which read more planes twice, are
// for grids that would leave SMs idle.  us per step at 2 / 8 / 16 planes: 40^3
// 5.9 / 9.5 / 14.7, 80^3 11.0 / 11.1 / 15.9, 100^3 17.3 / 16.4 / 19.0, 128^3
// 25.4 / 23.3 / 25.4, 187^3 70.7 / 59.0 / 58.9, 256^3 179 / 146 / 147.
constexpr int kC32Planes = 8;
constexpr long long kC32Long = 1000000;   // cells from which on the runs are that long

// Constants of both forms.
struct C64 {
    double wx, wy, wz;    // Laplacian weights of padded axes X, Y, Z
    double kappa, dtm, u;
    double w2;            // 2 (wx + wy + wz) over the real axes: the centre weight
    double poly0;         // contracted mu: 2 + kappa*w2 (CH) or -r + kappa*w2 (CH_POLY)
    double upd0;          // contracted update: -dt*M*w2
    double four, six;     // contracted CH: set in the kernel
};

// The constants of the expressions in registers (Ar::reg).
static __device__ __forceinline__ C64 held(const Ar<double>& A, C64 q)
{
    q.wx = A.reg(q.wx);
    q.wy = A.reg(q.wy);
    q.wz = A.reg(q.wz);
    q.kappa = A.reg(q.kappa);
    q.dtm = A.reg(q.dtm);
    q.u = A.reg(q.u);
    q.poly0 = A.reg(q.poly0);
    q.upd0 = A.reg(q.upd0);
    q.four = A.reg(4.0);
    q.six = A.reg(6.0);
    return q;
}

// Weighted sum of the neighbour pairs (sx, sy, sz: sums of the two
// neighbours along X, Y, Z), the contracted Laplacian without its centre term.
template <int DIM, bool UNIT>
static __device__ __forceinline__ double nsum(const Ar<double>& A, double sx, double sy, double sz, const C64& q)
{
    if (UNIT) return DIM == 3 ? A.add(A.add(sx, sy), sz) : A.add(sy, sz);
    return DIM == 3 ? fma(q.wx, sx, fma(q.wy, sy, A.mul(q.wz, sz))) : fma(q.wy, sy, A.mul(q.wz, sz));
}

// Contracted mu from the neighbours' sum: f'(c) - kappa (S - w2 c) = c * (poly0 + ...) - kappa S
template <int MODEL, bool KONE>
static __device__ __forceinline__ double mu_sum(const Ar<double>& A, double c, double s, const C64& q)
{
    double t;
    if (MODEL == MMSP_GPU_CH) {   // 2c(1-c)(1-2c) = c (2 + c (-6 + 4c))
        t = fma(fma(q.four, c, -q.six), c, q.poly0);
    } else {                      // -r c + u c^3 = c (-r + u c^2)
        t = fma(q.u, A.mul(c, c), q.poly0);
    }
    return KONE ? fma(t, c, -s) : fma(-q.kappa, s, A.mul(t, c));
}

template <int DIM, int MODEL, bool UNIT, bool KONE, bool EXACT>
static __device__ __forceinline__ double mu_cell(const Ar<double>& A, double c, double xh, double xl, double yh, double yl,
                                                 double zh, double zl, const C64& q, const P<double>& p)
{
    if (EXACT) {
        // temp = mu(c) in the reference's order (pf_device.cuh: lap_ref, ch_mu)
        const double lap = lap_ref<double, UNIT, DIM>(A, twice(c), xh, xl, yh, yl, zh, zl, p.wx, p.wy, p.wz);
        P<double> pk = p;
        if (KONE) pk.kappa = 1.0;   // constant: kappa_times folds to lap
        return ch_mu<double, MODEL>(A, c, lap, pk);
    }
    return mu_sum<MODEL, KONE>(A, c, nsum<DIM, UNIT>(A, A.add(xh, xl), A.add(yh, yl), A.add(zh, zl), q), q);
}

template <int DIM, int MODEL, bool UNIT, bool KONE, bool EXACT, bool NOISE>
__global__ void __launch_bounds__(kC64Z * kC64Y)
ch64_mu(const double* __restrict__ cin, double* __restrict__ mu, Geom g, C64 q0, P<double> p0, int planes)
{
    const Ar<double> A(g.dim);
    const C64 q = held(A, q0);
    const P<double> p = held(A, p0);
    const int z = blockIdx.x * kC64Z + threadIdx.x;
    const int y = blockIdx.y * kC64Y + threadIdx.y;
    if (z >= g.Z || y >= g.Y) return;   // no barrier in this kernel
    const int zl = z == 0 ? g.Z - 1 : z - 1, zh = z + 1 == g.Z ? 0 : z + 1;
    const long long row = (long long)y * g.Z;
    const long long rl = (long long)(y == 0 ? g.Y - 1 : y - 1) * g.Z;
    const long long rh = (long long)(y + 1 == g.Y ? 0 : y + 1) * g.Z;
    const int xs = blockIdx.z * planes;
    const int xe = min(xs + planes, g.X);
    auto plane = [&](int x) { return cin + (long long)x * g.YZ; };
    double a = 0.0, b = __ldg(plane(xs) + row + z);
    if (DIM == 3) a = __ldg(plane(xs == 0 ? g.X - 1 : xs - 1) + row + z);
    for (int x = xs; x < xe; x++) {
        const double* pc = plane(x);
        double n = 0.0;
        if (DIM == 3) n = __ldg(plane(x + 1 == g.X ? 0 : x + 1) + row + z);
        const double vyh = __ldg(pc + rh + z), vyl = __ldg(pc + rl + z);
        const double vzh = __ldg(pc + row + zh), vzl = __ldg(pc + row + zl);
        double m = mu_cell<DIM, MODEL, UNIT, KONE, EXACT>(A, b, n, a, vyh, vyl, vzh, vzl, q, p);
        // thermal noise of the stochastic forms (model_B.cpp:100-101, spinodal.cpp:95-97): mu + noise
        if (NOISE) m = A.add(m, noise_at(p, g.cells, (long long)x * g.YZ + row + z));
        mu[(long long)x * g.YZ + row + z] = m;
        a = b;
        b = n;
    }
}

template <int DIM, bool UNIT, bool EXACT>
__global__ void __launch_bounds__(kC64Z * kC64Y)
ch64_update(const double* __restrict__ cin, const double* __restrict__ mu, double* __restrict__ cout, Geom g, C64 q0,
            P<double> p0, int planes)
{
    const Ar<double> A(g.dim);
    const C64 q = held(A, q0);
    const P<double> p = held(A, p0);
    const int z = blockIdx.x * kC64Z + threadIdx.x;
    const int y = blockIdx.y * kC64Y + threadIdx.y;
    if (z >= g.Z || y >= g.Y) return;
    const int zl = z == 0 ? g.Z - 1 : z - 1, zh = z + 1 == g.Z ? 0 : z + 1;
    const long long row = (long long)y * g.Z;
    const long long rl = (long long)(y == 0 ? g.Y - 1 : y - 1) * g.Z;
    const long long rh = (long long)(y + 1 == g.Y ? 0 : y + 1) * g.Z;
    const int xs = blockIdx.z * planes;
    const int xe = min(xs + planes, g.X);
    auto plane = [&](int x) { return mu + (long long)x * g.YZ; };
    double a = 0.0, b = __ldg(plane(xs) + row + z);
    if (DIM == 3) a = __ldg(plane(xs == 0 ? g.X - 1 : xs - 1) + row + z);
    for (int x = xs; x < xe; x++) {
        const long long i = (long long)x * g.YZ + row + z;
        const double* pm = plane(x);
        double n = 0.0;
        if (DIM == 3) n = __ldg(plane(x + 1 == g.X ? 0 : x + 1) + row + z);
        const double myh = __ldg(pm + rh + z), myl = __ldg(pm + rl + z);
        const double mzh = __ldg(pm + row + zh), mzl = __ldg(pm + row + zl);
        const double c = __ldg(cin + i);
        double o;
        if (EXACT) {
            // newGrid(n) = GRID(n) + dt*M*lap(temp)   (cahn-hilliard.cpp:75-76)
            const double lap = lap_ref<double, UNIT, DIM>(A, twice(b), n, a, myh, myl, mzh, mzl, p.wx, p.wy, p.wz);
            o = A.add(c, A.mul(p.dtm, lap));
        } else {
            // c + dtM (S - w2 mu) = fma(dtM, S, c - dtM w2 mu)
            const double s = nsum<DIM, UNIT>(A, A.add(n, a), A.add(myh, myl), A.add(mzh, mzl), q);
            o = fma(q.dtm, s, fma(q.upd0, b, c));
        }
        cout[i] = o;
        a = b;
        b = n;
    }
}

// Contracted form on unit spacing, 3D: the same two passes with fewer additions.
//
// With D(x, y) = f(x+1, y) + f(x, y+1), the four neighbours along X and Y of a
// cell are D(x, y) + D(x-1, y-1): one addition a cell for D, one for the sum, in
// place of three.  A thread owns kC64Rows rows and walks X, so D(x-1, y-1) is
// the D of its row above from the plane before; only the first row's, and a
// run's first plane's, are added up anew: a Laplacian takes 4 + 1/R + 1/planes
// additions for 5, a step 14.3 operations for 15.  Bound by the FP64 pipe as the
// two passes above.  256^3: 412 -> 395 us per step, 16.8 M * 14.3 / 395 us =
// 0.61 T operations per second.  us per step by rows (planes of the best run):
// 256^3 394 (2 rows, 8 planes), 392 (4, 8), 389 (6, 5), but 187^3 164 (2, 6),
// 165 (4, 4), 165 (6, 4) and 160^3 103 (2, 6), 104 (4, 3), 103 (6, 3): more rows
// want a length of run for each grid, so that no SM gets a block more than the
// others.  One warp a block: those blocks are the smallest.
constexpr int kC64Rows = 2, kC64PairPlanes = 6;
constexpr long long kC64PairCells = 1LL << 22;

template <typename F>
static __device__ __forceinline__ void walk_pairs(const Ar<double>& A, const double* __restrict__ f, const Geom& g,
                                                  int planes, F out)
{
    constexpr int R = kC64Rows;
    const int z = blockIdx.x * kC64Z + threadIdx.x;
    if (z >= g.Z) return;   // no barrier
    const int y0 = min((int)blockIdx.y * R, g.Y - R);   // the last strip may repeat a row of the one before
    const int dzl = z == 0 ? g.Z - 1 : -1, dzh = z + 1 == g.Z ? -z : 1;
    const long long row = (long long)y0 * g.Z + z;
    const long long rl = (long long)(y0 == 0 ? g.Y - 1 : y0 - 1) * g.Z + z;
    const long long rh = (long long)(y0 + R == g.Y ? 0 : y0 + R) * g.Z + z;
    const int xs = blockIdx.z * planes, xe = min(xs + planes, g.X);
    double c[R + 1], d[R];   // plane x on rows y0 .. y0+R; D(x-1, y-1) on rows y0 .. y0+R-1
    {
        const double* pl = f + (long long)(xs == 0 ? g.X - 1 : xs - 1) * g.YZ;
        const double* pc = f + (long long)xs * g.YZ;
#pragma unroll
        for (int r = 0; r < R; r++) c[r] = __ldg(pc + row + (long long)r * g.Z);
        c[R] = __ldg(pc + rh);
#pragma unroll
        for (int r = 0; r < R; r++) d[r] = A.add(r == 0 ? __ldg(pc + rl) : c[r - 1], __ldg(pl + row + (long long)r * g.Z));
    }
    for (int x = xs; x < xe; x++) {
        const double* pc = f + (long long)x * g.YZ + row;
        const double* ph = f + (long long)(x + 1 == g.X ? 0 : x + 1) * g.YZ;
        double n[R + 1], e[R];
#pragma unroll
        for (int r = 0; r < R; r++) n[r] = __ldg(ph + row + (long long)r * g.Z);
        n[R] = __ldg(ph + rh);
        const double nl = __ldg(ph + rl);
#pragma unroll
        for (int r = 0; r < R; r++) {
            const double* pz = pc + (long long)r * g.Z;
            const double sz = A.add(__ldg(pz + dzh), __ldg(pz + dzl));
            e[r] = A.add(n[r], c[r + 1]);
            out((long long)x * g.YZ + row + (long long)r * g.Z, c[r], A.add(A.add(e[r], d[r]), sz));
        }
        d[0] = A.add(nl, c[0]);
#pragma unroll
        for (int r = 1; r < R; r++) d[r] = e[r - 1];
#pragma unroll
        for (int r = 0; r <= R; r++) c[r] = n[r];
    }
}

template <int MODEL, bool KONE>
__global__ void __launch_bounds__(kC64Z)
ch64_mu_pairs(const double* __restrict__ cin, double* __restrict__ mu, Geom g, C64 q0, P<double>, int planes)
{
    const Ar<double> A(g.dim);
    const C64 q = held(A, q0);
    walk_pairs(A, cin, g, planes, [&](long long i, double c, double s) { mu[i] = mu_sum<MODEL, KONE>(A, c, s, q); });
}

__global__ void __launch_bounds__(kC64Z)
ch64_update_pairs(const double* __restrict__ cin, const double* __restrict__ mu, double* __restrict__ cout, Geom g, C64 q0,
                  P<double>, int planes)
{
    const Ar<double> A(g.dim);
    const C64 q = held(A, q0);
    walk_pairs(A, mu, g, planes,
               [&](long long i, double m, double s) { cout[i] = fma(q.dtm, s, fma(q.upd0, m, __ldg(cin + i))); });
}

// Small 2D grids: many steps in one cooperative launch.  The two passes above
// cost two launches a step, 1.6 us each however small the grid; here a block
// per SM keeps its tile of c in shared memory, computes mu on the tile and one
// cell around it, updates in place, and exchanges only the two outer cells of
// each side with its neighbours, through the state buffers in turn, past a
// grid barrier per step.  While the barrier's arrivals travel (1.3 us), a block
// computes mu where it needs no neighbour.  (Announcing the outer cells before
// the others are updated measured slower: 256^2 4.35 us per step, one more
// phase to wait through.)  Each mu is computed with the
// operations of ch64_mu, so the rim that two blocks both compute has the same
// bits, and the states are those of the two passes.
constexpr int kC64StepThreads = 512;

struct C64Tiles {
    int h, w, nz;   // rows and columns of a tile, tiles along Z
};

// Cell e of a frame two cells wide around an h x w interior: its row and column
// in the (h+4) x (w+4) frame.
static __device__ __forceinline__ void frame_cell(int e, int h, int w, int& r, int& c)
{
    if (e < 4 * (w + 4)) {
        r = e / (w + 4);
        c = e - r * (w + 4);
        r = r < 2 ? r : h + r;
    } else {
        const int m = e - 4 * (w + 4);
        r = 2 + (m >> 2);
        c = (m & 3) < 2 ? (m & 3) : w + (m & 3);
    }
}

template <int MODEL, bool UNIT, bool KONE, bool EXACT>
__global__ void __launch_bounds__(kC64StepThreads)
ch64_steps(double* s0, double* s1, Geom g, C64 q0, P<double> p0, C64Tiles tl, int steps, unsigned* count, unsigned base,
           int* err)
{
    const Ar<double> A(g.dim);
    const C64 q = held(A, q0);
    const P<double> p = held(A, p0);
    extern __shared__ double tile_sm[];
    __shared__ int s_ok;
    const int tid = threadIdx.x;
    const int y0 = (int)(blockIdx.x / tl.nz) * tl.h, z0 = (int)(blockIdx.x % tl.nz) * tl.w;
    const int h = min(tl.h, g.Y - y0), w = min(tl.w, g.Z - z0);
    const int CW = tl.w + 4, MW = tl.w + 2;
    double* C = tile_sm;                       // c with two cells around: [h+4][CW]
    double* M = C + (tl.h + 4) * CW;           // mu with one cell around: [h+2][MW]
    auto where = [&](int r, int c) {           // cell (r, c) of C in a state buffer
        return (long long)wrapi(y0 - 2 + r, g.Y) * g.Z + wrapi(z0 - 2 + c, g.Z);
    };
    auto mu_at = [&](int r, int c) {           // mu of cell (r, c) of M
        const double* k = C + (r + 1) * CW + c + 1;
        M[r * MW + c] = mu_cell<2, MODEL, UNIT, KONE, EXACT>(A, k[0], 0.0, 0.0, k[CW], k[-CW], k[1], k[-1], q, p);
    };
    // mu without neighbours' cells: the (h-2) x (w-2) cells two inside M
    const int ih = h - 2, iw = w - 2;
    const bool inner = ih > 0 && iw > 0;
    const int inner_n = inner ? ih * iw : 0, rim_n = inner ? (h + 2) * (w + 2) - inner_n : 0;

    for (int e = tid; e < (h + 4) * (w + 4); e += kC64StepThreads) {
        const int r = e / (w + 4), c = e - r * (w + 4);
        C[r * CW + c] = __ldcg(s0 + where(r, c));
    }
    __syncthreads();
    for (int e = tid; e < inner_n; e += kC64StepThreads) {
        const int r = e / iw;
        mu_at(r + 2, e - r * iw + 2);
    }
    for (int s = 0; s < steps; s++) {
        // the rest of mu
        if (inner) {
            for (int e = tid; e < rim_n; e += kC64StepThreads) {
                int r, c;
                frame_cell(e, ih, iw, r, c);
                mu_at(r, c);
            }
        } else {
            for (int e = tid; e < (h + 2) * (w + 2); e += kC64StepThreads) {
                const int r = e / (w + 2);
                mu_at(r, e - r * (w + 2));
            }
        }
        __syncthreads();
        // the update in place; a cell that a neighbour will read, or any at the end, to the next state buffer
        double* dst = s & 1 ? s0 : s1;
        const bool last = s + 1 == steps;
        for (int e = tid; e < h * w; e += kC64StepThreads) {
            const int r = e / w, c = e - r * w;
            const double* m = M + (r + 1) * MW + c + 1;
            double* k = C + (r + 2) * CW + c + 2;
            double o;
            if (EXACT) {
                const double lap = lap_ref<double, UNIT, 2>(A, twice(m[0]), 0.0, 0.0, m[MW], m[-MW], m[1], m[-1], p.wx, p.wy, p.wz);
                o = A.add(*k, A.mul(p.dtm, lap));
            } else {
                o = fma(q.dtm, nsum<2, UNIT>(A, 0.0, A.add(m[MW], m[-MW]), A.add(m[1], m[-1]), q), fma(q.upd0, m[0], *k));
            }
            *k = o;
            if (last || r < 2 || r >= h - 2 || c < 2 || c >= w - 2) dst[(long long)(y0 + r) * g.Z + z0 + c] = o;
        }
        if (last) break;
        // arrive, compute what needs no other block, wait
        __syncthreads();
        if (tid == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
        for (int e = tid; e < inner_n; e += kC64StepThreads) {
            const int r = e / iw;
            mu_at(r + 2, e - r * iw + 2);
        }
        if (tid == 0) {
            const unsigned target = base + (unsigned)(s + 1) * gridDim.x;
            const uint64_t t0 = global_ns();
            bool done = false;
            for (unsigned spin = 0; !done; spin++) {
                unsigned v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
                done = (int)(v - target) >= 0;
                if (!done && (spin & 255u) == 255u && global_ns() - t0 > kWaitNs) break;
            }
            s_ok = done;
        }
        __syncthreads();
        if (!s_ok) {   // the other blocks' waits run out too
            if (tid == 0) atomicExch(err, 1);
            return;
        }
        for (int e = tid; e < 4 * (w + 4) + 4 * h; e += kC64StepThreads) {
            int r, c;
            frame_cell(e, h, w, r, c);
            C[r * CW + c] = __ldcg(dst + where(r, c));
        }
        __syncthreads();
    }
}

// The stochastic 3D Cahn-Hilliard form in FP32 (model B, spinodal: CH_POLY
// with noise) takes the same two passes: the noise term costs two SplitMix64
// draws, a logarithm, a cosine and a square root per cell, and a fused kernel
// would draw it again on every halo; here each deviate is drawn once, in the
// mu pass, at 8 B per cell of extra traffic (128^3 x 500 steps: 11.5 ms
// against 15.2 ms for the fused row kernel; in 2D the fused tile kernel
// stays faster, 7.1 ms against 8.3 ms on 1024^2, 6.5 ms by now).  Arithmetic as the FP32 form's:
// mu = c (-r + kappa w2 + u c^2) - kappa S + noise, c' = c + dtM (S_mu - w2 mu).
struct C32 {
    float wx, wy, wz, kappa, u, dtm, poly0, upd0;
};

template <int DIM, bool UNIT>
static __device__ __forceinline__ float nsum_f(float sx, float sy, float sz, const C32& q)
{
    if (UNIT) return DIM == 3 ? (sx + sy) + sz : sy + sz;
    return DIM == 3 ? fmaf(q.wx, sx, fmaf(q.wy, sy, q.wz * sz)) : fmaf(q.wy, sy, q.wz * sz);
}

template <int DIM, bool UNIT>
__global__ void __launch_bounds__(kC64Z * kC64Y)
chf_noise_mu(const float* __restrict__ cin, float* __restrict__ mu, Geom g, C32 q, P<float> p, int planes)
{
    const int z = blockIdx.x * kC64Z + threadIdx.x;
    const int y = blockIdx.y * kC64Y + threadIdx.y;
    if (z >= g.Z || y >= g.Y) return;   // no barrier in this kernel
    const int zl = z == 0 ? g.Z - 1 : z - 1, zh = z + 1 == g.Z ? 0 : z + 1;
    const long long row = (long long)y * g.Z;
    const long long rl = (long long)(y == 0 ? g.Y - 1 : y - 1) * g.Z;
    const long long rh = (long long)(y + 1 == g.Y ? 0 : y + 1) * g.Z;
    const int xs = blockIdx.z * planes;
    const int xe = min(xs + planes, g.X);
    auto plane = [&](int x) { return cin + (long long)x * g.YZ; };
    float a = 0.0f, b = __ldg(plane(xs) + row + z);
    if (DIM == 3) a = __ldg(plane(xs == 0 ? g.X - 1 : xs - 1) + row + z);
    for (int x = xs; x < xe; x++) {
        const float* pc = plane(x);
        float n = 0.0f;
        if (DIM == 3) n = __ldg(plane(x + 1 == g.X ? 0 : x + 1) + row + z);
        const float s = nsum_f<DIM, UNIT>(n + a, __ldg(pc + rh + z) + __ldg(pc + rl + z),
                                          __ldg(pc + row + zh) + __ldg(pc + row + zl), q);
        const long long i = (long long)x * g.YZ + row + z;
        const float m = fmaf(-q.kappa, s, fmaf(q.u, b * b, q.poly0) * b);
        mu[i] = m + noise_at(p, g.cells, i);
        a = b;
        b = n;
    }
}

template <int DIM, bool UNIT>
__global__ void __launch_bounds__(kC64Z * kC64Y)
chf_update(const float* __restrict__ cin, const float* __restrict__ mu, float* __restrict__ cout, Geom g, C32 q,
           int planes)
{
    const int z = blockIdx.x * kC64Z + threadIdx.x;
    const int y = blockIdx.y * kC64Y + threadIdx.y;
    if (z >= g.Z || y >= g.Y) return;
    const int zl = z == 0 ? g.Z - 1 : z - 1, zh = z + 1 == g.Z ? 0 : z + 1;
    const long long row = (long long)y * g.Z;
    const long long rl = (long long)(y == 0 ? g.Y - 1 : y - 1) * g.Z;
    const long long rh = (long long)(y + 1 == g.Y ? 0 : y + 1) * g.Z;
    const int xs = blockIdx.z * planes;
    const int xe = min(xs + planes, g.X);
    auto plane = [&](int x) { return mu + (long long)x * g.YZ; };
    float a = 0.0f, b = __ldg(plane(xs) + row + z);
    if (DIM == 3) a = __ldg(plane(xs == 0 ? g.X - 1 : xs - 1) + row + z);
    for (int x = xs; x < xe; x++) {
        const long long i = (long long)x * g.YZ + row + z;
        const float* pm = plane(x);
        float n = 0.0f;
        if (DIM == 3) n = __ldg(plane(x + 1 == g.X ? 0 : x + 1) + row + z);
        const float s = nsum_f<DIM, UNIT>(n + a, __ldg(pm + rh + z) + __ldg(pm + rl + z),
                                          __ldg(pm + row + zh) + __ldg(pm + row + zl), q);
        cout[i] = fmaf(q.dtm, s, fmaf(q.upd0, b, __ldg(cin + i)));
        a = b;
        b = n;
    }
}

bool ch64_eligible(const mmsp_gpu_desc& d, const Geom& g)
{
    // grid dimensions y and z of the launch stay within 65535 blocks (z with runs of up to kC64MostPlanes planes)
    const long long by = (g.Y + kC64Y - 1) / kC64Y;
    const long long bz = g.dim == 3 ? (g.X + kC64MostPlanes - 1) / kC64MostPlanes : 1;
    const bool fp64 = d.dtype == MMSP_GPU_F64 && (d.model == MMSP_GPU_CH || d.model == MMSP_GPU_CH_POLY);
    const bool noisy32 = d.dtype == MMSP_GPU_F32 && d.model == MMSP_GPU_CH_POLY && g.dim == 3 && noisy(d);
    return (fp64 || noisy32) && (g.dim == 2 || g.dim == 3) && by <= 65535 && bz <= 65535;
}

namespace {

// Kernel tables indexed by the template switches.
template <int DIM, int MODEL, bool UNIT, bool KONE, bool EXACT>
const void* mu_fn_n(bool noise)
{
    return noise ? reinterpret_cast<const void*>(&ch64_mu<DIM, MODEL, UNIT, KONE, EXACT, true>)
                 : reinterpret_cast<const void*>(&ch64_mu<DIM, MODEL, UNIT, KONE, EXACT, false>);
}
template <int DIM, int MODEL, bool UNIT, bool KONE>
const void* mu_fn_e(bool exact, bool noise)
{
    return exact ? mu_fn_n<DIM, MODEL, UNIT, KONE, true>(noise) : mu_fn_n<DIM, MODEL, UNIT, KONE, false>(noise);
}
template <int DIM, int MODEL, bool UNIT>
const void* mu_fn_k(bool kone, bool exact, bool noise)
{
    return kone ? mu_fn_e<DIM, MODEL, UNIT, true>(exact, noise) : mu_fn_e<DIM, MODEL, UNIT, false>(exact, noise);
}
template <int DIM, int MODEL>
const void* mu_fn_u(bool unit, bool kone, bool exact, bool noise)
{
    return unit ? mu_fn_k<DIM, MODEL, true>(kone, exact, noise) : mu_fn_k<DIM, MODEL, false>(kone, exact, noise);
}
template <int DIM>
const void* mu_fn_m(int model, bool unit, bool kone, bool exact, bool noise)
{
    return model == MMSP_GPU_CH ? mu_fn_u<DIM, MMSP_GPU_CH>(unit, kone, exact, noise)
                                : mu_fn_u<DIM, MMSP_GPU_CH_POLY>(unit, kone, exact, noise);
}
template <int DIM>
const void* upd_fn(bool unit, bool exact)
{
    if (unit) return exact ? reinterpret_cast<const void*>(&ch64_update<DIM, true, true>)
                           : reinterpret_cast<const void*>(&ch64_update<DIM, true, false>);
    return exact ? reinterpret_cast<const void*>(&ch64_update<DIM, false, true>)
                 : reinterpret_cast<const void*>(&ch64_update<DIM, false, false>);
}

C64 c64_of(const Coeffs& c, int dim)
{
    const P<double> p = narrow<double>(c, dim);
    C64 q;
    q.wx = p.wx;
    q.wy = p.wy;
    q.wz = p.wz;
    q.kappa = c.kappa;
    q.dtm = c.dtm;
    q.u = c.u;
    q.w2 = 2.0 * (dim == 3 ? p.wx + p.wy + p.wz : p.wy + p.wz);
    q.poly0 = 0.0;   // set by the launcher per model
    q.upd0 = -c.dtm * q.w2;
    return q;
}

}  // namespace

// The mu kernel goes in p->fn, the update kernel in p->fn2.
cudaError_t plan_ch64(const mmsp_gpu_desc& d, const Geom& g, StepPlan* p)
{
    const Coeffs c = make_coeffs(d);
    const bool exact = !(d.flags & MMSP_GPU_FLAG_CONTRACT);
    const bool kone = c.kappa == 1.0;
    const bool noise = noisy(d);
    if (d.dtype == MMSP_GPU_F32) {   // the noisy FP32 form, 3D only (ch64_eligible)
        p->fn = c.unit_w ? (const void*)&chf_noise_mu<3, true> : (const void*)&chf_noise_mu<3, false>;
        p->fn2 = c.unit_w ? (const void*)&chf_update<3, true> : (const void*)&chf_update<3, false>;
    } else {
        p->fn = g.dim == 3 ? mu_fn_m<3>(d.model, c.unit_w, kone, exact, noise)
                           : mu_fn_m<2>(d.model, c.unit_w, kone, exact, noise);
        p->fn2 = g.dim == 3 ? upd_fn<3>(c.unit_w, exact) : upd_fn<2>(c.unit_w, exact);
    }
    p->planes = g.dim != 3 ? 1 : d.dtype == MMSP_GPU_F32 && g.cells >= kC32Long ? kC32Planes : kC64Planes;
    unsigned warps_y = kC64Y, rows = 1;
    // Fewer additions a cell, but threads with more to do: 256^3 412 -> 395 us
    // per step, 224^3 278 -> 269, 187^3 168 -> 164, 160^3 104.5 -> 102.8; but 128^3 55 -> 58.
    if (d.dtype == MMSP_GPU_F64 && g.dim == 3 && !exact && !noise && c.unit_w && g.cells >= kC64PairCells &&
        g.Y >= kC64Rows && g.Y <= 65535 * kC64Rows) {
        p->fn = d.model == MMSP_GPU_CH ? (kone ? (const void*)&ch64_mu_pairs<MMSP_GPU_CH, true>
                                               : (const void*)&ch64_mu_pairs<MMSP_GPU_CH, false>)
                                       : (kone ? (const void*)&ch64_mu_pairs<MMSP_GPU_CH_POLY, true>
                                               : (const void*)&ch64_mu_pairs<MMSP_GPU_CH_POLY, false>);
        p->fn2 = (const void*)&ch64_update_pairs;
        p->planes = kC64PairPlanes;
        warps_y = 1;
        rows = kC64Rows;
    }
    p->planes = std::max(p->planes, (g.X + 65534) / 65535);
    p->block = dim3(kC64Z, warps_y, 1);
    const int segs = (g.X + p->planes - 1) / p->planes;
    p->grid = dim3((g.Z + kC64Z - 1) / kC64Z, (g.Y + warps_y * rows - 1) / (warps_y * rows), segs);
    p->smem = 0;
    p->fields = 1;
    p->kind = 6;
    p->ok = true;
    return cudaSuccess;
}

cudaError_t launch_ch64(const StepPlan& p, const mmsp_gpu_desc& d, const Geom& g, const Coeffs& c, const void* in,
                        void* out, void* work, int* err, cudaStream_t s)
{
    C64 q = c64_of(c, g.dim);
    q.poly0 = (d.model == MMSP_GPU_CH ? 2.0 : c.neg_r) + c.kappa * q.w2;
    int planes = p.planes;
    if (d.dtype == MMSP_GPU_F32) {
        C32 f;
        f.wx = (float)q.wx;
        f.wy = (float)q.wy;
        f.wz = (float)q.wz;
        f.kappa = (float)q.kappa;
        f.u = (float)q.u;
        f.dtm = (float)q.dtm;
        f.poly0 = (float)q.poly0;
        f.upd0 = (float)q.upd0;
        P<float> pf = narrow<float>(c, g.dim);
        pf.stepp = step_word(err);
        void* a1[] = {(void*)&in, (void*)&work, (void*)&g, (void*)&f, (void*)&pf, (void*)&planes};
        cudaError_t e = cudaLaunchKernel(p.fn, p.grid, p.block, a1, 0, s);
        if (e != cudaSuccess) return e;
        const void* mu = work;
        void* a2[] = {(void*)&in, (void*)&mu, (void*)&out, (void*)&g, (void*)&f, (void*)&planes};
        return cudaLaunchKernel(p.fn2, p.grid, p.block, a2, 0, s);
    }
    P<double> pp = narrow<double>(c, g.dim);
    if (noisy(d)) pp.stepp = step_word(err);
    void* a1[] = {(void*)&in, (void*)&work, (void*)&g, (void*)&q, (void*)&pp, (void*)&planes};
    cudaError_t e = cudaLaunchKernel(p.fn, p.grid, p.block, a1, 0, s);
    if (e != cudaSuccess) return e;
    const void* mu = work;
    void* a2[] = {(void*)&in, (void*)&mu, (void*)&out, (void*)&g, (void*)&q, (void*)&pp, (void*)&planes};
    return cudaLaunchKernel(p.fn2, p.grid, p.block, a2, 0, s);
}

namespace {

template <int MODEL, bool UNIT>
const void* steps_fn_u(bool kone, bool exact)
{
    if (kone) return exact ? (const void*)&ch64_steps<MODEL, UNIT, true, true> : (const void*)&ch64_steps<MODEL, UNIT, true, false>;
    return exact ? (const void*)&ch64_steps<MODEL, UNIT, false, true> : (const void*)&ch64_steps<MODEL, UNIT, false, false>;
}

template <int MODEL>
const void* steps_fn(bool unit, bool kone, bool exact)
{
    return unit ? steps_fn_u<MODEL, true>(kone, exact) : steps_fn_u<MODEL, false>(kone, exact);
}

}  // namespace

// us per step, two passes / here (256 steps a call): 64^2 3.6 / 3.1, 256^2 5.1 /
// 4.0 (contracted 4.2 / 3.2), 400^2 7.9 / 7.1, 512^2 10.9 / 10.3, 640x600 14.2 /
// 13.2; in calls of 20 steps, which the two passes launch one by one, 8.5 /
// 3.5 at 64^2 and 18.7 / 13.8 at 640x600.  Above, the FP64 work of the tiles'
// rims outweighs the launches.
constexpr long long kC64StepsMost = 400LL << 10;

bool plan_ch64_steps(const mmsp_gpu_desc& d, const Geom& g, Ch64Steps* p)
{
    if (d.dtype != MMSP_GPU_F64 || g.dim != 2 || noisy(d) || g.cells > kC64StepsMost ||
        (d.model != MMSP_GPU_CH && d.model != MMSP_GPU_CH_POLY))
        return false;
    const Coeffs c = make_coeffs(d);
    const bool exact = !(d.flags & MMSP_GPU_FLAG_CONTRACT), kone = c.kappa == 1.0;
    p->fn = d.model == MMSP_GPU_CH ? steps_fn<MMSP_GPU_CH>(c.unit_w, kone, exact)
                                   : steps_fn<MMSP_GPU_CH_POLY>(c.unit_w, kone, exact);
    // tiles that leave an SM the least FP64 work: 10 operations per mu, 7 per update
    const int sms = sm_count();
    long long best = -1;
    for (int nz = 1; nz <= std::min(sms, g.Z); nz++) {
        const int ny = std::min(sms / nz, g.Y);
        const int h = (g.Y + ny - 1) / ny, w = (g.Z + nz - 1) / nz;
        const long long work = 10LL * (h + 2) * (w + 2) + 7LL * h * w;
        if (best < 0 || work < best) {
            best = work;
            p->h = h;
            p->w = w;
        }
    }
    p->nz = (g.Z + p->w - 1) / p->w;
    p->blocks = (g.Y + p->h - 1) / p->h * p->nz;
    p->smem = sizeof(double) * ((size_t)(p->h + 4) * (p->w + 4) + (size_t)(p->h + 2) * (p->w + 2));
    // one block per SM fits at 512 threads of at most 64 registers
    if (p->smem > 200 * 1024) return false;
    if (p->smem > 40 * 1024 && ensure_smem(p->fn, p->smem) != cudaSuccess) {   // (48 KB with the static part)
        cudaGetLastError();
        return false;
    }
    return true;
}

cudaError_t launch_ch64_steps(const Ch64Steps& p, const mmsp_gpu_desc& d, const Geom& g, const Coeffs& c, void* in,
                              void* other, int steps, unsigned* count, unsigned base, int* err, cudaStream_t s)
{
    C64 q = c64_of(c, g.dim);
    q.poly0 = (d.model == MMSP_GPU_CH ? 2.0 : c.neg_r) + c.kappa * q.w2;
    P<double> pp = narrow<double>(c, g.dim);
    C64Tiles tl{p.h, p.w, p.nz};
    if (take_stall()) base += 1u << 30;   // counts that no block will see
    void* args[] = {(void*)&in, (void*)&other, (void*)&g, (void*)&q, (void*)&pp, (void*)&tl, (void*)&steps, (void*)&count,
                    (void*)&base, (void*)&err};
    return cudaLaunchCooperativeKernel(p.fn, dim3(p.blocks), dim3(kC64StepThreads), args, p.smem, s);
}

}  // namespace pf
