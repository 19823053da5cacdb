// pf_convex.cu -- semi-implicit convex-splitting Cahn-Hilliard, FP64.
//
// The reference (examples/phase_transitions/cahn-hilliard/convex_splitting/
// cahn-hilliard.cpp:273-463) solves, each step, the linearised system for
// (c, mu) at every cell by red-black Gauss-Seidel with over-relaxation,
// checking the relative residual of the original system after iterations
// 1-4 and every 5th one.  With a 5/7-point stencil a cell reads only cells
// of the other color, so a sweep over one color is independent of its
// visiting order once every periodic extent is even: one thread per cell of
// the color gives the serial sweep's values.
//
// A step is one cooperative launch: its blocks, at most one per SM, hold the
// cells of each color as even shares of the flat list of that color, run all
// iterations of the solve and meet at a grid barrier after every sweep.  Each
// block adds up its residual (Neumaier sums, fixed order) and, past a barrier,
// every block adds the blocks' sums in the same order, so all take the same
// decision to go on or stop.  Where a thread has one cell of each color
// (up to 512 * SMs cells per color) it keeps their values, the old
// composition and its expansive term in registers.
//
// Bound: the FP64 pipe and the barrier (1.3 us).  400x200: 11 us per iteration,
// of which 2 sweeps of 40000 cells are 2 * 2.2 us of FP64 work; 64x64 7.3 us,
// 600x500 29 us.  A launch per sweep, with the checks in conditional graph
// nodes, took 30, 18 and 54 us.  (A word per block that every block polls,
// instead of one count of arrivals, took 22 us at 400x200: the polls of all
// words crowd out the arrivals.)
//
// Arithmetic: the example's expressions regrouped into fused multiply-adds
// (30 FP64 operations per cell and sweep instead of 45), with what a cell
// needs of its own guess alone done while the blocks meet.  The two quotients
// share one reciprocal.  A stop can fall one check apart from the serial
// program's, as its residual's sum is rounded differently anyway.
#include <algorithm>

#include "pf_async.cuh"
#include "pf_device.cuh"
#include "pf_internal.h"

namespace pf {

struct CsArgs {
    CsConst q;
    double wx, wy, wz;   // 1/dx^2 of padded axes X, Y, Z
    double a0, d0, d1;   // A21 = -(QA c^2 + a0) and det A = d1 c^2 + d0
};

// The constants of the expressions in registers (Ar::reg).
static __device__ __forceinline__ CsArgs held(const Ar<double>& A, CsArgs a)
{
    double* v = &a.q.A12;
#pragma unroll
    for (int i = 0; i < (int)(sizeof(CsArgs) / sizeof(double)); i++) v[i] = A.reg(v[i]);
    return a;
}

// A cell's neighbours as offsets from it.
struct CsNb {
    long long xh, xl, yh, yl;
    int zh, zl;
};

// Cell k of the color that a sweep with `skip` updates (cells whose coordinate
// sum has the parity `skip` are left alone, as the example's `continue` does):
// its index, and its neighbours.
static __device__ __forceinline__ long long cs_cell(const Geom& g, long long k, int skip, CsNb& n)
{
    const int hz = g.Z >> 1;   // every extent is even
    const long long row = k / hz;
    const int j = (int)(k - row * hz);
    const int x = (int)(row / g.Y), y = (int)(row - (long long)x * g.Y);
    const int z = 2 * j + ((x + y + skip + 1) & 1);
    n.xh = (x + 1 == g.X ? -(long long)x : 1LL) * g.YZ;
    n.xl = (x == 0 ? (long long)(g.X - 1) : -1LL) * g.YZ;
    n.yh = (y + 1 == g.Y ? -(long long)y : 1LL) * g.Z;
    n.yl = (y == 0 ? (long long)(g.Y - 1) : -1LL) * g.Z;
    n.zh = z + 1 == g.Z ? -z : 1;
    n.zl = z == 0 ? g.Z - 1 : -1;
    return row * g.Z + z;
}

// Other blocks write the cells between barriers: loads go to L2 (ld.cg).
static __device__ __forceinline__ double at(const double* p) { return __ldcg(p); }

// fringe_laplacian (cahn-hilliard.cpp:155-170): sum over axes of
// weight * (yh + yl), the Laplacian without its central term.
template <int DIM, bool UNIT>
static __device__ __forceinline__ double fringe(const Ar<double>& A, const double* f, const CsNb& n, const CsArgs& a)
{
    auto w = [&](double weight, double t) { return UNIT ? t : A.mul(weight, t); };   // 1.0*t is t
    double s = 0.0;
    if (DIM == 3) s = plus_zero(w(a.wx, A.add(at(f + n.xh), at(f + n.xl))));
    if (DIM == 3) s = A.add(s, w(a.wy, A.add(at(f + n.yh), at(f + n.yl))));
    if (DIM == 2) s = plus_zero(w(a.wy, A.add(at(f + n.yh), at(f + n.yl))));
    const double tz = w(a.wz, A.add(at(f + n.zh), at(f + n.zl)));
    return DIM == 1 ? plus_zero(tz) : A.add(s, tz);
}

template <int DIM, bool UNIT>
static __device__ __forceinline__ double field_lap(const Ar<double>& A, const double* f, double v, const CsNb& n,
                                                   const CsArgs& a)
{
    double xh = 0.0, xl = 0.0, yh = 0.0, yl = 0.0;
    if (DIM == 3) xh = at(f + n.xh), xl = at(f + n.xl);
    if (DIM >= 2) yh = at(f + n.yh), yl = at(f + n.yl);
    return lap_ref<double, UNIT, DIM>(A, twice(v), xh, xl, yh, yl, at(f + n.zh), at(f + n.zl), a.wx, a.wy, a.wz);
}

// expansive_dfdc (cahn-hilliard.cpp:92-96): -A*(C-C0) - QB*pow(C,2.0) - QD
static __device__ __forceinline__ double expansive(const Ar<double>& A, double C, const CsConst& q)
{
    return A.sub(A.sub(A.mul(-q.A, A.sub(C, q.C0)), A.mul(q.QB, A.mul(C, C))), q.QD);
}

// What a cell's update needs of its own guess alone (cahn-hilliard.cpp:325-334):
// the system's A21, its determinant and the determinant's reciprocal.
struct CsOwn {
    double A21, det, r;
};

// A21 = -(QA c^2 + QC) - KL, det = 1 - A12 A21
static __device__ __forceinline__ CsOwn cs_own(const Ar<double>& A, double c, const CsArgs& a)
{
    CsOwn o;
    const double c2 = A.mul(c, c);
    o.A21 = fma(-a.q.QA, c2, -a.a0);
    o.det = fma(a.d1, c2, a.d0);
    o.r = __drcp_rn(o.det);
    return o;
}

// a/d by the reciprocal r = 1/d: the quotient a*r corrected by its exact
// remainder (P. Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", IBM J. Res. Dev. 34, 1990).  Far from the middle
// of d's range, where r or the remainder would lose bits: the division.
static __device__ __forceinline__ double quotient(const Ar<double>& A, double a, const CsOwn& o)
{
    const unsigned e = ((unsigned)__double2hiint(o.det) >> 20) & 0x7ffu;
    if (e - 523u >= 1000u) return __ddiv_rn(a, o.det);   // |d| below 2^-500 or above 2^500
    const double t = A.mul(a, o.r);
    return __fma_rn(__fma_rn(-o.det, t, a), o.r, t);
}

// The sweep's update of one cell (cahn-hilliard.cpp:325-345): f1 and f2 point
// at the cell in the guess's two fields, c and u are its values there.
template <int DIM, bool UNIT>
static __device__ __forceinline__ void cs_update(const Ar<double>& A, const CsOwn& o, double cOld, double ex,
                                                 const double* f1, const double* f2, const CsNb& n, const CsArgs& a,
                                                 double& c, double& u)
{
    const CsConst& q = a.q;
    const double B1 = fma(q.Ddt, fringe<DIM, UNIT>(A, f2, n, a), cOld);
    const double B2 = fma(-q.K, fringe<DIM, UNIT>(A, f1, n, a), ex);
    const double cNew = quotient(A, fma(-q.A12, B2, B1), o);
    const double uNew = quotient(A, fma(-o.A21, B1, B2), o);
    c = fma(q.omega, cNew, A.mul(q.om1, c));
    u = fma(q.omega, uNew, A.mul(q.om1, u));
}

// Residual of the original system at one cell (cahn-hilliard.cpp:353-380):
// R1 = cOld - (cNew - D*dt*lap u), R2 = expansive(cOld) - (uNew -
// contractive(cNew) + K*lap c); returns R1^2 + R2^2.
template <int DIM, bool UNIT>
static __device__ __forceinline__ double cs_residual(const Ar<double>& A, double cOld, double ex, const double* f1,
                                                     const double* f2, const CsNb& n, const CsArgs& a, double c, double u)
{
    const CsConst& q = a.q;
    const double lapC = field_lap<DIM, UNIT>(A, f1, c, n, a);
    const double lapU = field_lap<DIM, UNIT>(A, f2, u, n, a);
    const double AX1 = fma(-q.Ddt, lapU, c);
    const double contr = A.mul(fma(q.QA, A.mul(c, c), q.QC), c);   // contractive_dfdc: QA c^3 + QC c
    const double AX2 = fma(q.K, lapC, A.sub(u, contr));
    const double R1 = A.sub(cOld, AX1), R2 = A.sub(ex, AX2);
    return fma(R1, R1, A.mul(R2, R2));
}

// A compensated sum: the rounding error of every addition, exact by Knuth's
// TwoSum, is added up beside it (no compare, so the additions of s follow each
// other without waiting for it).
struct CsNS {
    double s, c;
};

static __device__ __forceinline__ void cs_add(const Ar<double>& A, CsNS& a, double x)
{
    const double t = A.add(a.s, x), z = A.sub(t, a.s);
    a.c = A.add(a.c, A.add(A.sub(a.s, A.sub(t, z)), A.sub(x, z)));
    a.s = t;
}

// The lanes' sums of a warp, in a fixed order, on lane 0.
static __device__ __forceinline__ CsNS cs_warp_sum(const Ar<double>& A, CsNS v)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const CsNS o{__shfl_down_sync(0xffffffffu, v.s, off), __shfl_down_sync(0xffffffffu, v.c, off)};
        cs_add(A, v, o.s);
        v.c = A.add(v.c, o.c);
    }
    return v;
}

// The threads' sums of a block on its first thread.
static __device__ __forceinline__ CsNS cs_block_sum(const Ar<double>& A, CsNS v, CsNS* sh)
{
    v = cs_warp_sum(A, v);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    if (warp == 0) v = cs_warp_sum(A, lane < (int)(blockDim.x >> 5) ? sh[lane] : CsNS{0.0, 0.0});
    __syncthreads();
    return v;
}

// The blocks' sums on lane 0 of one warp of every block: lane l adds blocks l,
// l+32, ..., then the lanes' sums are added, the same way in every block.
static __device__ __forceinline__ double cs_grid_sum(const Ar<double>& A, const double* parts, int blocks)
{
    CsNS v{0.0, 0.0};
    for (int k = threadIdx.x & 31; k < blocks; k += 32) {
        cs_add(A, v, __ldcg(parts + 4 * k));
        v.c = A.add(v.c, __ldcg(parts + 4 * k + 1));
    }
    v = cs_warp_sum(A, v);
    return v.s + v.c;
}

// Grid barrier of a cooperative launch, in two halves so that work which needs
// no other block fits between them: a block adds itself to the count of
// arrivals (zero at the launch) ...
static __device__ __forceinline__ void cs_arrive(unsigned* count)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
    }
}

// ... and waits until all blocks of barrier `turn` have.  False when the wait
// ran out (2 s), for every thread of the block; the block then leaves, and the
// others' waits run out too.
static __device__ __forceinline__ bool cs_wait(const unsigned* count, unsigned turn, int* ok)
{
    if (threadIdx.x == 0) {
        const unsigned target = turn * gridDim.x;
        const uint64_t t0 = global_ns();
        bool done = false;
        for (unsigned spin = 0; !done; spin++) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
            done = (int)(v - target) >= 0;
            if (!done && (spin & 255u) == 255u && global_ns() - t0 > kWaitNs) break;
        }
        *ok = done;
    }
    __syncthreads();
    return *ok != 0;
}

constexpr int kCsThreads = 512;   // 128 registers, which the ONE form needs


// One step: the guess nw is iterated until the residual is at most tol or
// max_iter is reached.  parts: 4 doubles per block (residual sum and its
// compensation).  ONE: a thread has at most one cell of each color.
template <int DIM, bool UNIT, bool ONE>
__global__ void __launch_bounds__(kCsThreads)
cs_solve(const double* __restrict__ old, double* nw, Geom g, CsArgs a0, double* parts, CsLoop* L, unsigned* count,
         int* err, unsigned max_iter, unsigned first_checks)
{
    const Ar<double> A(g.dim);
    const CsArgs a = held(A, a0);
    __shared__ CsNS sh[kCsThreads / 32];
    __shared__ int s_ok;
    __shared__ double s_res;
    const long long per_color = g.cells >> 1;
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long k0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool on = k0 < per_color;
    double* f2 = nw + g.cells;
    unsigned turns = 0;   // barriers arrived at

    // the thread's cells of color 1 and of color 0, in the example's order (cahn-hilliard.cpp:321)
    CsNb n[2];
    long long i[2] = {0, 0};
    double cO[2], ex[2], c[2], u[2];
    if (ONE && on) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            i[h] = cs_cell(g, k0, 1 - h, n[h]);
            cO[h] = old[i[h]];
            ex[h] = expansive(A, cO[h], a.q);
            c[h] = at(nw + i[h]);
            u[h] = at(f2 + i[h]);
        }
    }
    // visits every cell of the thread: f(half sweep, slot), after loading what is not in registers
    auto each = [&](int h, auto f) {
        if (ONE) {
            if (on) f(h);
        } else {
            for (long long k = k0; k < per_color; k += stride) {
                i[h] = cs_cell(g, k, 1 - h, n[h]);
                cO[h] = old[i[h]];
                ex[h] = expansive(A, cO[h], a.q);
                c[h] = at(nw + i[h]);
                u[h] = at(f2 + i[h]);
                f(h);
            }
        }
    };

    // the norm of the right-hand side does not change during the solve
    CsNS b{0.0, 0.0};
#pragma unroll
    for (int h = 0; h < 2; h++) each(h, [&](int s) { cs_add(A, b, A.add(A.mul(cO[s], cO[s]), A.mul(ex[s], ex[s]))); });
    b = cs_block_sum(A, b, sh);
    if (threadIdx.x == 0) {
        parts[4 * blockIdx.x + 2] = b.s;
        parts[4 * blockIdx.x + 3] = b.c;
    }

    unsigned iter = 0;
    double res = 1.0, norm = 0.0;
    CsOwn own{};
    if (ONE) own = cs_own(A, c[0], a);
    while (iter < max_iter && res > a0.q.tol) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            each(h, [&](int s) {
                if (!ONE) own = cs_own(A, c[s], a);
                cs_update<DIM, UNIT>(A, own, cO[s], ex[s], nw + i[s], f2 + i[s], n[s], a, c[s], u[s]);
                nw[i[s]] = c[s];
                f2[i[s]] = u[s];
            });
            cs_arrive(count);
            turns++;
            if (ONE) own = cs_own(A, c[1 - h], a);   // the next sweep's, while the other blocks arrive
            if (!cs_wait(count, turns, &s_ok)) {
                if (threadIdx.x == 0) atomicExch(err, 1);
                return;
            }
        }
        iter++;
        if (iter >= first_checks && iter % first_checks) continue;
        CsNS r{0.0, 0.0};
#pragma unroll
        for (int h = 0; h < 2; h++)
            each(h, [&](int s) {
                cs_add(A, r, cs_residual<DIM, UNIT>(A, cO[s], ex[s], nw + i[s], f2 + i[s], n[s], a, c[s], u[s]));
            });
        r = cs_block_sum(A, r, sh);
        if (threadIdx.x == 0) {
            parts[4 * blockIdx.x + 0] = r.s;
            parts[4 * blockIdx.x + 1] = r.c;
        }
        cs_arrive(count);
            turns++;
        if (!cs_wait(count, turns, &s_ok)) {
            if (threadIdx.x == 0) atomicExch(err, 1);
            return;
        }
        if (threadIdx.x < 32) {
            if (iter == 1) norm = cs_grid_sum(A, parts + 2, gridDim.x);
            const double sum = cs_grid_sum(A, parts, gridDim.x);
            if (threadIdx.x == 0) s_res = sqrt(sum / norm) / (2.0 * a0.q.cells);
        }
        __syncthreads();
        res = s_res;
        // (s_res and parts are next written past two grid barriers)
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        L->last_iters = iter;
        L->residual = res;
        if (iter >= max_iter) L->hit_max = 1;
    }
}

static CsArgs cs_args(const Coeffs& c, const Geom& g)
{
    CsArgs a;
    a.q = c.cs;
    double w[3] = {1.0, 1.0, 1.0};
    for (int k = 0; k < g.dim; k++) w[3 - g.dim + k] = c.w[k];
    a.wx = w[0];
    a.wy = w[1];
    a.wz = w[2];
    a.a0 = a.q.QC + a.q.KL;
    a.d0 = 1.0 + a.q.A12 * a.a0;
    a.d1 = a.q.A12 * a.q.QA;
    return a;
}

template <int DIM, bool UNIT>
static const void* cs_pick(bool one)
{
    return one ? (const void*)&cs_solve<DIM, UNIT, true> : (const void*)&cs_solve<DIM, UNIT, false>;
}

cudaError_t launch_convex_step(const Geom& g, const Coeffs& c, const void* old, void* nw, double* partials, CsLoop* L,
                               int* err, unsigned max_iter, unsigned first_checks, cudaStream_t s)
{
    CsArgs a = cs_args(c, g);
    const bool unit = c.unit_w;
    // even shares of a color over the SMs, and of a share over its rounds, in whole warps
    const long long per_color = g.cells / 2, sms = std::min(sm_count(), kReduceBlocks);
    const long long share = (per_color + sms - 1) / sms, rounds = (share + kCsThreads - 1) / kCsThreads;
    const int threads = (int)(((share + rounds - 1) / rounds + 31) / 32 * 32);
    int blocks = (int)std::min(sms, (per_color + threads - 1) / threads);
    auto pick = [&](bool one) {
        return g.dim == 3   ? (unit ? cs_pick<3, true>(one) : cs_pick<3, false>(one))
               : g.dim == 2 ? (unit ? cs_pick<2, true>(one) : cs_pick<2, false>(one))
                            : (unit ? cs_pick<1, true>(one) : cs_pick<1, false>(one));
    };
    const void* fn = pick(rounds == 1);
    // the reduction scratch: 4 doubles per block, the barrier's count in its last words
    unsigned* count = reinterpret_cast<unsigned*>(partials + 4 * kReduceBlocks);
    // (from 0x80808080 it does not get to the count that the waits are for)
    cudaError_t e = cudaMemsetAsync(count, take_stall() ? 0x80 : 0, sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
    void* args[] = {(void*)&old, (void*)&nw, (void*)&g, (void*)&a, (void*)&partials, (void*)&L, (void*)&count, (void*)&err,
                    (void*)&max_iter, (void*)&first_checks};
    e = cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(threads), args, 0, s);
    // a stream with a part of the SMs: fewer blocks, each of which then takes more cells
    while (e == cudaErrorCooperativeLaunchTooLarge && blocks > 1) {
        cudaGetLastError();
        blocks = (blocks + 1) / 2;
        e = cudaLaunchCooperativeKernel(pick(false), dim3(blocks), dim3(threads), args, 0, s);
    }
    return e;
}

}  // namespace pf
