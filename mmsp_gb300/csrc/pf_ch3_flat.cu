// pf_ch3_flat.cu -- FP32 3D Cahn-Hilliard step, one independent warp per window of rows.
//
// A warp owns R rows (axis Y) of a window of 60 cells (axis Z) and a run of X
// planes: 32 lanes of two adjacent cells, the outer lane of each side a halo.
// Everything a cell needs lies in its own lane's registers or one lane away:
// c of planes x-1 .. x+2 and mu of planes x-2 .. x on R rows and the halo rows
// of the strip (Y neighbours are neighbouring registers, X neighbours the
// other planes' registers), Z neighbours by shuffle.  So there is no shared
// memory and no barrier, the warps of an SM drift apart, and the loads of one
// cover the arithmetic of the others.  Plane x+2 is loaded before plane x-1 is
// written out, so the warp's own output arithmetic covers its loads too.
//
// Rows of any length: a plane's rows are taken as virtual rows of Z + 4 cells
// (-2 .. Z+1, Z+5 when Z is odd), wrapped periodically on load, and the
// windows run over the pairs of all virtual rows without a gap; a window may
// span two rows, because a virtual row carries its own halo.  The last strip
// starts at Y - R where Y is no multiple of R, and writes some rows twice
// (the same values).  Odd rows load and store their pairs as two single cells.
//
// mu is computed on R + 2 rows for R: the price of keeping it in registers.
// 187^3: 13.0 us per step = 4.0 TB/s of algorithmic traffic (in L2), bound by
// load latency at 12 warps per SM; staging whole rows in a shared-memory ring
// with a barrier per plane took 22.6 us (62 instructions per cell against
// 21).  243^3 42.6 -> 28.1, 242^3 34.3 -> 26.5, 208^3 25.9 -> 14.9, 140^3 12.6
// -> 7.4, 61^3 4.9 -> 4.0, 40^3 4.9 -> 2.7.
#include <algorithm>

#include "pf_device.cuh"
#include "pf_internal.h"

namespace pf {

struct ChFlat {
    float wx, wy, wz, w2;   // Laplacian weights, w2 = 2 (wx + wy + wz)
    float kappa, dtm, neg_r, u;
};

static __device__ __forceinline__ float2 p2(float a, float b) { return make_float2(a, b); }
static __device__ __forceinline__ float2 p2(float a) { return make_float2(a, a); }

// The Laplacian and mu from sums of neighbours and regrouped terms, or (DIFF) as
// the reference writes them: differences (hi - 2 c) + lo, whose rounding follows
// the differences and not the cells' own size, and f' as a product.  DIFF is for
// rows above 512 cells, which had the reference's form when all others had
// sums: RMS error against 64 bits after 40 steps of dt = 0.01, sums /
// differences, 45x45x513 2.05e-8 / 1.86e-8 (dt = 0.002: 3.01e-8 / 2.99e-8).
template <bool UNIT>
static __device__ __forceinline__ float2 flat_lap(float2 sx, float2 sy, float2 sz, float2 c, const ChFlat& q)
{
    if (UNIT) return __ffma2_rn(p2(-6.0f), c, __fadd2_rn(__fadd2_rn(sx, sy), sz));
    return __ffma2_rn(p2(q.wx), sx, __ffma2_rn(p2(q.wy), sy, __ffma2_rn(p2(q.wz), sz, __fmul2_rn(p2(-q.w2), c))));
}

static __device__ __forceinline__ float2 diff2(float2 lo, float2 c, float2 hi)
{
    return __fadd2_rn(__ffma2_rn(p2(-2.0f), c, hi), lo);
}

template <bool UNIT>
static __device__ __forceinline__ float2 flat_lap_diff(float2 dx, float2 dy, float2 dz, const ChFlat& q)
{
    if (UNIT) return __fadd2_rn(__fadd2_rn(dx, dy), dz);
    return __ffma2_rn(p2(q.wz), dz, __ffma2_rn(p2(q.wy), dy, __fmul2_rn(p2(q.wx), dx)));
}

template <int MODEL, bool DIFF>
static __device__ __forceinline__ float2 flat_mu(float2 c, float2 lap, const ChFlat& q)
{
    float2 fp;
    if (MODEL == MMSP_GPU_CH) {
        if (DIFF) {   // 2c (1-c) (1-2c)
            const float2 one = p2(1.0f);
            fp = __fmul2_rn(__fmul2_rn(__fadd2_rn(c, c), __ffma2_rn(p2(-1.0f), c, one)), __ffma2_rn(p2(-2.0f), c, one));
        } else {
            fp = __fmul2_rn(c, __ffma2_rn(__ffma2_rn(p2(4.0f), c, p2(-6.0f)), c, p2(2.0f)));
        }
    } else {
        if (DIFF) fp = __ffma2_rn(p2(q.u), __fmul2_rn(__fmul2_rn(c, c), c), __fmul2_rn(p2(q.neg_r), c));
        else fp = __fmul2_rn(c, __ffma2_rn(p2(q.u), __fmul2_rn(c, c), p2(q.neg_r)));
    }
    return __ffma2_rn(p2(-q.kappa), lap, fp);
}

// sums, or differences, of the two Z neighbours of a lane's pair
static __device__ __forceinline__ float2 zsum(float2 c)
{
    const float left = __shfl_up_sync(0xffffffffu, c.y, 1), right = __shfl_down_sync(0xffffffffu, c.x, 1);
    return p2(left + c.y, c.x + right);
}
static __device__ __forceinline__ float2 zdiff(float2 c)
{
    const float left = __shfl_up_sync(0xffffffffu, c.y, 1), right = __shfl_down_sync(0xffffffffu, c.x, 1);
    return p2(fmaf(-2.0f, c.x, c.y) + left, fmaf(-2.0f, c.y, right) + c.x);
}

constexpr int kFlatThreads = 128;

// Warps per SM that the registers are held to: 12 (6 rows), 16 (4 rows), 28 (2
// rows).  One more block spills.
template <int R>
constexpr int flat_min_blocks()
{
    return R == 6 ? 3 : R == 4 ? 4 : 7;
}

// PRE: prefetch the warp's rows of plane x+4 into L2 (states above L2).
template <int R, bool ODD, int MODEL, bool UNIT, bool PRE, bool DIFF>
__global__ void __launch_bounds__(kFlatThreads, flat_min_blocks<R>())
ch3_flat_f32(const float* __restrict__ cin, float* __restrict__ cout, Geom g, ChFlat q, int planes, int mirror)
{
    constexpr bool PIPE = R > 2;   // two rows: the output is too short to cover loads, registers count more
    const int lane = threadIdx.x & 31;
    const int warp = (int)((blockIdx.x * kFlatThreads + threadIdx.x) >> 5);
    const int Z = g.Z, half = (Z + 5) >> 1;   // pairs of a virtual row
    const int total = (g.Y + R - 1) / R * half;
    const int pr = warp * 30 + lane - 1;      // this lane's pair among all virtual rows of the plane
    const bool mine = lane >= 1 && lane <= 30 && pr < total;
    const int pc = min(max(pr, 0), total - 1);
    const int strip = pc / half, zz = 2 * (pc - strip * half) - 2;
    const int y0 = min(strip * R, g.Y - R);
    const int za = wrap_near(zz, Z), zb = wrap_near(zz + 1, Z);
    const bool ok0 = mine && zz >= 0 && zz < Z, ok1 = mine && zz + 1 >= 0 && zz + 1 < Z;
    // byte offsets in a plane: the strip's rows, the two rows above and below it
    const unsigned rb = 4u * (unsigned)Z;
    auto row = [&](int y) { return (unsigned)wrap_near(y, g.Y) * rb + 4u * (unsigned)za; };
    const unsigned om = row(y0), ot2 = row(y0 - 2), ot1 = row(y0 - 1), ob0 = row(y0 + R), ob1 = row(y0 + R + 1);
    const int dz = 4 * (zb - za);             // odd rows: the pair's second cell
    const int xs = blockIdx.y * planes, xe = min(xs + planes, g.X);
    const long long pb = 4LL * g.YZ;
    // mirror: the walk runs through X downwards.  Successive steps alternate,
    // so a step starts with the planes that the one before touched last, which
    // are still in L2.
    auto plane = [&](int x) {
        const int xw = wrapi(x, g.X);
        return (mirror ? g.X - 1 - xw : xw) * pb;
    };
    const char* in = reinterpret_cast<const char*>(cin);
    char* out = reinterpret_cast<char*>(cout);

    auto ld = [&](const char* base, unsigned off) -> float2 {
        if (ODD)
            return p2(__ldg(reinterpret_cast<const float*>(base + off)),
                      __ldg(reinterpret_cast<const float*>(base + (off + (unsigned)dz))));
        return __ldg(reinterpret_cast<const float2*>(base + off));
    };
    auto load = [&](int x, float2 (&c)[R + 4]) {
        const char* base = in + plane(x);
        c[0] = ld(base, ot2);
        c[1] = ld(base, ot1);
#pragma unroll
        for (int r = 0; r < R; r++) c[r + 2] = ld(base + (size_t)r * rb, om);
        c[R + 2] = ld(base, ob0);
        c[R + 3] = ld(base, ob1);
    };
    auto output = [&](int x, const float2 (&c)[R + 4], const float2 (&ml)[R + 2], const float2 (&m)[R + 2],
                      const float2 (&mh)[R + 2]) {
        char* base = out + plane(x);
#pragma unroll
        for (int r = 0; r < R; r++) {
            const float2 v = m[r + 1];
            const float2 lap =
                DIFF ? flat_lap_diff<UNIT>(diff2(ml[r + 1], v, mh[r + 1]), diff2(m[r], v, m[r + 2]), zdiff(v), q)
                     : flat_lap<UNIT>(__fadd2_rn(ml[r + 1], mh[r + 1]), __fadd2_rn(m[r], m[r + 2]), zsum(v), v, q);
            const float2 o = __ffma2_rn(p2(q.dtm), lap, c[r + 2]);
            char* dst = base + (size_t)r * rb;
            if (ODD) {
                if (ok0) *reinterpret_cast<float*>(dst + om) = o.x;
                if (ok1) *reinterpret_cast<float*>(dst + (om + (unsigned)dz)) = o.y;
            } else {
                if (ok0) *reinterpret_cast<float2*>(dst + om) = o;
            }
        }
    };
    auto chem = [&](const float2 (&cl)[R + 4], const float2 (&c)[R + 4], const float2 (&ch)[R + 4], float2 (&m)[R + 2]) {
#pragma unroll
        for (int r = 0; r < R + 2; r++) {
            const float2 v = c[r + 1];
            const float2 lap =
                DIFF ? flat_lap_diff<UNIT>(diff2(cl[r + 1], v, ch[r + 1]), diff2(c[r], v, c[r + 2]), zdiff(v), q)
                     : flat_lap<UNIT>(__fadd2_rn(cl[r + 1], ch[r + 1]), __fadd2_rn(c[r], c[r + 2]), zsum(v), v, q);
            m[r] = flat_mu<MODEL, DIFF>(v, lap, q);
        }
    };
    // one plane: c0 = c(x-1), c1 = c(x), c2 = c(x+1), n = c(x+2); m0 = mu(x-2), m1 = mu(x-1), m2 = mu(x)
    auto iter = [&](int x, float2 (&c0)[R + 4], float2 (&c1)[R + 4], float2 (&c2)[R + 4], float2 (&n)[R + 4],
                    float2 (&m0)[R + 2], float2 (&m1)[R + 2], float2 (&m2)[R + 2], float2 (&m3)[R + 2]) {
        if (PRE) {
            const char* base = in + plane(x + 4);
#pragma unroll
            for (int r = 0; r < R; r++) asm volatile("prefetch.global.L2 [%0];" ::"l"(base + (size_t)r * rb + om));
        }
        if (PIPE) load(x + 2, n);
        if (x - 1 >= xs) output(x - 1, c0, m0, m1, m2);
        if (!PIPE) load(x + 2, n);
        chem(c1, c2, n, m3);
    };
    float2 cA[R + 4], cB[R + 4], cC[R + 4], cD[R + 4];
    float2 mA[R + 2], mB[R + 2], mC[R + 2], mD[R + 2];
#pragma unroll
    for (int i = 0; i < R + 4; i++) cA[i] = p2(0.0f);
#pragma unroll
    for (int i = 0; i < R + 2; i++) mA[i] = mB[i] = mC[i] = p2(0.0f);
    load(xs - 2, cB);
    load(xs - 1, cC);
    // the arrays' roles rotate by one per plane
    for (int x = xs - 2;;) {
        if (x == xe) {
            output(xe - 1, cA, mA, mB, mC);
            break;
        }
        iter(x++, cA, cB, cC, cD, mA, mB, mC, mD);
        if (x == xe) {
            output(xe - 1, cB, mB, mC, mD);
            break;
        }
        iter(x++, cB, cC, cD, cA, mB, mC, mD, mA);
        if (x == xe) {
            output(xe - 1, cC, mC, mD, mA);
            break;
        }
        iter(x++, cC, cD, cA, cB, mC, mD, mA, mB);
        if (x == xe) {
            output(xe - 1, cD, mD, mA, mB);
            break;
        }
        iter(x++, cD, cA, cB, cC, mD, mA, mB, mC);
    }
}

namespace {

template <int R, bool ODD, int MODEL, bool UNIT, bool DIFF>
const void* flat_pre(bool pre)
{
    // strips of 2 and 4 rows are for grids far below L2
    if constexpr (R < 6) return (const void*)&ch3_flat_f32<R, ODD, MODEL, UNIT, false, DIFF>;
    else return pre ? (const void*)&ch3_flat_f32<R, ODD, MODEL, UNIT, true, DIFF>
                    : (const void*)&ch3_flat_f32<R, ODD, MODEL, UNIT, false, DIFF>;
}

template <int R, bool ODD, int MODEL, bool UNIT>
const void* flat_diff(bool pre, bool diff)
{
    return diff ? flat_pre<R, ODD, MODEL, UNIT, true>(pre) : flat_pre<R, ODD, MODEL, UNIT, false>(pre);
}

template <int R, bool ODD>
const void* flat_model(int model, bool unit, bool pre, bool diff)
{
    if (model == MMSP_GPU_CH)
        return unit ? flat_diff<R, ODD, MMSP_GPU_CH, true>(pre, diff) : flat_diff<R, ODD, MMSP_GPU_CH, false>(pre, diff);
    return unit ? flat_diff<R, ODD, MMSP_GPU_CH_POLY, true>(pre, diff)
                : flat_diff<R, ODD, MMSP_GPU_CH_POLY, false>(pre, diff);
}

template <int R>
const void* flat_fn(bool odd, int model, bool unit, bool pre, bool diff)
{
    return odd ? flat_model<R, true>(model, unit, pre, diff) : flat_model<R, false>(model, unit, pre, diff);
}

// Rows per strip: few rows give many short warps, which small grids need;
// many rows recompute less of mu.  us per step at 2 / 4 / 6 rows: 40^3 2.7 /
// 3.2 / 3.4, 64^3 3.7 / 3.7 / 3.5, 140^3 8.5 / 6.8 / 7.0, 160^3 - / 8.9 / 8.0,
// 187^3 18.8 / 12.7 / 12.2, 240^3 - / 25.2 / 22.9.
int flat_rows(const Geom& g)
{
    return g.cells < (100LL << 10) || g.Y < 4 ? 2 : g.cells < (7LL << 19) || g.Y < 6 ? 4 : 6;
}

// Prefetching and mirrored walks are for pairs of states that do not fit the
// 129 MB L2: 240^3 (111 MB) 23.3 -> 22.9 us per step with prefetch, 256^3 31.9
// -> 28.5, 255^3 33.4 -> 30.6; but 224^3 (90 MB) 18.2 -> 18.7, 187^3 12.2 -> 13.2.
constexpr long long kFlatL2 = 96LL << 20;

}  // namespace

bool ch3_flat_eligible(const mmsp_gpu_desc& d, const Geom& g)
{
    return d.dtype == MMSP_GPU_F32 && g.dim == 3 && g.Z >= 4 && g.Y >= 2 && g.YZ < (1LL << 30) &&
           (d.model == MMSP_GPU_CH || d.model == MMSP_GPU_CH_POLY) && !noisy(d);
}

cudaError_t plan_ch3_flat(const mmsp_gpu_desc& d, const Geom& g, StepPlan* p)
{
    const Coeffs c = make_coeffs(d);
    const int R = flat_rows(g);
    const bool odd = g.Z % 2 != 0, pre = 8LL * g.cells > kFlatL2;
    const bool diff = g.Z > 512;
    p->fn = R == 6   ? flat_fn<6>(odd, d.model, c.unit_w, pre, diff)
            : R == 4 ? flat_fn<4>(odd, d.model, c.unit_w, pre, diff)
                     : flat_fn<2>(odd, d.model, c.unit_w, pre, diff);
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, p->fn, kFlatThreads, 0);
    if (e != cudaSuccess) return e;
    const long long pairs = (long long)((g.Y + R - 1) / R) * ((g.Z + 5) / 2);
    const long long warps = (pairs + 29) / 30, per_block = kFlatThreads / 32;
    const long long blocks = (warps + per_block - 1) / per_block;
    // one wave: windows * runs <= resident blocks (each run starts with 2 planes of mu that its neighbour has too)
    const long long segs = std::max(1LL, std::min((long long)g.X, (long long)sm_count() * std::max(1, per_sm) / blocks));
    p->planes = (int)((g.X + segs - 1) / segs);
    p->grid = dim3((unsigned)blocks, (unsigned)((g.X + p->planes - 1) / p->planes), 1);
    p->block = dim3(kFlatThreads, 1, 1);
    p->smem = 0;
    p->fields = 1;
    p->kind = 2;
    p->ok = true;
    return cudaSuccess;
}

cudaError_t launch_ch3_flat(const StepPlan& p, const Geom& g, const Coeffs& c, const void* in, void* out, cudaStream_t s)
{
    ChFlat q;
    q.wx = (float)c.w[0];
    q.wy = (float)c.w[1];
    q.wz = (float)c.w[2];
    q.w2 = 2.0f * (q.wx + q.wy + q.wz);
    q.kappa = (float)c.kappa;
    q.dtm = (float)c.dtm;
    q.neg_r = (float)c.neg_r;
    q.u = (float)c.u;
    int planes = p.planes, mirror = in > out;
    void* args[] = {(void*)&in, (void*)&out, (void*)&g, (void*)&q, (void*)&planes, (void*)&mirror};
    return cudaLaunchKernel(p.fn, p.grid, p.block, args, 0, s);
}

}  // namespace pf
