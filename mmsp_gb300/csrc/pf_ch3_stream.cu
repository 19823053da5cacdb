// pf_ch3_stream.cu -- FP32 3D Cahn-Hilliard step on rows of 256 cells, register streaming along X.
//
// A block owns R consecutive rows (axis Y) of full Z extent and a run of X
// planes; each thread owns two adjacent cells of a row.
//
// For every plane the block's R+4 rows (2 halo rows on each side, wrapped
// periodically) arrive in shared memory by cp.async.bulk on an mbarrier ring,
// several planes ahead of the one being computed.  Each thread keeps its
// cells of c for planes x, x+1, x+2 and of mu for x-1, x, x+1 in registers:
// Y neighbours are neighbouring registers, X neighbours the neighbouring
// planes' registers, Z neighbours inside a thread are registers, Z
// neighbours across threads come from shared memory (c) or warp shuffles
// (mu), and the first and last cells of each warp exchange mu through a small
// shared array that wraps periodically across the row.  mu is recomputed only
// on the 2 halo rows of the strip; a block spans whole rows, so there is no Z
// halo.
//
// FP32 arithmetic is reassociated for throughput (six-neighbour sums and
// Horner's form of f'(c)); the result is checked against the FP64 oracle
// with a tolerance, not bitwise.
#include <atomic>
#include <stdlib.h>

#include "pf_async.cuh"
#include "pf_device.cuh"
#include "pf_internal.h"

namespace pf {

constexpr int kRing = 4;      // planes staged in shared memory (kRing-1 in flight)
constexpr int kStreamR = 8;   // rows per block strip

struct F32Coef {
    float wx, wy, wz, w2;   // Laplacian weights, w2 = 2(wx+wy+wz)
    float kappa, dtm, neg_r, u;
};

// A thread's two adjacent cells: packed FP32x2 arithmetic, one instruction for both.
static __device__ __forceinline__ float2 vadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
static __device__ __forceinline__ float2 vmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
static __device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
static __device__ __forceinline__ float2 vset(float k) { return make_float2(k, k); }
// Sum of the two Z neighbours of each cell, given the cells just left and
// just right of the thread's pair.
static __device__ __forceinline__ float2 vzsum(float2 c, float left, float right)
{
    return __fadd2_rn(make_float2(left, c.x), make_float2(c.y, right));
}

template <int MODEL>
static __device__ __forceinline__ float2 mu_v(float2 c, float2 lap, const F32Coef& q)
{
    float2 fp;
    if (MODEL == MMSP_GPU_CH)   // 2c(1-c)(1-2c) = c*(2 + c*(-6 + 4c))
        fp = vmul(c, vfma(vfma(vset(4.0f), c, vset(-6.0f)), c, vset(2.0f)));
    else                        // -r c + u c^3 = c*(u c^2 - r)
        fp = vmul(c, vfma(vset(q.u), vmul(c, c), vset(q.neg_r)));
    return vfma(vset(-q.kappa), lap, fp);
}

// wx*sx + wy*sy + wz*sz - 2(wx+wy+wz)*c, with sx, sy, sz the sums of the two
// neighbours along each axis.
template <bool UNIT>
static __device__ __forceinline__ float2 lap_v(float2 sx, float2 sy, float2 sz, float2 c, const F32Coef& q)
{
    if (UNIT) return vfma(vset(-6.0f), c, vadd(vadd(sx, sy), sz));
    return vfma(vset(q.wx), sx, vfma(vset(q.wy), sy, vfma(vset(q.wz), sz, vmul(vset(-q.w2), c))));
}

// Shared memory: kRing slots of (R+4) x Z floats, the warp-end mu buffers
// [parity][warp][side][R], then kRing mbarriers.
static size_t ch3_smem(int R, int Z)
{
    const int warps = Z / 64;
    return sizeof(float) * (size_t)kRing * (R + 4) * Z + sizeof(float) * 2 * warps * 2 * R + sizeof(uint64_t) * kRing;
}

// STALL: the failure-detection test (never in normal use).  The plane fills
// expect their bytes without issuing the copies and every wait is capped at
// 4 polls, so the waits run out with no copy in flight and the launch takes
// its timed-out exit (error word, bounded drain, return).  The host selects
// it only through MMSP_GPU_TEST_STALL_LAUNCHES.
template <int R, int Z, int MODEL, bool UNIT, bool STALL>
__global__ void __launch_bounds__(Z / 2, 3)
ch3_stream_f32(const float* __restrict__ cin, float* __restrict__ cout, Geom g, F32Coef q, int planes,
               int mirror, int* __restrict__ err)
{
    constexpr int RR = R + 4, V = 2, TM = Z / V, W = TM / 32;   // threads and warps per block
    static_assert(TM % 32 == 0 && R % 4 == 0, "row split");
    const int t = threadIdx.x;
    const int lane = t & 31, warp = t >> 5;
    const int z0 = t * V;        // first cell of this thread
    const int wlast = W - 1;
    extern __shared__ __align__(128) unsigned char sm[];
    float* slots = reinterpret_cast<float*>(sm);
    float* edges = slots + (size_t)kRing * RR * Z;
    uint64_t* bars = reinterpret_cast<uint64_t*>(edges + 2 * W * 2 * R);
    __shared__ int s_err;

    const int y0 = blockIdx.x * R;
    const int xs = blockIdx.y * planes;
    const int xe = min(xs + planes, g.X);
    if (xs >= xe) return;
    const int zl = z0 == 0 ? Z - 1 : z0 - 1;            // cell left of this thread's first
    const int zh = z0 + V == Z ? 0 : z0 + V;            // cell right of its last
    const int wl = warp == 0 ? wlast : warp - 1;
    const int wh = warp == wlast ? 0 : warp + 1;
    const int x_first = xs - 2, x_last = xe + 1;        // planes read from global memory

    // stage plane pl (wrapped) into its ring slot: thread 0
    auto fill = [&](int pl) {
        const int k = pl - x_first, s = k % kRing;
        uint64_t* bar = &bars[s];
        float* dst = slots + (size_t)s * RR * Z;
        // mirror: the walk runs through X downwards.  Successive steps
        // alternate, so a step starts with the planes that the one before
        // touched last, which are still in L2.
        const int xw = wrapi(pl, g.X);
        const float* base = cin + (long long)(mirror ? g.X - 1 - xw : xw) * g.YZ;
        const uint32_t row = (uint32_t)Z * sizeof(float);
        fence_proxy_async();
        mbar_expect_tx(bar, RR * row);
        if (STALL) return;   // failure-detection test: the bytes never arrive
        const int a = y0 - 2, b = y0 + R + 2;
        if (a >= 0 && b <= g.Y) {
            bulk_g2s(dst, base + (long long)a * Z, RR * row, bar);
        } else if (a < 0) {
            const int n1 = -a;   // rows Y-n1 .. Y-1 first, then 0 ..
            bulk_g2s(dst, base + (long long)(g.Y - n1) * Z, n1 * row, bar);
            bulk_g2s(dst + n1 * Z, base, (RR - n1) * row, bar);
        } else {
            const int n1 = g.Y - a;   // rows a .. Y-1, then 0 ..
            bulk_g2s(dst, base + (long long)a * Z, n1 * row, bar);
            bulk_g2s(dst + n1 * Z, base, (RR - n1) * row, bar);
        }
    };
    auto slot_of = [&](int pl) -> const float* { return slots + (size_t)((pl - x_first) % kRing) * RR * Z; };
    auto wait_plane = [&](int pl) {
        const int k = pl - x_first;
        if (!mbar_wait(&bars[k % kRing], (uint32_t)(k / kRing) & 1u, STALL ? 4u : kSpinLimit)) {
            s_err = 1;
            atomicExch(err, 1);
        }
    };

    if (t == 0) {
        for (int s = 0; s < kRing; s++) mbar_init(&bars[s], 1);
        mbar_fence_init();
        s_err = 0;
    }
    __syncthreads();
    if (t == 0)
        for (int pl = x_first; pl < x_first + kRing && pl <= x_last; pl++) fill(pl);

    using VT = float2;
    VT cA[RR], cB[RR], cC[RR];
    VT mA[R + 2], mB[R + 2], mC[R + 2];
    wait_plane(x_first);
    wait_plane(x_first + 1);
    {
        const float* s0 = slot_of(x_first) + z0;
        const float* s1 = slot_of(x_first + 1) + z0;
#pragma unroll
        for (int i = 0; i < RR; i++) {
            cA[i] = *reinterpret_cast<const VT*>(s0 + i * Z);
            cB[i] = *reinterpret_cast<const VT*>(s1 + i * Z);
        }
    }
#pragma unroll
    for (int i = 0; i < R + 2; i++) mA[i] = mB[i] = vset(0.0f);
    __syncthreads();
    if (t == 0 && !s_err && x_first + kRing <= x_last) fill(x_first + kRing);   // slot of x_first is free

    // One plane: a = c(x), b = c(x+1), c = c(x+2) (loaded here); ma = mu(x-1),
    // mb = mu(x), mc = mu(x+1) (computed here); writes c'(x) when x >= xs.
    auto iter = [&](int x, VT (&a)[RR], VT (&b)[RR], VT (&c)[RR], VT (&ma)[R + 2], VT (&mb)[R + 2],
                    VT (&mc)[R + 2]) -> bool {
        wait_plane(x + 2);
        const float* s2 = slot_of(x + 2) + z0;
#pragma unroll
        for (int i = 0; i < RR; i++) c[i] = *reinterpret_cast<const VT*>(s2 + i * Z);
        const float* s1 = slot_of(x + 1);
#pragma unroll
        for (int r = -1; r <= R; r++) {
            const int i = r + 2;
            const float left = s1[i * Z + zl];
            const float right = s1[i * Z + zh];
            const VT cc = b[i];
            const VT lap = lap_v<UNIT>(vadd(a[i], c[i]), vadd(b[i - 1], b[i + 1]), vzsum(cc, left, right), cc, q);
            mc[r + 1] = mu_v<MODEL>(cc, lap, q);
        }
        // warp ends publish mu(x+1) of rows 0..R-1 for the neighbouring warps:
        // lane 0 its first cell, the warp's last real lane its last
        float* e1 = edges + (((x + 1) & 1) * W + warp) * 2 * R;
        if (lane == 0 || lane == 31) {
            // (selects keep mc in registers)
            const bool first = lane == 0;
            float* dst = e1 + (first ? 0 : R);
#pragma unroll
            for (int r = 0; r < R; r += 4)
                *reinterpret_cast<float4*>(dst + r) = make_float4(
                    first ? mc[r + 1].x : mc[r + 1].y, first ? mc[r + 2].x : mc[r + 2].y,
                    first ? mc[r + 3].x : mc[r + 3].y, first ? mc[r + 4].x : mc[r + 4].y);
        }
        if (x >= xs) {
            // the neighbouring warps' end cells: every lane reads the same
            // words (broadcast) and lanes 0 / 31 select them, without branches
            const float4* eL = reinterpret_cast<const float4*>(edges + ((x & 1) * W + wl) * 2 * R + R);
            const float4* eH = reinterpret_cast<const float4*>(edges + ((x & 1) * W + wh) * 2 * R);
            float el[R], eh[R];
#pragma unroll
            for (int r = 0; r < R; r += 4) {
                const float4 u = eL[r / 4], v = eH[r / 4];
                el[r] = u.x, el[r + 1] = u.y, el[r + 2] = u.z, el[r + 3] = u.w;
                eh[r] = v.x, eh[r + 1] = v.y, eh[r + 2] = v.z, eh[r + 3] = v.w;
            }
            float* dst = cout + (long long)(mirror ? g.X - 1 - x : x) * g.YZ + (long long)y0 * Z + z0;
            const int rows = min(R, g.Y - y0);
#pragma unroll
            for (int r = 0; r < R; r++) {
                const VT m = mb[r + 1];
                const float up = __shfl_up_sync(0xffffffffu, m.y, 1);
                const float down = __shfl_down_sync(0xffffffffu, m.x, 1);
                const float left = lane == 0 ? el[r] : up;
                const float right = lane == 31 ? eh[r] : down;
                const VT lap = lap_v<UNIT>(vadd(ma[r + 1], mc[r + 1]), vadd(mb[r], mb[r + 2]), vzsum(m, left, right), m, q);
                const VT o = vfma(vset(q.dtm), lap, a[r + 2]);
                if (r < rows) *reinterpret_cast<VT*>(dst + (long long)r * Z) = o;
            }
        }
        __syncthreads();
        if (s_err) return false;
        if (t == 0 && x + 1 + kRing <= x_last) fill(x + 1 + kRing);   // slot of x+1 is free now
        return true;
    };

    int x = x_first;
    while (!s_err) {
        if (x >= xe || !iter(x, cA, cB, cC, mA, mB, mC)) break;
        x++;
        if (x >= xe || !iter(x, cB, cC, cA, mB, mC, mA)) break;
        x++;
        if (x >= xe || !iter(x, cC, cA, cB, mC, mA, mB)) break;
        x++;
    }
    if (s_err && t == 0) {
        // leave no copy in flight: wait (bounded) for every issued fill
        for (int pl = max(x, x_first); pl <= min(x + kRing, x_last); pl++) {
            const int k = pl - x_first;
            mbar_wait(&bars[k % kRing], (uint32_t)(k / kRing) & 1u, STALL ? 4u : kSpinLimit);
        }
    }
}

static F32Coef f32coef(const Coeffs& c)
{
    F32Coef q;
    q.wx = (float)c.w[0];
    q.wy = (float)c.w[1];
    q.wz = (float)c.w[2];
    q.w2 = 2.0f * (q.wx + q.wy + q.wz);
    q.kappa = (float)c.kappa;
    q.dtm = (float)c.dtm;
    q.neg_r = (float)c.neg_r;
    q.u = (float)c.u;
    return q;
}

// MMSP_GPU_TEST_STALL_LAUNCHES=n: in the next n launches of this kernel and of
// the ones with a grid barrier in the process the waits run out, and grids with
// rows of 64 cells take this kernel too (the failure-detection tests).  Read
// once; unset in normal use.
static std::atomic<int> g_stall_left{-1};
static int stall_left()
{
    int left = g_stall_left.load();
    if (left < 0) {
        const char* v = getenv("MMSP_GPU_TEST_STALL_LAUNCHES");
        int n = v ? atoi(v) : 0;
        g_stall_left.compare_exchange_strong(left, n > 0 ? n : 0);
        left = g_stall_left.load();
    }
    return left;
}
int take_stall()
{
    int cur = stall_left();
    while (cur > 0 && !g_stall_left.compare_exchange_weak(cur, cur - 1)) {
    }
    return cur > 0 ? 1 : 0;
}

// Rows of 256 cells whose two states fill L2 or do not fit it: there the
// ring's bulk copies keep more of HBM and L2 busy than the loads of
// pf_ch3_flat.cu.  us per step, here / there: 256^3 (128 MB) 24.6 / 28.7,
// 512x256x256 45.0 / 52.5, 200x256x256 (100 MB) 20.5 / 23.9, 160x256x256 (80
// MB) 17.2 / 18.2; 128x256x256 (64 MB) 14.9 / 14.2.  Every other row length is
// faster there (rows of 512 in a ring that walked X one way only: 64x512x512
// 33.0 / 31.8, 130x512x512 59.7 / 57.7).
constexpr long long kStreamL2 = 72LL << 20;
bool ch3_stream_eligible(const mmsp_gpu_desc& d, const Geom& g)
{
    const bool ch = d.dtype == MMSP_GPU_F32 && g.dim == 3 && g.Y >= kStreamR + 4 &&
                    (d.model == MMSP_GPU_CH || d.model == MMSP_GPU_CH_POLY);
    return ch && ((g.Z == 256 && 8LL * g.cells > kStreamL2) || (g.Z == 64 && stall_left() > 0));
}

template <int Z, bool STALL>
static const void* pick_stream(bool ch, bool unit)
{
    if (ch)
        return unit ? (const void*)&ch3_stream_f32<kStreamR, Z, MMSP_GPU_CH, true, STALL>
                    : (const void*)&ch3_stream_f32<kStreamR, Z, MMSP_GPU_CH, false, STALL>;
    return unit ? (const void*)&ch3_stream_f32<kStreamR, Z, MMSP_GPU_CH_POLY, true, STALL>
                : (const void*)&ch3_stream_f32<kStreamR, Z, MMSP_GPU_CH_POLY, false, STALL>;
}

cudaError_t plan_ch3_stream(const mmsp_gpu_desc& d, const Geom& g, StepPlan* p)
{
    const Coeffs c = make_coeffs(d);
    const bool ch = d.model == MMSP_GPU_CH;
    const int threads = g.Z / 2;
    p->fn = g.Z == 64 ? pick_stream<64, false>(ch, c.unit_w) : pick_stream<256, false>(ch, c.unit_w);
    p->fn2 = g.Z == 64 ? pick_stream<64, true>(ch, c.unit_w) : pick_stream<256, true>(ch, c.unit_w);   // the test's form
    p->smem = ch3_smem(kStreamR, g.Z);
    p->block = dim3(threads, 1, 1);
    cudaError_t e = ensure_smem(p->fn, p->smem);
    if (e == cudaSuccess) e = ensure_smem(p->fn2, p->smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, p->fn, threads, p->smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    const int strips = (g.Y + kStreamR - 1) / kStreamR;
    // one wave: strips * segments <= resident blocks, segments >= 1
    long long slots = (long long)sm_count() * per_sm;
    int segs = (int)(slots / strips);
    if (segs < 1) segs = 1;
    if (segs > g.X) segs = g.X;
    p->planes = (g.X + segs - 1) / segs;
    segs = (g.X + p->planes - 1) / p->planes;
    p->grid = dim3(strips, segs, 1);
    p->fields = 1;
    p->kind = 1;
    p->ok = true;
    return cudaSuccess;
}

cudaError_t launch_ch3_stream(const StepPlan& p, const Geom& g, const Coeffs& c, const void* in, void* out,
                              int* err, cudaStream_t s)
{
    F32Coef q = f32coef(c);
    int planes = p.planes, mirror = in > out;
    void* args[] = {(void*)&in, (void*)&out, (void*)&g, (void*)&q, (void*)&planes, (void*)&mirror, (void*)&err};
    return cudaLaunchKernel(take_stall() ? p.fn2 : p.fn, p.grid, p.block, args, p.smem, s);
}

}  // namespace pf
