// pf_ac_cols.cu -- multi-order Allen-Cahn steps on the columns of the flat (Y, Z) plane.
//
// FP32: a thread owns V adjacent cells of the (Y, Z) plane and walks a run of
// X planes.  The plane is taken flat (cell y*Z + z), so every lane works
// whatever the row length, and the index is split into y and z once per
// thread.  The values of all N fields at planes x-1 and x roll through
// registers; plane x+1 and the four in-plane neighbours come straight from
// global memory, the neighbours out of L1 where the next rows' threads of the
// block have just read them.  No shared memory, no barrier, no copy pipeline:
// the loads of the unrolled fields overlap each other, and the other warps of
// the SM cover what is left.  The sum of squares needs no loads (the centres
// are in registers), so a cell of a field costs 5 loads, one store and about
// a dozen arithmetic instructions for V = 1.  Offsets within a plane are
// 32-bit byte offsets, the same for every field and plane; the plane bases
// are uniform.  Bound: HBM where the two states exceed L2 (128^3 x 8: 24.8 us
// per step = 5.4 TB/s; x 16: 55 us), else the L1/L2 latency that the resident
// warps leave uncovered.  Streaming whole rows of all fields through a
// shared-memory ring, one warp per row, took 32.1 and 75.2 us there (it holds
// 8 to 16 warps per SM), one thread per cell of a row 28.9 us against 10.3 on
// 74^3 x 14, 22.4 against 8.9 on 65^3 x 14, 64.6 against 38.8 on 127^3 x 9.
//
// FP64, and the FP32 forms that the kernel above does not take (thermal
// noise, planes of 2^30 cells and more): one thread per cell, the fields in a
// loop.  In FP64 the pipe (2 lanes per clock and SM) is the bound by far, so
// loads are free beside it and the kernel only saves FP64 operations: the
// square of a field is kept in shared memory between the sum and the update,
// doubling is integer arithmetic, and a gradient coefficient of 1 or 2 costs
// nothing.  19 operations per cell and field for MMSP_GPU_AC with kappa = 2
// in the reference's order, every one rounded on its own: bit-identical to
// the reference.  128^3 x 8: 515 us per step, 19 * 16.8 M / 515 us = 0.62 T
// operations per second; a tile of shared memory with a halo of 1 on a
// 4-plane ring, 22 operations, took 1100 us (its warps idle at the barriers
// of each plane), 40x41x42 x 5 14.1 against 84.8, 32^3 x 16 21.7 against 253.
#include <algorithm>

#include "pf_device.cuh"
#include "pf_internal.h"

namespace pf {

struct AcColF32 {
    float wx, wy, wz, w2;   // Laplacian weights (DIFF: negative), w2 = 2 (wx + wy + wz)
    float kappa, dtm, gamma2, neg_r, u;
};

constexpr int kAcColThreads = 128;

static __device__ __forceinline__ float ldo(const char* base, unsigned off)
{
    return __ldg(reinterpret_cast<const float*>(base + off));
}

template <int V> struct ColVec;
template <> struct ColVec<1> {
    float v[1];
    __device__ __forceinline__ void load(const char* base, unsigned off) { v[0] = ldo(base, off); }
    __device__ __forceinline__ void store(char* base, unsigned off) const { *reinterpret_cast<float*>(base + off) = v[0]; }
};
template <> struct ColVec<2> {
    float v[2];
    __device__ __forceinline__ void load(const char* base, unsigned off)
    {
        const float2 a = __ldg(reinterpret_cast<const float2*>(base + off));
        v[0] = a.x, v[1] = a.y;
    }
    __device__ __forceinline__ void store(char* base, unsigned off) const
    {
        *reinterpret_cast<float2*>(base + off) = make_float2(v[0], v[1]);
    }
};
template <> struct ColVec<4> {
    float v[4];
    __device__ __forceinline__ void load(const char* base, unsigned off)
    {
        const float4 a = __ldg(reinterpret_cast<const float4*>(base + off));
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
    }
    __device__ __forceinline__ void store(char* base, unsigned off) const
    {
        *reinterpret_cast<float4*>(base + off) = make_float4(v[0], v[1], v[2], v[3]);
    }
};

// The new value of one cell, or of a pair in packed FP32x2 instructions.
//
// SUMS: the Laplacian from the sums sx, sy, sz of the two neighbours along each
// axis, w (hi + lo) - 2 w c, and the polynomial's terms regrouped into fewer
// multiply-adds.  DIFF: the reference's expressions in its order, the Laplacian
// from (hi - 2 c) + lo, whose rounding follows the differences and not the
// cells' own size.  cols_sums below says which grids take which.
static __device__ __forceinline__ float cfma(float a, float b, float c) { return fmaf(a, b, c); }
static __device__ __forceinline__ float cmul(float a, float b) { return a * b; }
static __device__ __forceinline__ float cadd(float a, float b) { return a + b; }
static __device__ __forceinline__ float2 cfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
static __device__ __forceinline__ float2 cmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
static __device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
template <typename VT> static __device__ __forceinline__ VT cset(float k);
template <> __device__ __forceinline__ float cset<float>(float k) { return k; }
template <> __device__ __forceinline__ float2 cset<float2>(float k) { return make_float2(k, k); }

template <typename VT>
static __device__ __forceinline__ VT diff2(VT c, VT lo, VT hi)
{
    return cadd(cfma(cset<VT>(-2.0f), c, hi), lo);
}

template <int MODEL, typename VT>
static __device__ __forceinline__ VT col_new_sums(VT c, VT sum, VT sx, VT sy, VT sz, const AcColF32& q)
{
    const VT lap = cfma(cset<VT>(q.wx), sx, cfma(cset<VT>(q.wy), sy, cfma(cset<VT>(q.wz), sz, cmul(cset<VT>(-q.w2), c))));
    const VT c2 = cmul(c, c);
    if (MODEL == MMSP_GPU_AC) {
        // c' = c - dt L (c (gamma2 sum + (1 - gamma2) c^2 - 1) - kappa lap)
        const VT df = cmul(c, cfma(cset<VT>(q.gamma2), sum, cfma(cset<VT>(1.0f - q.gamma2), c2, cset<VT>(-1.0f))));
        return cfma(cset<VT>(-q.dtm), cfma(cset<VT>(-q.kappa), lap, df), c);
    } else if (MODEL == MMSP_GPU_GG || MODEL == MMSP_GPU_ZENER) {
        // c' = c - dt L (2 (c sum - lap) - c (c^2 + 1)): the change first, rounded once at the cell's size
        const VT t = cfma(c, sum, cmul(lap, cset<VT>(-1.0f)));
        const VT m = cmul(c, cfma(cset<VT>(-1.0f), c2, cset<VT>(-1.0f)));
        return cfma(cset<VT>(-q.dtm), cfma(cset<VT>(2.0f), t, m), c);
    } else {
        // c' = c - dt L (c (u c^2 - r) - kappa lap)
        const VT e = cfma(cset<VT>(-q.kappa), lap, cmul(c, cfma(cset<VT>(q.u), c2, cset<VT>(q.neg_r))));
        return cfma(cset<VT>(-q.dtm), e, c);
    }
}

// dx, dy, dz: diff2 along each axis.  The Laplacian and the centre enter with
// the sign that saves a negation.
template <int MODEL, typename VT>
static __device__ __forceinline__ VT col_new_diff(VT c, VT sum, VT dx, VT dy, VT dz, const AcColF32& q)
{
    const VT neg_lap = cfma(cset<VT>(q.wz), dz, cfma(cset<VT>(q.wy), dy, cmul(cset<VT>(q.wx), dx)));
    const VT c2 = cmul(c, c);
    VT e;
    if (MODEL == MMSP_GPU_AC) {
        // -c + c^3 + 2 gamma c (sum - c^2) - kappa lap
        const VT nc = cmul(cset<VT>(-1.0f), c);
        e = cfma(cmul(cset<VT>(q.gamma2), c), cfma(nc, c, sum), cfma(c2, c, nc));
        e = cfma(cset<VT>(q.kappa), neg_lap, e);
    } else if (MODEL == MMSP_GPU_GG || MODEL == MMSP_GPU_ZENER) {
        // -(-c - c^3 + 2 (c sum - lap))
        e = cfma(cset<VT>(-2.0f), cfma(c, sum, neg_lap), cfma(c2, c, c));
        return cfma(cset<VT>(q.dtm), e, c);
    } else {
        // -r c + u c^3 - kappa lap
        e = cfma(cset<VT>(q.kappa), neg_lap, cfma(cset<VT>(q.u), cmul(c2, c), cmul(cset<VT>(q.neg_r), c)));
    }
    return cfma(cset<VT>(-q.dtm), e, c);
}

// Blocks per SM that the registers are held to: 3 (168 registers) where the
// rolled planes are small, so that the loads of several fields are in flight
// at once, 4 or 5 where many fields fill the registers.  Measured, us per
// step (best of the plane runs): 128^3 x 8, V = 2: 24.5 at 3, 28.1 at 4, 28.9
// unbounded; 128^3 x 16, V = 2: 57.0 at 3, 55.0 at 4, 64.8 at 5; 74^3 x 14,
// V = 2: 10.1 / 10.5 / 14.5; 127^3 x 9, V = 1: 37.4 at 3, 39.6 at 4, 37.5 at
// 5; 65^3 x 14, V = 1: 9.8 / 8.3 / 8.9; 128^3 x 7, V = 4: 23.0 / 23.3 / 26.7.
template <int N, int V>
constexpr int cols_min_blocks()
{
    return V == 4 || N <= 8 ? 3 : V == 1 && N <= 16 ? 5 : N <= 16 ? 4 : 3;
}

// PRE: ask L2 for the cells of plane x+2 while plane x is worked on.  Only few
// rolled values leave registers for several fields' loads in flight, and only
// a dozen warps share an SM; the loads of plane x+1 then find L2 instead of
// waiting for HBM.
template <int N, int V, int MODEL, bool DIFF, bool PRE>
__global__ void __launch_bounds__(kAcColThreads, cols_min_blocks<N, V>())
ac_cols_f32(const float* __restrict__ ein, float* __restrict__ eout, Geom g, AcColF32 q, int planes, int flip)
{
    const unsigned YZ = (unsigned)g.YZ;
    const unsigned i = (blockIdx.x * kAcColThreads + threadIdx.x) * V;
    if (i >= YZ) return;
    const int Z = g.Z;
    const int y = (int)(i / (unsigned)Z), z = (int)(i - (unsigned)y * Z);
    // byte offsets in a plane: the cells, the rows above and below, the cells left and right
    const unsigned o = 4u * i;
    const unsigned oyl = 4u * (unsigned)((y == 0 ? g.Y - 1 : y - 1) * (long long)Z + z);
    const unsigned oyh = 4u * (unsigned)((y + 1 == g.Y ? 0 : y + 1) * (long long)Z + z);
    const unsigned ozl = z == 0 ? o + 4u * (unsigned)(Z - 1) : o - 4u;
    const unsigned ozh = z + V == Z ? o - 4u * (unsigned)z : o + 4u * V;
    // successive steps sweep X in opposite directions: a step then starts with
    // the planes that the one before wrote last, which are still in L2
    const int seg = flip ? (int)(gridDim.y - 1 - blockIdx.y) : (int)blockIdx.y;
    const int xs = seg * planes, xe = min(xs + planes, g.X);
    const long long pb = 4LL * g.YZ, fb = 4LL * g.cells;   // bytes of a plane and of a field
    const char* in = reinterpret_cast<const char*>(ein);
    char* out = reinterpret_cast<char*>(eout);

    ColVec<V> xl[N], cc[N];
    {
        const char* pl = in + (xs == 0 ? g.X - 1 : xs - 1) * pb;
        const char* pc = in + xs * pb;
#pragma unroll
        for (int f = 0; f < N; f++) {
            xl[f].load(pl + f * fb, o);
            cc[f].load(pc + f * fb, o);
        }
    }
#pragma unroll 1
    for (int x = xs; x < xe; x++) {
        const char* pc = in + x * pb;
        const char* ph = in + (x + 1 == g.X ? 0 : x + 1) * pb;
        char* po = out + x * pb;
        if (PRE) {
            const char* pn = in + (x + 2 >= g.X ? (x + 2) % g.X : x + 2) * pb;
#pragma unroll
            for (int f = 0; f < N; f++) asm volatile("prefetch.global.L2 [%0];" ::"l"(pn + f * fb + o));
        }
        float sum[V];
#pragma unroll
        for (int k = 0; k < V; k++) {
            float s0 = 0.0f, s1 = 0.0f;   // two chains: even and odd fields
#pragma unroll
            for (int f = 0; f < N; f += 2) {
                s0 = fmaf(cc[f].v[k], cc[f].v[k], s0);
                if (f + 1 < N) s1 = fmaf(cc[f + 1].v[k], cc[f + 1].v[k], s1);
            }
            sum[k] = s0 + s1;
        }
#pragma unroll
        for (int f = 0; f < N; f++) {
            ColVec<V> xh, yl, yh, w;
            xh.load(ph + f * fb, o);
            yl.load(pc + f * fb, oyl);
            yh.load(pc + f * fb, oyh);
            const float zl = ldo(pc + f * fb, ozl), zh = ldo(pc + f * fb, ozh);
            if (MODEL == MMSP_GPU_ZENER && f == 0) {
                w = cc[f];   // Zener pinning: the particles (field 0) have zero mobility
            } else if constexpr (V == 1) {
                const float c = cc[f].v[0], xl0 = xl[f].v[0], xh0 = xh.v[0], yl0 = yl.v[0], yh0 = yh.v[0];
                w.v[0] = DIFF ? col_new_diff<MODEL, float>(c, sum[0], diff2(c, xl0, xh0), diff2(c, yl0, yh0), diff2(c, zl, zh), q)
                              : col_new_sums<MODEL, float>(c, sum[0], xl0 + xh0, yl0 + yh0, zl + zh, q);
            } else {
#pragma unroll
                for (int k = 0; k < V; k += 2) {
                    const float2 c2 = make_float2(cc[f].v[k], cc[f].v[k + 1]), s2 = make_float2(sum[k], sum[k + 1]);
                    const float2 x0 = make_float2(xl[f].v[k], xl[f].v[k + 1]), x1 = make_float2(xh.v[k], xh.v[k + 1]);
                    const float2 y0 = make_float2(yl.v[k], yl.v[k + 1]), y1 = make_float2(yh.v[k], yh.v[k + 1]);
                    const float left = k == 0 ? zl : cc[f].v[k - 1], right = k + 2 == V ? zh : cc[f].v[k + 2];
                    float2 nv;
                    if (DIFF) {   // (along Z cell by cell: pairs of left and right neighbours would cost moves)
                        const float2 dz = make_float2(diff2(c2.x, left, c2.y), diff2(c2.y, c2.x, right));
                        nv = col_new_diff<MODEL, float2>(c2, s2, diff2(c2, x0, x1), diff2(c2, y0, y1), dz, q);
                    } else {
                        nv = col_new_sums<MODEL, float2>(c2, s2, cadd(x0, x1), cadd(y0, y1),
                                                         make_float2(left + c2.y, c2.x + right), q);
                    }
                    w.v[k] = nv.x;
                    w.v[k + 1] = nv.y;
                }
            }
            w.store(po + f * fb, o);
            xl[f] = cc[f];
            cc[f] = xh;
        }
    }
}


// ---------------------------------------------------------------------------
// The new value of one order parameter in the reference's order, with the
// square p2 = phi*phi at hand.  KAPPA: 1 or 2 when kappa is exactly that
// (1.0*x is x, 2.0*x is exact), 0 for any other value.
template <typename T, int MODEL, int KAPPA, bool NOISE>
static __device__ __forceinline__ T ac_new_p2(const Ar<T>& A, T phi, T p2, T sum, T lap, T noise, const P<T>& p)
{
    const T kl = KAPPA == 1 ? lap : KAPPA == 2 ? twice(lap) : A.mul(p.kappa, lap);
    if (MODEL == MMSP_GPU_AC) {
        // phi - dt*L*(-phi + phi*phi*phi + 2.0*gamma*phi*(sum - phi*phi) - kappa*lap)
        const T a = A.add(-phi, A.mul(p2, phi));
        const T g = A.mul(A.mul(p.gamma2, phi), A.sub(sum, p2));
        return A.sub(phi, A.mul(p.dtm, A.sub(A.add(a, g), kl)));
    } else if (MODEL == MMSP_GPU_GG || MODEL == MMSP_GPU_ZENER) {
        // phi - dt*(-phi - pow(phi,3) + 2.0*(phi*sum - lap))   (graingrowth.cpp:105, zener.cpp:135)
        const T e = A.add(A.sub(-phi, cube_p2(A, phi, p2)), twice(A.sub(A.mul(phi, sum), lap)));
        return A.sub(phi, A.mul(p.dtm, e));
    } else {
        // phi - dt*M*(-r*phi + u*pow(phi,3) - K*lap + noise)   (allen-cahn.cpp:70, model_A.cpp:99-100)
        T e = A.sub(A.add(A.mul(p.neg_r, phi), A.mul(p.u, cube_p2(A, phi, p2))), kl);
        if (NOISE) e = A.add(e, noise);
        return A.sub(phi, A.mul(p.dtm, e));
    }
}

// Threads per block: 128, or 32 on grids of few cells, whose warps then
// spread evenly over the SMs (one FP64 pipe each): 32^3 x 16 fields 25.4 ->
// 23.0 us per step, 40x41x42 x 5 16.9 -> 15.9 (before the arithmetic of
// pf_device.cuh, which takes them to 21.7 and 14.1); no difference on large grids.
constexpr int kAcAnyThreads = 128;
constexpr long long kAcAnySmall = 1LL << 17;

template <typename T, int DIM, int MODEL, bool UNIT, int KAPPA, bool NOISE>
__global__ void __launch_bounds__(kAcAnyThreads)
ac_cols_any(const T* __restrict__ ein, T* __restrict__ eout, Geom g, P<T> pc0, int N)
{
    const Ar<T> A(g.dim);
    const P<T> p = held(A, pc0);
    extern __shared__ __align__(8) unsigned char sq_raw[];
    T* mine = reinterpret_cast<T*>(sq_raw) + threadIdx.x;   // [field][thread]: this thread's squares
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.YZ) return;           // no barrier in this kernel
    const int y = (int)(i / g.Z), z = (int)(i - (long long)y * g.Z);
    const long long dyl = (y == 0 ? (long long)(g.Y - 1) : -1LL) * g.Z, dyh = (y + 1 == g.Y ? -(long long)y : 1LL) * g.Z;
    const int dzl = z == 0 ? g.Z - 1 : -1, dzh = z + 1 == g.Z ? -z : 1;
    for (int x = blockIdx.y; x < g.X; x += gridDim.y) {
        const T* pc = ein + (long long)x * g.YZ + i;
        T* po = eout + (long long)x * g.YZ + i;
        const long long dxl = (x == 0 ? (long long)(g.X - 1) : -1LL) * g.YZ;
        const long long dxh = (x + 1 == g.X ? -(long long)x : 1LL) * g.YZ;
        const T noise = NOISE ? noise_at(p, g.cells, (long long)x * g.YZ + i) : T(0);
        // sum of squares in field order (graingrowth.cpp:98-101); 0.0 + p0^2 == p0^2
        T sum = T(0);
#pragma unroll 4
        for (int f = 0; f < N; f++) {
            const T c = __ldg(pc + f * g.cells);
            const T p2 = A.mul(c, c);
            sum = f == 0 ? p2 : A.add(sum, p2);
            mine[f * blockDim.x] = p2;
        }
#pragma unroll 2
        for (int f = 0; f < N; f++) {
            const T* q = pc + f * g.cells;
            const T c = __ldg(q);
            T xl = T(0), xh = T(0), yl = T(0), yh = T(0);
            if (DIM == 3) xl = __ldg(q + dxl), xh = __ldg(q + dxh);
            if (DIM >= 2) yl = __ldg(q + dyl), yh = __ldg(q + dyh);
            const T lap = lap_ref<T, UNIT, DIM>(A, twice(c), xh, xl, yh, yl, __ldg(q + dzh), __ldg(q + dzl), p.wx, p.wy, p.wz);
            const T v = ac_new_p2<T, MODEL, KAPPA, NOISE>(A, c, mine[f * blockDim.x], sum, lap, noise, p);
            // Zener pinning: the particles (field 0) have zero mobility (zener.cpp:134)
            po[f * g.cells] = (MODEL == MMSP_GPU_ZENER && f == 0) ? c : v;
        }
    }
}

namespace {

template <int N, int V, bool DIFF, bool PRE>
const void* cols_model(int model)
{
    if (model == MMSP_GPU_AC) return (const void*)&ac_cols_f32<N, V, MMSP_GPU_AC, DIFF, PRE>;
    if (model == MMSP_GPU_GG) return (const void*)&ac_cols_f32<N, V, MMSP_GPU_GG, DIFF, PRE>;
    if (model == MMSP_GPU_ZENER) return (const void*)&ac_cols_f32<N, V, MMSP_GPU_ZENER, DIFF, PRE>;
    if (N == 1 && model == MMSP_GPU_AC_POLY) return (const void*)&ac_cols_f32<1, V, MMSP_GPU_AC_POLY, DIFF, PRE>;
    return nullptr;
}

// Prefetch (us per step without / with): V = 4 with 6 and 7 fields always,
// 128^3 x 6 22.3 / 18.8, x 7 24.8 / 22.7, 80^3 x 6 8.3 / 8.3; 4 and 5 fields
// never, 160^3 x 4 24.7 / 26.7, 148^3 x 5 25.8 / 26.7.  V = 1 with 5 to 9 fields
// where the states exceed L2, 127^3 x 6 35.0 / 25.5, x 8 36.9 / 34.8, but 91^3
// x 7 (42 MB) 12.4 / 13.1 and 127^3 x 10 43.4 / 45.3.  V = 2 never, 128^3 x 8
// 24.1 / 26.0, 126^3 x 12 44.2 / 45.2.
template <int N, int V, bool DIFF>
const void* cols_pre(int model, bool big)
{
    if constexpr (V == 4) return cols_model<N, V, DIFF, (N >= 6)>(model);
    else if constexpr (V == 1 && N >= 5 && N <= 9)
        return big ? cols_model<N, V, DIFF, true>(model) : cols_model<N, V, DIFF, false>(model);
    else return cols_model<N, V, DIFF, false>(model);
}

// V cells per thread, by the row length and the field count: vectors need
// rows of a multiple of V cells (every row, plane and field then starts on
// the vector's alignment), and V*N rolled values must fit the registers.
// Measured, us per step: 128^3 x 7: 21.7 (V = 4), 31.9 (2), 31.6 (1); x 8:
// 27.5 / 24.5 / 36.9; x 16: 62 / 55 / 85; 74^3 x 14: 10.3 (V = 2), 12.4 (1).
template <int V, bool DIFF, int LO, int HI>
const void* cols_fn(int n, int model, bool big)
{
    if constexpr (LO > HI) {
        return nullptr;
    } else {
        return n == LO ? cols_pre<LO, V, DIFF>(model, big) : cols_fn<V, DIFF, LO + 1, HI>(n, model, big);
    }
}

template <bool DIFF>
const void* cols_pick(int Z, int n, int model, bool big, int* v)
{
    *v = Z % 4 == 0 && n <= 7 ? 4 : Z % 2 == 0 && n <= 16 ? 2 : 1;
    return *v == 4   ? cols_fn<4, DIFF, 1, 7>(n, model, big)
           : *v == 2 ? cols_fn<2, DIFF, 1, 16>(n, model, big)
                     : cols_fn<1, DIFF, 1, 32>(n, model, big);
}

// Sums of neighbours on 3D grids of rows of up to 256 cells, unless a plane is
// one or two rows or a row of all fields more than 5600 values; differences on
// all others.  Sums are faster where the registers are full, differences round
// less.  us per step and RMS error against 64 bits after 40 steps, sums /
// differences: 128^3 x 8 25.0, 1.08e-8 / 29.0, 0.86e-8; 40x50x1000 x 8 27.0,
// 1.08e-8 / 31.1, 0.84e-8; 30x40x300 x 4 4.1, 1.56e-8 / 4.1, 1.21e-8; 1024^2 x
// 16 32.9, 0.79e-8 / 32.9, 0.73e-8.
bool cols_sums(const Geom& g, int n)
{
    return g.dim == 3 && g.Z <= 256 && g.Y >= 3 && (long long)g.Z * n <= 5600;
}

template <typename T, int DIM, bool UNIT>
const void* any_model(int model, int kappa, bool noise)
{
    // grain growth and Zener pinning have no gradient coefficient; FP32 multiplies by any coefficient
    constexpr int K1 = sizeof(T) == 8 ? 1 : 0, K2 = sizeof(T) == 8 ? 2 : 0;
    if (model == MMSP_GPU_GG) return (const void*)&ac_cols_any<T, DIM, MMSP_GPU_GG, UNIT, 1, false>;
    if (model == MMSP_GPU_ZENER) return (const void*)&ac_cols_any<T, DIM, MMSP_GPU_ZENER, UNIT, 1, false>;
    if (model == MMSP_GPU_AC)
        return kappa == 2 ? (const void*)&ac_cols_any<T, DIM, MMSP_GPU_AC, UNIT, K2, false>
               : kappa == 1 ? (const void*)&ac_cols_any<T, DIM, MMSP_GPU_AC, UNIT, K1, false>
                            : (const void*)&ac_cols_any<T, DIM, MMSP_GPU_AC, UNIT, 0, false>;
    if (noise) return (const void*)&ac_cols_any<T, DIM, MMSP_GPU_AC_POLY, UNIT, 0, true>;
    return kappa == 1 ? (const void*)&ac_cols_any<T, DIM, MMSP_GPU_AC_POLY, UNIT, K1, false>
                      : (const void*)&ac_cols_any<T, DIM, MMSP_GPU_AC_POLY, UNIT, 0, false>;
}

template <typename T>
const void* any_pick(int dim, bool unit, int model, double kappa, bool noise)
{
    const int k = kappa == 1.0 ? 1 : kappa == 2.0 ? 2 : 0;
    if (dim == 3) return unit ? any_model<T, 3, true>(model, k, noise) : any_model<T, 3, false>(model, k, noise);
    if (dim == 2) return unit ? any_model<T, 2, true>(model, k, noise) : any_model<T, 2, false>(model, k, noise);
    return unit ? any_model<T, 1, true>(model, k, noise) : any_model<T, 1, false>(model, k, noise);
}

}  // namespace

// FP32: one wave of blocks where the two states stay in L2 (planes per block
// as few as that allows); above, short runs of 2 or 3 planes, so that the
// blocks run through X in order and a step finds the last planes of the step
// before in L2 (the direction alternates).  Measured, us per step, one wave
// against short runs: 128^3 x 8 (134 MB) 28.3 / 24.5 (29.0 with a fixed
// direction), 128^3 x 16 73.3 / 55.0, 128^3 x 7 (117 MB) 24.4 / 21.7; 128^3 x
// 4 (67 MB) 9.6 / 10.5, 74^3 x 14 (45 MB) 10.5 / 11.8, 65^3 x 14 8.9 / 9.5.
constexpr long long kAcColL2 = 96LL << 20;

cudaError_t plan_ac(const mmsp_gpu_desc& d, const Geom& g, StepPlan* p)
{
    p->fields = d.fields;
    p->kind = 0;
    p->planes = 0;
    // 32-bit byte offsets within a plane need fewer than 2^30 cells
    if (d.dtype == MMSP_GPU_F64 || noisy(d) || g.YZ >= (1LL << 30)) {
        const Coeffs c = make_coeffs(d);
        const bool dbl = d.dtype == MMSP_GPU_F64;
        p->fn = dbl ? any_pick<double>(g.dim, c.unit_w, d.model, c.kappa, noisy(d))
                    : any_pick<float>(g.dim, c.unit_w, d.model, c.kappa, noisy(d));
        const int threads = g.cells < kAcAnySmall ? 32 : kAcAnyThreads;
        p->smem = (dbl ? sizeof(double) : sizeof(float)) * (size_t)d.fields * threads;   // at most 32 KB
        p->block = dim3(threads, 1, 1);
        p->grid = dim3((unsigned)((g.YZ + threads - 1) / threads), std::min(g.X, 65535), 1);
        p->ok = true;
        return cudaSuccess;
    }
    const bool big = 2LL * g.cells * d.fields * (long long)sizeof(float) > kAcColL2;
    int v = 1;
    p->fn = cols_sums(g, d.fields) ? cols_pick<false>(g.Z, d.fields, d.model, big, &v)
                                   : cols_pick<true>(g.Z, d.fields, d.model, big, &v);
    if (!p->fn) return cudaErrorInvalidConfiguration;
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, p->fn, kAcColThreads, 0);
    if (e != cudaSuccess) return e;
    const long long cols = (g.YZ / v + kAcColThreads - 1) / kAcColThreads;
    const long long slots = (long long)sm_count() * std::max(1, per_sm);
    long long planes = big ? (d.fields <= 8 ? 3 : 2) : (cols * g.X + slots - 1) / slots;
    planes = std::max(planes, (long long)(g.X + 65534) / 65535);
    planes = std::min(std::max(planes, 1LL), (long long)g.X);
    p->planes = (int)planes;
    p->block = dim3(kAcColThreads, 1, 1);
    p->grid = dim3((unsigned)cols, (unsigned)((g.X + planes - 1) / planes), 1);
    p->smem = 0;
    p->ok = true;
    return cudaSuccess;
}

cudaError_t launch_ac(const StepPlan& p, const mmsp_gpu_desc& d, const Geom& g, const Coeffs& c, const void* in,
                      void* out, int* err, cudaStream_t s)
{
    int n = p.fields, planes = p.planes;
    if (d.dtype == MMSP_GPU_F64) {
        P<double> q = narrow<double>(c, g.dim);
        if (noisy(d)) q.stepp = step_word(err);
        void* args[] = {(void*)&in, (void*)&out, (void*)&g, (void*)&q, (void*)&n};
        return cudaLaunchKernel(p.fn, p.grid, p.block, args, p.smem, s);
    }
    P<float> w = narrow<float>(c, g.dim);
    if (planes == 0) {
        if (noisy(d)) w.stepp = step_word(err);
        void* args[] = {(void*)&in, (void*)&out, (void*)&g, (void*)&w, (void*)&n};
        return cudaLaunchKernel(p.fn, p.grid, p.block, args, p.smem, s);
    }
    // axes that the grid does not have weigh nothing (their neighbours are the cell itself)
    const float sign = cols_sums(g, n) ? 1.0f : -1.0f;
    AcColF32 q;
    q.wx = g.dim == 3 ? sign * w.wx : 0.0f;
    q.wy = g.dim >= 2 ? sign * w.wy : 0.0f;
    q.wz = sign * w.wz;
    q.w2 = 2.0f * (q.wx + q.wy + q.wz);
    q.kappa = w.kappa;
    q.dtm = w.dtm;
    q.gamma2 = w.gamma2;
    q.neg_r = w.neg_r;
    q.u = w.u;
    int flip = in > out;
    void* args[] = {(void*)&in, (void*)&out, (void*)&g, (void*)&q, (void*)&planes, (void*)&flip};
    return cudaLaunchKernel(p.fn, p.grid, p.block, args, 0, s);
}

}  // namespace pf
