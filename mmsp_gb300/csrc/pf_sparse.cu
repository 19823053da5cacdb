// pf_sparse.cu -- isotropic sparse phase-field grain growth (the sparsePF example).
//
// The reference keeps, per cell, a list of (grain index, value) items in
// insertion order (class sparse, include/MMSP.sparse.h:19; set() overwrites
// an item or appends one, operator[] reads 0 for an absent index), and its
// update (examples/coarsening/grain_growth/isotropic/sparsePF/graingrowth.cpp:58-120)
// works per cell on the union of the indices of the cell and its 2*dim face
// neighbours.
//
// Device format: a state buffer holds the lists slot-major, so that slot h
// of neighbouring cells is one coalesced line:
//   count[cells]           int32 items per cell
//   index[K][cells]        int32 grain index of slot h
//   value[K][cells]        T value of slot h
// with K = mmsp_gpu_desc.fields slots per cell.  A list that would outgrow K
// sets the overflow word and leaves that item out (the host reports
// MMSP_GPU_EOVERFLOW; the state is then invalid).
//
// The example's newGrid starts with empty cells and is never cleared:
// after swap() the buffer written at step s holds the state of
// step s-2, and set() keeps the items it does not overwrite.  The ping-pong
// buffers do the same (the host clears the idle buffer's counts at the start
// of each step call, as each update() call builds a fresh newGrid), so the
// stale items that enter later neighbour sets and sums are the reference's.
//
// Arithmetic: the sparse Laplacian (include/MMSP.grid.cpp:2110-2128) adds and
// subtracts item lists through sparse operator+/- that start each index at 0;
// where an index is absent each operation is exact, so its value is the
// dense weight*((yh - 2y) + yl) summed from 0.0 over axes with absent items
// read as 0 -- computed here in that order with every operation rounded on
// its own.  pow(phi,3) is the compensated cube of pf_device.cuh (within the
// C library's 1 ulp), so values are held to 1e-12 relative and counts and
// indices exactly.
#include "pf_device.cuh"
#include "pf_internal.h"

namespace pf {

constexpr int kSparseSet = 64;   // largest neighbour set (union of 2*dim+1 lists)

struct SpView {
    int* cnt;
    int* idx;        // idx[h * cells + c]
    double* val;     // val[h * cells + c]
};

SparseLayout sparse_layout(long long cells, int K)
{
    SparseLayout L;
    auto pad = [](size_t b) { return (b + 255) / 256 * 256; };
    L.idx_off = pad(sizeof(int) * (size_t)cells);
    L.val_off = L.idx_off + pad(sizeof(int) * (size_t)cells * K);
    L.bytes = L.val_off + sizeof(double) * (size_t)cells * K;
    return L;
}

static SpView view_of(void* buf, long long cells, int K)
{
    const SparseLayout L = sparse_layout(cells, K);
    SpView v;
    v.cnt = static_cast<int*>(buf);
    v.idx = reinterpret_cast<int*>(static_cast<char*>(buf) + L.idx_off);
    v.val = reinterpret_cast<double*>(static_cast<char*>(buf) + L.val_off);
    return v;
}

// Value of index i in cell c's list (0 when absent), as sparse::operator[].
static __device__ __forceinline__ double sp_get(const SpView& s, long long cells, long long c, int i)
{
    const int n = __ldg(s.cnt + c);
    for (int h = 0; h < n; h++)
        if (__ldg(s.idx + h * cells + c) == i) return __ldg(s.val + h * cells + c);
    return 0.0;
}

struct SpConst {
    double w[3];     // 1/(dx*dx) per real axis
    double eps;      // epsilon: values at or below it are not stored
    P<double> p;     // dtm = dt for the update expression
};

// The padded coordinates' neighbours of one cell in the reference's axis order
// (real axis 0 first), then the update of its lists, list by list in global
// memory: any number of grains.
template <int DIM, bool UNIT>
static __device__ __noinline__ void sparse_cell(SpView in, SpView out, Geom g, SpConst q, int K, long long c, int* err)
{
    const long long cells = g.cells;
    const Ar<double> A(g.dim);
    const int x = (int)(c / g.YZ);
    const int r = (int)(c - (long long)x * g.YZ);
    const int y = r / g.Z;
    const int z = r - y * g.Z;
    long long lo[3], hi[3];
    {
        const int xl = x == 0 ? g.X - 1 : x - 1, xh = x + 1 == g.X ? 0 : x + 1;
        const int yl = y == 0 ? g.Y - 1 : y - 1, yh = y + 1 == g.Y ? 0 : y + 1;
        const int zl = z == 0 ? g.Z - 1 : z - 1, zh = z + 1 == g.Z ? 0 : z + 1;
        const long long px[3] = {c + (long long)(xl - x) * g.YZ, c + (long long)(yl - y) * g.Z, c + (zl - z)};
        const long long qx[3] = {c + (long long)(xh - x) * g.YZ, c + (long long)(yh - y) * g.Z, c + (zh - z)};
        for (int ra = 0; ra < DIM; ra++) {
            lo[ra] = px[3 - DIM + ra];
            hi[ra] = qx[3 - DIM + ra];
        }
    }
    // nonzero fields of the neighbourhood, in the example's visiting order:
    // per axis the low neighbour, the cell itself, the high neighbour
    int S[kSparseSet];
    int ns = 0;
    bool ovf = false;
#pragma unroll
    for (int ra = 0; ra < DIM; ra++) {
        for (int k = 0; k < 3; k++) {
            const long long nc = k == 0 ? lo[ra] : k == 1 ? c : hi[ra];
            const int n = __ldg(in.cnt + nc);
            for (int h = 0; h < n; h++) {
                const int i = __ldg(in.idx + h * cells + nc);
                bool seen = false;
                for (int s = 0; s < ns; s++) seen |= S[s] == i;
                if (!seen) {
                    if (ns == kSparseSet) ovf = true;
                    else S[ns++] = i;
                }
            }
        }
    }
    const int own = __ldg(in.cnt + c);
    if (ns < 2) {
        // newGrid(n) = oldGrid(n): the whole list
        out.cnt[c] = own;
        for (int h = 0; h < own; h++) {
            out.idx[h * cells + c] = __ldg(in.idx + h * cells + c);
            out.val[h * cells + c] = __ldg(in.val + h * cells + c);
        }
    } else {
        double sum = 0.0;
        for (int h = 0; h < own; h++) {
            const double phi = __ldg(in.val + h * cells + c);
            sum = A.add(sum, A.mul(phi, phi));
        }
        // newGrid(n) as it stands: the state of two steps back
        int dn = out.cnt[c];
        for (int s = 0; s < ns; s++) {
            const int i = S[s];
            const double phi = sp_get(in, cells, c, i);
            const double y2 = twice(phi);
            double lap = 0.0;
#pragma unroll
            for (int ra = 0; ra < DIM; ra++) {
                double t = A.add(A.sub(sp_get(in, cells, hi[ra], i), y2), sp_get(in, cells, lo[ra], i));
                if (!UNIT) t = A.mul(q.w[ra], t);
                lap = ra == 0 ? plus_zero(t) : A.add(lap, t);
            }
            const double v = gg_new(A, phi, sum, lap, q.p);
            if (v > q.eps) {
                int h = 0;
                while (h < dn && out.idx[h * cells + c] != i) h++;
                if (h == dn) {
                    if (dn == K) {
                        ovf = true;
                        continue;
                    }
                    out.idx[h * cells + c] = i;
                    dn++;
                }
                out.val[h * cells + c] = v;
            }
        }
        out.cnt[c] = dn;
    }
    if (ovf) atomicExch(err, 1);
}

// One thread per cell.  The neighbour lists are read once: the union is built
// in shared memory, one column per thread, and beside each of its grains the
// slots that the grain has in the cell's, the neighbours' and the destination
// list, 6 bits each.  Every value is then one direct load, and the loads of a
// grain are independent of each other.  A union of more than kSpUnion grains
// goes through sparse_cell.
//
// Bound: the FP64 pipe (about 18 operations per cell and grain, and a warp
// takes as many rounds as its busiest cell; 55% busy) and load latency.  us per
// step, walking the lists in global memory for every value / here with a row of
// cells a warp: 512x512 cells of 160 grains 78.5 / 54.9 (500 steps from one item
// per cell), 2048x2048 of 32 grains 201 / 157, 48^3 of 12 grains 100 / 55.8.
// (A dense table of a tile's grains in shared memory, behind a hashed
// dictionary, took 65, 64, 229 and 82: its set-up costs more than the walks.)
// 64-thread blocks of at most 64 registers: with 128 threads 60.9, with 72
// registers 58.6.
// BAND: a warp's cells are a patch of the plane, BAND rows by 32 / BAND columns,
// instead of 32 in a row: they lie closer together, so their numbers of grains
// differ less.  us per step in a row / in bands of 2 / 4 / 8 rows: 512x512 54.9
// / 50.6 / 48.5 / 49.4, 2048x2048 157 / 151 / 144 / 148, 48^3 55.8 / 51.8 / 50.1
// / 51.3, 41^3 55.4 / 54.9 / 54.7 / 54.7; but 25^3 55.2 / 56.0 / 56.5 / 56.5 and
// 33x50x27 42.0 / 42.4 / 42.5 / 42.7, one wave of blocks: small grids, and 1D,
// keep the row (kSpBandCells).
constexpr int kSpThreads = 64;
constexpr int kSpUnion = 16;
constexpr int kSpBatch = 4;   // items of a list that are loaded at once
constexpr long long kSpBandCells = 1LL << 16;

template <int DIM, bool UNIT, int BAND>
__global__ void __launch_bounds__(kSpThreads, 16)
sparse_gg_step(SpView in, SpView out, Geom g, SpConst q0, int K, int* __restrict__ err)
{
    __shared__ int s_key[kSpUnion][kSpThreads];
    __shared__ unsigned long long s_pos[kSpUnion][kSpThreads];   // slot + 1 in list l at bit 6*l, 0: not there
    const int tid = threadIdx.x;
    const long long k0 = (long long)blockIdx.x * kSpThreads + tid;
    if (k0 >= g.cells) return;   // no barrier in this kernel
    const long long cells = g.cells;
    // the cells of a plane in bands of BAND rows (the last may have fewer), down each column of a band in turn
    const int x = (int)(k0 / g.YZ);
    const int r = (int)(k0 - (long long)x * g.YZ);
    int y = r / g.Z / BAND * BAND, z = r - y * g.Z;
    if constexpr (BAND > 1) {
        const int e = z, rows = min(BAND, g.Y - y);
        z = rows == BAND ? e / BAND : e / rows;
        y += e - z * rows;
    }
    const long long c = (long long)x * g.YZ + (long long)y * g.Z + z;
    // padded coordinates and the periodic face neighbours of the real axes,
    // in the reference's axis order (real axis 0 first); list 0 is the cell's
    // own, 1 + 2 ra and 2 + 2 ra the low and high neighbour's on axis ra, 7 the
    // destination's
    long long nb[1 + 2 * DIM];
    nb[0] = c;
    nb[2 * DIM - 1] = c + (z == 0 ? g.Z - 1 : -1);
    nb[2 * DIM] = c + (z + 1 == g.Z ? -z : 1);
    if constexpr (DIM >= 2) {
        nb[2 * DIM - 3] = c + (long long)(y == 0 ? g.Y - 1 : -1) * g.Z;
        nb[2 * DIM - 2] = c + (long long)(y + 1 == g.Y ? -y : 1) * g.Z;
    }
    if constexpr (DIM == 3) {
        nb[1] = c + (long long)(x == 0 ? g.X - 1 : -1) * g.YZ;
        nb[2] = c + (long long)(x + 1 == g.X ? -x : 1) * g.YZ;
    }
    int n[1 + 2 * DIM];
#pragma unroll
    for (int l = 0; l < 1 + 2 * DIM; l++) n[l] = __ldg(in.cnt + nb[l]);

    int ns = 0;
    // items of list l into the union (JOIN), or only their slots
    auto read = [&](const int* idx, long long cell, int items, int l, bool join) {
        for (int h0 = 0; h0 < items; h0 += kSpBatch) {
            int key[kSpBatch];
#pragma unroll
            for (int k = 0; k < kSpBatch; k++) key[k] = h0 + k < items ? idx[(h0 + k) * cells + cell] : 0;
#pragma unroll
            for (int k = 0; k < kSpBatch; k++) {
                if (h0 + k >= items) break;
                int s = 0;
                while (s < ns && s_key[s][tid] != key[k]) s++;
                const unsigned long long slot = (unsigned long long)(h0 + k + 1) << (6 * l);
                if (s < ns) {
                    // (of a repeated index the first item counts)
                    const unsigned long long have = s_pos[s][tid];
                    if (!(have >> (6 * l) & 63)) s_pos[s][tid] = have | slot;
                } else if (join) {
                    if (ns < kSpUnion) {
                        s_key[ns][tid] = key[k];
                        s_pos[ns][tid] = slot;
                    }
                    if (ns <= kSpUnion) ns++;
                    if (ns > kSpUnion) return;
                }
            }
        }
    };
    // the example's visiting order: per axis the low neighbour, the cell itself, the high neighbour
#pragma unroll
    for (int ra = 0; ra < DIM; ra++) {
        if (ns <= kSpUnion) read(in.idx, nb[1 + 2 * ra], n[1 + 2 * ra], 1 + 2 * ra, true);
        if (ra == 0 && ns <= kSpUnion) read(in.idx, c, n[0], 0, true);
        if (ns <= kSpUnion) read(in.idx, nb[2 + 2 * ra], n[2 + 2 * ra], 2 + 2 * ra, true);
    }
    if (ns > kSpUnion) {
        sparse_cell<DIM, UNIT>(in, out, g, q0, K, c, err);
        return;
    }
    if (ns < 2) {
        // newGrid(n) = oldGrid(n): the whole list
        out.cnt[c] = n[0];
        for (int h = 0; h < n[0]; h++) {
            out.idx[h * cells + c] = __ldg(in.idx + h * cells + c);
            out.val[h * cells + c] = __ldg(in.val + h * cells + c);
        }
        return;
    }
    const Ar<double> A(g.dim);
    const P<double> p = held(A, q0.p);
    double sum = 0.0;
    for (int h0 = 0; h0 < n[0]; h0 += kSpBatch) {
        double v[kSpBatch];
#pragma unroll
        for (int k = 0; k < kSpBatch; k++) v[k] = h0 + k < n[0] ? __ldg(in.val + (h0 + k) * cells + c) : 0.0;
#pragma unroll
        for (int k = 0; k < kSpBatch; k++) {
            if (h0 + k >= n[0]) break;
            sum = A.add(sum, A.mul(v[k], v[k]));
        }
    }
    // newGrid(n) as it stands: the state of two steps back
    int dn = out.cnt[c];
    read(out.idx, c, dn, 7, false);
    bool ovf = false;
    // the values of grain s in the cell's and the neighbours' lists
    auto fetch = [&](int s, double (&f)[1 + 2 * DIM]) {
        const unsigned long long pos = s_pos[s][tid];
#pragma unroll
        for (int l = 0; l < 1 + 2 * DIM; l++) {
            const int slot = (int)(pos >> (6 * l)) & 63;
            f[l] = slot ? __ldg(in.val + (slot - 1) * cells + nb[l]) : 0.0;
        }
    };
    double next[1 + 2 * DIM];   // loaded one grain ahead
    fetch(0, next);
    for (int s = 0; s < ns; s++) {
        double f[1 + 2 * DIM];
#pragma unroll
        for (int l = 0; l < 1 + 2 * DIM; l++) f[l] = next[l];
        if (s + 1 < ns) fetch(s + 1, next);
        const double phi = f[0], y2 = twice(phi);
        double lap = 0.0;
#pragma unroll
        for (int ra = 0; ra < DIM; ra++) {
            double t = A.add(A.sub(f[2 + 2 * ra], y2), f[1 + 2 * ra]);
            if (!UNIT) t = A.mul(A.reg(q0.w[ra]), t);
            lap = ra == 0 ? plus_zero(t) : A.add(lap, t);
        }
        const double v = gg_new(A, phi, sum, lap, p);
        if (v > q0.eps) {
            int h = (int)(s_pos[s][tid] >> 42) & 63;
            if (!h) {
                if (dn == K) {
                    ovf = true;
                    continue;
                }
                out.idx[dn * cells + c] = s_key[s][tid];
                h = ++dn;
            }
            out.val[(h - 1) * cells + c] = v;
        }
    }
    out.cnt[c] = dn;
    if (ovf) atomicExch(err, 1);
}

// Host cell-major slots (count[cells], index[cells*K], value[cells*K]) <->
// the device's slot-major buffer, through a staging buffer that holds the
// three host arrays at the offsets of sparse_layout.
__global__ void sparse_pack(const int* __restrict__ hcnt, const int* __restrict__ hidx, const double* __restrict__ hval,
                            SpView d, long long cells, int K)
{
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= cells) return;
    const int n = min(max(hcnt[c], 0), K);   // the host has checked 0 <= n <= K
    d.cnt[c] = n;
    for (int h = 0; h < K; h++) {
        d.idx[h * cells + c] = h < n ? hidx[c * K + h] : 0;
        d.val[h * cells + c] = h < n ? hval[c * K + h] : 0.0;
    }
}

__global__ void sparse_unpack(SpView d, int* __restrict__ hcnt, int* __restrict__ hidx, double* __restrict__ hval,
                              long long cells, int K)
{
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= cells) return;
    const int n = d.cnt[c];
    hcnt[c] = n;
    for (int h = 0; h < K; h++) {
        hidx[c * K + h] = h < n ? d.idx[h * cells + c] : 0;
        hval[c * K + h] = h < n ? d.val[h * cells + c] : 0.0;
    }
}

static unsigned blocks_for(long long cells, int threads = 128) { return (unsigned)((cells + threads - 1) / threads); }

template <int DIM>
static const void* sparse_fn(bool unit, bool band)
{
    if constexpr (DIM > 1) {
        if (band)
            return unit ? (const void*)&sparse_gg_step<DIM, true, 4> : (const void*)&sparse_gg_step<DIM, false, 4>;
    }
    return unit ? (const void*)&sparse_gg_step<DIM, true, 1> : (const void*)&sparse_gg_step<DIM, false, 1>;
}

cudaError_t launch_sparse_gg(const mmsp_gpu_desc& d, const Geom& g, const Coeffs& c, const void* in, void* out,
                             int* err, cudaStream_t s)
{
    const int K = d.fields;
    SpView vi = view_of(const_cast<void*>(in), g.cells, K), vo = view_of(out, g.cells, K);
    SpConst q;
    for (int a = 0; a < 3; a++) q.w[a] = a < d.dim ? c.w[a] : 1.0;
    q.eps = d.aux[0];
    q.p = narrow<double>(c, g.dim);
    const bool band = g.dim > 1 && g.cells >= kSpBandCells;
    const void* fn = g.dim == 3   ? sparse_fn<3>(c.unit_w, band)
                     : g.dim == 2 ? sparse_fn<2>(c.unit_w, band)
                                  : sparse_fn<1>(c.unit_w, false);
    int* ovf = err + 1;
    void* args[] = {(void*)&vi, (void*)&vo, (void*)&g, (void*)&q, (void*)&K, (void*)&ovf};
    return cudaLaunchKernel(fn, dim3(blocks_for(g.cells, kSpThreads)), dim3(kSpThreads), args, 0, s);
}

cudaError_t launch_sparse_pack(const void* staging, void* state, long long cells, int K, cudaStream_t s)
{
    const SpView h = view_of(const_cast<void*>(staging), cells, K);
    sparse_pack<<<blocks_for(cells), 128, 0, s>>>(h.cnt, h.idx, h.val, view_of(state, cells, K), cells, K);
    return cudaGetLastError();
}

cudaError_t launch_sparse_unpack(const void* state, void* staging, long long cells, int K, cudaStream_t s)
{
    const SpView h = view_of(staging, cells, K);
    sparse_unpack<<<blocks_for(cells), 128, 0, s>>>(view_of(const_cast<void*>(state), cells, K), h.cnt, h.idx, h.val,
                                                    cells, K);
    return cudaGetLastError();
}

}  // namespace pf
