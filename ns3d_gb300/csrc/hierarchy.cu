// hierarchy.cu -- the aggregation hierarchy of a pressure system (MIXED_MG),
// built on the device from the row -> cell table.
//
// Level k+1 groups the rows of level k by the 2x2x2 block of their cell
// coordinates and numbers the blocks in ascending (i, j, k) order.  Rows of
// every level are numbered in that order too, so a block's members in
// ascending row order are its occupied octants in ascending octant order:
// one 8-bit occupancy mask per block gives the member count (popc) and each
// member's place (popc of the lower octants), and no sort is needed.
//
// What bounds it: bytes and launches.  Per level one pass over the rows sets
// the masks, a three-pass scan over the dense block grid (1/8 of the cells)
// numbers the blocks, and two passes write the member lists and the
// neighbour table.  The sort-based host build this replaces took 280 ms at
// 3.6 M rows (the image's whole six-iteration solve: 280 ms) and 17 ms at
// 205 K rows.
#include <cstring>

#include "mixed.h"
#include "runtime.h"

namespace ns3d {

constexpr int HB_THREADS = 256;
constexpr int HB_PER_THREAD = 4;
constexpr int HB_TILE = HB_THREADS * HB_PER_THREAD;  // dense blocks per scan tile

struct CellBox {  // extents of a level's cell grid (cell = (i ny + j) nz + k)
    int nx, ny, nz;
    __host__ __device__ CellBox coarse() const { return {(nx + 1) / 2, (ny + 1) / 2, (nz + 1) / 2}; }
    __host__ __device__ long cells() const { return (long)nx * ny * nz; }
};

// block of a cell in the coarse grid, and its octant in the block
__device__ __forceinline__ int block_of(int c, CellBox f, int &oct) {
    const int k = c % f.nz, t = c / f.nz, j = t % f.ny, i = t / f.ny;
    const CellBox b = f.coarse();
    oct = ((i & 1) << 2) | ((j & 1) << 1) | (k & 1);
    return ((i >> 1) * b.ny + (j >> 1)) * b.nz + (k >> 1);
}

__global__ void k_hb_mark(const int *__restrict__ cell, int n, CellBox f, unsigned int *__restrict__ mask) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        int oct;
        const int b = block_of(cell[r], f, oct);
        atomicOr(mask + b, 1u << oct);
    }
}

__device__ __forceinline__ int2 add2(int2 a, int2 b) { return make_int2(a.x + b.x, a.y + b.y); }

// (occupied blocks, members) of this thread's blocks of a tile
__device__ __forceinline__ int2 hb_counts(const unsigned int *mask, long base, long nb) {
    int2 s = make_int2(0, 0);
#pragma unroll
    for (int m = 0; m < HB_PER_THREAD; ++m)
        if (base + m < nb) {
            const unsigned int v = mask[base + m];
            s = add2(s, make_int2(v != 0, __popc(v)));
        }
    return s;
}

// exclusive scan over the block's threads; every thread gets the total
__device__ int2 hb_exscan(int2 v, int2 &total) {
    __shared__ int2 wt[HB_THREADS / 32 + 1];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int2 inc = v;
    for (int d = 1; d < 32; d <<= 1) {
        const int2 o = make_int2(__shfl_up_sync(0xffffffffu, inc.x, d), __shfl_up_sync(0xffffffffu, inc.y, d));
        if (lane >= d) inc = add2(inc, o);
    }
    __syncthreads();  // the totals of a previous call are read
    if (lane == 31) wt[wid] = inc;
    __syncthreads();
    if (threadIdx.x == 0) {
        int2 run = make_int2(0, 0);
        for (int q = 0; q < HB_THREADS / 32; ++q) {
            const int2 t = wt[q];
            wt[q] = run;
            run = add2(run, t);
        }
        wt[HB_THREADS / 32] = run;
    }
    __syncthreads();
    total = wt[HB_THREADS / 32];
    return make_int2(wt[wid].x + inc.x - v.x, wt[wid].y + inc.y - v.y);
}

__global__ void __launch_bounds__(HB_THREADS) k_hb_tiles(const unsigned int *__restrict__ mask, long nb,
                                                         int2 *__restrict__ tiles) {
    int2 total;
    hb_exscan(hb_counts(mask, (long)blockIdx.x * HB_TILE + threadIdx.x * HB_PER_THREAD, nb), total);
    if (threadIdx.x == 0) tiles[blockIdx.x] = total;
}

// one block: exclusive scan of the tile totals in place; tiles[ntiles] = total
__global__ void __launch_bounds__(HB_THREADS) k_hb_scan(int2 *__restrict__ tiles, int ntiles) {
    int2 carry = make_int2(0, 0);
    for (int b0 = 0; b0 < ntiles; b0 += HB_THREADS) {
        const int b = b0 + threadIdx.x;
        int2 total;
        const int2 ex = hb_exscan(b < ntiles ? tiles[b] : make_int2(0, 0), total);
        if (b < ntiles) tiles[b] = add2(carry, ex);
        carry = add2(carry, total);
    }
    if (threadIdx.x == 0) tiles[ntiles] = carry;
}

// coarse row of every dense block (-1: empty), and per coarse row its block
// and its first member's place
__global__ void __launch_bounds__(HB_THREADS)
    k_hb_number(const unsigned int *__restrict__ mask, long nb, const int2 *__restrict__ tiles, int ntiles,
                int *__restrict__ index, int *__restrict__ ccell, int *__restrict__ mstart) {
    const long base = (long)blockIdx.x * HB_TILE + threadIdx.x * HB_PER_THREAD;
    int2 total;
    int2 at = add2(tiles[blockIdx.x], hb_exscan(hb_counts(mask, base, nb), total));
#pragma unroll
    for (int m = 0; m < HB_PER_THREAD; ++m) {
        if (base + m >= nb) break;
        const unsigned int v = mask[base + m];
        index[base + m] = v ? at.x : -1;
        if (v) {
            ccell[at.x] = (int)(base + m);
            mstart[at.x] = at.y;
        }
        at = add2(at, make_int2(v != 0, __popc(v)));
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) mstart[tiles[ntiles].x] = tiles[ntiles].y;
}

__global__ void k_hb_members(const int *__restrict__ cell, int n, CellBox f, const unsigned int *__restrict__ mask,
                             const int *__restrict__ index, const int *__restrict__ mstart, int *__restrict__ pos,
                             int *__restrict__ members) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        int oct;
        const int b = block_of(cell[r], f, oct), I = index[b];
        const int rank = __popc(mask[b] & ((1u << oct) - 1u));
        pos[r] = 8 * I + rank;
        members[mstart[I] + rank] = r;
    }
}

// directions W, E, S, N, B, T
__global__ void k_hb_nbr(const int *__restrict__ ccell, int nc, int npad, CellBox g, const int *__restrict__ index,
                         int *__restrict__ nbr) {
    for (int I = blockIdx.x * blockDim.x + threadIdx.x; I < npad; I += gridDim.x * blockDim.x) {
        int v[6] = {-1, -1, -1, -1, -1, -1};
        if (I < nc) {
            const int c = ccell[I], k = c % g.nz, t = c / g.nz, j = t % g.ny, i = t / g.ny, si = g.ny * g.nz;
            if (i > 0) v[0] = index[c - si];
            if (i + 1 < g.nx) v[1] = index[c + si];
            if (j > 0) v[2] = index[c - g.nz];
            if (j + 1 < g.ny) v[3] = index[c + g.nz];
            if (k > 0) v[4] = index[c - 1];
            if (k + 1 < g.nz) v[5] = index[c + 1];
        }
#pragma unroll
        for (int d = 0; d < 6; ++d) nbr[(size_t)d * npad + I] = v[d];
    }
}

// The six columns of a row in 8 bytes (packed_columns).  *far is set when one
// does not fit; the table is not used then.
__global__ void k_pack_columns(const int *__restrict__ nbr, int npad, ushort4 *__restrict__ pack, int *far) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < npad; r += gridDim.x * blockDim.x) {
        int d[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const int c = nbr[(size_t)k * npad + r];
            d[k] = c < 0 ? 0 : (k & 1) ? c - r : r - c;
        }
        if (d[0] < 0 || d[0] > 0xffff || d[1] < 0 || d[1] > 0xffff || d[2] < 0 || d[2] > 0x7fff || d[3] < 0 ||
            d[3] > 0x7fff || d[4] < 0 || d[4] > 1 || d[5] < 0 || d[5] > 1)
            *far = 1;
        pack[r] = make_ushort4((unsigned short)d[0], (unsigned short)d[1], (unsigned short)(d[2] | d[4] << 15),
                               (unsigned short)(d[3] | d[5] << 15));
    }
}

static int hb_grid(long n) { return (int)std::max(1L, std::min((n + 255) / 256, (long)device_sm_count() * 16)); }

void build_hierarchy(DevSys &S, cudaStream_t st) {
    std::unique_ptr<MGHost> H(new MGHost());
    CellBox box = {S.d0, S.cell_ny, S.cell_nz};
    DBuf<int> cells[2];  // the row -> cell tables of the level being aggregated and of the new one
    const int *cell = S.cell.p;
    int nf = S.n, flip = 0;
    DBuf<int> dfar;
    int far = 0;
    if (nf >= kPackRows) {
        H->pack.alloc((size_t)S.npad, st);
        dfar.alloc_zero(1, st);
        count_launches(1);
        k_pack_columns<<<hb_grid(S.npad), 256, 0, st>>>(S.nbr.p, S.npad, H->pack.p, dfar.p);
        NS3D_CUDA_CHECK(cudaMemcpyAsync(&far, dfar.p, sizeof far, cudaMemcpyDeviceToHost, st));
    }
    while (H->nlev < MG_MAX && nf > kMGCoarsest) {
        const CellBox cbox = box.coarse();
        const long nb = cbox.cells();
        const int ntiles = (int)((nb + HB_TILE - 1) / HB_TILE);
        DBuf<unsigned int> mask;
        DBuf<int> index;
        DBuf<int2> tiles;
        mask.alloc_zero((size_t)nb, st);
        index.alloc((size_t)nb, st);
        tiles.alloc((size_t)ntiles + 1, st);
        count_launches(3);
        k_hb_mark<<<hb_grid(nf), 256, 0, st>>>(cell, nf, box, mask.p);
        k_hb_tiles<<<ntiles, HB_THREADS, 0, st>>>(mask.p, nb, tiles.p);
        k_hb_scan<<<1, HB_THREADS, 0, st>>>(tiles.p, ntiles);
        int2 total;
        NS3D_CUDA_CHECK(cudaMemcpyAsync(&total, tiles.p + ntiles, sizeof total, cudaMemcpyDeviceToHost, st));
        NS3D_CUDA_CHECK(cudaStreamSynchronize(st));
        if (far) {  // (copied before the totals)
            H->pack.release();
            far = 0;
        }
        const int nc = total.x;
        MGHostLevel &L = H->lev[++H->nlev];
        L.n = nc;
        L.npad = (nc + 255) / 256 * 256;
        L.nbr.alloc((size_t)6 * L.npad, st);
        L.pos.alloc((size_t)nf, st);
        L.mstart.alloc((size_t)nc + 1, st);
        L.members.alloc((size_t)nf, st);
        DBuf<int> &ccell = cells[flip];
        ccell.alloc((size_t)nc, st);
        count_launches(3);
        k_hb_number<<<ntiles, HB_THREADS, 0, st>>>(mask.p, nb, tiles.p, ntiles, index.p, ccell.p, L.mstart.p);
        k_hb_members<<<hb_grid(nf), 256, 0, st>>>(cell, nf, box, mask.p, index.p, L.mstart.p, L.pos.p, L.members.p);
        k_hb_nbr<<<hb_grid(L.npad), 256, 0, st>>>(ccell.p, nc, L.npad, cbox, index.p, L.nbr.p);
        L.coef.alloc_zero((size_t)7 * L.npad, st);
        L.t8.alloc_zero((size_t)8 * L.npad, st);
        for (DBuf<float> *b : {&L.invdiag, &L.x, &L.b, &L.t, &L.xo}) b->alloc_zero((size_t)L.npad, st);
        cell = ccell.p;
        box = cbox;
        nf = nc;
        flip ^= 1;
    }
    NS3D_CUDA_CHECK(cudaGetLastError());
    S.mg = std::move(H);
}

}  // namespace ns3d
