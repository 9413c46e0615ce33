// Differentiable mode, short-range kernels: the brick of grid points a block
// owns and the receptor atoms it can reach.
#pragma once
#include "agb_device.cuh"
#include "diff.h"

namespace agb {

constexpr int DF_WARPS = DF_THREADS / 32;
constexpr int DF_MAXSEG = 64;  // rows of cells (y, z) around a brick; at most 7 x 7 are in reach

struct Brick {
    int ix0, iy0, iz0;
    int ix, iy, iz;
    int conf;
    bool valid;
    long long lin;
};

// blockIdx.z runs over (z bricks) x (conformers).  A warp's lanes are a 4x4x2
// corner of the brick: its box grown by 8 A is 8% smaller than that of an
// 8x4x1 slice, so fewer of a warp's candidates lie beyond the cutoff of a lane.
__device__ __forceinline__ Brick brick_of(const DiffArgs &a)
{
    static_assert(DF_BRICK_X == 8 && DF_BRICK_Y == 8 && DF_BRICK_Z == 4, "lane layout below");
    Brick b;
    const int nbz = (a.n1z + DF_BRICK_Z - 1) / DF_BRICK_Z;
    b.conf = blockIdx.z / nbz;
    b.ix0 = blockIdx.x * DF_BRICK_X;
    b.iy0 = blockIdx.y * DF_BRICK_Y;
    b.iz0 = (blockIdx.z % nbz) * DF_BRICK_Z;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    b.ix = b.ix0 + (lane & 3) + 4 * (w & 1);
    b.iy = b.iy0 + ((lane >> 2) & 3) + 4 * ((w >> 1) & 1);
    b.iz = b.iz0 + (lane >> 4) + 2 * (w >> 2);
    b.valid = b.ix < a.n1x && b.iy < a.n1y && b.iz < a.n1z;
    b.lin = b.valid ? (long long)b.ix + (long long)a.n1x * (b.iy + (long long)a.n1y * b.iz) : 0;
    return b;
}

// The candidate atoms of a brick: one run of cell_atoms per row of cells.
struct BrickSegs {
    int start[DF_MAXSEG], off[DF_MAXSEG + 1];
    int n, total;
};

// Per row (y, z) of cells around the brick, the run of x cells within
// DF_RADIUS of the brick's box (cells of a row are consecutive in the cell
// list), with the running offsets of their atoms.  All threads call it; it
// ends with a barrier.
__device__ __forceinline__ void brick_segments(const DiffArgs &a, const ConfView &v, const Brick &bk, BrickSegs &sg)
{
    const int ix1 = min(bk.ix0 + DF_BRICK_X - 1, a.n1x - 1), iy1 = min(bk.iy0 + DF_BRICK_Y - 1, a.n1y - 1),
              iz1 = min(bk.iz0 + DF_BRICK_Z - 1, a.n1z - 1);
    const double lo[3] = {(bk.ix0 - a.nex) * a.spacing, (bk.iy0 - a.ney) * a.spacing, (bk.iz0 - a.nez) * a.spacing};
    const double hi[3] = {(ix1 - a.nex) * a.spacing, (iy1 - a.ney) * a.spacing, (iz1 - a.nez) * a.spacing};
    const int nc[3] = {a.ncx, a.ncy, a.ncz};
    int c0[3], c1[3];
    bool empty = false;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        c0[i] = max((int)floor((lo[i] - DF_RADIUS - a.cell0[i]) / a.cell_size), 0);
        c1[i] = min((int)floor((hi[i] + DF_RADIUS - a.cell0[i]) / a.cell_size), nc[i] - 1);
        if (c0[i] > c1[i]) empty = true;
    }
    // squared gap between cell c of axis i and the brick's box
    auto gap2 = [&](int i, int c) {
        const double blo = a.cell0[i] + c * a.cell_size, bhi = blo + a.cell_size;
        const double g = fmax(fmax(blo - hi[i], lo[i] - bhi), 0.0);
        return g * g;
    };
    const int wy = c1[1] - c0[1] + 1, wz = c1[2] - c0[2] + 1;
    const int n = empty ? 0 : min(wy * wz, DF_MAXSEG);
    for (int k = threadIdx.x; k < n; k += DF_THREADS) {
        const int cy = c0[1] + k % wy, cz = c0[2] + k / wy;
        const double left = DF_RADIUS * DF_RADIUS - gap2(1, cy) - gap2(2, cz);
        int x0 = c0[0], x1 = c1[0];
        while (x0 <= x1 && gap2(0, x0) > left) x0++;
        while (x1 >= x0 && gap2(0, x1) > left) x1--;
        const int row = a.ncx * (cy + a.ncy * cz);
        const int s = x0 <= x1 ? v.cell_start[row + x0] : 0, e = x0 <= x1 ? v.cell_start[row + x1 + 1] : 0;
        sg.start[k] = s;
        sg.off[k] = e - s;
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // exclusive scan of the run lengths, two per lane
        static_assert(DF_MAXSEG == 64, "two runs per lane");
        const int l = threadIdx.x;
        const int u = 2 * l < n ? sg.off[2 * l] : 0, w = 2 * l + 1 < n ? sg.off[2 * l + 1] : 0;
        int incl = u + w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (l >= o) incl += t;
        }
        __syncwarp();
        sg.off[2 * l] = incl - u - w;
        sg.off[2 * l + 1] = incl - w;
        if (l == 31) {
            sg.off[DF_MAXSEG] = incl;
            sg.total = incl;
            sg.n = n;
        }
    }
    __syncthreads();
}

// File index of candidate k (< total) of the brick.
__device__ __forceinline__ int brick_atom(const ConfView &v, const BrickSegs &sg, int k)
{
    int lo = 0, hi = sg.n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (sg.off[mid] <= k) lo = mid;
        else hi = mid - 1;
    }
    return v.cell_atoms[sg.start[lo] + (k - sg.off[lo])];
}

// Covalent map of a point, main.cpp:2866-2879.
template <class R> __device__ __forceinline__ R covalent_value(const DiffArgs &a, R px, R py, R pz)
{
    const R d0 = (R)a.cov_pos[0] - px, d1 = (R)a.cov_pos[1] - py, d2 = (R)a.cov_pos[2] - pz;
    R rc = dfm::sqrt_(d0 * d0 + d1 * d1 + d2 * d2) / (R)a.cov_half_width;
    if (rc < (R)dfm::DF_TINY) rc = (R)dfm::DF_TINY;
    return (R)a.cov_barrier * ((R)1 - dfm::exp_((R)-0.69314718055994531 * rc * rc));
}

inline dim3 brick_grid(const DiffArgs &a)
{
    return dim3((unsigned)((a.n1x + DF_BRICK_X - 1) / DF_BRICK_X), (unsigned)((a.n1y + DF_BRICK_Y - 1) / DF_BRICK_Y),
                (unsigned)((a.n1z + DF_BRICK_Z - 1) / DF_BRICK_Z * a.n_conf));
}

}  // namespace agb
