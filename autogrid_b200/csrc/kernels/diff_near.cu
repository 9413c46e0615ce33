// Differentiable mode, short-range maps, FP64 twin: LOOP 2 of
// main.cpp:3017-3431 with linearly interpolated tables and the 8 A switch
// (kernels/diff.h), and its adjoint, with the per-pair code of diff_pair.cuh.
// (The FP32 kernels are in diff_rows.cu.)
//   k_closest_h         closest DS/D1 atom of each point, FP64, the reference's
//                       scan (main.cpp:2986-3015: file order, strict <)
//   k_near_lin          forward: a brick of 8x8x4 points per block, one point per
//                       thread; candidate atoms of the cells within 8.05 A of the
//                       brick staged through shared memory; records for each
//                       H-bond min/max slot the atoms attaining the min and max
//   k_near_lin_adj      adjoint: same bricks and staging, pair terms recomputed;
//                       per candidate the 32 points of a warp are reduced with
//                       shuffles and one lane adds the atom's gradient (FP64
//                       atomics); the Hramp gradient on the closest hydrogen's
//                       bond vector is added per point.
#include "agb_device.cuh"
#include "diff.h"
#include "diff_pair.cuh"

#include "diff_brick.cuh"

namespace agb {

using namespace dfm;

namespace {

struct NearLinSmem {
    Atom<double> at[DF_STAGE];
    BrickSegs sg;
    unsigned short wl[DF_WARPS][DF_STAGE];  // per warp: staged slots near its points
    double wbox[DF_WARPS][6];               // per warp: its points' box (lo xyz, hi xyz), A
};

// This warp's points as a box (lanes outside the grid do not count), kept in
// shared memory for warp_candidates.
__device__ __forceinline__ void warp_box(const Brick &bk, double px, double py, double pz, NearLinSmem &sm)
{
    const double big = 3.0e38f;
    double lo[3] = {bk.valid ? px : big, bk.valid ? py : big, bk.valid ? pz : big};
    double hi[3] = {bk.valid ? px : -big, bk.valid ? py : -big, bk.valid ? pz : -big};
#pragma unroll
    for (int d = 0; d < 3; d++)
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const double a = __shfl_xor_sync(0xffffffffu, lo[d], o), b = __shfl_xor_sync(0xffffffffu, hi[d], o);
            lo[d] = a < lo[d] ? a : lo[d];
            hi[d] = b > hi[d] ? b : hi[d];
        }
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0)
        for (int d = 0; d < 3; d++) {
            sm.wbox[w][d] = lo[d];
            sm.wbox[w][3 + d] = hi[d];
        }
    __syncwarp();
}

// Slots j < n of the staged chunk whose atom lies within the cutoff + 0.01 A
// of this warp's box, in staged order (called by all 32 lanes).  Every pair a
// lane of the warp evaluates (r^2 <= 64 in geom) is on the list, so the pairs
// and their order are those of the whole chunk.
__device__ __forceinline__ int warp_candidates(NearLinSmem &sm, int n)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const double *bx = sm.wbox[w];
    const double lim2 = (AG_NBC + 0.01) * (AG_NBC + 0.01);
    int cnt = 0;
    for (int j0 = 0; j0 < n; j0 += 32) {
        const int j = j0 + lane;
        bool keep = false;
        if (j < n) {
            const Atom<double> &at = sm.at[j];
            double e[3];
            const double c[3] = {at.x, at.y, at.z};
#pragma unroll
            for (int d = 0; d < 3; d++) {
                const double u = bx[d] - c[d], v = c[d] - bx[3 + d];
                const double m = u > v ? u : v;
                e[d] = m > 0.0 ? m : 0.0;
            }
            keep = e[0] * e[0] + e[1] * e[1] + e[2] * e[2] <= lim2;
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) sm.wl[w][cnt + __popc(m & ((1u << lane) - 1u))] = (unsigned short)j;
        cnt += __popc(m);
    }
    __syncwarp();
    return cnt;
}

// Stage candidates [c0, c0 + DF_STAGE) of the brick into shared memory.
__device__ void stage_chunk(const DiffArgs &a, const ConfView &v, NearLinSmem &sm, int c0)
{
    const int k = c0 + threadIdx.x;
    if (threadIdx.x < DF_STAGE && k < sm.sg.total) {
        const int ia = brick_atom(v, sm.sg, k);
        Atom<double> &t = sm.at[threadIdx.x];
        t.x = v.x[ia]; t.y = v.y[ia]; t.z = v.z[ia];
        t.q = v.q[ia]; t.vol = a.vol[ia]; t.solpar = a.solpar[ia];
        for (int i = 0; i < 3; i++) {
            t.rv[i] = v.rv[3 * ia + i];
            t.rv2[i] = v.rv2[3 * ia + i];
        }
        t.meta = a.meta[ia];
        t.idx = ia;
    }
}

// MS slots and MM min/max registers per point.
template <int MS, int MM, int MINB>
__global__ void __launch_bounds__(DF_THREADS, MINB)
k_near_lin(DiffArgs a, const R2<double> *__restrict__ vdw, const R2<double> *__restrict__ sol, double *__restrict__ maps,
           const int *__restrict__ chs, int *__restrict__ mmarg)
{
    constexpr int MMA = MM > 0 ? MM : 1;
    __shared__ NearLinSmem sm;
    const Brick bk = brick_of(a);
    const ConfView v = conf_view(a, DiffGrads{}, bk.conf);
    chs += bk.conf * a.P;
    maps += (long long)bk.conf * a.n_maps_out * a.P;
    mmarg += 2LL * bk.conf * a.n_mm * a.P;
    const double px = (bk.ix - a.nex) * a.spacing, py = (bk.iy - a.ney) * a.spacing, pz = (bk.iz - a.nez) * a.spacing;
    const int ch = bk.valid ? chs[bk.lin] : -1;
    double rvh[3] = {0, 0, 0};
    if (ch >= 0)
        for (int i = 0; i < 3; i++) rvh[i] = v.rv[3 * ch + i];
    double E[MS], hmin[MMA], hmax[MMA];
    int amin[MMA], amax[MMA];
#pragma unroll
    for (int s = 0; s < MS; s++) E[s] = 0;
#pragma unroll
    for (int s = 0; s < MMA; s++) { hmin[s] = 999999.; hmax[s] = -999999.; amin[s] = -1; amax[s] = -1; }

    brick_segments(a, v, bk, sm.sg);
    warp_box(bk, px, py, pz, sm);
    for (int c0 = 0; c0 < sm.sg.total; c0 += DF_STAGE) {
        __syncthreads();
        stage_chunk(a, v, sm, c0);
        __syncthreads();
        const int n = min(DF_STAGE, sm.sg.total - c0);
        const int cnt = warp_candidates(sm, n);
        if (!bk.valid) continue;
        const unsigned short *wl = sm.wl[threadIdx.x >> 5];
        for (int k = 0; k < cnt; k++) {
            const Atom<double> at = sm.at[wl[k]];
            Geom<double> g;
            if (!geom(a.need_sol ? sol : nullptr, at, px, py, pz, g)) continue;
            Ang<double> an;
            angular((at.meta >> DM_HB_SHIFT) & 7, (at.meta >> DM_REXP_SHIFT) & 7, (at.meta & DM_DIS) != 0,
                    ch >= 0 && at.idx != ch, g.dn, at.rv, at.rv2, rvh, an);
            pair_fwd<double, MS, MM>(a, vdw, g, at, an, E, hmin, hmax, amin, amax);
        }
    }
    if (!bk.valid) return;
#pragma unroll
    for (int s = 0; s < MS; s++) {
        if (s >= a.n_slots) break;
        double v = E[s];
        if (s < MM && s < a.n_mm) {
            // H-bond finaliser, main.cpp:3420-3431
            if (amin[s] >= 0) v += hmin[s] + (hmax[s] > 0.0 ? hmax[s] : 0.0);
            mmarg[(2LL * s) * a.P + bk.lin] = amin[s];
            mmarg[(2LL * s + 1) * a.P + bk.lin] = hmax[s] > 0.0 ? amax[s] : -1;
        }
        if (a.slot_kind[s] == DK_COV) v += covalent_value<double>(a, px, py, pz);
        maps[(long long)a.slot_map[s] * a.P + bk.lin] = v;
    }
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <int MS, int MM, int MINB>
__global__ void __launch_bounds__(DF_THREADS, MINB)
k_near_lin_adj(DiffArgs a, const R2<double> *__restrict__ vdw, const R2<double> *__restrict__ sol,
               const double *__restrict__ g_maps, const int *__restrict__ chs, const int *__restrict__ mmarg,
               DiffGrads gr_all)
{
    constexpr int MMA = MM > 0 ? MM : 1;
    __shared__ NearLinSmem sm;
    const Brick bk = brick_of(a);
    const ConfView v = conf_view(a, gr_all, bk.conf);
    const DiffGrads gr = v.g;
    chs += bk.conf * a.P;
    g_maps += (long long)bk.conf * a.n_maps_out * a.P;
    mmarg += 2LL * bk.conf * a.n_mm * a.P;
    const double px = (bk.ix - a.nex) * a.spacing, py = (bk.iy - a.ney) * a.spacing, pz = (bk.iz - a.nez) * a.spacing;
    const int ch = bk.valid ? chs[bk.lin] : -1;
    double rvh[3] = {0, 0, 0}, g_rvh[3] = {0, 0, 0};
    if (ch >= 0)
        for (int i = 0; i < 3; i++) rvh[i] = v.rv[3 * ch + i];
    double gs[MS];
    int amin[MMA], amax[MMA];
#pragma unroll
    for (int s = 0; s < MS; s++)
        gs[s] = (bk.valid && s < a.n_slots) ? g_maps[(long long)a.slot_map[s] * a.P + bk.lin] : 0.0;
#pragma unroll
    for (int s = 0; s < MMA; s++) {
        const bool has = bk.valid && s < MM && s < a.n_mm;
        amin[s] = has ? mmarg[(2LL * s) * a.P + bk.lin] : -1;
        amax[s] = has ? mmarg[(2LL * s + 1) * a.P + bk.lin] : -1;
    }
    const int lane = threadIdx.x & 31;

    brick_segments(a, v, bk, sm.sg);
    warp_box(bk, px, py, pz, sm);
    for (int c0 = 0; c0 < sm.sg.total; c0 += DF_STAGE) {
        __syncthreads();
        stage_chunk(a, v, sm, c0);
        __syncthreads();
        const int n = min(DF_STAGE, sm.sg.total - c0);
        const int cnt = warp_candidates(sm, n);
        const unsigned short *wl = sm.wl[threadIdx.x >> 5];
        for (int k = 0; k < cnt; k++) {
            const Atom<double> at = sm.at[wl[k]];
            Geom<double> g;
            const bool in = bk.valid && geom(a.need_sol ? sol : nullptr, at, px, py, pz, g);
            if (!__any_sync(0xffffffffu, in)) continue;
            const int hb = (at.meta >> DM_HB_SHIFT) & 7;
            const bool dis = (at.meta & DM_DIS) != 0;
            double g_d[3] = {0, 0, 0}, g_rv[3] = {0, 0, 0}, g_rv2[3] = {0, 0, 0}, G_q = 0;
            if (in) {
                Ang<double> an;
                angular(hb, (at.meta >> DM_REXP_SHIFT) & 7, dis, ch >= 0 && at.idx != ch, g.dn, at.rv, at.rv2, rvh, an);
                double G_x = 0, G_racc = 0, G_rdon = 0, G_H = 0;
                pair_bwd<double, MS, MM>(a, vdw, g, at, an, gs, amin, amax, G_x, G_racc, G_rdon, G_H, G_q);
                double g_dn[3] = {0, 0, 0};
                angular_bwd(hb, dis, an, G_racc, G_rdon, G_H, g.dn, at.rv, at.rv2, rvh, g_dn, g_rv, g_rv2, g_rvh);
                geom_bwd(g, G_x, g_dn, g_d);
            }
            // the candidate is the same for the whole warp: reduce, one lane adds
            // G_q comes from desolvation terms only
            const double sx = warp_sum(g_d[0]), sy = warp_sum(g_d[1]), sz = warp_sum(g_d[2]);
            const double sq = a.need_sol ? warp_sum(G_q) : 0.0;
            double sr[3] = {0, 0, 0}, sr2[3] = {0, 0, 0};
            const bool has_rv = hb == 2 || hb == 4 || hb == 5;
            const bool has_rv2 = hb == 5 && !dis;
            if (has_rv)
                for (int i = 0; i < 3; i++) sr[i] = warp_sum(g_rv[i]);
            if (has_rv2)
                for (int i = 0; i < 3; i++) sr2[i] = warp_sum(g_rv2[i]);
            if (lane == 0) {
                const long long ia = at.idx;
                atomicAdd(gr.xyz + 3 * ia, sx);
                atomicAdd(gr.xyz + 3 * ia + 1, sy);
                atomicAdd(gr.xyz + 3 * ia + 2, sz);
                if (sq != 0.0) atomicAdd(gr.q + ia, sq);
                if (has_rv)
                    for (int i = 0; i < 3; i++) atomicAdd(gr.rv + 3 * ia + i, sr[i]);
                if (has_rv2)
                    for (int i = 0; i < 3; i++) atomicAdd(gr.rv2 + 3 * ia + i, sr2[i]);
            }
        }
    }
    if (ch >= 0 && (g_rvh[0] != 0.0 || g_rvh[1] != 0.0 || g_rvh[2] != 0.0))
        for (int i = 0; i < 3; i++) atomicAdd(gr.rv + 3LL * ch + i, g_rvh[i]);
}

constexpr int CH_THREADS = 256;

__global__ void __launch_bounds__(CH_THREADS) k_closest_h(DiffArgs a, int *__restrict__ ch)
{
    __shared__ double sx[CH_THREADS], sy[CH_THREADS], sz[CH_THREADS];
    __shared__ int sidx[CH_THREADS];
    const ConfView v = conf_view(a, DiffGrads{}, blockIdx.y);
    ch += blockIdx.y * a.P;
    const long long lin = (long long)blockIdx.x * CH_THREADS + threadIdx.x;
    const bool valid = lin < a.P;
    const long long l = valid ? lin : 0;
    const int ix = (int)(l % a.n1x), iy = (int)((l / a.n1x) % a.n1y), iz = (int)(l / ((long long)a.n1x * a.n1y));
    const double cx = (double)(ix - a.nex) * a.spacing, cy = (double)(iy - a.ney) * a.spacing,
                 cz = (double)(iz - a.nez) * a.spacing;
    // The reference keeps the first H atom in file order with the strictly
    // smallest r = sqrt(d0^2 + d1^2 + d2^2).  sqrt is monotonic, so only a
    // strictly smaller square can give a strictly smaller r; when the squares
    // differ by more than 2^-48 relative, the correctly rounded roots differ
    // too, and only closer squares need the roots themselves compared.
    double best2 = 999999. * 999999.;  // rmin = 999999, exactly
    int best = -1;
    for (int h0 = 0; h0 < a.n_h; h0 += CH_THREADS) {
        const int nh = min(CH_THREADS, a.n_h - h0);
        __syncthreads();
        if (threadIdx.x < nh) {
            const int ia = a.h_index[h0 + threadIdx.x];
            sx[threadIdx.x] = v.x[ia]; sy[threadIdx.x] = v.y[ia]; sz[threadIdx.x] = v.z[ia];
            sidx[threadIdx.x] = ia;
        }
        __syncthreads();
        for (int j = 0; j < nh; j++) {
            const double d0 = __dsub_rn(sx[j], cx), d1 = __dsub_rn(sy[j], cy), d2 = __dsub_rn(sz[j], cz);
            const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2));
            if (r2 < best2 &&
                (best2 - r2 > best2 * 3.552713678800501e-15 /* 2^-48 */ || __dsqrt_rn(r2) < __dsqrt_rn(best2))) {
                best2 = r2;
                best = sidx[j];
            }
        }
    }
    if (valid) ch[lin] = best;
}

}  // namespace

cudaError_t launch_closest_h(const DiffArgs &a, int *ch, cudaStream_t s)
{
    if (a.P == 0) return cudaSuccess;
    k_closest_h<<<dim3((unsigned)((a.P + CH_THREADS - 1) / CH_THREADS), (unsigned)a.n_conf), CH_THREADS, 0, s>>>(a, ch);
    return cudaGetLastError();
}

// The kernels are bound by the latency of the pair's FP64 operations at few
// warps per SM.  Up to 8 slots with 4 min/max fit 128 registers with few
// spills, for 2 blocks per SM (1,000 atoms x 33^3 points, 8 maps: forward
// 300 -> 267 us, adjoint 457 -> 397; one block 1.07 ms for the whole call
// against 0.99); with 16 slots the spills cost more than the second block
// gives (16 maps: 1.96 ms against 1.70 with one block).
static bool near_lin_small(const DiffArgs &a) { return a.n_slots <= 8 && a.n_mm <= 4; }

cudaError_t launch_near_lin(const DiffArgs &a, const void *vdw, const void *sol, double *maps, const int *ch, int *mmarg,
                            cudaStream_t s)
{
    if (a.P == 0 || a.n_slots == 0) return cudaSuccess;
    const auto kernel = near_lin_small(a) ? k_near_lin<8, 4, 2> : k_near_lin<DF_MAXS, DF_MAXMM, 1>;
    kernel<<<brick_grid(a), DF_THREADS, 0, s>>>(a, (const R2<double> *)vdw, (const R2<double> *)sol, maps, ch, mmarg);
    return cudaGetLastError();
}

cudaError_t launch_near_lin_adj(const DiffArgs &a, const void *vdw, const void *sol, const double *g_maps, const int *ch,
                                const int *mmarg, DiffGrads g, cudaStream_t s)
{
    if (a.P == 0 || a.n_slots == 0) return cudaSuccess;
    const auto kernel = near_lin_small(a) ? k_near_lin_adj<8, 4, 2> : k_near_lin_adj<DF_MAXS, DF_MAXMM, 1>;
    kernel<<<brick_grid(a), DF_THREADS, 0, s>>>(a, (const R2<double> *)vdw, (const R2<double> *)sol, g_maps, ch, mmarg, g);
    return cudaGetLastError();
}

}  // namespace agb
