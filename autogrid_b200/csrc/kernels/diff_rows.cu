// Differentiable mode, short-range maps in FP32: LOOP 2 of main.cpp:3017-3431
// with linearly interpolated tables and the 8 A switch (kernels/diff.h), and
// its adjoint.  (The FP64 twin is in diff_near.cu.)
//   k_rows       forward: a brick of 8x8x4 points per block, one point per
//                thread; candidate atoms of the cells within 8.05 A staged
//                through shared memory; records for each H-bond min/max slot
//                the atoms attaining the min and max
//   k_rows_adj   adjoint: same bricks and staging, pair terms recomputed; per
//                candidate the 32 points of a warp are summed by shuffles and
//                the sums added to the atom's gradient (FP64 atomics); the
//                Hramp gradient on the closest hydrogen is added per point.
//
// Table rows.  Row (type, bin) of row_v and row_d holds the value and the step
// to the next bin of every slot, 8 (or 16) floats, one 32-byte load each.  The
// forward reads the value rows of the bin and the next one and subtracts (the
// steps exactly, as the tables are FP32), which keeps its tables at half the
// size in L1; candidates are staged in the order of their types for the same
// reason.  For most receptor classes every slot is the plain T = v + f d, and
// the row is 4 (8) packed multiply-adds; only classes with an H-bond action
// walk the slots one by one.  The desolvation terms of all slots factor into two sums
// per point, D1 = sum w sol vol and D2 = sum w sol (solpar + qasp |q|):
// slot s ends with sp_s D1 + vp_s D2.  In the adjoint a plain pair below the
// last bin (w = 1, dw = 0) needs the steps alone: half the bytes.
//
// What bounds it: the forward, the L1 data path of the row gathers (85% busy, at
// one wavefront per lane for a 32-byte gather that hits L1, two for a miss);
// the adjoint, issue (64%) and that path (69%).  Eight conformers of 8,000
// atoms, 101^3 points, 8 Vina maps: forward 2.8 ms, adjoint 2.8 ms; kernels that
// walked the slots of every pair one by one took 8.6 and 12.8 ms (295 and 475
// instructions per warp and candidate, now 65 and 101).  Rows in the order of
// the candidates' cells instead of their types, and step rows in the forward,
// hit L1 for 58% instead of 89%: the forward took 3.6 ms in place of 3.1.  4,000 atoms, 61^3 points,
// 8 AD4 maps: 0.39 -> 0.17 ms and 0.75 -> 0.33 ms.
#include "diff_pair.cuh"

#include "diff_brick.cuh"
#include "table_row.cuh"
#include "type_sort.cuh"
#include "warp_sums.cuh"

namespace agb {

using namespace dfm;

namespace {

__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }

template <bool ANG, bool SOL> struct RowsSmem {
    float4 pos[DF_STAGE];                       // x, y, z, meta
    float4 aux[SOL || ANG ? DF_STAGE : 1];      // vol, solpar + qasp |q|, qasp sgn(q), -
    int idx[DF_STAGE];
    float4 rv[ANG ? DF_STAGE : 1], rv2[ANG ? DF_STAGE : 1];
    union {
        unsigned short wl[DF_WARPS][DF_STAGE];  // per warp: staged slots near its points
        int tcnt[DF_WARPS][32];                 // staging by receptor type (type_sorted_place)
    };
    float wbox[DF_WARPS][6];                    // per warp: its points' box (lo xyz, hi xyz), A
    float2 sol[SOL ? AG_NEINT : 1];
    unsigned long long act[ANG ? 16 : 1];
    BrickSegs sg;
};

template <bool ANG, bool SOL>
__device__ __forceinline__ void rows_setup(const DiffArgs &a, const float2 *sol, RowsSmem<ANG, SOL> &sm)
{
    if (SOL)
        for (int i = threadIdx.x; i < AG_NEINT / 2; i += DF_THREADS) ((float4 *)sm.sol)[i] = __ldg((const float4 *)sol + i);
    if (ANG && threadIdx.x < 16) sm.act[threadIdx.x] = a.cls_act[threadIdx.x];
}

// This warp's points as a box (lanes outside the grid do not count).
template <class SM>
__device__ __forceinline__ void rows_box(const Brick &bk, float px, float py, float pz, SM &sm)
{
    float lo[3] = {bk.valid ? px : 3.0e38f, bk.valid ? py : 3.0e38f, bk.valid ? pz : 3.0e38f};
    float hi[3] = {bk.valid ? px : -3.0e38f, bk.valid ? py : -3.0e38f, bk.valid ? pz : -3.0e38f};
#pragma unroll
    for (int d = 0; d < 3; d++)
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
            hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
        }
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0)
        for (int d = 0; d < 3; d++) {
            sm.wbox[w][d] = lo[d];
            sm.wbox[w][3 + d] = hi[d];
        }
    __syncwarp();
}

// Stage candidates [c0, c0 + DF_STAGE) of the brick, ordered by receptor type
// (cell order within a type), so that the warps walk the table of one type at
// a time.  All threads call it; it ends with a barrier.
template <bool ANG, bool SOL>
__device__ __forceinline__ void rows_stage(const DiffArgs &a, const ConfView &v, RowsSmem<ANG, SOL> &sm, int c0)
{
    static_assert(DF_STAGE == DF_THREADS, "one candidate per thread");
    const int t = threadIdx.x;
    const bool in = c0 + t < sm.sg.total;
    const int ia = in ? brick_atom(v, sm.sg, c0 + t) : 0;
    const int meta = in ? a.meta[ia] : 0;
    const int j = type_sorted_place<DF_WARPS>(sm.tcnt, in ? meta & DM_TYPE_MASK : 32, in);
    if (in) {
        sm.pos[j] = make_float4((float)v.x[ia], (float)v.y[ia], (float)v.z[ia], __int_as_float(meta));
        sm.idx[j] = ia;
        if (SOL) {
            const float q = (float)v.q[ia], qasp = (float)a.solpar_q;
            sm.aux[j] = make_float4((float)a.vol[ia], (float)a.solpar[ia] + qasp * fabsf(q),
                                    q > 0.f ? qasp : (q < 0.f ? -qasp : 0.f), 0.f);
        }
        if (ANG) {
            sm.rv[j] = make_float4((float)v.rv[3 * ia], (float)v.rv[3 * ia + 1], (float)v.rv[3 * ia + 2], 0.f);
            sm.rv2[j] = make_float4((float)v.rv2[3 * ia], (float)v.rv2[3 * ia + 1], (float)v.rv2[3 * ia + 2], 0.f);
        }
    }
    __syncthreads();
}

// Slots j < n of the staged chunk whose atom lies within the cutoff + 0.01 A
// of this warp's box and is not skipped by LOOP 2 (main.cpp:3052), in staged
// order (called by all 32 lanes).
template <class SM> __device__ __forceinline__ int rows_candidates(SM &sm, int n)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const float *bx = sm.wbox[w];
    const float lim2 = (float)((AG_NBC + 0.01) * (AG_NBC + 0.01));
    int cnt = 0;
    for (int j0 = 0; j0 < n; j0 += 32) {
        const int j = j0 + lane;
        bool keep = false;
        if (j < n) {
            const float4 A = sm.pos[j];
            const float ex = fmaxf(fmaxf(bx[0] - A.x, A.x - bx[3]), 0.f);
            const float ey = fmaxf(fmaxf(bx[1] - A.y, A.y - bx[4]), 0.f);
            const float ez = fmaxf(fmaxf(bx[2] - A.z, A.z - bx[5]), 0.f);
            keep = ex * ex + ey * ey + ez * ez <= lim2 && !(__float_as_int(A.w) & DM_SKIP);
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) sm.wl[w][cnt + __popc(m & ((1u << lane) - 1u))] = (unsigned short)j;
        cnt += __popc(m);
    }
    __syncwarp();
    return cnt;
}

// Geometry of one pair; false beyond 8 A.
struct RowGeom {
    float d[3], inv, x, fx, w;
    int b;
};
__device__ __forceinline__ bool rows_geom(const float4 &A, float px, float py, float pz, RowGeom &g)
{
    g.d[0] = A.x - px;
    g.d[1] = A.y - py;
    g.d[2] = A.z - pz;
    // r picks the table bin, where the slopes jump: its rounding is pinned, so
    // that forward and adjoint (and later builds) take the same bins
    const float r2 = __fmaf_rn(g.d[2], g.d[2], __fmaf_rn(g.d[1], g.d[1], __fmul_rn(g.d[0], g.d[0])));
    if (r2 > (float)(AG_NBC * AG_NBC)) return false;
    const float r = sqrt_markstein(fmaxf(r2, 1.0e-12f), g.inv);  // at least 1e-6 A
    g.x = r * (float)AG_A_DIV;
    g.b = min((int)g.x, AG_NEINT - 1);
    g.fx = g.x - (float)g.b;
    g.w = fminf((float)AG_NEINT - g.x, 1.f);
    return true;
}

// What slot s does for a class: 4 bits of its action word.
__device__ __forceinline__ int slot_act(unsigned long long act, int s) { return (int)(act >> (4 * s)) & 15; }

// T_H(r - 1.10) of slot s: the hydrogen row at xh = A_DIV (r - 1.10)
// (main.cpp:3309-3313), and its slope.
__device__ __forceinline__ float th_row(const DiffArgs &a, int s, float x, float &dth)
{
    dth = 0.f;
    if (a.hydrogen_type < 0 || a.hydrogen_type >= a.n_rec_types) return 0.f;
    const float xh = x - (float)(1.10 * AG_A_DIV);
    const int bh = xh <= 0.f ? 0 : min((int)xh, AG_NEINT - 1);
    const size_t o = ((size_t)a.hydrogen_type * DF_ROWS + bh) * a.row_stride + s;
    const float v = __ldg(a.row_v + o);
    if (xh <= 0.f) return v;
    dth = __ldg(a.row_d + o);
    return fmaf(xh - (float)bh, dth, v);
}

__device__ __forceinline__ float lane_of(const Row8 *r, int s) { return (s & 1) ? r[s >> 3].p[(s >> 1) & 3].y : r[s >> 3].p[(s >> 1) & 3].x; }

template <int MS, int MM, int MINB, bool ANG, bool SOL>
__global__ void __launch_bounds__(DF_THREADS, MINB)
k_rows(DiffArgs a, const float2 *__restrict__ sol, float *__restrict__ maps, const int *__restrict__ chs,
       int *__restrict__ mmarg)
{
    constexpr int MMA = MM > 0 ? MM : 1, NB = MS / 8;
    __shared__ RowsSmem<ANG, SOL> sm;
    const Brick bk = brick_of(a);
    const ConfView v = conf_view(a, DiffGrads{}, bk.conf);
    rows_setup(a, sol, sm);
    const float px = (float)((bk.ix - a.nex) * a.spacing), py = (float)((bk.iy - a.ney) * a.spacing),
                pz = (float)((bk.iz - a.nez) * a.spacing);
    int ch = -1;
    float rvh[3] = {0.f, 0.f, 0.f};
    if (ANG && bk.valid) {
        ch = chs[bk.conf * a.P + bk.lin];
        if (ch >= 0)
            for (int i = 0; i < 3; i++) rvh[i] = (float)v.rv[3 * ch + i];
    }
    float2 E[MS / 2];
    float hmin[MMA], hmax[MMA], D1 = 0.f, D2 = 0.f;
    int amin[MMA], amax[MMA];
#pragma unroll
    for (int k = 0; k < MS / 2; k++) E[k] = both(0.f);
#pragma unroll
    for (int s = 0; s < MMA; s++) { hmin[s] = 999999.f; hmax[s] = -999999.f; amin[s] = -1; amax[s] = -1; }

    brick_segments(a, v, bk, sm.sg);
    rows_box(bk, px, py, pz, sm);
    const unsigned short *wl = sm.wl[threadIdx.x >> 5];
    for (int c0 = 0; c0 < sm.sg.total; c0 += DF_STAGE) {
        if (c0) __syncthreads();
        rows_stage(a, v, sm, c0);
        const int cnt = rows_candidates(sm, min(DF_STAGE, sm.sg.total - c0));
        if (!bk.valid) continue;
        for (int k = 0; k < cnt; k++) {
            const int j = wl[k];
            const float4 A = sm.pos[j];
            RowGeom g;
            if (!rows_geom(A, px, py, pz, g)) continue;
            const int meta = __float_as_int(A.w);
            const unsigned ro = (unsigned)((meta & DM_TYPE_MASK) * DF_ROWS + g.b) * (unsigned)a.row_stride;
            Row8 rv8[NB], rd8[NB];
#pragma unroll
            for (int k8 = 0; k8 < NB; k8++)
                if (8 * k8 < a.n_slots) {
                    rv8[k8] = load_row8(a.row_v + ro + 8 * k8);
                    rd8[k8] = load_row8(a.row_v + ro + a.row_stride + 8 * k8);  // the next bin's values
                }
            if (SOL) {
                const float2 t = sm.sol[g.b];
                const float4 x = sm.aux[j];
                const float ws = g.w * fmaf(g.fx, t.y, t.x);
                D1 = fmaf(ws, x.x, D1);
                D2 = fmaf(ws, x.y, D2);
            }
#pragma unroll
            for (int k8 = 0; k8 < NB; k8++)
                if (8 * k8 < a.n_slots)
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        rd8[k8].p[i] = __fadd2_rn(rd8[k8].p[i], make_float2(-rv8[k8].p[i].x, -rv8[k8].p[i].y));
            const float2 f2 = both(g.fx), w2 = both(g.w);
            const int cls = ANG ? ((meta >> DM_HB_SHIFT) & 7) + ((meta & DM_DIS) ? 8 : 0) : 0;
            if (!ANG || ((a.cls_plain >> cls) & 1u)) {
#pragma unroll
                for (int k8 = 0; k8 < NB; k8++)
                    if (8 * k8 < a.n_slots)
#pragma unroll
                        for (int i = 0; i < 4; i++)
                            E[4 * k8 + i] = __ffma2_rn(w2, __ffma2_rn(f2, rd8[k8].p[i], rv8[k8].p[i]), E[4 * k8 + i]);
                continue;
            }
            const float4 r1 = sm.rv[j], r2 = sm.rv2[j];
            const float rv[3] = {r1.x, r1.y, r1.z}, rv2[3] = {r2.x, r2.y, r2.z};
            const float dn[3] = {g.d[0] * g.inv, g.d[1] * g.inv, g.d[2] * g.inv};
            const int ia = sm.idx[j];
            Ang<float> an;
            angular(cls & 7, (meta >> DM_REXP_SHIFT) & 7, cls > 7, ch >= 0 && ia != ch, dn, rv, rv2, rvh, an);
            const unsigned long long act = sm.act[cls];
#pragma unroll
            for (int s = 0; s < MS; s++) {
                if (s >= a.n_slots) break;
                const float T = fmaf(g.fx, lane_of(rd8, s), lane_of(rv8, s));
                float val = g.w * T;
                const int ac = s < a.n_hb ? slot_act(act, s) : DA_PLAIN;
                if (ac != DA_PLAIN && ac != DA_NONE) {
                    const float rs = __saturatef(T * 0.01f);
                    const bool don = ac == DA_MMD || ac == DA_SUMD_DIS;
                    const float fa = don ? an.rdon : an.racc;
                    const float f = fmaf(1.f - fa, rs, fa);
                    if (ac == DA_MMA || ac == DA_MMD) {
                        if (s < MM) {  // min/max slots come first
                            val *= f;
                            if (val <= hmin[s < MM ? s : 0]) { hmin[s < MM ? s : 0] = val; amin[s < MM ? s : 0] = ia; }
                            if (val >= hmax[s < MM ? s : 0]) { hmax[s < MM ? s : 0] = val; amax[s < MM ? s : 0] = ia; }
                        }
                        continue;
                    }
                    float dth;
                    if (ac != DA_SUMA) val = g.w * th_row(a, s, g.x, dth);
                    val *= an.H * f;
                }
                if (s & 1) E[s >> 1].y += val;
                else E[s >> 1].x += val;
            }
        }
    }
    if (!bk.valid) return;
    maps += (long long)bk.conf * a.n_maps_out * a.P;
    mmarg += 2LL * bk.conf * a.n_mm * a.P;
#pragma unroll
    for (int s = 0; s < MS; s++) {
        if (s >= a.n_slots) break;
        float val = (s & 1) ? E[s >> 1].y : E[s >> 1].x;
        if (s < MM && s < a.n_mm) {
            // H-bond finaliser, main.cpp:3420-3431
            if (amin[s < MM ? s : 0] >= 0) val += hmin[s < MM ? s : 0] + fmaxf(hmax[s < MM ? s : 0], 0.f);
            mmarg[(2LL * s) * a.P + bk.lin] = amin[s < MM ? s : 0];
            mmarg[(2LL * s + 1) * a.P + bk.lin] = hmax[s < MM ? s : 0] > 0.f ? amax[s < MM ? s : 0] : -1;
        }
        if (SOL) {
            if (a.slot_kind[s] == DK_D) val += (float)a.solpar_q * D1;                                   // main.cpp:3393-3404
            else if (a.slot_desolv[s]) val += fmaf((float)a.slot_sp[s], D1, (float)a.slot_vp[s] * D2);   // :3381-3389
        }
        if (a.slot_kind[s] == DK_COV) val += covalent_value<float>(a, px, py, pz);
        maps[(long long)a.slot_map[s] * a.P + bk.lin] = val;
    }
}

// A slot of weight 0 adds nothing, also where its table entry is no number: the
// entries of such slots become 0.  Most map sets need none of it (ALL,
// DiffArgs::weigh_all; a test at run time took 8 us of the 2.13 ms step of 4,000 atoms).
template <int NB>
__device__ __forceinline__ void drop_unweighted(const float2 (&gs)[4 * NB], Row8 &r, int k8)
{
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if (gs[4 * k8 + i].x == 0.f) r.p[i].x = 0.f;
        if (gs[4 * k8 + i].y == 0.f) r.p[i].y = 0.f;
    }
}

// Adjoint of one in-range pair of a class whose slots are all plain:
// dL/d(atom position) and, with desolvation, dL/dq.
template <int NB, bool SOL, bool ALL>
__device__ __forceinline__ void plain_adjoint(const DiffArgs &a, const RowGeom &g, unsigned ro, const float2 *sol,
                                              const float4 *aux, const float2 (&gs)[4 * NB], float gD1, float gD2,
                                              float *out)
{
    const float dw = (float)AG_NEINT - g.x < 1.f ? -1.f : 0.f;
    float G_x = 0.f;
    Row8 rd8[NB];
#pragma unroll
    for (int k8 = 0; k8 < NB; k8++)
        if (8 * k8 < a.n_slots) {
            rd8[k8] = load_row8(a.row_d + ro + 8 * k8);
            if (!ALL) drop_unweighted<NB>(gs, rd8[k8], k8);
        }
    if (SOL) {
        const float2 t = sol[g.b];
        const float4 x = *aux;
        const float so = fmaf(g.fx, t.y, t.x);
        G_x = fmaf(dw, so, g.w * t.y) * fmaf(x.y, gD2, x.x * gD1);
        out[3] = g.w * so * x.z * gD2;
    }
    float2 S = both(0.f);
#pragma unroll
    for (int k8 = 0; k8 < NB; k8++)
        if (8 * k8 < a.n_slots)
#pragma unroll
            for (int i = 0; i < 4; i++) S = __ffma2_rn(gs[4 * k8 + i], rd8[k8].p[i], S);
    G_x = fmaf(g.w, S.x + S.y, G_x);
    if (dw != 0.f) {  // the last bin: the switch's own slope
        const float2 f2 = both(g.fx);
        S = both(0.f);
#pragma unroll
        for (int k8 = 0; k8 < NB; k8++)
            if (8 * k8 < a.n_slots) {
                Row8 r = load_row8(a.row_v + ro + 8 * k8);
                if (!ALL) drop_unweighted<NB>(gs, r, k8);
#pragma unroll
                for (int i = 0; i < 4; i++) S = __ffma2_rn(gs[4 * k8 + i], __ffma2_rn(f2, rd8[k8].p[i], r.p[i]), S);
            }
        G_x -= S.x + S.y;
    }
    const float gx = G_x * (float)AG_A_DIV * g.inv;
    out[0] = gx * g.d[0];
    out[1] = gx * g.d[1];
    out[2] = gx * g.d[2];
}

template <int MS, int MM, int MINB, bool ANG, bool SOL, bool ALL>
__global__ void __launch_bounds__(DF_THREADS, MINB)
k_rows_adj(DiffArgs a, const float2 *__restrict__ sol, const float *__restrict__ g_maps, const int *__restrict__ chs,
           const int *__restrict__ mmarg, DiffGrads gr_all)
{
    constexpr int MMA = MM > 0 ? MM : 1, NB = MS / 8;
    __shared__ RowsSmem<ANG, SOL> sm;
    const Brick bk = brick_of(a);
    const ConfView v = conf_view(a, gr_all, bk.conf);
    rows_setup(a, sol, sm);
    const float px = (float)((bk.ix - a.nex) * a.spacing), py = (float)((bk.iy - a.ney) * a.spacing),
                pz = (float)((bk.iz - a.nez) * a.spacing);
    int ch = -1;
    float rvh[3] = {0.f, 0.f, 0.f}, g_rvh[3] = {0.f, 0.f, 0.f};
    if (ANG && bk.valid) {
        ch = chs[bk.conf * a.P + bk.lin];
        if (ch >= 0)
            for (int i = 0; i < 3; i++) rvh[i] = (float)v.rv[3 * ch + i];
    }
    // loss weights per slot, and of the two desolvation sums
    float2 gs[MS / 2];
    float gD1 = 0.f, gD2 = 0.f;
    int amin[MMA], amax[MMA];
    g_maps += (long long)bk.conf * a.n_maps_out * a.P;
    mmarg += 2LL * bk.conf * a.n_mm * a.P;
#pragma unroll
    for (int s = 0; s < MS; s++) {
        float w = 0.f;
        if (bk.valid && s < a.n_slots) {
            w = g_maps[(long long)a.slot_map[s] * a.P + bk.lin];
            if (SOL) {
                if (a.slot_kind[s] == DK_D) gD1 = fmaf(w, (float)a.solpar_q, gD1);
                else if (a.slot_desolv[s]) {
                    gD1 = fmaf(w, (float)a.slot_sp[s], gD1);
                    gD2 = fmaf(w, (float)a.slot_vp[s], gD2);
                }
            }
            if (!ALL && a.slot_tab[s] < 0) w = 0.f;  // no pair term: the weight goes nowhere else
        }
        if (s & 1) gs[s >> 1].y = w;
        else gs[s >> 1].x = w;
    }
#pragma unroll
    for (int s = 0; s < MMA; s++) {
        const bool has = bk.valid && s < MM && s < a.n_mm;
        amin[s] = has ? mmarg[(2LL * s) * a.P + bk.lin] : -1;
        amax[s] = has ? mmarg[(2LL * s + 1) * a.P + bk.lin] : -1;
    }
    const int lane = threadIdx.x & 31;
    const DiffGrads gr = v.g;

    brick_segments(a, v, bk, sm.sg);
    rows_box(bk, px, py, pz, sm);
    const unsigned short *wl = sm.wl[threadIdx.x >> 5];
    for (int c0 = 0; c0 < sm.sg.total; c0 += DF_STAGE) {
        if (c0) __syncthreads();
        rows_stage(a, v, sm, c0);
        const int cnt = rows_candidates(sm, min(DF_STAGE, sm.sg.total - c0));
        if (!ANG) {
            // two candidates at a time: their chains overlap, and one pass of
            // shuffles sums both
            for (int k = 0; k < cnt; k += 2) {
                float out[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const int j = wl[min(k + u, cnt - 1)];
                    const float4 A = sm.pos[j];
                    RowGeom g;
                    if (!rows_geom(A, px, py, pz, g) || !bk.valid || k + u >= cnt) continue;
                    const unsigned ro = (unsigned)((__float_as_int(A.w) & DM_TYPE_MASK) * DF_ROWS + g.b) * (unsigned)a.row_stride;
                    plain_adjoint<NB, SOL, ALL>(a, g, ro, sm.sol, sm.aux + (SOL ? j : 0), gs, gD1, gD2, out + 4 * u);
                }
                const float sum = warp_sums(out, lane);
                const int n = (lane >> 2) & 3, u = lane >> 4;
                if ((lane & 3) == 0 && (SOL || n < 3) && k + u < cnt && sum != 0.f) {
                    const long long ia = sm.idx[wl[k + u]];
                    atomicAdd(n < 3 ? gr.xyz + 3 * ia + n : gr.q + ia, (double)sum);
                }
            }
            continue;
        }
        for (int k = 0; k < cnt; k++) {
            const int j = wl[k];
            const float4 A = sm.pos[j];
            RowGeom g;
            const bool in = rows_geom(A, px, py, pz, g) && bk.valid;
            if (!__any_sync(0xffffffffu, in)) continue;
            const int meta = __float_as_int(A.w), ia = sm.idx[j];
            const int cls = ANG ? ((meta >> DM_HB_SHIFT) & 7) + ((meta & DM_DIS) ? 8 : 0) : 0;
            const bool plain = !ANG || ((a.cls_plain >> cls) & 1u);
            float out[4] = {0.f, 0.f, 0.f, 0.f};
            float g_rv[3] = {0.f, 0.f, 0.f}, g_rv2[3] = {0.f, 0.f, 0.f};
            const unsigned ro = (unsigned)((meta & DM_TYPE_MASK) * DF_ROWS + g.b) * (unsigned)a.row_stride;
            if (in) {
                if (plain) {
                    plain_adjoint<NB, SOL, ALL>(a, g, ro, sm.sol, sm.aux + (SOL ? j : 0), gs, gD1, gD2, out);
                } else {
                    const float dw = (float)AG_NEINT - g.x < 1.f ? -1.f : 0.f;
                    const float dn[3] = {g.d[0] * g.inv, g.d[1] * g.inv, g.d[2] * g.inv};
                    float G_x = 0.f;
                    Row8 rd8[NB], rv8[NB];
#pragma unroll
                    for (int k8 = 0; k8 < NB; k8++)
                        if (8 * k8 < a.n_slots) {
                            rd8[k8] = load_row8(a.row_d + ro + 8 * k8);
                            rv8[k8] = load_row8(a.row_v + ro + 8 * k8);
                            if (!ALL) {
                                drop_unweighted<NB>(gs, rd8[k8], k8);
                                drop_unweighted<NB>(gs, rv8[k8], k8);
                            }
                        }
                    if (SOL) {
                        const float2 t = sm.sol[g.b];
                        const float4 x = sm.aux[j];
                        const float so = fmaf(g.fx, t.y, t.x);
                        G_x = fmaf(dw, so, g.w * t.y) * fmaf(x.y, gD2, x.x * gD1);
                        out[3] = g.w * so * x.z * gD2;
                    }
                    const float4 r1 = sm.rv[j], r2 = sm.rv2[j];
                    const float rv[3] = {r1.x, r1.y, r1.z}, rv2[3] = {r2.x, r2.y, r2.z};
                    const int hb = cls & 7;
                    const bool dis = cls > 7;
                    Ang<float> an;
                    angular(hb, (meta >> DM_REXP_SHIFT) & 7, dis, ch >= 0 && ia != ch, dn, rv, rv2, rvh, an);
                    const unsigned long long act = sm.act[cls];
                    float G_racc = 0.f, G_rdon = 0.f, G_H = 0.f;
#pragma unroll
                    for (int s = 0; s < MS; s++) {
                        if (s >= a.n_slots) break;
                        const float d = lane_of(rd8, s), T = fmaf(g.fx, d, lane_of(rv8, s));
                        float gv = (s & 1) ? gs[s >> 1].y : gs[s >> 1].x;
                        const int ac = s < a.n_hb ? slot_act(act, s) : DA_PLAIN;
                        if (ac == DA_PLAIN || ac == DA_NONE) {
                            G_x = fmaf(gv, fmaf(dw, T, g.w * d), G_x);
                            continue;
                        }
                        if (ac == DA_MMA || ac == DA_MMD) {
                            const float n = s < MM ? (amin[s < MM ? s : 0] == ia ? 1.f : 0.f) + (amax[s < MM ? s : 0] == ia ? 1.f : 0.f) : 0.f;
                            gv *= n;
                        }
                        if (gv == 0.f) continue;
                        Term<float> t;
                        term_of(ac, T, d, an, [&](float &dth) { return th_row(a, s, g.x, dth); }, t);
                        G_x = fmaf(gv, fmaf(dw, t.v, g.w * t.dx), G_x);
                        const float gw = gv * g.w;
                        G_racc = fmaf(gw, t.dracc, G_racc);
                        G_rdon = fmaf(gw, t.drdon, G_rdon);
                        G_H = fmaf(gw, t.dH, G_H);
                    }
                    float g_dn[3] = {0.f, 0.f, 0.f};
                    angular_bwd(hb, dis, an, G_racc, G_rdon, G_H, dn, rv, rv2, rvh, g_dn, g_rv, g_rv2, g_rvh);
                    const float gx = G_x * (float)AG_A_DIV;
                    const float dot = dn[0] * g_dn[0] + dn[1] * g_dn[1] + dn[2] * g_dn[2];
#pragma unroll
                    for (int i = 0; i < 3; i++) out[i] = gx * dn[i] + (g_dn[i] - dn[i] * dot) * g.inv;
                }
            }
            // the candidate is the same for the whole warp: sum over its points
            const int hb = cls & 7;
            if (ANG && !plain && (hb == 2 || hb == 4 || hb == 5)) {
                // position, charge, rv and (ordered A2 atoms) rv2
                if (hb == 5 && cls < 8) {
                    float all[16] = {out[0], out[1], out[2], out[3], g_rv[0], g_rv[1], g_rv[2], g_rv2[0],
                                     g_rv2[1], g_rv2[2], 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                    const float sum = warp_sums(all, lane);
                    const int n = lane >> 1;
                    if ((lane & 1) == 0 && n < 10)
                        atomicAdd(n < 3 ? gr.xyz + 3LL * ia + n : n == 3 ? gr.q + ia
                                  : n < 7 ? gr.rv + 3LL * ia + (n - 4) : gr.rv2 + 3LL * ia + (n - 7), (double)sum);
                } else {
                    float all[8] = {out[0], out[1], out[2], out[3], g_rv[0], g_rv[1], g_rv[2], 0.f};
                    const float sum = warp_sums(all, lane);
                    const int n = lane >> 2;
                    if ((lane & 3) == 0 && n < 7)
                        atomicAdd(n < 3 ? gr.xyz + 3LL * ia + n : n == 3 ? gr.q + ia : gr.rv + 3LL * ia + (n - 4),
                                  (double)sum);
                }
            } else {
                const float sum = warp_sums(out, lane);
                const int n = lane >> 3;
                if ((lane & 7) == 0 && (SOL || n < 3))
                    atomicAdd(n < 3 ? gr.xyz + 3LL * ia + n : gr.q + ia, (double)sum);
            }
        }
    }
    if (ANG && ch >= 0 && (g_rvh[0] != 0.f || g_rvh[1] != 0.f || g_rvh[2] != 0.f))
        for (int i = 0; i < 3; i++) atomicAdd(gr.rv + 3LL * ch + i, (double)g_rvh[i]);
}

// The instantiation of a map set: 8 or 16 slots; no, at most 2 or at most 8
// min/max slots; directional factors or not; desolvation terms or not; the
// adjoint for map sets with weigh_all or any.
// <MS, MM, blocks per SM>: the Vina maps measured the same with 3 and 4 blocks
// and 3-5% slower with 5 and 6 (the registers spill); the 8-slot AD4 forward
// the same with 2 and 3, its adjoint 10% faster with 2 (it spills with 3).
#define ROWS_LAUNCH(KERNEL, AD4, ...)                                                                          \
    do {                                                                                                  \
        const bool small = a.n_slots <= 8;                                                                \
        if (!a.need_ang && small && !a.need_sol) KERNEL(8, 0, 4, false, false)<<<brick_grid(a), DF_THREADS, 0, s>>>(__VA_ARGS__);  \
        else if (!a.need_ang && small) KERNEL(8, 0, 4, false, true)<<<brick_grid(a), DF_THREADS, 0, s>>>(__VA_ARGS__);             \
        else if (!a.need_ang) KERNEL(16, 0, 3, false, true)<<<brick_grid(a), DF_THREADS, 0, s>>>(__VA_ARGS__);                     \
        else if (small && a.n_mm <= 2) KERNEL(8, 2, AD4, true, true)<<<brick_grid(a), DF_THREADS, 0, s>>>(__VA_ARGS__);              \
        else if (a.n_mm <= 2) KERNEL(16, 2, 2, true, true)<<<brick_grid(a), DF_THREADS, 0, s>>>(__VA_ARGS__);                      \
        else KERNEL(16, DF_MAXMM, 2, true, true)<<<brick_grid(a), DF_THREADS, 0, s>>>(__VA_ARGS__);                                \
    } while (0)
#define FORWARD(...) k_rows<__VA_ARGS__>
#define ADJOINT(...) k_rows_adj<__VA_ARGS__, true>
#define ADJOINT_ANY(...) k_rows_adj<__VA_ARGS__, false>

}  // namespace

cudaError_t launch_rows(const DiffArgs &a, const void *sol, float *maps, const int *ch, int *mmarg, cudaStream_t s)
{
    if (a.P == 0 || a.n_slots == 0) return cudaSuccess;
    ROWS_LAUNCH(FORWARD, 3, a, (const float2 *)sol, maps, ch, mmarg);
    return cudaGetLastError();
}

cudaError_t launch_rows_adj(const DiffArgs &a, const void *sol, const float *g_maps, const int *ch, const int *mmarg,
                            DiffGrads g, cudaStream_t s)
{
    if (a.P == 0 || a.n_slots == 0) return cudaSuccess;
    if (a.weigh_all) ROWS_LAUNCH(ADJOINT, 2, a, (const float2 *)sol, g_maps, ch, mmarg, g);
    else ROWS_LAUNCH(ADJOINT_ANY, 2, a, (const float2 *)sol, g_maps, ch, mmarg, g);
    return cudaGetLastError();
}

}  // namespace agb
