// Near-field kernel in FP32 (production path): everything of the reference
// grid loop except the far-field electrostatics, i.e. the short-range AD4 terms
// of LOOP 2 (main.cpp:3030-3404), the d map, and the near part of the e map
// (the pairs the far-field kernel leaves out).  (The FP64 twin is in near.cu.)
//
//   One thread per grid point, bricks of 256 points that lie inside one far
//   frame.  Per brick:
//     stage  candidate atoms of the cells within 8.05 A (one run of the cell
//            list per row of cells), with their canonical frame-relative FP32
//            coordinates, ordered by receptor type (cell order within a type)
//     A      closest DS/D1 atom per point (main.cpp:2986-3015): FP32
//            prefilter, then FP64 with the reference's order, among the
//            candidates (no pair reads one further away)
//     B      per warp the staged atoms near its points, then the pair terms
//   Distances come from the same canonical FP32 arithmetic as the far-field
//   kernel.  Whenever an FP32 quantity lies within its error bound of a
//   discontinuity of the reference (table-bin edge, the 8 A cutoff, the cos=0
//   branch of the D1 and A2 factors, a disordered-hydrogen bin edge) it is
//   decided in FP64, so table bins equal the FP64 reference's.
//   Desolvation is factored: sum_a sol(r)(sp_m vol_a + (solpar_a+qasp|q_a|) vp_m)
//   = sp_m*D1 + vp_m*D2 with D1 = sum vol_a sol, D2 = sum (solpar_a+qasp|q_a|) sol,
//   and the d map is qasp*D1 (main.cpp:3381-3404).
//
// What bounds it: latency (42% of issue slots at 16 warps per SM: the directional
// factors' dependency chains and the row gathers) and the L1 data path (59%).
// 127^3 points x 10,000 atoms x 16 maps: 2.54 -> 1.94 ms (1.74 without
// the scan described at phase A); the gain came from
// 32-byte row loads, the ambiguous pairs' FP64 code behind calls (their guard
// now the proven error bound: 0.12% instead of 0.4% of pairs take it), the
// brick's geometry out of the pair loop's registers, H-bond maps gathered in
// the first table rows and 4x4x2-point warps.
#include <algorithm>

#include "near_exact.cuh"

namespace agb {

namespace {

constexpr int NR_THREADS = 256;
// Resident CTAs per SM the register allocation targets: with 2 (128 registers)
// nothing spills and L1 keeps 156 KB for the table rows; 3 (80 registers)
// take 2.40 against 1.94 ms (127^3 points, 10,000 atoms, 16 maps), 4 2.87 ms.
constexpr int NEAR_MIN_CTAS = 2;
// Candidates staged at once.  Most bricks need one chunk at 0.026 atoms per A^3;
// at 0.06, the inside of a protein with its hydrogens, most need two (10,000
// atoms, 127^3 points, 16 maps, serial: 1.75 ms at 0.026, 2.78 at 0.042, 3.76 at 0.06).
constexpr int NR_CHUNK = 320;
constexpr int NR_WARPS = NR_THREADS / 32;
constexpr int NR_SEGS = NB_SEGS_MAX;    // cell rows laid out at once
constexpr float GUARD_COS = 5.0e-5f;

struct RowsNearSmem {
    float4 pos[NR_CHUNK];                  // frame-relative bins, w = q
    int4 im[NR_CHUNK];                     // file index, metadata, vol, solpar + qasp|q| (float bits)
    float4 a[NR_CHUNK], b[NR_CHUNK];       // bond vector, lone-pair normal
    unsigned short hl[NR_CHUNK];           // staged DS/D1 candidates (slots in this chunk), any order
    union {
        unsigned short wl[NR_WARPS][NR_CHUNK];  // per warp: slots of the staged atoms near its points, in staged order
        int tcnt[NR_CHUNK / 32][32];            // staging by receptor type: per 32-candidate slice and type
    };
    float wbox[NR_WARPS][6];               // per warp: its points' box in frame bins (lo xyz, hi xyz)
    float2 es[NT_SMALL];                   // near e table, desolvation table
    // per thread: the running H-bond min/max of the MM maps (out of the pair
    // loop's register budget)
    float hmin[NG_MM][NR_THREADS], hmax[NG_MM][NR_THREADS];
    // per thread: bond vector of the closest DS/D1 atom and its file index
    float rvh[3][NR_THREADS];
    int ch[NR_THREADS];
    int seg_start[NR_SEGS], seg_off[NR_SEGS + 1];
    int total, nh;
    // the brick: its box (A), the far frame's middle point and its place (bins),
    // and the range of cells in reach.  Here and not in registers, because
    // the staging needs them again when the candidates take several chunks.
    double lo[3], hi[3], org[3];
    int c0[3], c1[3], frame[3];
};

struct PairAng {
    float racc, rdon, Hramp;
};

// FP32 directional factors (racc, rdon, Hramp) from the unit pair vector and
// the atom's staged bond vectors.  Returns false when cos_theta lies within
// its error bound of the D1/A2 branch at 0; the caller then uses pair_exact().
__device__ __forceinline__ bool angular_fast(int meta, float4 rvA, float4 rvB, int ia, float dX, float dY, float dZ,
                                             float rs, int ch, float3 rvh, PairAng &o)
{
    o.racc = 1.f; o.rdon = 1.f; o.Hramp = 1.f;
    const bool dis = (meta & META_DIS) != 0;
    const int hb = (meta >> META_HB_SHIFT) & 7;
    if (hb != 2 && hb != 4 && hb != 5) return true;
    const float dn0 = dX * rs, dn1 = dY * rs, dn2 = dZ * rs;
    const float rv0 = rvA.x, rv1 = rvA.y, rv2 = rvA.z;
    const float cos_theta = ((0.f - dn0 * rv0) - dn1 * rv1) - dn2 * rv2;
    // An atom without bonded neighbours keeps a zero bond vector; its cos_theta
    // is exactly 0 in every precision, so the branch at 0 is not ambiguous.
    const bool rv_zero = (meta & META_RVZERO) != 0;
    if (hb == 2) {
        if (fabsf(cos_theta) < GUARD_COS && !rv_zero) return false;
        if (cos_theta <= 0.f) {
            o.racc = 0.f;
        } else {
            const int e = (meta >> META_REXP_SHIFT) & 7;
            o.racc = (e == 2) ? cos_theta * cos_theta
                   : (e == 4) ? (cos_theta * cos_theta) * (cos_theta * cos_theta) : cos_theta;
            if (ia != ch && ch >= 0) {
                float ct = rvh.x * rv0 + rvh.y * rv1 + rvh.z * rv2;
                ct = fminf(fmaxf(ct, -1.f), 1.f);
                // 0.5 - 0.5 cos(x) = 0.5 + 0.5 cos(x - pi), x - pi in [-pi, pi/3]: the
                // range on which __cosf's absolute error is within 2^-21.4
                o.Hramp = 0.5f + 0.5f * __cosf(acosf(ct) * (120.f / 90.f) - 3.14159265f);
            }
        }
    } else if (hb == 4) {
        o.rdon = (cos_theta <= 0.f) ? 0.f : cos_theta * cos_theta;
    } else if (!dis) {  // A2 ordered (main.cpp:3163-3246)
        if (fabsf(cos_theta) < GUARD_COS && !rv_zero) return false;
        const float w0 = rvB.x, w1 = rvB.y, w2 = rvB.z;
        float t0 = dn0 * w0 + dn1 * w1 + dn2 * w2;
        t0 = fminf(fmaxf(t0, -1.f), 1.f);
        // cos(pi/2 - acos(t0)) = sqrt(1 - t0^2)
        const float cos_t0 = sqrt_approx(fmaxf(1.f - t0 * t0, 0.f));
        const float c0 = dn1 * w2 - dn2 * w1, c1 = dn2 * w0 - dn0 * w2, c2 = dn0 * w1 - dn1 * w0;
        float rd2 = c0 * c0 + c1 * c1 + c2 * c2;
        rd2 = fmaxf(rd2, 1.0e-6f);
        const float inv_rd = rsqrtf(rd2);
        float ti = (c0 * rv0 + c1 * rv1 + c2 * rv2) * inv_rd;
        o.rdon = 0.f;
        if (cos_theta >= 0.f) {
            ti = fminf(fmaxf(ti, -1.f), 1.f);
            // sin(2|acos(ti) - pi/2|) = |sin(2 acos(ti))| = 2|ti|sqrt(1 - ti^2)
            const float s2 = 2.f * fabsf(ti) * sqrt_approx(fmaxf(1.f - ti * ti, 0.f));
            o.rdon = (0.9f + 0.1f * s2) * cos_t0;
        } else if (cos_theta >= -0.34202f) {
            const float b = 0.116978f - cos_theta * cos_theta;
            o.rdon = 562.25f * (b * b * b) * cos_t0;
        }
    } else {  // A2 disordered, cylindrical hydroxyl (main.cpp:3247-3272)
        const float ct = fminf(fmaxf(cos_theta, -1.f), 1.f);
        o.racc = 0.f; o.rdon = 0.f;
        // theta = acos(ct) <= 1.24791 + pi/2  <=>  ct >= -sin(1.24791); the value is 0 at the edge
        if (ct >= -0.94832352f) {
            // cos(theta - a) = ct cos(a) + sin(theta) sin(a), a = 1.24791
            const float c = ct * 0.31730505f + sqrtf(fmaxf(1.f - ct * ct, 0.f)) * 0.94832352f;
            o.rdon = (c * c) * (c * c);
            o.racc = o.rdon;
        }
    }
    return true;
}


// The FP64 point coordinate (main.cpp:2815-2859) behind a frame coordinate P,
// whose rounding is far below half a spacing.
__device__ __forceinline__ double point_coord(const DevProblem &p, int frame, int ne, float P)
{
    return (double)(frame + __double2int_rn(P / (p.spacing * AG_A_DIV)) - ne) * p.spacing;
}

// The cold paths of a pair are calls that take and return values: with their
// code in line, or results by address, the pair loop keeps 30 more registers
// alive or spilled.

struct PairBins {  // x: bin; y: LOOP 1 bin, negative when beyond 8 A; z: disordered-hydrogen row bin; w: 1/max(r, 0.5)
    int4 v;
};

// The bins of a pair whose FP32 distance t (bins) lies within its error bound
// of an edge.  e = rint(t) is the edge: the FP64 squared distance in bins
// (exactly 2^14 times the reference's) against e^2 decides, unless the two
// are within 1e-12 of each other or the hydrogen-row bin is in doubt, where
// the reference's own expressions do.
__device__ __noinline__ PairBins near_bins_exact(const DevProblem &p, int fx, int fy, int fz, int ia, float PX, float PY,
                                                 float PZ, float t, float inv_rmax, int kh, bool kh_clear)
{
    const double cx = point_coord(p, fx, p.nex, PX), cy = point_coord(p, fy, p.ney, PY), cz = point_coord(p, fz, p.nez, PZ);
    const double d0 = __dsub_rn(p.x[ia], cx), d1 = __dsub_rn(p.y[ia], cy), d2 = __dsub_rn(p.z[ia], cz);
    const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2));
    const int e = __float2int_rn(t);
    const double t2 = r2 * (double)(AG_A_DIV * AG_A_DIV), e2 = (double)(e * e);
    PairBins o;
    if (kh_clear && t >= 1.0f && fabs(t2 - e2) > 1.0e-12 * e2) {
        const int kb = t2 >= e2 ? e : e - 1;
        o.v = make_int4(kb, kb < AG_NEINT ? kb : -1 - kb, kh, __float_as_int(inv_rmax));
        return o;
    }
    PairQ<float> q;
    dist_exact_f(p, ia, cx, cy, cz, q);
    o.v = make_int4(q.bin, q.ad4_in ? q.bin_e : -1 - q.bin_e, q.ih, __float_as_int(q.inv_rmax));
    return o;
}

__device__ __noinline__ float3 near_angles_exact(const DevProblem &p, int fx, int fy, int fz, int ia, int ch, float PX,
                                                 float PY, float PZ)
{
    double d0, d1, d2;
    const double r = loop2_dist(p, ia, point_coord(p, fx, p.nex, PX), point_coord(p, fy, p.ney, PY),
                                point_coord(p, fz, p.nez, PZ), d0, d1, d2);
    PairQ<double> q;
    angular_exact(p, ia, ch, d0, d1, d2, r, q);
    return make_float3((float)q.racc, (float)q.rdon, (float)q.Hramp);
}

// One brick `b` of one instance (p, g).
template <int BX, int BY, int BZ, int NGK>
__device__ __forceinline__ void near_rows_unit(const DevProblem &p, const NearGroup &g, const NearPtrs &ptr, int b,
                                               RowsNearSmem &S)
{
    static_assert(BX * BY * BZ == NR_THREADS, "one thread per brick point");
    static_assert(BX % 4 == 0 && BY % 4 == 0 && BZ % 2 == 0, "warps of 4x4x2 points");
    static_assert(FRAME_X % BX == 0 && FRAME_Y % BY == 0 && FRAME_Z % BZ == 0, "bricks tile far frames");
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (int i = tid; i < NT_SMALL; i += NR_THREADS) S.es[i] = make_float2(ptr.etab[i], ptr.solf[i]);
    const int nbx = (p.n1x + BX - 1) / BX, nby = (p.n1y + BY - 1) / BY;
    const int bx = b % nbx, by = (b / nbx) % nby, bz = b / (nbx * nby);
    // A whole brick's warps are 4x4x2 corners: their box grown by 8 A holds
    // fewer atoms out of a lane's reach than that of an 8x4x1 slice.  A brick cut by
    // the box's edge packs its points inside the box into its first threads
    // (x fastest), so that whole warps idle instead of lanes in every warp.
    const int wx = min(BX, p.n1x - bx * BX), wy = min(BY, p.n1y - by * BY), wz = min(BZ, p.n1z - bz * BZ);
    int lx, ly, lz;
    if (wx * wy * wz == NR_THREADS) {
        constexpr int TX = BX / 4, TY = BY / 4;
        lx = (lane & 3) + 4 * (wid % TX);
        ly = ((lane >> 2) & 3) + 4 * ((wid / TX) % TY);
        lz = (lane >> 4) + 2 * (wid / (TX * TY));
    } else {
        lx = tid % wx;
        ly = (tid / wx) % wy;
        lz = tid / (wx * wy);
    }
    const int ix = bx * BX + lx, iy = by * BY + ly, iz = bz * BZ + lz;
    const bool valid = lz < wz;
    const long long lin = ((long long)iz * p.n1y + iy) * p.n1x + ix;

    if (tid < 3) {
        const int n1 = tid == 0 ? p.n1x : tid == 1 ? p.n1y : p.n1z, ne = tid == 0 ? p.nex : tid == 1 ? p.ney : p.nez;
        const int first = tid == 0 ? bx * BX : tid == 1 ? by * BY : bz * BZ, step = tid == 0 ? BX : tid == 1 ? BY : BZ;
        const int fr = tid == 0 ? FRAME_X : tid == 1 ? FRAME_Y : FRAME_Z, nc = tid == 0 ? p.ncx : tid == 1 ? p.ncy : p.ncz;
        const int o = first / fr * fr + fr / 2;
        const double lo = (double)(first - ne) * p.spacing, hi = (double)(min(first + step, n1) - 1 - ne) * p.spacing;
        S.lo[tid] = lo;
        S.hi[tid] = hi;
        S.frame[tid] = o;
        S.org[tid] = frame_origin_bins(o, ne, p.spacing * AG_A_DIV);
        // cells within the candidate radius of the brick
        S.c0[tid] = max(0, min(nc - 1, (int)floor((lo - AGB_NEAR_RADIUS - p.cell0[tid]) / p.cell_size)));
        S.c1[tid] = max(0, min(nc - 1, (int)floor((hi + AGB_NEAR_RADIUS - p.cell0[tid]) / p.cell_size)));
    }
    __syncthreads();
    // the point's canonical coordinates in its far frame
    const float PX = frame_point_coord(ix - S.frame[0], p.spacing * AG_A_DIV),
                PY = frame_point_coord(iy - S.frame[1], p.spacing * AG_A_DIV),
                PZ = frame_point_coord(iz - S.frame[2], p.spacing * AG_A_DIV);
    auto cx = [&]() { return point_coord(p, S.frame[0], p.nex, PX); };
    auto cy = [&]() { return point_coord(p, S.frame[1], p.ney, PY); };
    auto cz = [&]() { return point_coord(p, S.frame[2], p.nez, PZ); };

    const bool need_h = p.n_atom_maps > 0;
    const bool do_e = g.write_special && p.elec_map >= 0;
    const bool need_pairs = g.ng > 0 || (g.write_special && p.dsolv_map >= 0) || do_e;

    auto nrow_y = [&]() { return S.c1[1] - S.c0[1] + 1; };
    auto nseg_total = [&]() { return (need_pairs || need_h) ? nrow_y() * (S.c1[2] - S.c0[2] + 1) : 0; };

    // Rows [sb, sb + nseg) of cells: each row's run of x cells within the
    // radius of the brick (cells of a row are consecutive in the cell list),
    // and the running offsets of their atoms.  All threads call it; it ends
    // with a barrier.
    auto layout_segments = [&](int sb, int nseg) {
        auto gap2 = [&](int i, int c) {  // squared gap between cell c of axis i and the brick's box
            const double blo = p.cell0[i] + c * p.cell_size, bhi = blo + p.cell_size;
            const double gp = fmax(fmax(blo - S.hi[i], S.lo[i] - bhi), 0.0);
            return gp * gp;
        };
        for (int k = tid; k < nseg; k += NR_THREADS) {
            const int cyy = S.c0[1] + (sb + k) % nrow_y(), czz = S.c0[2] + (sb + k) / nrow_y();
            const double left = AGB_NEAR_RADIUS * AGB_NEAR_RADIUS - gap2(1, cyy) - gap2(2, czz);
            int x0 = S.c0[0], x1 = S.c1[0];
            // an edge cell also holds the atoms past the last cell boundary (none is dropped by its box)
            while (x0 <= x1 && x0 > 0 && gap2(0, x0) > left) x0++;
            while (x1 >= x0 && x1 < p.ncx - 1 && gap2(0, x1) > left) x1--;
            const int row = (czz * p.ncy + cyy) * p.ncx;
            const int st = x0 <= x1 ? p.cell_start[row + x0] : 0;
            S.seg_start[k] = st;
            S.seg_off[k] = (x0 <= x1 ? p.cell_start[row + x1 + 1] : 0) - st;
        }
        __syncthreads();
        if (tid < 32) {  // exclusive scan of the run lengths, two per lane
            static_assert(NR_SEGS == 64, "two runs per lane");
            const int u = 2 * tid < nseg ? S.seg_off[2 * tid] : 0, w = 2 * tid + 1 < nseg ? S.seg_off[2 * tid + 1] : 0;
            int incl = u + w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (tid >= o) incl += v;
            }
            __syncwarp();
            S.seg_off[2 * tid] = incl - u - w;
            S.seg_off[2 * tid + 1] = incl - w;
            if (tid == 31) {
                S.seg_off[NR_SEGS] = incl;
                S.total = incl;
            }
            if (tid == 0) S.nh = 0;
        }
        __syncthreads();
    };
    // Stage chunk `k0` (n candidates) of the laid-out rows, ordered by
    // receptor type by a stable counting sort (cell order within a type), so
    // that a warp's consecutive pairs read the table rows of one type, which
    // then stay in L1.  Slice k (candidates [32k, 32k + 32) of the chunk) is
    // ranked by one warp; S.tcnt[k][t] holds the slice's count of type t,
    // then the slot of its first such candidate.  All threads call it.
    static_assert(NR_CHUNK <= 2 * NR_THREADS && NR_CHUNK % 32 == 0, "two candidates per thread at most");
    auto stage = [&](int k0, int n) {
        constexpr int NSL = NR_CHUNK / 32;
        for (int i = tid; i < NSL * 32; i += NR_THREADS) S.tcnt[i >> 5][i & 31] = 0;
        __syncthreads();
        int ca[2], ct[2], cr[2], cm[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int i = u * NR_THREADS + tid;
            int a = -1, t = 32, m = 0;  // lanes past the chunk form a group of their own
            if (i < n) {
                const int c = k0 + i;
                int s = 0, e = NR_SEGS - 1;  // the last row that starts at or before c
#pragma unroll
                for (int o = NR_SEGS / 2; o; o >>= 1) {
                    const int mid = s + o;
                    if (mid <= e && S.seg_off[mid] <= c) s = mid;
                }
                a = p.cell_atoms[S.seg_start[s] + (c - S.seg_off[s])];
                m = ptr.meta[a];
                t = m & META_TYPE_MASK;
            }
            const unsigned same = __match_any_sync(0xffffffffu, t);
            cr[u] = __popc(same & ((1u << lane) - 1u));
            if (i < n && cr[u] == 0) S.tcnt[i >> 5][t] = __popc(same);
            ca[u] = a;
            ct[u] = t;
            cm[u] = m;
        }
        __syncthreads();
        if (tid < 32) {  // thread t: type t's slots, slices in order, after every lower type
            int cnt[NSL], run = 0;
#pragma unroll
            for (int k = 0; k < NSL; k++) {
                cnt[k] = S.tcnt[k][tid];
                run += cnt[k];
            }
            int incl = run;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (tid >= o) incl += v;
            }
            incl -= run;
#pragma unroll
            for (int k = 0; k < NSL; k++) {
                S.tcnt[k][tid] = incl;
                incl += cnt[k];
            }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int i = u * NR_THREADS + tid;
            if (i >= n) continue;
            const int a = ca[u], j = S.tcnt[i >> 5][ct[u]] + cr[u];
            S.pos[j] = make_float4(frame_atom_coord(p.x[a] * AG_A_DIV, S.org[0]),
                                   frame_atom_coord(p.y[a] * AG_A_DIV, S.org[1]),
                                   frame_atom_coord(p.z[a] * AG_A_DIV, S.org[2]), (float)p.q[a]);
            const float4 va = ptr.atomA[a], vb = ptr.atomB[a];
            S.a[j] = va;
            S.b[j] = vb;
            S.im[j] = make_int4(a, cm[u], __float_as_int(va.w), __float_as_int(vb.w));
            const int hb = (cm[u] >> META_HB_SHIFT) & 7;
            if (hb == 1 || hb == 2) S.hl[atomicAdd(&S.nh, 1)] = (unsigned short)j;
        }
        __syncthreads();
    };
    // the candidate list fits one chunk in the common case: stage it once
    bool resident = false;
    if (nseg_total() > 0 && nseg_total() <= NR_SEGS) {
        layout_segments(0, nseg_total());
        if (S.total <= NR_CHUNK) {
            stage(0, S.total);
            resident = true;
        }
    }
    // visit every candidate chunk: fn(n) with the chunk staged in shared memory.
    // One call site for fn, so its body is instantiated once.
    auto for_each_chunk = [&](auto &&fn) {
        const int nsb = resident ? 1 : (nseg_total() + NR_SEGS - 1) / NR_SEGS;
        for (int sbi = 0; sbi < nsb; sbi++) {
            if (!resident) {
                const int sb = sbi * NR_SEGS;
                __syncthreads();
                layout_segments(sb, min(NR_SEGS, nseg_total() - sb));
            }
            const int total = S.total;
            for (int k0 = 0; k0 < total; k0 += NR_CHUNK) {
                const int n = min(NR_CHUNK, total - k0);
                if (!resident) {
                    __syncthreads();
                    if (tid == 0) S.nh = 0;
                    stage(k0, n);
                }
                fn(n);
            }
        }
    };
    // ---- A: closest DS/D1 hydrogen (main.cpp:2986-3015).  Only pairs with a D1
    // atom in range use it, and such an atom is among the candidates: where none
    // of these is a DS/D1 atom (ch = -1), and beyond the candidates' radius,
    // nothing reads it.  (Scanning every DS/D1 atom there, thread by thread, held
    // up to 30% of the SM time idle behind a few bricks of empty space:
    // 10,000 atoms, 16 maps, 127^3 points 1.95 -> 1.74 ms, 127x127x49 points
    // 1.11 -> 0.74 ms.)
    int ch = -1;
    if (need_h) {
        // FP32 prefilter: the two smallest squared distances (bins^2) and the
        // atom of the smallest.  Every candidate within `lim` of the smallest
        // is re-checked in FP64; when the second smallest lies beyond `lim`,
        // that is the smallest's atom alone, and the FP64 pass over the
        // candidates reduces to its own distance.
        float best2 = 3.0e38f, next2 = 3.0e38f;
        int best_a = -1;
        for_each_chunk([&](int) {
            if (!valid) return;
            for (int k = 0; k < S.nh; k++) {
                const int j = S.hl[k];
                const float4 A = S.pos[j];
                const float dx = A.x - PX, dy = A.y - PY, dz = A.z - PZ;
                const float d2 = dx * dx + dy * dy + dz * dz;
                next2 = fminf(next2, fmaxf(best2, d2));
                if (d2 < best2) {
                    best2 = d2;
                    best_a = S.im[j].x;
                }
            }
        });
        const float lim = best2 * (1.0f + 2.0e-5f) + 4.0f;
        double rmin = 999999.;
        const bool several = valid && best_a >= 0 && next2 <= lim;
        if (!several) ch = best_a;
        if (__syncthreads_or(several))
            for_each_chunk([&](int) {
                if (!several) return;
                for (int k = 0; k < S.nh; k++) {
                    const int j = S.hl[k];
                    const float4 A = S.pos[j];
                    const float dx = A.x - PX, dy = A.y - PY, dz = A.z - PZ;
                    if (dx * dx + dy * dy + dz * dz > lim) continue;
                    const int a = S.im[j].x;
                    const double r = h_dist(p, a, cx(), cy(), cz());
                    if (r < rmin || (r == rmin && a < ch)) { rmin = r; ch = a; }
                }
            });
    }
    if (need_h && valid) {
        S.ch[tid] = ch;
        const float4 v = ch >= 0 ? ptr.atomA[ch] : make_float4(0.f, 0.f, 0.f, 0.f);
        S.rvh[0][tid] = v.x;
        S.rvh[1][tid] = v.y;
        S.rvh[2][tid] = v.z;
    }

    // ---- B: pair terms
    static_assert(NGK % 8 == 0 && NGK >= NG_MM && NGK <= NG_MAX, "accumulator count");
    float2 E[NGK / 2];
#pragma unroll
    for (int k = 0; k < NGK / 2; k++) E[k] = make_float2(0.f, 0.f);
    for (int m = 0; m < NG_MM; m++) {
        S.hmin[m][tid] = 999999.f;
        S.hmax[m][tid] = -999999.f;
    }
    float D1 = 0.f, D2 = 0.f, e_near = 0.f;
    unsigned n_near = 0, n_fb = 0;
    if (need_pairs) {
        // This warp's points as a box in frame bins (lanes outside the grid do
        // not count).  Per chunk, the warp keeps the staged atoms whose
        // distance to the box is within the near radius plus 2 bins, in staged
        // order: every pair a lane evaluates below (FP32 t < 1024 + the guard)
        // lies inside that margin, so the pairs and their summation order are
        // those of the full staged list.
        {
            float blo[3] = {valid ? PX : 3.0e38f, valid ? PY : 3.0e38f, valid ? PZ : 3.0e38f};
            float bhi[3] = {valid ? PX : -3.0e38f, valid ? PY : -3.0e38f, valid ? PZ : -3.0e38f};
#pragma unroll
            for (int d = 0; d < 3; d++)
#pragma unroll
                for (int o = 16; o; o >>= 1) {
                    blo[d] = fminf(blo[d], __shfl_xor_sync(0xffffffffu, blo[d], o));
                    bhi[d] = fmaxf(bhi[d], __shfl_xor_sync(0xffffffffu, bhi[d], o));
                }
            if (lane == 0)
                for (int d = 0; d < 3; d++) {
                    S.wbox[wid][d] = blo[d];
                    S.wbox[wid][3 + d] = bhi[d];
                }
            __syncwarp();
        }
        const float keep2 = (FAR_T0 + 2.0f) * (FAR_T0 + 2.0f);
        const float guard = p.near_guard;
        unsigned short *wl = S.wl[wid];
        for_each_chunk([&](int n) {
            int cnt = 0;
            for (int j0 = 0; j0 < n; j0 += 32) {
                const int jj = j0 + lane;
                bool keep = false;
                if (jj < n) {
                    const float4 A = S.pos[jj];
                    const float *bx_ = S.wbox[wid];
                    const float ex = fmaxf(fmaxf(bx_[0] - A.x, A.x - bx_[3]), 0.f);
                    const float ey = fmaxf(fmaxf(bx_[1] - A.y, A.y - bx_[4]), 0.f);
                    const float ez = fmaxf(fmaxf(bx_[2] - A.z, A.z - bx_[5]), 0.f);
                    keep = ex * ex + ey * ey + ez * ez <= keep2;
                }
                const unsigned m = __ballot_sync(0xffffffffu, keep);
                if (keep) wl[cnt + __popc(m & ((1u << lane) - 1u))] = (unsigned short)jj;
                cnt += __popc(m);
            }
            __syncwarp();
            if (!valid) return;
            for (int k = 0; k < cnt; k++) {
                const int j = wl[k];
                const float4 A = S.pos[j];
                const float dY = __fsub_rn(A.y, PY), dZ = __fsub_rn(A.z, PZ);
                const float s = __fmaf_rn(dY, dY, __fmaf_rn(dZ, dZ, TINY_T2));
                const float dX = __fsub_rn(A.x, PX);
                const float t2 = __fmaf_rn(dX, dX, s);
                const float rs = rsqrt_approx(t2);
                const float t = __fmul_rn(t2, rs);
                if (t >= FAR_T0 + guard) continue;
                const int4 im = S.im[j];
                const int meta = im.y;
                const bool dis = (meta & META_DIS) != 0;
                // bin: floor(t), unless t lies within its error bound of an edge
                const float tm = __fadd_rz(t, 8388608.f);  // 2^23 + floor(t)
                int kb = __float_as_int(tm) - (int)MAGIC_BITS, kh = 0;
                const float fr = t - (tm - 8388608.f);
                float inv_rmax = fminf((float)AG_A_DIV * rs, 2.0f);
                bool clear = fminf(fr, 1.f - fr) >= guard && t >= 1.0f, kh_clear = true;
                if (dis) {  // the disordered-hydrogen row bin, (r - 1.10) * A_DIV
                    const float xh = t - 140.8f, hm = floorf(xh);
                    kh = max(0, min((int)hm, AG_NEINT - 1));
                    kh_clear = xh <= 0.5f || fminf(xh - hm, hm + 1.f - xh) >= guard + 1.0e-4f;
                    clear &= kh_clear;
                }
                bool in = kb < AG_NEINT;  // r <= 8 A (r = 8 A exactly: decided in FP64)
                int ke = kb;
                if (!clear) {
                    const int4 x = near_bins_exact(p, S.frame[0], S.frame[1], S.frame[2], im.x, PX, PY, PZ, t, inv_rmax, kh,
                                                   kh_clear).v;
                    kb = x.x;
                    in = x.y >= 0;
                    ke = in ? x.y : -1 - x.y;
                    kh = x.z;
                    inv_rmax = __int_as_float(x.w);
                    n_fb++;
                }
                const float2 es = S.es[min(kb, NT_SMALL - 1)];
                // the far-field kernel skips exactly the pairs with t < FAR_T0
                if (t < FAR_T0 && do_e) {
                    const float eb = ke == kb ? es.x : S.es[min(ke, NT_SMALL - 1)].x;
                    e_near += (eb * A.w) * inv_rmax;
                }
                if (!in || (meta & META_SKIP_AD4)) continue;
                n_near++;
                D1 += __int_as_float(im.z) * es.y;  // vol
                D2 += __int_as_float(im.w) * es.y;  // solpar + qasp|q|
                if (g.ng == 0) continue;
                const int hb = (meta >> META_HB_SHIFT) & 7, ta = meta & META_TYPE_MASK;
                const int kn = min(kb, AG_NEINT - 1);
                const float *Trow = ptr.vdwT + (unsigned)(ta * AG_NEINT + kn) * (unsigned)ptr.mpad + g.col0;
                Row8 T[NGK / 8];
#pragma unroll
                for (int k8 = 0; k8 < NGK / 8; k8++)
                    if (8 * k8 < g.ng) T[k8] = load_row8(Trow + 8 * k8);
                if ((g.plain_hb >> hb) & 1u) {  // every map a plain sum for this class (most atoms)
#pragma unroll
                    for (int i = 0; i < NGK / 2; i++)
                        if (8 * (i / 4) < g.ng) E[i] = __fadd2_rn(E[i], T[i / 4].p[i % 4]);
                    continue;
                }
                PairAng q;
                const int chp = S.ch[tid];
                const float3 rvh = make_float3(S.rvh[0][tid], S.rvh[1][tid], S.rvh[2][tid]);
                if (!angular_fast(meta, S.a[j], S.b[j], im.x, dX, dY, dZ, rs, chp, rvh, q)) {
                    const float3 x = near_angles_exact(p, S.frame[0], S.frame[1], S.frame[2], im.x, chp, PX, PY, PZ);
                    q.racc = x.x;
                    q.rdon = x.y;
                    q.Hramp = x.z;
                    n_fb++;
                }
                const float *Hrow = (g.has_hrow && dis && p.hydrogen_type >= 0)
                    ? ptr.vdwT + (unsigned)(p.hydrogen_type * AG_NEINT + kh) * (unsigned)ptr.mpad + g.col0 : Trow;
                const unsigned long long aw = g.actw[hb];
                const unsigned rows_plain = (g.plain4 >> (4 * hb)) & 15u;
#pragma unroll
                for (int k8 = 0; k8 < NGK / 8; k8++) {
                    if (8 * k8 >= g.ng) break;
#pragma unroll
                    for (int h4 = 0; h4 < 2; h4++) {
                        const int m4 = 2 * k8 + h4;
                        if ((rows_plain >> m4) & 1u) {  // the same adds as the per-map chain below
                            E[2 * m4] = __fadd2_rn(E[2 * m4], T[k8].p[2 * h4]);
                            E[2 * m4 + 1] = __fadd2_rn(E[2 * m4 + 1], T[k8].p[2 * h4 + 1]);
                            continue;
                        }
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            const int m = 4 * m4 + u;
                            if (m >= g.ng) break;
                            const int act = (int)(aw >> (3 * m)) & 7;
                            if (act == ACT_SKIP) continue;
                            float v = (u & 1) ? T[k8].p[2 * h4 + u / 2].y : T[k8].p[2 * h4 + u / 2].x;
                            if (act != ACT_PLAIN) {
                                // a product with 0.01f is within 1.5 ulp of the quotient
                                const float rsph = __saturatef(v * 0.01f);
                                const float f = (act == ACT_SUMA || act == ACT_MMA) ? q.racc : q.rdon;
                                const float fac = f + (1.f - f) * rsph;
                                if (act == ACT_SUMA || (act == ACT_MMD && dis)) {
                                    if (dis) v = __ldg(Hrow + m);
                                    v = v * q.Hramp * fac;
                                } else {
                                    if (m < NG_MM) {  // min/max maps are placed first by the host
                                        v *= fac;
                                        // comparisons as the reference's: a NaN is stored
                                        const float lo = S.hmin[m < NG_MM ? m : 0][tid], hi = S.hmax[m < NG_MM ? m : 0][tid];
                                        S.hmin[m < NG_MM ? m : 0][tid] = lo < v ? lo : v;
                                        S.hmax[m < NG_MM ? m : 0][tid] = hi > v ? hi : v;
                                    }
                                    continue;
                                }
                            }
                            if (u & 1) E[m / 2].y += v;
                            else E[m / 2].x += v;
                        }
                    }
                }
            }
        });
    }

    // finalise (main.cpp:3420-3431) and store
    if (valid) {
#pragma unroll
        for (int m = 0; m < NGK; m++) {
            if (m >= g.ng) break;
            float v = (m & 1) ? E[m / 2].y : E[m / 2].x;
            // some pair entered (also where it left a NaN): until then min > max
            if (m < NG_MM && !(S.hmin[m < NG_MM ? m : 0][tid] > S.hmax[m < NG_MM ? m : 0][tid]))
                v += S.hmin[m < NG_MM ? m : 0][tid] + fmaxf(S.hmax[m < NG_MM ? m : 0][tid], 0.f);
            v += (float)g.sp[m] * D1 + (float)g.vp[m] * D2;
            const size_t o = (size_t)g.out_map[m] * (size_t)p.P + (size_t)lin;
            ptr.out32[o] = g.cov[m] ? (float)ptr.cov_map[lin] : v;
        }
        if (g.write_special) {
            if (p.dsolv_map >= 0) ptr.out32[(size_t)p.dsolv_map * (size_t)p.P + (size_t)lin] = (float)p.solpar_q * D1;
            if (do_e)  // the near part of the e map; k_emap_reduce adds the far-field chunks
                ptr.out32[(size_t)p.elec_map * (size_t)p.P + (size_t)lin] = e_near;
        }
    }
    if (ptr.counters) {  // one atomic per counter and warp
        const unsigned n0 = __reduce_add_sync(0xffffffffu, n_near), n1 = __reduce_add_sync(0xffffffffu, n_fb);
        if (lane == 0) {
            if (n0) atomicAdd(ptr.counters + 0, (unsigned long long)n0);
            if (n1) atomicAdd(ptr.counters + 1, (unsigned long long)n1);
        }
    }
}

// Single instance: one CTA per brick.  The problem is read through a
// shared-memory copy: the FP64 fallbacks take it by reference, and a reference
// to the kernel parameter would make every thread copy it into local memory.
template <int BX, int BY, int BZ, int NGK>
__global__ void __launch_bounds__(NR_THREADS, NEAR_MIN_CTAS) k_near(DevProblem p, NearGroup g, NearPtrs ptr, int brick0)
{
    __shared__ RowsNearSmem S;
    __shared__ DevProblem s_p;
    if (threadIdx.x == 0) s_p = p;
    __syncthreads();
    near_rows_unit<BX, BY, BZ, NGK>(s_p, g, ptr, brick0 + blockIdx.x, S);
}

// Many instances, persistent: (instance-group, brick) units from an atomic
// counter; units never wait on each other.
template <int BX, int BY, int BZ, int NGK>
__global__ void __launch_bounds__(NR_THREADS, NEAR_MIN_CTAS)
k_near_batch(const NearInst *__restrict__ insts, const long long *__restrict__ unit_begin, int n_inst,
             unsigned long long *__restrict__ counter)
{
    __shared__ RowsNearSmem S;
    __shared__ NearInst s_i;
    __shared__ long long s_unit;
    int cur = -1;
    const long long total = unit_begin[n_inst];
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_unit = (long long)atomicAdd(counter, 1ull);
        __syncthreads();
        const long long u = s_unit;
        if (u >= total) break;
        int lo = 0, hi = n_inst - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (unit_begin[mid] <= u) lo = mid; else hi = mid - 1;
        }
        if (lo != cur) {
            __syncthreads();
            for (int i = threadIdx.x; i < (int)(sizeof(NearInst) / 4); i += NR_THREADS)
                ((int *)&s_i)[i] = ((const int *)&insts[lo])[i];
            __syncthreads();
            cur = lo;
        }
        near_rows_unit<BX, BY, BZ, NGK>(s_i.p, s_i.g, s_i.ptr, (int)(u - unit_begin[lo]), S);
    }
}

// Accumulators a launch holds per point: groups of at most 8 maps (the
// 8-map sets of batched ensembles) run with 8, one row load per pair instead of
// two; larger groups with NG_MAX.
constexpr int NGK_SMALL = 8;

template <int BX, int BY, int BZ>
cudaError_t near_single(const DevProblem &p, const NearGroup &g, const NearPtrs &ptr, cudaStream_t s, int bz0, int bz1)
{
    const int nbx = (p.n1x + BX - 1) / BX, nby = (p.n1y + BY - 1) / BY, nbz = (p.n1z + BZ - 1) / BZ;
    if (bz1 < 0 || bz1 > nbz) bz1 = nbz;
    if (bz0 >= bz1) return cudaSuccess;
    const unsigned nb = (unsigned)(nbx * nby * (bz1 - bz0));
    const int b0 = bz0 * nbx * nby;
    if (g.ng <= NGK_SMALL) k_near<BX, BY, BZ, NGK_SMALL><<<nb, NR_THREADS, 0, s>>>(p, g, ptr, b0);
    else k_near<BX, BY, BZ, NG_MAX><<<nb, NR_THREADS, 0, s>>>(p, g, ptr, b0);
    return cudaGetLastError();
}

template <int BX, int BY, int BZ, int NGK>
cudaError_t near_batch_t(const NearInst *insts, const long long *unit_begin, int n_inst, unsigned long long *counter,
                         int ctas_per_sm, cudaStream_t s)
{
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_near_batch<BX, BY, BZ, NGK>, NR_THREADS, 0);
    const int per_sm = std::max(1, std::min(ctas_per_sm, occ));
    k_near_batch<BX, BY, BZ, NGK><<<current_device_sms() * per_sm, NR_THREADS, 0, s>>>(insts, unit_begin, n_inst, counter);
    return cudaGetLastError();
}

template <int NGK>
cudaError_t near_batch_shape(const NearInst *insts, const long long *unit_begin, int n_inst, unsigned long long *counter,
                             int shape, int ctas_per_sm, cudaStream_t s)
{
    if (shape == 1) return near_batch_t<8, 4, 8, NGK>(insts, unit_begin, n_inst, counter, ctas_per_sm, s);
    if (shape == 2) return near_batch_t<4, 8, 8, NGK>(insts, unit_begin, n_inst, counter, ctas_per_sm, s);
    return near_batch_t<8, 8, 4, NGK>(insts, unit_begin, n_inst, counter, ctas_per_sm, s);
}

}  // namespace

// Brick z-rows [bz0, bz1) (bz1 < 0: through the last).
cudaError_t launch_near(const DevProblem &p, const NearGroup &g, const NearPtrs &ptr, cudaStream_t s, int bz0, int bz1)
{
    return near_single<8, 8, 4>(p, g, ptr, s, bz0, bz1);
}

cudaError_t launch_near_batch(const NearInst *insts, const long long *unit_begin, int n_inst,
                              unsigned long long *counter, int shape, int ctas_per_sm, int max_ng, cudaStream_t s)
{
    if (max_ng <= NGK_SMALL)
        return near_batch_shape<NGK_SMALL>(insts, unit_begin, n_inst, counter, shape, ctas_per_sm, s);
    return near_batch_shape<NG_MAX>(insts, unit_begin, n_inst, counter, shape, ctas_per_sm, s);
}

}  // namespace agb
