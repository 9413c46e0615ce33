// Near-field kernel, FP64 twin: LOOP 2 of the reference (main.cpp:3030-3404)
// with every quantity in FP64 exactly as the reference, and the covalent map.
// (The FP32 production kernel is in near_rows.cu.)
#include <algorithm>

#include "near_exact.cuh"

namespace agb {

constexpr int NB_THREADS = 256;   // one thread per brick point
constexpr int NB_CHUNK = NB_CHUNK_MAX;   // candidates staged at once (most bricks need one chunk)
constexpr int NB_SEGS = NB_SEGS_MAX;

struct NearSmem {
    float4 pos[NB_CHUNK_MAX];
    int meta[NB_CHUNK_MAX], idx[NB_CHUNK_MAX];
    int hl[NB_CHUNK_MAX], nh;  // staged DS/D1 candidates (slots in this chunk), any order
    // per warp: slots of the staged atoms near that warp's points, in staged order
    unsigned short wl[NB_WARPS_MAX][NB_CHUNK_MAX];
    float wbox[NB_WARPS_MAX][6];  // per warp: its points' box in frame bins (lo xyz, hi xyz)
    int seg_start[NB_SEGS_MAX], seg_off[NB_SEGS_MAX + 1];
    int total;
};

// One 8x8x4 brick of points, one thread per point:
//   stage  candidate atoms of the cells within 8.05 A of the brick, with
//          frame-relative FP32 coordinates for the filters
//   A      closest DS/D1 atom per point (main.cpp:2986-3015) among the candidates:
//          any DS/D1 atom within 8.05 A of the point is one, so a best distance
//          <= 8 A is the global minimum; strict '<' in file order == lowest
//          index on a tie.  Where no DS/D1 atom is a candidate, no pair asks for it
//   B      pair terms of every candidate inside 8 A
// Only classes with an H-bond action evaluate the directional factors.
__global__ void __launch_bounds__(NB_THREADS, 2) k_near_exact(DevProblem p_, NearGroup g, NearPtrs ptr)
{
    __shared__ NearSmem S;
    __shared__ DevProblem p;  // functions take it by reference (see k_near)
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (tid == 0) p = p_;
    __syncthreads();
    constexpr int BX = 8, BY = 8, BZ = 4;
    const int b = blockIdx.x;
    const int nbx = (p.n1x + BX - 1) / BX, nby = (p.n1y + BY - 1) / BY;
    const int bx = b % nbx, by = (b / nbx) % nby, bz = b / (nbx * nby);
    const int ix = bx * BX + (lane & 3) + 4 * (wid & 1), iy = by * BY + ((lane >> 2) & 3) + 4 * ((wid >> 1) & 1),
              iz = bz * BZ + (lane >> 4) + 2 * (wid >> 2);
    const bool valid = ix < p.n1x && iy < p.n1y && iz < p.n1z;
    const long long lin = ((long long)iz * p.n1y + iy) * p.n1x + ix;
    const double sp128 = p.spacing * AG_A_DIV;
    const int ox = ((bx * BX) / FRAME_X) * FRAME_X + FRAME_X / 2, oy = ((by * BY) / FRAME_Y) * FRAME_Y + FRAME_Y / 2,
              oz = ((bz * BZ) / FRAME_Z) * FRAME_Z + FRAME_Z / 2;
    const double X0 = frame_origin_bins(ox, p.nex, sp128), Y0 = frame_origin_bins(oy, p.ney, sp128),
                 Z0 = frame_origin_bins(oz, p.nez, sp128);
    const float PX = frame_point_coord(ix - ox, sp128), PY = frame_point_coord(iy - oy, sp128),
                PZ = frame_point_coord(iz - oz, sp128);
    // FP64 point coordinates (main.cpp:2815-2859)
    const double cx = (double)(ix - p.nex) * p.spacing, cy = (double)(iy - p.ney) * p.spacing,
                 cz = (double)(iz - p.nez) * p.spacing;
    const bool need_h = p.n_atom_maps > 0;
    const bool need_pairs = g.ng > 0 || (g.write_special && p.dsolv_map >= 0);

    // candidate cells: brick bounding box grown by the candidate radius
    const double rc = AGB_NEAR_RADIUS;
    const int last[3] = {min(bx * BX + BX - 1, p.n1x - 1), min(by * BY + BY - 1, p.n1y - 1), min(bz * BZ + BZ - 1, p.n1z - 1)};
    const int first[3] = {bx * BX, by * BY, bz * BZ}, ne[3] = {p.nex, p.ney, p.nez}, nc[3] = {p.ncx, p.ncy, p.ncz};
    int c0[3], c1[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const double lo = (double)(first[i] - ne[i]) * p.spacing, hi = (double)(last[i] - ne[i]) * p.spacing;
        c0[i] = max(0, min(nc[i] - 1, (int)floor((lo - rc - p.cell0[i]) / p.cell_size)));
        c1[i] = max(0, min(nc[i] - 1, (int)floor((hi + rc - p.cell0[i]) / p.cell_size)));
    }
    const int nrow_y = c1[1] - c0[1] + 1;
    const int nseg_total = (need_pairs || need_h) ? nrow_y * (c1[2] - c0[2] + 1) : 0;

    auto layout_segments = [&](int sb, int nseg) {
        if (tid < nseg) {
            const int k = sb + tid, row = ((c0[2] + k / nrow_y) * p.ncy + c0[1] + k % nrow_y) * p.ncx;
            const int st = p.cell_start[row + c0[0]];
            S.seg_start[tid] = st;
            S.seg_off[tid + 1] = p.cell_start[row + c1[0] + 1] - st;
        }
        __syncthreads();
        if (tid == 0) {
            S.seg_off[0] = 0;
            for (int k = 0; k < nseg; k++) S.seg_off[k + 1] += S.seg_off[k];
            S.total = S.seg_off[nseg];
            S.nh = 0;
        }
        __syncthreads();
    };
    auto stage = [&](int k0, int n) {
        for (int i = tid; i < n; i += NB_THREADS) {
            const int c = k0 + i;
            int s = 0;
            while (S.seg_off[s + 1] <= c) s++;
            const int a = p.cell_atoms[S.seg_start[s] + (c - S.seg_off[s])];
            const int m = ptr.meta[a], hb = (m >> META_HB_SHIFT) & 7;
            S.idx[i] = a;
            S.meta[i] = m;
            S.pos[i] = make_float4(frame_atom_coord(p.x[a] * AG_A_DIV, X0), frame_atom_coord(p.y[a] * AG_A_DIV, Y0),
                                   frame_atom_coord(p.z[a] * AG_A_DIV, Z0), 0.f);
            if (hb == 1 || hb == 2) S.hl[atomicAdd(&S.nh, 1)] = i;
        }
        __syncthreads();
    };
    // visit every candidate chunk: fn(n) with the chunk staged
    auto for_each_chunk = [&](auto &&fn) {
        for (int sb = 0; sb < nseg_total; sb += NB_SEGS) {
            __syncthreads();
            layout_segments(sb, min(NB_SEGS, nseg_total - sb));
            const int total = S.total;
            for (int k0 = 0; k0 < total; k0 += NB_CHUNK) {
                const int n = min(NB_CHUNK, total - k0);
                if (k0) {
                    __syncthreads();
                    if (tid == 0) S.nh = 0;
                    __syncthreads();
                }
                stage(k0, n);
                fn(n);
            }
        }
    };
    // ---- A: closest DS/D1 hydrogen.  Only pairs with a D1 atom in range use it,
    // and such an atom is among the candidates.
    int ch = -1;
    if (need_h) {
        // the FP32 filter leaves the atoms whose distance can be the smallest;
        // the smallest seen so far only shrinks, so one pass is enough
        float best2 = 3.0e38f;
        double rmin = 999999.;
        for_each_chunk([&](int) {
            if (!valid) return;
            for (int k = 0; k < S.nh; k++) {
                const int j = S.hl[k];
                const float4 A = S.pos[j];
                const float dx = A.x - PX, dy = A.y - PY, dz = A.z - PZ;
                const float d2 = dx * dx + dy * dy + dz * dz;
                if (d2 > best2 * (1.0f + 2.0e-5f) + 4.0f) continue;
                best2 = fminf(best2, d2);
                const int a = S.idx[j];
                const double r = h_dist(p, a, cx, cy, cz);
                if (r < rmin || (r == rmin && a < ch)) { rmin = r; ch = a; }
            }
        });
    }

    // ---- B: pair terms
    double E[NG_MAX], hmin[NG_MM], hmax[NG_MM];
#pragma unroll
    for (int m = 0; m < NG_MAX; m++) E[m] = 0.;
#pragma unroll
    for (int m = 0; m < NG_MM; m++) { hmin[m] = 999999.; hmax[m] = -999999.; }
    uint32_t hflag = 0;
    double D1 = 0., D2 = 0.;
    unsigned n_near = 0;
    if (need_pairs) {
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
        unsigned short *wl = S.wl[wid];
        for_each_chunk([&](int n) {
            int cnt = 0;
            for (int j0 = 0; j0 < n; j0 += 32) {
                const int jj = j0 + lane;
                bool keep = false;
                if (jj < n) {
                    const float4 A = S.pos[jj];
                    const float *w = S.wbox[wid];
                    const float ex = fmaxf(fmaxf(w[0] - A.x, A.x - w[3]), 0.f);
                    const float ey = fmaxf(fmaxf(w[1] - A.y, A.y - w[4]), 0.f);
                    const float ez = fmaxf(fmaxf(w[2] - A.z, A.z - w[5]), 0.f);
                    // LOOP 2 skips disordered hydrogens (main.cpp:3052)
                    keep = ex * ex + ey * ey + ez * ez <= keep2 && !(S.meta[jj] & META_SKIP_AD4);
                }
                const unsigned m = __ballot_sync(0xffffffffu, keep);
                if (keep) wl[cnt + __popc(m & ((1u << lane) - 1u))] = (unsigned short)jj;
                cnt += __popc(m);
            }
            __syncwarp();
            if (!valid) return;
            for (int k = 0; k < cnt; k++) {
                const int j = wl[k];
                // the FP32 distance is off by less than 2 bins
                const float4 A = S.pos[j];
                const float fx = A.x - PX, fy = A.y - PY, fz = A.z - PZ;
                if (fx * fx + fy * fy + fz * fz > keep2) continue;
                const int ia = S.idx[j], meta = S.meta[j];
                double d0, d1, d2;
                const double r = loop2_dist(p, ia, cx, cy, cz, d0, d1, d2);
                if (r > AG_NBC) continue;
                n_near++;
                const int bin = __double2int_rz(__dmul_rn(r, (double)AG_A_DIV));
                const double sol = p.sol_fn[bin];
                D1 += p.vol[ia] * sol;
                D2 += (p.solpar[ia] + p.solpar_q * fabs(p.q[ia])) * sol;
                if (g.ng == 0) continue;
                const int hb = (meta >> META_HB_SHIFT) & 7, ta = meta & META_TYPE_MASK;
                const bool dis = (meta & META_DIS) != 0;
                const float *Trow = ptr.vdwT + ((size_t)ta * AG_NEINT + min(bin, AG_NEINT - 1)) * ptr.mpad + g.col0;
                Row8 T8[NG_MAX / 8];
#pragma unroll
                for (int k8 = 0; k8 < NG_MAX / 8; k8++)
                    if (8 * k8 < g.ng) T8[k8] = load_row8(Trow + 8 * k8);
                auto T_of = [&](int m) { const float2 v = T8[m / 8].p[(m / 2) % 4]; return (double)((m & 1) ? v.y : v.x); };
                if ((g.plain_hb >> hb) & 1u) {  // every map a plain sum for this class (most atoms)
#pragma unroll
                    for (int m = 0; m < NG_MAX; m++)
                        if (8 * (m / 8) < g.ng) E[m] += T_of(m);
                    continue;
                }
                PairQ<double> q;
                angular_exact(p, ia, ch, d0, d1, d2, r, q);
                const float *Hrow = Trow;
                if (g.has_hrow && dis && p.hydrogen_type >= 0) {
                    int ih = __double2int_rz(__dmul_rn(__dsub_rn(r, 1.10), (double)AG_A_DIV));
                    ih = min(max(ih, 0), AG_NEINT - 1);
                    Hrow = ptr.vdwT + ((size_t)p.hydrogen_type * AG_NEINT + ih) * ptr.mpad + g.col0;
                }
                const unsigned long long aw = g.actw[hb];
#pragma unroll
                for (int m = 0; m < NG_MAX; m++) {
                    if (m >= g.ng) break;
                    const int act = (int)((aw >> (3 * m)) & 7ull);
                    if (act == ACT_SKIP) continue;
                    const double T = T_of(m);
                    if (act == ACT_PLAIN) { E[m] += T; continue; }
                    double rsph = T / 100.;
                    rsph = rsph > 0. ? rsph : 0.;
                    rsph = rsph < 1. ? rsph : 1.;
                    if (act == ACT_SUMA) {
                        const double Th = dis ? (double)__ldg(Hrow + m) : T;
                        E[m] += Th * q.Hramp * (q.racc + (1. - q.racc) * rsph);
                    } else if (act == ACT_MMD && dis) {
                        E[m] += (double)__ldg(Hrow + m) * q.Hramp * (q.rdon + (1. - q.rdon) * rsph);
                    } else if (m < NG_MM) {  // min/max maps are placed first by the host
                        const double f = (act == ACT_MMA) ? q.racc : q.rdon;
                        const double v = T * (f + (1. - f) * rsph);
                        hmin[m < NG_MM ? m : 0] = hmin[m < NG_MM ? m : 0] < v ? hmin[m < NG_MM ? m : 0] : v;
                        hmax[m < NG_MM ? m : 0] = hmax[m < NG_MM ? m : 0] > v ? hmax[m < NG_MM ? m : 0] : v;
                        hflag |= 1u << m;
                    }
                }
            }
        });
    }

    // finalise (main.cpp:3420-3431) and store
    if (valid) {
#pragma unroll
        for (int m = 0; m < NG_MAX; m++) {
            if (m >= g.ng) break;
            double v = E[m];
            if (m < NG_MM && (hflag & (1u << m))) {
                const double lo = hmin[m < NG_MM ? m : 0], hi = hmax[m < NG_MM ? m : 0];
                v += lo + (hi > 0. ? hi : 0.);
            }
            v += g.sp[m] * D1 + g.vp[m] * D2;
            ptr.out64[(size_t)g.out_map[m] * (size_t)p.P + (size_t)lin] = g.cov[m] ? ptr.cov_map[lin] : v;
        }
        if (g.write_special && p.dsolv_map >= 0)
            ptr.out64[(size_t)p.dsolv_map * (size_t)p.P + (size_t)lin] = p.solpar_q * D1;
    }
    if (ptr.counters) {
        const unsigned n = __reduce_add_sync(0xffffffffu, n_near);
        if (lane == 0 && n) atomicAdd(ptr.counters + 0, (unsigned long long)n);
    }
}

// Covalent map(s), main.cpp:2866-2879, in FP64 (a handful of flops per point).
__global__ void k_covalent(DevProblem p, double *__restrict__ cov)
{
    const long long lin = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (lin >= p.P) return;
    const int ix = (int)(lin % p.n1x), iy = (int)((lin / p.n1x) % p.n1y), iz = (int)(lin / ((long long)p.n1x * p.n1y));
    const double d0 = __dsub_rn(p.cov_pos[0], (double)(ix - p.nex) * p.spacing);
    const double d1 = __dsub_rn(p.cov_pos[1], (double)(iy - p.ney) * p.spacing);
    const double d2 = __dsub_rn(p.cov_pos[2], (double)(iz - p.nez) * p.spacing);
    double rcov = __ddiv_rn(__dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2))),
                            p.cov_half_width);
    if (rcov < APPROX_ZERO_D) rcov = APPROX_ZERO_D;
    cov[lin] = __dmul_rn(p.cov_barrier, __dsub_rn(1., exp(__dmul_rn(__dmul_rn(log(0.5), rcov), rcov))));
}

int near_bricks(const DevProblem &p, int shape)
{
    int bx = 8, by = 8, bz = 4;
    if (shape == 1) { by = 4; bz = 8; }
    else if (shape == 2) { bx = 4; bz = 8; }
    return ((p.n1x + bx - 1) / bx) * ((p.n1y + by - 1) / by) * ((p.n1z + bz - 1) / bz);
}

cudaError_t launch_covalent(const DevProblem &p, double *cov, cudaStream_t s)
{
    k_covalent<<<(unsigned)((p.P + 255) / 256), 256, 0, s>>>(p, cov);
    return cudaGetLastError();
}

cudaError_t launch_near_exact(const DevProblem &p, const NearGroup &g, const NearPtrs &ptr, cudaStream_t s)
{
    k_near_exact<<<(unsigned)near_bricks(p, 0), NB_THREADS, 0, s>>>(p, g, ptr);
    return cudaGetLastError();
}

}  // namespace agb
