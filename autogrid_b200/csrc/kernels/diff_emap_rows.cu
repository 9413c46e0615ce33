// Differentiable mode, electrostatic map in FP32: LOOP 1 of main.cpp:2940-2982
// with the dielectric table read by linear interpolation (kernels/diff.h):
//     e(p) = sum_a q_a F(r_pa),   F(r) = T(A_DIV r) / max(r, 0.5),
// T the table of eps factor * coeff_estat, constant past its last bin.
// (The FP64 twin is in diff_emap.cu.)
//   k_elin      forward; sums of an atom chunk per point
//   k_elin_adj  adjoint: dL/dq_a = sum_p g(p) F(r),
//               dL/dx_a = sum_p g(p) q_a F'(r) (x_a - x_p) / r
// Both tile the grid in the far-field kernel's frames of 32x8x8 points and
// work like it (emap.cu): coordinates relative to the frame in table bins, a
// thread holds 16 points of two x-rows, a warp's points are a compact block so
// that its gathers of the table meet few bank conflicts, and each half of a
// block takes every other run of 32 atoms.  Value and step of a bin are two
// 32-bit gathers from separate arrays: 2.8 wavefronts each on that block,
// where a 64-bit gather of 32 points in a row took 8.  The forward reads
// the value of the next bin instead of the step, one table less.
// The adjoint sums an atom's four derivatives over a warp's 512 points in
// registers, then by shuffles, then by one FP64 atomic add each.
// A quarter of the gathers go through the texture unit, which has a pipe of its
// own (ER_TEX).  Atoms within 0.5 A of a row's line have a code path apart
// (1/max(r, 0.5)); inside the common one it cost 5 instructions per pair.
// 4,000 atoms, 61^3 points: forward 0.80 -> 0.57 ms (shared-memory pipe 88%
// busy), adjoint 1.02 -> 0.85 ms (67%, issue 61%, FMA 59%), against one point
// or one atom per thread with 64-bit gathers.  Without the texture unit 0.69
// and 0.98 ms; sums of two atoms at a time over the warp: no faster.
#include <algorithm>
#include <type_traits>

#include "agb_device.cuh"
#include "diff.h"
#include "warp_sums.cuh"

namespace agb {

namespace {

constexpr int ER_THREADS = 256, ER_GROUP = ER_THREADS / 2;  // a group holds a frame's points
constexpr int ER_TILE = 512;
constexpr int ER_CTAS = 2;
constexpr int ER_PAIRS = FRAME_X / 8;  // pairs of points per row and thread
constexpr int ER_TAB = AG_NDIEL + 4;   // floats of a table in shared memory
constexpr float ER_MIN_T2 = 1.0e-12f * AG_A_DIV * AG_A_DIV;  // r >= 1e-6 A
// Packed pairs (of 8 per atom and thread) whose table entries come through
// the texture unit: a gather of (value, step) takes it 12.6 clocks, beside the
// shared-memory pipe's 5.5 for two 32-bit gathers.  0, 1, 2, 3 of 8: forward and
// adjoint step (with the other kernels) 2.47, 2.37, 2.30, 2.33 ms.
constexpr int ER_TEX = 2;
constexpr float ER_LAST = (float)(AG_NDIEL - 1);

__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }

__device__ __forceinline__ float lds(uint32_t addr)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}

// A thread's place in a frame: rows y and y + 4 of one plane, x = tx + 8j and
// tx + 8j + 4 (negated frame coordinates in bins).
struct ErPoints {
    float2 npx[ER_PAIRS], npy;
    float npz;
    int ix, iy, iz;    // first point of the first row
    bool warp_in;      // some row and plane of the warp lie inside the box
};
__device__ __forceinline__ ErPoints er_points(const DiffArgs &a, int f)
{
    const int nfx = (a.n1x + FRAME_X - 1) / FRAME_X, nfy = (a.n1y + FRAME_Y - 1) / FRAME_Y;
    const int lane = threadIdx.x & 31, v = (threadIdx.x >> 5) & 3;
    const int tx = lane & 3, ty = (lane >> 2) & 3, tz = (lane >> 4) + 2 * v;
    const double bin = a.spacing * AG_A_DIV;
    ErPoints p;
    const int oz = f / (nfx * nfy) * FRAME_Z;
    p.ix = f % nfx * FRAME_X + tx;
    p.iy = f / nfx % nfy * FRAME_Y + ty;
    p.iz = oz + tz;
    p.warp_in = oz + 2 * v < a.n1z;
    // a point of the frame past the box takes the coordinates of the box's last:
    // the distances are then those of points in the box, and its weight of 0
    // meets no table value (which may be no number) that these do not
    const int lx = a.n1x - 1 - (p.ix - tx), ly = a.n1y - 1 - (p.iy - ty), lz = a.n1z - 1 - oz;
#pragma unroll
    for (int j = 0; j < ER_PAIRS; j++)
        p.npx[j] = make_float2(-frame_point_coord(min(tx + 8 * j, lx), bin), -frame_point_coord(min(tx + 8 * j + 4, lx), bin));
    p.npy = make_float2(-frame_point_coord(min(ty, ly), bin), -frame_point_coord(min(ty + 4, ly), bin));
    p.npz = -frame_point_coord(min(tz, lz), bin);
    return p;
}

// Stage atoms [a0, a0 + n): frame-relative (Y, Z, X) in bins and the charge.
__device__ __forceinline__ void er_stage(const DiffArgs &a, const ConfView &v, int f, int a0, int n, float4 *s_atom)
{
    const int nfx = (a.n1x + FRAME_X - 1) / FRAME_X, nfy = (a.n1y + FRAME_Y - 1) / FRAME_Y;
    const double bin = a.spacing * AG_A_DIV;
    const double X0 = frame_origin_bins(f % nfx * FRAME_X, a.nex, bin), Y0 = frame_origin_bins(f / nfx % nfy * FRAME_Y, a.ney, bin),
                 Z0 = frame_origin_bins(f / (nfx * nfy) * FRAME_Z, a.nez, bin);
    for (int i = threadIdx.x; i < n; i += ER_THREADS)
        s_atom[i] = make_float4(frame_atom_coord(v.y[a0 + i] * AG_A_DIV, Y0), frame_atom_coord(v.z[a0 + i] * AG_A_DIV, Z0),
                                frame_atom_coord(v.x[a0 + i] * AG_A_DIV, X0), (float)v.q[a0 + i]);
}

// The value column of the (value, step) table, its last entry repeated, and
// (steps != null) the step column.
__device__ __forceinline__ void er_table(const float2 *gtab, float *vals, float *steps)
{
    for (int i = threadIdx.x; i < ER_TAB; i += ER_THREADS) {
        const float2 e = __ldg(gtab + min(i, AG_NDIEL - 1));
        vals[i] = e.x;
        if (steps) steps[i] = e.y;
    }
}

// Distance in bins, clamped to the last bin, as whole bins (float bits minus
// those of 2^23) and fraction.
__device__ __forceinline__ void er_bin(float2 t2, float2 rs, float2 &frac, uint32_t &b0, uint32_t &b1)
{
    float2 t = __fmul2_rn(t2, rs);
    t = make_float2(fminf(t.x, ER_LAST), fminf(t.y, ER_LAST));
    const float2 m = __fadd2_rz(t, both(8388608.f));
    frac = __fadd2_rn(t, __fadd2_rn(both(8388608.f), make_float2(-m.x, -m.y)));
    b0 = __float_as_uint(m.x);
    b1 = __float_as_uint(m.y);
}

__global__ void __launch_bounds__(ER_THREADS, ER_CTAS)
k_elin(DiffArgs a, const float2 *__restrict__ gtab, cudaTextureObject_t tex, int chunk_atoms, float *__restrict__ out, long long out_conf,
       long long out_chunk)
{
    extern __shared__ float4 er_smem[];
    float4 *s_atom = er_smem;
    float *s_val = (float *)(er_smem + ER_TILE);
    er_table(gtab, s_val, nullptr);
    const ConfView v = conf_view(a, DiffGrads{}, blockIdx.z);
    const ErPoints P = er_points(a, blockIdx.x);
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(s_val) - (MAGIC_BITS << 2);
    const int half = threadIdx.x / ER_GROUP;
    const int a_begin = blockIdx.y * chunk_atoms, a_end = min(a.n_atoms, a_begin + chunk_atoms);
    float2 tot[2][ER_PAIRS];
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
        for (int j = 0; j < ER_PAIRS; j++) tot[r][j] = both(0.f);
    for (int t0 = a_begin; t0 < a_end; t0 += ER_TILE) {
        const int na = min(ER_TILE, a_end - t0);
        __syncthreads();
        er_stage(a, v, blockIdx.x, t0, na, s_atom);
        __syncthreads();
        if (!P.warp_in) continue;
        float2 acc[2][ER_PAIRS];
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
            for (int j = 0; j < ER_PAIRS; j++) acc[r][j] = both(0.f);
        for (int ib = 32 * half; ib < na; ib += 64) {
            const int nb = min(32, na - ib);
#pragma unroll 1
            for (int ii = 0; ii < nb; ii++) {
                const float4 A = s_atom[ib + ii];
                const float2 dy = __fadd2_rn(both(A.x), P.npy);
                const float dz = A.y + P.npz;
                const float2 s = __ffma2_rn(dy, dy, both(__fmaf_rn(dz, dz, TINY_T2)));
                // 1/max(r, 0.5) differs from 1/r only for atoms within 64 bins of a row
                const bool close = __any_sync(0xffffffffu, fminf(s.x, s.y) < 4096.f);
                auto pairs = [&](auto near) {
                    constexpr bool CLOSE = decltype(near)::value;
                    const float2 q2 = both(A.w);
                    float2 tx[ER_TEX], ty[ER_TEX], tf[ER_TEX], tw[ER_TEX];
#pragma unroll
                    for (int j = 0; j < ER_PAIRS; j++) {
                        const float2 dx = __fadd2_rn(both(A.z), P.npx[j]);
#pragma unroll
                        for (int r = 0; r < 2; r++) {
                            const int n = 2 * j + r;
                            float2 t2 = __ffma2_rn(dx, dx, both(r ? s.y : s.x));
                            if (CLOSE) t2 = make_float2(fmaxf(t2.x, ER_MIN_T2), fmaxf(t2.y, ER_MIN_T2));
                            float2 rs = make_float2(rsqrt_approx(t2.x), rsqrt_approx(t2.y)), f;
                            uint32_t b0, b1;
                            er_bin(t2, rs, f, b0, b1);
                            if (n < ER_TEX) {
                                tx[n < ER_TEX ? n : 0] = tex1Dfetch<float2>(tex, (int)(b0 - MAGIC_BITS));
                                ty[n < ER_TEX ? n : 0] = tex1Dfetch<float2>(tex, (int)(b1 - MAGIC_BITS));
                            }
                            if (CLOSE) rs = make_float2(fminf(rs.x, 0.015625f), fminf(rs.y, 0.015625f));
                            const float2 w = __fmul2_rn(q2, rs);
                            if (n < ER_TEX) {
                                tf[n < ER_TEX ? n : 0] = f;
                                tw[n < ER_TEX ? n : 0] = w;
                                continue;
                            }
                            const uint32_t a0 = base + (b0 << 2), a1 = base + (b1 << 2);
                            const float2 v0 = make_float2(lds(a0), lds(a1)), v1 = make_float2(lds(a0 + 4), lds(a1 + 4));
                            const float2 T = __ffma2_rn(f, __fadd2_rn(v1, make_float2(-v0.x, -v0.y)), v0);
                            acc[r][j] = __ffma2_rn(w, T, acc[r][j]);
                        }
                    }
#pragma unroll
                    for (int n = 0; n < ER_TEX; n++)
                        acc[n & 1][n >> 1] = __ffma2_rn(tw[n], __ffma2_rn(tf[n], make_float2(tx[n].y, ty[n].y), make_float2(tx[n].x, ty[n].x)),
                                                        acc[n & 1][n >> 1]);
                };
                if (close) pairs(std::true_type{});
                else pairs(std::false_type{});
            }
        }
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
            for (int j = 0; j < ER_PAIRS; j++) tot[r][j] = __fadd2_rn(tot[r][j], acc[r][j]);
    }
    // the second half's sums through the atom tile
    static_assert(ER_TILE * sizeof(float4) >= 16 * ER_GROUP * sizeof(float), "the tile holds one half's sums");
    float *ex = (float *)s_atom + (threadIdx.x & (ER_GROUP - 1));
    __syncthreads();
    if (half)
#pragma unroll
        for (int k = 0; k < 2 * ER_PAIRS; k++) {
            ex[(2 * k) * ER_GROUP] = tot[k / ER_PAIRS][k % ER_PAIRS].x;
            ex[(2 * k + 1) * ER_GROUP] = tot[k / ER_PAIRS][k % ER_PAIRS].y;
        }
    __syncthreads();
    if (half || P.iz >= a.n1z) return;
    out += blockIdx.z * out_conf + blockIdx.y * out_chunk;
#pragma unroll
    for (int r = 0; r < 2; r++) {
        if (P.iy + 4 * r >= a.n1y) continue;
        float *row = out + ((size_t)P.iz * a.n1y + P.iy + 4 * r) * a.n1x + P.ix;
#pragma unroll
        for (int j = 0; j < ER_PAIRS; j++) {
            const int k = r * ER_PAIRS + j;
            if (P.ix + 8 * j < a.n1x) row[8 * j] = (float)AG_A_DIV * (tot[r][j].x + ex[2 * k * ER_GROUP]);
            if (P.ix + 8 * j + 4 < a.n1x) row[8 * j + 4] = (float)AG_A_DIV * (tot[r][j].y + ex[(2 * k + 1) * ER_GROUP]);
        }
    }
}

// The e map from its atom chunks' sums, in chunk order.
__global__ void __launch_bounds__(256)
k_elin_sum(const float *__restrict__ partial, int chunks, long long P, float *__restrict__ emap, long long map_conf)
{
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= P) return;
    partial += (long long)blockIdx.y * chunks * P;
    float e = 0.f;
    for (int c = 0; c < chunks; c++) e += partial[c * P + i];
    emap[blockIdx.y * map_conf + i] = e;
}

__global__ void __launch_bounds__(ER_THREADS, ER_CTAS)
k_elin_adj(DiffArgs a, const float2 *__restrict__ gtab, cudaTextureObject_t tex, int chunk_atoms,
           const float *__restrict__ g_e, DiffGrads g_all)
{
    extern __shared__ float4 er_smem[];
    float4 *s_atom = er_smem;
    float *s_val = (float *)(er_smem + ER_TILE), *s_step = s_val + ER_TAB;
    er_table(gtab, s_val, s_step);
    const ConfView v = conf_view(a, g_all, blockIdx.z);
    const ErPoints P = er_points(a, blockIdx.x);
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(s_val) - (MAGIC_BITS << 2);
    const int half = threadIdx.x / ER_GROUP, lane = threadIdx.x & 31;
    const int a_begin = blockIdx.y * chunk_atoms, a_end = min(a.n_atoms, a_begin + chunk_atoms);
    // the points' weights (0 outside the box)
    float2 w[2][ER_PAIRS];
    g_e += (long long)blockIdx.z * a.n_maps_out * a.P;
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const bool row_in = P.iy + 4 * r < a.n1y && P.iz < a.n1z;
        const float *row = g_e + ((size_t)P.iz * a.n1y + P.iy + 4 * r) * a.n1x + P.ix;
#pragma unroll
        for (int j = 0; j < ER_PAIRS; j++)
            w[r][j] = make_float2(row_in && P.ix + 8 * j < a.n1x ? row[8 * j] : 0.f,
                                  row_in && P.ix + 8 * j + 4 < a.n1x ? row[8 * j + 4] : 0.f);
    }
    for (int t0 = a_begin; t0 < a_end; t0 += ER_TILE) {
        const int na = min(ER_TILE, a_end - t0);
        __syncthreads();
        er_stage(a, v, blockIdx.x, t0, na, s_atom);
        __syncthreads();
        if (!P.warp_in) continue;
        for (int ib = 32 * half; ib < na; ib += 64) {
            const int nb = min(32, na - ib);
#pragma unroll 1
            for (int ii = 0; ii < nb; ii++) {
                const float4 A = s_atom[ib + ii];
                const float2 dy = __fadd2_rn(both(A.x), P.npy);
                const float dz = A.y + P.npz;
                const float2 s = __ffma2_rn(dy, dy, both(__fmaf_rn(dz, dz, TINY_T2)));
                const bool close = __any_sync(0xffffffffu, fminf(s.x, s.y) < 4096.f);
                // in bins, with inv = min(1/r, 1/64): sum of w inv T, and of
                // k = w inv / r (T' - T / r) (without T / r where r < 64), k dx
                float2 aq = both(0.f), ax = both(0.f), k0 = both(0.f), k1 = both(0.f);
                auto pairs = [&](auto near) {
                    constexpr bool CLOSE = decltype(near)::value;
                    auto add = [&](int r, float2 h, float2 rs, float2 T, float2 d, float2 dx) {
                        float2 out = rs;
                        if (CLOSE) out = make_float2(rs.x < 0.015625f ? rs.x : 0.f, rs.y < 0.015625f ? rs.y : 0.f);
                        aq = __ffma2_rn(h, T, aq);
                        const float2 u = __fmul2_rn(T, out);
                        const float2 k = __fmul2_rn(__fmul2_rn(h, rs), __fadd2_rn(d, make_float2(-u.x, -u.y)));
                        ax = __ffma2_rn(k, dx, ax);
                        if (r) k1 = __fadd2_rn(k1, k);
                        else k0 = __fadd2_rn(k0, k);
                    };
                    float2 tx[ER_TEX], ty[ER_TEX], tf[ER_TEX], th[ER_TEX], trs[ER_TEX];
#pragma unroll
                    for (int j = 0; j < ER_PAIRS; j++) {
                        const float2 dx = __fadd2_rn(both(A.z), P.npx[j]);
#pragma unroll
                        for (int r = 0; r < 2; r++) {
                            const int n = 2 * j + r;
                            float2 t2 = __ffma2_rn(dx, dx, both(r ? s.y : s.x));
                            if (CLOSE) t2 = make_float2(fmaxf(t2.x, ER_MIN_T2), fmaxf(t2.y, ER_MIN_T2));
                            const float2 rs = make_float2(rsqrt_approx(t2.x), rsqrt_approx(t2.y));
                            float2 f, inv = rs;
                            uint32_t b0, b1;
                            er_bin(t2, rs, f, b0, b1);
                            if (n < ER_TEX) {
                                tx[n < ER_TEX ? n : 0] = tex1Dfetch<float2>(tex, (int)(b0 - MAGIC_BITS));
                                ty[n < ER_TEX ? n : 0] = tex1Dfetch<float2>(tex, (int)(b1 - MAGIC_BITS));
                            }
                            if (CLOSE) inv = make_float2(fminf(rs.x, 0.015625f), fminf(rs.y, 0.015625f));
                            const float2 h = __fmul2_rn(w[r][j], inv);
                            if (n < ER_TEX) {
                                tf[n < ER_TEX ? n : 0] = f;
                                th[n < ER_TEX ? n : 0] = h;
                                trs[n < ER_TEX ? n : 0] = rs;
                                continue;
                            }
                            const uint32_t a0 = base + (b0 << 2), a1 = base + (b1 << 2);
                            const float2 d = make_float2(lds(a0 + 4 * ER_TAB), lds(a1 + 4 * ER_TAB));
                            add(r, h, rs, __ffma2_rn(f, d, make_float2(lds(a0), lds(a1))), d, dx);
                        }
                    }
#pragma unroll
                    for (int n = 0; n < ER_TEX; n++) {
                        const float2 d = make_float2(tx[n].y, ty[n].y);
                        add(n & 1, th[n], trs[n], __ffma2_rn(tf[n], d, make_float2(tx[n].x, ty[n].x)), d,
                            __fadd2_rn(both(A.z), P.npx[n >> 1]));
                    }
                };
                if (close) pairs(std::true_type{});
                else pairs(std::false_type{});
                const float s0 = k0.x + k0.y, s1 = k1.x + k1.y;
                float sum[4] = {ax.x + ax.y, fmaf(dy.x, s0, dy.y * s1), dz * (s0 + s1), aq.x + aq.y};
                const float total = warp_sums(sum, lane);
                if ((lane & 7) == 0) {
                    const int n = lane >> 3, at = t0 + ib + ii;
                    const float c = n < 3 ? A.w * (float)(AG_A_DIV * AG_A_DIV) : (float)AG_A_DIV;
                    atomicAdd(n < 3 ? v.g.xyz + 3LL * at + n : v.g.q + at, (double)(total * c));
                }
            }
        }
    }
}

long long er_frames(const DiffArgs &a)
{
    return (long long)((a.n1x + FRAME_X - 1) / FRAME_X) * ((a.n1y + FRAME_Y - 1) / FRAME_Y) * ((a.n1z + FRAME_Z - 1) / FRAME_Z);
}

// Atoms per block: enough blocks for 4 waves, at least 128 atoms (a table load
// per block), whole pairs of 32-atom runs.
int er_chunk_atoms(const DiffArgs &a)
{
    const long long units = er_frames(a) * a.n_conf, want = 4LL * ER_CTAS * current_device_sms();
    const long long chunks = std::max(1LL, std::min<long long>((want + units - 1) / units, a.n_atoms / 128));
    return (int)(((a.n_atoms + chunks - 1) / chunks + 63) / 64 * 64);
}

size_t er_smem_bytes(int tables) { return ER_TILE * sizeof(float4) + (size_t)tables * ER_TAB * sizeof(float); }

}  // namespace

int elin_chunks(const DiffArgs &a)
{
    const int c = er_chunk_atoms(a);
    return a.n_atoms > 0 ? (a.n_atoms + c - 1) / c : 1;
}

cudaError_t prepare_elin()
{
    cudaError_t e = cudaFuncSetAttribute(k_elin, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)er_smem_bytes(1));
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_elin_adj, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)er_smem_bytes(2));
}

cudaError_t launch_elin(const DiffArgs &a, const void *eps, cudaTextureObject_t tex, float *emap, float *partial,
                        cudaStream_t s)
{
    if (a.P == 0) return cudaSuccess;
    const int chunks = elin_chunks(a);
    const long long map_conf = (long long)a.n_maps_out * a.P;
    const dim3 grid((unsigned)er_frames(a), (unsigned)chunks, (unsigned)a.n_conf);
    if (chunks == 1) {
        k_elin<<<grid, ER_THREADS, er_smem_bytes(1), s>>>(a, (const float2 *)eps, tex, er_chunk_atoms(a), emap, map_conf, 0);
        return cudaGetLastError();
    }
    k_elin<<<grid, ER_THREADS, er_smem_bytes(1), s>>>(a, (const float2 *)eps, tex, er_chunk_atoms(a), partial, chunks * a.P, a.P);
    k_elin_sum<<<dim3((unsigned)((a.P + 255) / 256), (unsigned)a.n_conf), 256, 0, s>>>(partial, chunks, a.P, emap, map_conf);
    return cudaGetLastError();
}

cudaError_t launch_elin_adj(const DiffArgs &a, const void *eps, cudaTextureObject_t tex, const float *g_e, DiffGrads g,
                            cudaStream_t s)
{
    if (a.n_atoms == 0 || a.P == 0) return cudaSuccess;
    const dim3 grid((unsigned)er_frames(a), (unsigned)elin_chunks(a), (unsigned)a.n_conf);
    k_elin_adj<<<grid, ER_THREADS, er_smem_bytes(2), s>>>(a, (const float2 *)eps, tex, er_chunk_atoms(a), g_e, g);
    return cudaGetLastError();
}

}  // namespace agb
