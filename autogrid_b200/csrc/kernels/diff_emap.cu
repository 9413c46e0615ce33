// Differentiable mode, electrostatic map, FP64 twin: LOOP 1 of
// main.cpp:2940-2982 with the dielectric table read by linear interpolation
// (kernels/diff.h):
//     e(p) = sum_a q_a F(r_pa),   F(r) = T(A_DIV r) / max(r, 0.5),
// T the table of eps factor * coeff_estat, constant past its last bin.
// (The FP32 kernels are in diff_emap_rows.cu.)
//   k_emap_lin      forward: 256 points per block, atoms staged through shared
//                   memory, the table resident in shared memory;
//   k_emap_lin_adj  adjoint: 256 atoms per block, points (with dL/de) staged
//                   through shared memory,
//                     dL/dq_a = sum_p g(p) F(r),
//                     dL/dx_a = sum_p g(p) q_a F'(r) (x_a - x_p) / r.
// The table takes 128 KB, so one block fits an SM; its 1,024 threads share each
// point's (atom's) sum out among EL_SPLIT of them, which meet in shared memory.
// With a thread for each, 8 warps per SM, the kernels waited on the chain of
// the distance's FP64 operations: 1,000 atoms x 33^3 points forward 153 -> 74
// us, adjoint 163 -> 97 us.
#include <algorithm>

#include "agb_device.cuh"
#include "diff.h"

namespace agb {

namespace {

constexpr int EL_SPLIT = 4, EL_OWNERS = 256, EL_THREADS = EL_SPLIT * EL_OWNERS, EL_TILE = 1024;

// Table value and slope at x = A_DIV r, and 1/r, from r^2 (FP64 reciprocal
// square root, about 2 ulp).
__device__ __forceinline__ void lin_eval(const R2<double> *tab, double r2, double &T, double &slope, double &rs)
{
    r2 = fmax(r2, 1.0e-12);
    rs = rsqrt_f64(r2);
    const double x = r2 * rs * (double)AG_A_DIV;
    const int b = min((int)x, AG_NDIEL - 1);
    const R2<double> e = tab[b];
    T = e.v + (x - (double)b) * e.d;
    slope = e.d * (double)AG_A_DIV;
}

__device__ __forceinline__ double point_coord(int i, int ne, double spacing) { return (double)(i - ne) * spacing; }

__global__ void __launch_bounds__(EL_THREADS) k_emap_lin(DiffArgs a, const R2<double> *__restrict__ gtab, double *__restrict__ emap)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R2<double> *s_tab = reinterpret_cast<R2<double> *>(smem_raw);
    double4 *s_atom = reinterpret_cast<double4 *>(smem_raw + sizeof(R2<double>) * AG_NDIEL);
    for (int i = threadIdx.x; i < AG_NDIEL; i += EL_THREADS) s_tab[i] = gtab[i];
    const ConfView v = conf_view(a, DiffGrads{}, blockIdx.y);  // blockIdx.y: conformer
    emap += (long long)blockIdx.y * a.n_maps_out * a.P;

    const int owner = threadIdx.x % EL_OWNERS, part = threadIdx.x / EL_OWNERS;
    const long long lin = (long long)blockIdx.x * EL_OWNERS + owner;
    const bool valid = lin < a.P;
    const long long l = valid ? lin : 0;
    const int ix = (int)(l % a.n1x), iy = (int)((l / a.n1x) % a.n1y), iz = (int)(l / ((long long)a.n1x * a.n1y));
    const double cx = point_coord(ix, a.nex, a.spacing), cy = point_coord(iy, a.ney, a.spacing),
            cz = point_coord(iz, a.nez, a.spacing);
    double e = 0;
    for (int a0 = 0; a0 < a.n_atoms; a0 += EL_TILE) {
        const int na = min(EL_TILE, a.n_atoms - a0);
        __syncthreads();
        for (int i = threadIdx.x; i < na; i += EL_THREADS) {
            double4 t;
            t.x = v.x[a0 + i]; t.y = v.y[a0 + i]; t.z = v.z[a0 + i]; t.w = v.q[a0 + i];
            s_atom[i] = t;
        }
        __syncthreads();
        double acc = 0;
#pragma unroll 4
        for (int i = part; i < na; i += EL_SPLIT) {
            const double4 at = s_atom[i];
            const double dx = at.x - cx, dy = at.y - cy, dz = at.z - cz;
            double T, slope, rs;
            lin_eval(s_tab, dx * dx + dy * dy + dz * dz, T, slope, rs);
            acc += at.w * (T * (rs < 2 ? rs : 2));
        }
        e += acc;
    }
    double *sum = (double *)s_atom + owner;
    __syncthreads();
    if (part) sum[(part - 1) * EL_OWNERS] = e;
    __syncthreads();
    if (part || !valid) return;
    for (int k = 0; k < EL_SPLIT - 1; k++) e += sum[k * EL_OWNERS];
    emap[lin] = e;
}

__global__ void __launch_bounds__(EL_THREADS)
k_emap_lin_adj(DiffArgs a, const R2<double> *__restrict__ gtab, const double *__restrict__ g_e, DiffGrads g_all,
               int points_per_block)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R2<double> *s_tab = reinterpret_cast<R2<double> *>(smem_raw);
    double4 *s_pt = reinterpret_cast<double4 *>(smem_raw + sizeof(R2<double>) * AG_NDIEL);
    for (int i = threadIdx.x; i < AG_NDIEL; i += EL_THREADS) s_tab[i] = gtab[i];
    const ConfView cv = conf_view(a, g_all, blockIdx.z);  // blockIdx.z: conformer
    const DiffGrads g = cv.g;
    g_e += (long long)blockIdx.z * a.n_maps_out * a.P;

    const int owner = threadIdx.x % EL_OWNERS, part = threadIdx.x / EL_OWNERS;
    const int at = blockIdx.x * EL_OWNERS + owner;
    const bool valid = at < a.n_atoms;
    const double xa = valid ? cv.x[at] : 0, ya = valid ? cv.y[at] : 0, za = valid ? cv.z[at] : 0;
    const double qa = valid ? cv.q[at] : 0;
    double gx = 0, gy = 0, gz = 0, gq = 0;
    const long long p_begin = (long long)blockIdx.y * points_per_block;
    const long long p_end = min(a.P, p_begin + points_per_block);
    for (long long p0 = p_begin; p0 < p_end; p0 += EL_TILE) {
        const int np = (int)min((long long)EL_TILE, p_end - p0);
        __syncthreads();
        for (int i = threadIdx.x; i < np; i += EL_THREADS) {
            const long long lin = p0 + i;
            const int ix = (int)(lin % a.n1x), iy = (int)((lin / a.n1x) % a.n1y),
                      iz = (int)(lin / ((long long)a.n1x * a.n1y));
            double4 v;
            v.x = point_coord(ix, a.nex, a.spacing);
            v.y = point_coord(iy, a.ney, a.spacing);
            v.z = point_coord(iz, a.nez, a.spacing);
            v.w = g_e[lin];
            s_pt[i] = v;
        }
        __syncthreads();
        double ax = 0, ay = 0, az = 0, aq = 0;
#pragma unroll 4
        for (int i = part; i < np; i += EL_SPLIT) {
            const double4 pt = s_pt[i];
            const double dx = xa - pt.x, dy = ya - pt.y, dz = za - pt.z;
            double T, slope, rs;
            lin_eval(s_tab, dx * dx + dy * dy + dz * dz, T, slope, rs);
            const bool outer = rs < 2;  // r > 0.5
            const double F = outer ? T * rs : T * 2;
            const double dF = outer ? (slope - T * rs) * rs : slope * 2;  // dF/dr
            aq += pt.w * F;
            const double s = pt.w * dF * rs;
            ax += s * dx; ay += s * dy; az += s * dz;
        }
        gx += ax; gy += ay; gz += az; gq += aq;
    }
    double4 *sum = s_pt + owner;
    __syncthreads();
    if (part) sum[(part - 1) * EL_OWNERS] = make_double4(gx, gy, gz, gq);
    __syncthreads();
    if (part == 0 && valid) {
        for (int k = 0; k < EL_SPLIT - 1; k++) {
            const double4 t = sum[k * EL_OWNERS];
            gx += t.x; gy += t.y; gz += t.z; gq += t.w;
        }
        atomicAdd(g.xyz + 3 * at, (double)(gx * qa));
        atomicAdd(g.xyz + 3 * at + 1, (double)(gy * qa));
        atomicAdd(g.xyz + 3 * at + 2, (double)(gz * qa));
        atomicAdd(g.q + at, (double)gq);
    }
}

static_assert((EL_SPLIT - 1) * EL_OWNERS <= EL_TILE, "the tile holds the parts' sums");
constexpr size_t kEmapSmem = sizeof(R2<double>) * AG_NDIEL + sizeof(double4) * EL_TILE;

}  // namespace

cudaError_t launch_emap_lin(const DiffArgs &a, const void *eps, double *emap, cudaStream_t s)
{
    if (a.P == 0) return cudaSuccess;
    const dim3 nb((unsigned)((a.P + EL_OWNERS - 1) / EL_OWNERS), (unsigned)a.n_conf);
    const cudaError_t e = cudaFuncSetAttribute(k_emap_lin, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kEmapSmem);
    if (e != cudaSuccess) return e;
    k_emap_lin<<<nb, EL_THREADS, kEmapSmem, s>>>(a, (const R2<double> *)eps, emap);
    return cudaGetLastError();
}

cudaError_t launch_emap_lin_adj(const DiffArgs &a, const void *eps, const double *g_e, DiffGrads g, cudaStream_t s)
{
    if (a.n_atoms == 0 || a.P == 0) return cudaSuccess;
    // about one block per SM over (atom blocks x point ranges x conformers): 2 and
    // 4 load the table more often and gain nothing (3,000 atoms x 61^3 points)
    const int atom_blocks = (a.n_atoms + EL_OWNERS - 1) / EL_OWNERS;
    long long ranges = std::max(1LL, (long long)current_device_sms() / ((long long)atom_blocks * a.n_conf));
    const long long ppb = std::max(((a.P + ranges - 1) / ranges + EL_SPLIT - 1) / EL_SPLIT * EL_SPLIT, 256LL);
    ranges = (a.P + ppb - 1) / ppb;
    dim3 grid((unsigned)atom_blocks, (unsigned)ranges, (unsigned)a.n_conf);
    const cudaError_t e = cudaFuncSetAttribute(k_emap_lin_adj, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kEmapSmem);
    if (e != cudaSuccess) return e;
    k_emap_lin_adj<<<grid, EL_THREADS, kEmapSmem, s>>>(a, (const R2<double> *)eps, g_e, g, (int)ppb);
    return cudaGetLastError();
}

}  // namespace agb
