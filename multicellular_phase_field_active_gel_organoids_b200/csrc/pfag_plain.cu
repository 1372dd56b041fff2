// Plain path: one kernel per reference function, full-grid passes wherever the
// reference makes them, cuFFT for the per-cell spectral solve (batched over
// cells).  This is the FP64 comparison path and what the drop-in layer calls
// function by function.  Each kernel cites the reference loop it computes.
#include "pfag_internal.cuh"
#include <algorithm>
#include <cmath>
#include <cstdlib>

namespace {

constexpr int TBX = 32, TBY = 8;

inline dim3 grid2d(int nx, int ny, int nz) {
    return dim3((unsigned)((ny + TBX - 1) / TBX), (unsigned)((nx + TBY - 1) / TBY), (unsigned)nz);
}

// ---- find_centres_cells (useful_functions.cpp:193-227) ---------------------
template <typename real>
__global__ void k_centres_accum(const real *__restrict__ phi, int N, long long *__restrict__ acc) {
    const int n = blockIdx.y;
    long long cnt = 0, sx = 0, sy = 0;
    const size_t base = (size_t)n * N * N;
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < (size_t)N * N;
         k += (size_t)gridDim.x * blockDim.x) {
        if (phi[base + k] > (real)0.5) {
            cnt++;
            sx += (long long)(k / N);
            sy += (long long)(k % N);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        cnt += __shfl_down_sync(0xffffffffu, cnt, o);
        sx += __shfl_down_sync(0xffffffffu, sx, o);
        sy += __shfl_down_sync(0xffffffffu, sy, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd((unsigned long long *)&acc[3 * n + 0], (unsigned long long)cnt);
        atomicAdd((unsigned long long *)&acc[3 * n + 1], (unsigned long long)sx);
        atomicAdd((unsigned long long *)&acc[3 * n + 2], (unsigned long long)sy);
    }
}

// xcenters = (int)(x_barycentre/count): integer division, as the reference.
// Zone / box bounds: the reference indexes phi[n][i+-1][j+-1] for i in
// [xc-z, xc+z) without checks, so it needs xc-z >= 1 and xc+z <= N-1.
__global__ void k_centres_finalize(const long long *__restrict__ acc, int Ntot, int N, int zone,
                                   int *__restrict__ xc, int *__restrict__ yc, unsigned *__restrict__ err) {
    int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= Ntot) return;
    long long c = acc[3 * n];
    if (c == 0) {
        atomicOr(err, ERRBIT_EMPTY_CELL);
        xc[n] = N / 2;
        yc[n] = N / 2;
        return;
    }
    int x = (int)(acc[3 * n + 1] / c), y = (int)(acc[3 * n + 2] / c);
    if (x - zone < 1 || x + zone > N - 1 || y - zone < 1 || y + zone > N - 1) {
        // flag it and clamp, so that no zone kernel can index outside the grid
        atomicOr(err, ERRBIT_ZONE);
        x = min(max(x, zone + 1), N - 1 - zone);
        y = min(max(y, zone + 1), N - 1 - zone);
    }
    xc[n] = x;
    yc[n] = y;
}

// ---- create_turnover_rates_tensions (rho_functions.cpp:286-405) -------------
// Winner among phi*lum (apical, 0), phi*ECM (basal, 1), phi*phi_{n-1},
// phi*phi_{n+1} (lateral, 2 and 3); index neighbours are cyclic.
template <typename real>
__device__ __forceinline__ int map_class(real ph, real l, real e, real pm, real pp) {
    real c1l = ph * l, c1e = ph * e;
    int index;
    real mx;
    if (c1l > c1e) { index = 0; mx = c1l; } else { index = 1; mx = c1e; }
    real c1c2 = ph * pm;
    if (c1c2 > mx) { index = 2; mx = c1c2; }
    real c1c3 = ph * pp;
    if (c1c3 > mx) { index = 3; }
    return index == 3 ? 2 : index;   // 2 and 3 both lateral
}

template <typename real>
__global__ void k_maps(const real *__restrict__ phi, const real *__restrict__ lum, const real *__restrict__ ecm,
                       const int *__restrict__ xc, const int *__restrict__ yc, DevParams P,
                       real *__restrict__ deg, real *__restrict__ gen, real *__restrict__ atan_,
                       real *__restrict__ aort, real *__restrict__ visc, real *__restrict__ bm) {
    const int n = blockIdx.z, N = P.N, z = P.zone;
    const int i = xc[n] - z + blockIdx.y * TBY + threadIdx.y;
    const int j = yc[n] - z + blockIdx.x * TBX + threadIdx.x;
    if (i >= xc[n] + z || j >= yc[n] + z) return;
    const int n1 = (n == 0) ? P.Ntot - 1 : n - 1;
    const int n2 = (n == P.Ntot - 1) ? 0 : n + 1;
    const size_t s = (size_t)i * N + j;
    const real ph = phi[(size_t)n * N * N + s];
    int c = map_class<real>(ph, lum[s], ecm[s], phi[(size_t)n1 * N * N + s], phi[(size_t)n2 * N * N + s]);
    // reference index order: 0 apical, 1 basal, 2/3 lateral; P arrays: 0 ap, 1 bas, 2 lat
    const size_t o = (size_t)n * N * N + s;
    deg[o] = (real)P.deg[c];
    gen[o] = (real)P.gen[c];
    aort[o] = (real)P.a_ort[c];
    atan_[o] = (real)P.a_tan[c];
    visc[o] = (real)P.visc[c];
    bm[o] = (real)P.bb[c];
}

// ---- compute_hfunc_3d_tables_kernels_loop_n (useful_functions.cpp:233-251) --
template <typename real>
__global__ void k_hfunc_zone(const real *__restrict__ phi, real *__restrict__ h, const int *__restrict__ xc,
                             const int *__restrict__ yc, int N, int z) {
    const int n = blockIdx.z;
    const int i = xc[n] - z + blockIdx.y * TBY + threadIdx.y;
    const int j = yc[n] - z + blockIdx.x * TBX + threadIdx.x;
    if (i >= xc[n] + z || j >= yc[n] + z) return;
    const size_t o = cidx(n, i, j, N);
    real f = phi[o];
    h[o] = f * f * ((real)3.0 - (real)2.0 * f);
}

// ---- compute_all_hfunc_2d_tables_kernels (useful_functions.cpp:272-285) -----
template <typename real>
__global__ void k_hfunc_2d(const real *__restrict__ lum, const real *__restrict__ ecm, real *__restrict__ hl,
                           real *__restrict__ he, size_t ng) {
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < ng; k += (size_t)gridDim.x * blockDim.x) {
        real a = lum[k], b = ecm[k];
        hl[k] = a * a * ((real)3.0 - (real)2.0 * a);
        he[k] = b * b * ((real)3.0 - (real)2.0 * b);
    }
}

// ---- compute_normal_grad_phi (useful_functions.cpp:326-354) -----------------
template <typename real>
__global__ void k_norm_grad(const real *__restrict__ phi, real *__restrict__ g, int N, real c4) {
    const int n = blockIdx.z;
    const int i = 1 + blockIdx.y * TBY + threadIdx.y;
    const int j = 1 + blockIdx.x * TBX + threadIdx.x;
    if (i > N - 2 || j > N - 2) return;
    const real *p = phi + (size_t)n * N * N;
    real a = p[(size_t)(i + 1) * N + j] - p[(size_t)(i - 1) * N + j];
    real b = p[(size_t)i * N + j + 1] - p[(size_t)i * N + j - 1];
    g[cidx(n, i, j, N)] = sqrt(c4 * (a * a + b * b));
}

// ---- boundary_conditions_cells (useful_functions.cpp:391-420) --------------
// All reads are interior sites, so the ghost ring can be written in any order.
template <typename real>
__global__ void k_bc_cells(real *__restrict__ t, int N, int ncells) {
    const int n = blockIdx.y;
    if (n >= ncells) return;
    real *p = t + (size_t)n * N * N;
    const int perim = 4 * N;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < perim; k += gridDim.x * blockDim.x) {
        int i, j;
        if (k < N) { i = 0; j = k; }
        else if (k < 2 * N) { i = N - 1; j = k - N; }
        else if (k < 3 * N) { i = k - 2 * N; j = 0; }
        else { i = k - 3 * N; j = N - 1; }
        if ((k >= 2 * N) && (i == 0 || i == N - 1)) continue;  // corners written once
        p[(size_t)i * N + j] = p[(size_t)ghost_src(i, N) * N + ghost_src(j, N)];
    }
}

// ---- compute_prod_norm_delta (rho_functions.cpp:13-30) ----------------------
template <typename real>
__global__ void k_prod_norm_delta(const real *__restrict__ g, const real *__restrict__ phi, real *__restrict__ pnd,
                                  const int *__restrict__ xc, const int *__restrict__ yc, int N, int z, real sigma) {
    const int n = blockIdx.z;
    const int i = xc[n] - z + blockIdx.y * TBY + threadIdx.y;
    const int j = yc[n] - z + blockIdx.x * TBX + threadIdx.x;
    if (i >= xc[n] + z || j >= yc[n] + z) return;
    const size_t o = cidx(n, i, j, N);
    real f = phi[o];
    pnd[o] = g[o] * exp(-(f - (real)0.5) * (f - (real)0.5) / (real)2.0 / sigma / sigma) /
             sqrt((real)(2.0 * M_PI)) / sigma;
}

// ---- compute_psi_kernels (useful_functions.cpp:305-322) ---------------------
template <typename real>
__global__ void k_psi(const real *__restrict__ h, real *__restrict__ psi, size_t ng, int ncells) {
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < ng; k += (size_t)gridDim.x * blockDim.x) {
        real s = (real)0.0;
        for (int n = 0; n < ncells; n++) s += h[(size_t)n * ng + k];
        psi[k] = s;
    }
}

// ---- sum_s_kernels (useful_functions.cpp:168-190): FP64 accumulation --------
// Deterministic: fixed-size per-block partials, then a fixed-order final sum.
constexpr int RED_THREADS = 256;
constexpr int RED_BLOCKS = 128;

__device__ __forceinline__ double block_sum(double v) {
    __shared__ double sh[32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sh[w] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x == 0)
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) r += sh[k];
    return r;
}

template <typename real>
__global__ void k_sum_cells(const real *__restrict__ h, size_t ng, double scale, double *__restrict__ part) {
    const int n = blockIdx.y;
    double acc = 0.0;
    const real *p = h + (size_t)n * ng;
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < ng; k += (size_t)gridDim.x * blockDim.x)
        acc += (double)p[k] * scale;
    double r = block_sum(acc);
    if (threadIdx.x == 0) part[(size_t)n * gridDim.x + blockIdx.x] = r;
}

__global__ void k_sum_s_finalize(const double *__restrict__ part, int nblk, int ncells, double alpha, double s0,
                                 double *__restrict__ s, double *__restrict__ f0) {
    int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= ncells) return;
    double a = 0.0;
    for (int b = 0; b < nblk; b++) a += part[(size_t)n * nblk + b];
    s[n] = a;
    f0[n] = alpha * (s0 - a);
}

// Serial-order sums (pfag_set_serial_sums): one thread per cell adds the terms
// in the order and with the expression of the reference's host loops, i-major
// with j inner.  sum_s_kernels (useful_functions.cpp:179-184):
// sum += h*dx*dx over the full grid; the reshaping check
// (cell_phase_functions.cpp:556-561): rdev += |phin-phi|*dx*dx/N_current over
// the zone; update_lumen_and_ECM's sum_ecm (:380-386) and the lumen/ECM check
// (:848-854): sum += v*dx*dx over the full grid.  Compiled without
// contraction, each partial sum then rounds as the host build's does.
template <typename real>
__global__ void k_serial_sum_cells(const real *__restrict__ h, int N, int ncells, double dx,
                                   double *__restrict__ out) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= ncells) return;
    const real *p = h + (size_t)n * N * N;
    double acc = 0.0;
    for (int i = 0; i < N; i++)
        for (int j = 0; j < N; j++) acc += (double)p[(size_t)i * N + j] * dx * dx;
    out[n] = acc;
}

template <typename real>
__global__ void k_serial_absdiff(const real *__restrict__ a, const real *__restrict__ b, int N, double dx,
                                 const int *__restrict__ active, double *__restrict__ out) {
    if (blockIdx.x != 0 || threadIdx.x != 0 || !*active) return;
    double acc = 0.0;
    for (int i = 0; i < N; i++)
        for (int j = 0; j < N; j++) {
            const size_t o = (size_t)i * N + j;
            acc += fabs((double)a[o] - (double)b[o]) * dx * dx;
        }
    *out = acc;
}

template <typename real>
__global__ void k_serial_cell_rdev(const real *__restrict__ pn, const real *__restrict__ p, bool compact,
                                   const int *__restrict__ xc, const int *__restrict__ yc, int N, int z, int ncells,
                                   double dx, double ncur, const int *__restrict__ active,
                                   double *__restrict__ out) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= ncells) return;
    double acc = 0.0;
    if (active[n])
        for (int i = 0; i < 2 * z; i++) {
            const real *a = p + cidx(n, xc[n] - z + i, yc[n] - z, N);
            const real *b = compact ? pn + cidx(n, i, 0, 2 * z) : pn + (a - p);                 // [Ntot][2z][2z]
            // eight loads of each before their additions, which wait for one another (a step
            // of seven cells on 256^2 106 -> 83 ms)
            for (int j0 = 0; j0 < 2 * z; j0 += 8) {
                const int m = min(8, 2 * z - j0);
                real u[8], v[8];
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (k < m) { u[k] = a[j0 + k]; v[k] = b[j0 + k]; }
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (k < m) acc += fabs((double)v[k] - (double)u[k]) * dx * dx / ncur;
            }
        }
    out[n] = acc;
}

// ---- update_all_cortices helpers (rho_functions.cpp:32-284, useful_functions.cpp:605-625)
template <typename real>
__global__ void k_pi(const real *__restrict__ rho, const real *__restrict__ g, const real *__restrict__ phi,
                     const real *__restrict__ atan_, const real *__restrict__ aort, const real *__restrict__ bm,
                     const int *__restrict__ xc, const int *__restrict__ yc, int N, int z, real c4,
                     real *__restrict__ pxx, real *__restrict__ pxy, real *__restrict__ pyy) {
    const int n = blockIdx.z;
    const int i = xc[n] - z + blockIdx.y * TBY + threadIdx.y;
    const int j = yc[n] - z + blockIdx.x * TBX + threadIdx.x;
    if (i >= xc[n] + z || j >= yc[n] + z) return;
    const size_t o = cidx(n, i, j, N);
    const real r = rho[o], at = atan_[o], ao = aort[o], b = bm[o], gg = g[o];
    const real *p = phi + (size_t)n * N * N;
    const real dxp = p[(size_t)(i + 1) * N + j] - p[(size_t)(i - 1) * N + j];
    const real dyp = p[(size_t)i * N + j + 1] - p[(size_t)i * N + j - 1];
    real xx = -at * r * r * r + b * r * r * r * r;
    real yy = xx;
    real xy = (real)0.0;
    if (gg > (real)0.0) {
        xx += (at - ao) * r * r * r * c4 * dxp * dxp / gg / gg;   // rho_functions.cpp:51
        yy += (at - ao) * r * r * r * c4 * dyp * dyp / gg / gg;   // :79
        xy += (at - ao) * r * r * r * c4 * dxp * dyp / gg / gg;   // :109
    }
    pxx[o] = xx;
    pxy[o] = xy;
    pyy[o] = yy;
}

// load_temp_fft: box[i][j] = table[n][i+1+xc-z][j+1+yc-z] + 0i
template <typename real>
__global__ void k_box_load(const real *__restrict__ t, typename Cplx<real>::type *__restrict__ box,
                           const int *__restrict__ xc, const int *__restrict__ yc, int N, int z, int M) {
    const int n = blockIdx.z;
    const int i = blockIdx.y * TBY + threadIdx.y, j = blockIdx.x * TBX + threadIdx.x;
    if (i >= M || j >= M) return;
    const int gi = i + 1 + xc[n] - z, gj = j + 1 + yc[n] - z;
    typename Cplx<real>::type v;
    v.x = t[cidx(n, gi, gj, N)];
    v.y = (real)0.0;
    box[((size_t)n * M + i) * M + j] = v;
}

// create_deg_gen (rho_functions.cpp:193-209): -deg*rho + gen*prod_norm_delta
template <typename real>
__global__ void k_box_deg_gen(const real *__restrict__ deg, const real *__restrict__ rho, const real *__restrict__ gen,
                              const real *__restrict__ pnd, typename Cplx<real>::type *__restrict__ box,
                              const int *__restrict__ xc, const int *__restrict__ yc, int N, int z, int M) {
    const int n = blockIdx.z;
    const int i = blockIdx.y * TBY + threadIdx.y, j = blockIdx.x * TBX + threadIdx.x;
    if (i >= M || j >= M) return;
    const size_t o = cidx(n, i + 1 + xc[n] - z, j + 1 + yc[n] - z, N);
    typename Cplx<real>::type v;
    v.x = -deg[o] * rho[o] + gen[o] * pnd[o];
    v.y = (real)0.0;
    box[((size_t)n * M + i) * M + j] = v;
}

// update_rho_velocity (rho_functions.cpp:133-190); viscosity is read at the
// real-space box site with the same (i, j) as the wavevector.
template <typename real>
__global__ void k_velocity(const typename Cplx<real>::type *__restrict__ fxx,
                           const typename Cplx<real>::type *__restrict__ fyy,
                           const typename Cplx<real>::type *__restrict__ fxy,
                           typename Cplx<real>::type *__restrict__ fvx, typename Cplx<real>::type *__restrict__ fvy,
                           const real *__restrict__ visc, const int *__restrict__ xc, const int *__restrict__ yc,
                           int N, int z, int M, double kfac, real friction) {
    const int n = blockIdx.z;
    const int i = blockIdx.y * TBY + threadIdx.y, j = blockIdx.x * TBX + threadIdx.x;
    if (i >= M || j >= M) return;
    const size_t b = ((size_t)n * M + i) * M + j;
    const int ir = (i < M / 2) ? i : i - M;
    const int jr = (j < M / 2) ? j : j - M;
    const real kx = (real)(kfac * ir), ky = (real)(kfac * jr);
    const real et = visc[cidx(n, i + 1 + xc[n] - z, j + 1 + yc[n] - z, N)];
    const auto pxx = fxx[b], pyy = fyy[b], pxy = fxy[b];
    const real A = friction + (real)2.0 * et * (kx * kx + ky * ky / (real)2.0);
    const real D = -((real)4.0 * et * et * kx * kx * ky * ky + friction * friction +
                     (real)3.0 * et * friction * (kx * kx + ky * ky) +
                     (real)2.0 * et * et * (kx * kx * kx * kx + ky * ky * ky * ky));
    typename Cplx<real>::type vx, vy;
    vy.x = (real)0.0 + et * kx * ky * (kx * pxx.y + ky * pxy.y);
    vy.x -= A * (ky * pyy.y + kx * pxy.y);
    vy.x /= D;
    vy.y = (real)0.0 - et * kx * ky * (kx * pxx.x + ky * pxy.x);
    vy.y += A * (ky * pyy.x + kx * pxy.x);
    vy.y /= D;
    vx.x = (real)0.0 + (kx * pxx.y + ky * pxy.y - et * kx * ky * vy.x);
    vx.x /= A;
    vx.y = (real)0.0 + (-kx * pxx.x - ky * pxy.x - et * kx * ky * vy.y);
    vx.y /= A;
    fvx[b] = vx;
    fvy[b] = vy;
}

// load_fft_rho_v (rho_functions.cpp:267-284): rho * Re(v) / (M*M) + 0i
template <typename real>
__global__ void k_load_rho_v(const real *__restrict__ rho, const typename Cplx<real>::type *__restrict__ tr,
                             typename Cplx<real>::type *__restrict__ box, const int *__restrict__ xc,
                             const int *__restrict__ yc, int N, int z, int M, real *__restrict__ vdbg) {
    const int n = blockIdx.z;
    const int i = blockIdx.y * TBY + threadIdx.y, j = blockIdx.x * TBX + threadIdx.x;
    if (i >= M || j >= M) return;
    const size_t b = ((size_t)n * M + i) * M + j;
    const real mm = (real)((double)M * (double)M);
    typename Cplx<real>::type v;
    v.x = rho[cidx(n, i + 1 + xc[n] - z, j + 1 + yc[n] - z, N)] * tr[b].x / mm;
    v.y = (real)0.0;
    box[b] = v;
    if (vdbg) vdbg[b] = tr[b].x / mm;
}

// update_fft_rho (rho_functions.cpp:213-251)
template <typename real>
__global__ void k_update_fft_rho(typename Cplx<real>::type *__restrict__ fr,
                                 const typename Cplx<real>::type *__restrict__ freact,
                                 const typename Cplx<real>::type *__restrict__ frvx,
                                 const typename Cplx<real>::type *__restrict__ frvy, int M, real dt, double kfac) {
    const int n = blockIdx.z;
    const int i = blockIdx.y * TBY + threadIdx.y, j = blockIdx.x * TBX + threadIdx.x;
    if (i >= M || j >= M) return;
    const size_t b = ((size_t)n * M + i) * M + j;
    const int ir = (i < M / 2) ? i : i - M;
    const int jr = (j < M / 2) ? j : j - M;
    auto r = fr[b];
    const auto q = freact[b];
    r.x += dt * q.x;
    r.y += dt * q.y;
    const real dk = (real)((double)dt * kfac);
    const auto a = frvx[b], c = frvy[b];
    r.x += dk * ((real)ir * a.y + (real)jr * c.y);
    r.y -= dk * ((real)ir * a.x + (real)jr * c.x);
    fr[b] = r;
}

// copy_to_rhon (rho_functions.cpp:253-265)
template <typename real>
__global__ void k_copy_to_rhon(const typename Cplx<real>::type *__restrict__ box, real *__restrict__ rhon,
                               const int *__restrict__ xc, const int *__restrict__ yc, int N, int z, int M) {
    const int n = blockIdx.z;
    const int i = blockIdx.y * TBY + threadIdx.y, j = blockIdx.x * TBX + threadIdx.x;
    if (i >= M || j >= M) return;
    rhon[cidx(n, i + 1 + xc[n] - z, j + 1 + yc[n] - z, N)] =
        box[((size_t)n * M + i) * M + j].x / (real)((double)M * (double)M);
}

// ---- update_lumen_and_ECM (cell_phase_functions.cpp:372-444) ---------------
template <typename real>
__global__ void k_lum_ecm_update(const real *__restrict__ lum, const real *__restrict__ ecm,
                                 const real *__restrict__ psi, const real *__restrict__ hl, const real *__restrict__ he,
                                 real *__restrict__ lumn, real *__restrict__ ecmn, DevParams P,
                                 const double *__restrict__ sum_ecm) {
    const int N = P.N;
    const int i = 1 + blockIdx.y * TBY + threadIdx.y, j = 1 + blockIdx.x * TBX + threadIdx.x;
    if (i > N - 2 || j > N - 2) return;
    const size_t c = (size_t)i * N + j;
    const real s = psi[c];
    const real L = lap9<real>(s, psi[c + N], psi[c - N], psi[c + 1], psi[c - 1], psi[c + N + 1], psi[c + N - 1],
                              psi[c - N - 1], psi[c - N + 1]);
    const real dx = (real)P.dx, dt = (real)P.dt;
    const real l = lum[c], e = ecm[c];
    real ln = l;
    ln += ((real)1.0 / (real)P.tau_lum) * l * ((real)1.0 - l) * dt *
          ((real)P.xi_lum - (real)P.beta_lum_cells * s + (real)P.eta_lum_cells * L / ((real)4.0 * dx * dx) -
           (real)P.beta_lum_ECM * he[c]);
    real en = e;
    const real elastic = (real)(P.alpha_ECM * ((double)N * (double)N * P.dx * P.dx - *sum_ecm));
    en += ((real)1.0 / (real)P.tau_ECM) * e * ((real)1.0 - e) * dt *
          (elastic + (real)P.xi_ECM - (real)P.beta_ECM_cells * s + (real)P.eta_ECM_cells * L / ((real)4.0 * dx * dx) -
           (real)P.beta_lum_ECM * hl[c]);
    lumn[c] = ln;
    ecmn[c] = en;
}

// boundary_conditions_lumen_and_ECM (useful_functions.cpp:439-462) and
// boundary_conditions_dirichlet (:422-437): sides to the side value, corners
// to `corner` (0 for the Dirichlet helper, the side value for the first one).
template <typename real>
__global__ void k_dirichlet(real *__restrict__ t, int N, real side, real corner) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < 4 * N; k += gridDim.x * blockDim.x) {
        int i, j;
        if (k < N) { i = 0; j = k; }
        else if (k < 2 * N) { i = N - 1; j = k - N; }
        else if (k < 3 * N) { i = k - 2 * N; j = 0; }
        else { i = k - 3 * N; j = N - 1; }
        if ((k >= 2 * N) && (i == 0 || i == N - 1)) continue;
        bool corner_site = (i == 0 || i == N - 1) && (j == 0 || j == N - 1);
        t[(size_t)i * N + j] = corner_site ? corner : side;
    }
}

// reshaping_lumen_or_ECM prologue (cell_phase_functions.cpp:722-771)
template <typename real>
__global__ void k_norm_grad_2d(const real *__restrict__ f, real *__restrict__ g, int N, real c4) {
    const int i = 1 + blockIdx.y * TBY + threadIdx.y, j = 1 + blockIdx.x * TBX + threadIdx.x;
    if (i > N - 2 || j > N - 2) return;
    const size_t c = (size_t)i * N + j;
    real a = f[c + N] - f[c - N], b = f[c + 1] - f[c - 1];
    g[c] = sqrt(c4 * (a * a + b * b));
}

template <typename real>
__global__ void k_lum_normals(const real *__restrict__ lumn, const real *__restrict__ ngl, real *__restrict__ jx,
                              real *__restrict__ jy, int N, real inv2dx) {
    const int i = 1 + blockIdx.y * TBY + threadIdx.y, j = 1 + blockIdx.x * TBX + threadIdx.x;
    if (i > N - 2 || j > N - 2) return;
    const size_t c = (size_t)i * N + j;
    const real g = ngl[c];
    jx[c] = (g != (real)0.0) ? inv2dx * (lumn[c + N] - lumn[c - N]) / g : (real)0.0;
    jy[c] = (g != (real)0.0) ? inv2dx * (lumn[c + 1] - lumn[c - 1]) / g : (real)0.0;
}

// One iteration of the lumen/ECM loop (:774-849): f <- P, Q = P + its
// relaxation update (interior; :802-838), the Dirichlet values on the boundary
// (useful_functions.cpp:422-437), and the block's sum of |Q - P| dx^2.  Does
// nothing once the loop has stopped (*active == 0).
template <typename real>
__global__ void k_lum_iter(const real *__restrict__ p, real *__restrict__ q, real *__restrict__ f,
                           const real *__restrict__ jx, const real *__restrict__ jy, int N, real A, real B, real side,
                           double scale, const int *__restrict__ active, double *__restrict__ part) {
    if (!*active) return;
    const int i = blockIdx.y * TBY + (threadIdx.x >> 5), j = blockIdx.x * TBX + (threadIdx.x & 31);
    double acc = 0.0;
    if (i < N && j < N) {
        const size_t c = (size_t)i * N + j;
        const real old = p[c];
        const bool ei = i == 0 || i == N - 1, ej = j == 0 || j == N - 1;
        real v;
        if (ei || ej) {
            v = ei && ej ? (real)0.0 : side;
        } else {
            real w[3][3];
            for (int a = 0; a < 3; a++)
                for (int b = 0; b < 3; b++) w[a][b] = p[c + (size_t)(a - 1) * N + (b - 1)];
            v = resh_update<real>(A, B, w, jx[c], jx[c + N], jx[c - N], jx[c + 1], jx[c - 1], jy[c], jy[c + N],
                                  jy[c - N], jy[c + 1], jy[c - 1], old);
        }
        q[c] = v;
        f[c] = old;
        acc = fabs((double)v - (double)old) * scale;
    }
    const double r = block_sum(acc);
    if (threadIdx.x == 0) part[blockIdx.y * gridDim.x + blockIdx.x] = r;
}

__global__ void k_lum_state(int *st, int active) {
    if (threadIdx.x < 4) st[threadIdx.x] = threadIdx.x == 0 ? active : 0;
}

// The loop's end test after it (:851-868): rdev from the blocks' sums in a fixed
// order.  st: [0] active, [1] ri, [2] iterations, [3] passed rimax.
__global__ void k_lum_check(const double *__restrict__ part, int npart, double thr, int rimax, int *__restrict__ st) {
    if (!st[0]) return;
    double a = 0.0;
    for (int k = threadIdx.x; k < npart; k += blockDim.x) a += part[k];
    a = block_sum(a);
    if (threadIdx.x == 0) {
        st[2]++;
        bool stop = !(a > thr);
        if (st[1] > rimax) { st[3] = 1; stop = true; }
        else st[1]++;
        if (stop) st[0] = 0;
    }
}
// the last iterate back into fn after an odd iteration count
template <typename real>
__global__ void k_lum_last(real *__restrict__ fn, const real *__restrict__ q, size_t n, const int *__restrict__ st) {
    if (!(st[2] & 1)) return;
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x)
        fn[k] = q[k];
}

__global__ void k_sum_partials(const double *__restrict__ part, int nblk, double *__restrict__ out) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        double a = 0.0;
        for (int b = 0; b < nblk; b++) a += part[b];
        *out = a;
    }
}

// ---- compute_normal_to_phi (useful_functions.cpp:356-388) -------------------
template <typename real>
__global__ void k_normals(const real *__restrict__ phi, const real *__restrict__ g, real *__restrict__ jx,
                          real *__restrict__ jy, int N, real inv2dx) {
    const int n = blockIdx.z;
    const int i = 1 + blockIdx.y * TBY + threadIdx.y, j = 1 + blockIdx.x * TBX + threadIdx.x;
    if (i > N - 2 || j > N - 2) return;
    const real *p = phi + (size_t)n * N * N;
    const size_t c = (size_t)i * N + j, o = (size_t)n * N * N + c;
    const real gg = g[o];
    jx[o] = (gg > (real)0.0) ? inv2dx * (p[c + N] - p[c - N]) / gg : (real)0.0;
    jy[o] = (gg > (real)0.0) ? inv2dx * (p[c + 1] - p[c - 1]) / gg : (real)0.0;
}

// ---- update_all_cells (cell_phase_functions.cpp:126-217) --------------------
// temp_phase = psi - hfunc_cell is formed on the fly at each stencil point.
template <typename real>
__global__ void k_update_cells(const real *__restrict__ phi, real *__restrict__ phin, const real *__restrict__ g,
                               const real *__restrict__ rho, const real *__restrict__ h, const double *__restrict__ f0,
                               const real *__restrict__ psi, const int *__restrict__ xc, const int *__restrict__ yc,
                               const real *__restrict__ hl, const real *__restrict__ he, DevParams P) {
    const int n = blockIdx.z, N = P.N, z = P.zone;
    const int i = xc[n] - z + blockIdx.y * TBY + threadIdx.y;
    const int j = yc[n] - z + blockIdx.x * TBX + threadIdx.x;
    if (i >= xc[n] + z || j >= yc[n] + z) return;
    const size_t c = (size_t)i * N + j, base = (size_t)n * N * N, o = base + c;
    const real dx = (real)P.dx, dt = (real)P.dt, tau = (real)P.tau, sigma = (real)P.sigma;
    const real f = phi[o];
    real pn = f;
    const real gg = g[o];
    if (gg > (real)0.0) {
        const real *p = phi + base, *r = rho + base;
        pn -= (real)P.cpl / tau * (dt / dx / dx / (real)4.0) *
              exp(-(f - (real)0.5) * (f - (real)0.5) / (real)2.0 / sigma / sigma) / sqrt((real)(2.0 * M_PI)) / sigma *
              ((r[c + N] - r[c - N]) * (p[c + N] - p[c - N]) + (r[c + 1] - r[c - 1]) * (p[c + 1] - p[c - 1])) / gg;
    }
    const real *hh = h + base;
    auto T = [&](size_t k) { return psi[k] - hh[k]; };
    const real Tc = T(c);
    const real LT = lap9<real>(Tc, T(c + N), T(c - N), T(c + 1), T(c - 1), T(c + N + 1), T(c + N - 1),
                               T(c - N - 1), T(c - N + 1));
    const real Ll = lap9<real>(hl[c], hl[c + N], hl[c - N], hl[c + 1], hl[c - 1], hl[c + N + 1], hl[c + N - 1],
                               hl[c - N - 1], hl[c - N + 1]);
    const real Le = lap9<real>(he[c], he[c + N], he[c - N], he[c + 1], he[c - 1], he[c + N + 1], he[c + N - 1],
                               he[c - N - 1], he[c - N + 1]);
    const real q4 = (real)4.0 * dx * dx;
    pn += ((real)1.0 / tau) * f * ((real)1.0 - f) * dt *
          ((real)f0[n] - (real)P.beta * Tc + (real)P.eta * LT / q4 - (real)P.beta_lum_cells * hl[c] +
           (real)P.eta_lum_cells * Ll / q4 - (real)P.beta_ECM_cells * he[c] + (real)P.eta_ECM_cells * Le / q4);
    phin[o] = pn;
}

// ---- reshaping_cells (cell_phase_functions.cpp:447-580) ---------------------
// Iteration k takes iterate k - 1 to iterate k: odd ones from phin into the
// compact planes T ([Ntot][2z][2z]), even ones back, so that reading and
// writing need no copy between them; each stores its input into phi (the copy
// at the top of the reference's loop).  active[n] != 0 while cell n is still
// iterating; a stopped cell's blocks return at once, so the host can enqueue
// several iterations between its looks at the flags.
template <typename real, bool ODD>
__global__ void k_cell_iter(real *__restrict__ phi, real *__restrict__ phin, real *__restrict__ T,
                            const real *__restrict__ jx, const real *__restrict__ jy, const int *__restrict__ xc,
                            const int *__restrict__ yc, int N, int z, real A, real B, double scale,
                            const int *__restrict__ active, double *__restrict__ part) {
    const int n = blockIdx.z;
    if (!active[n]) return;
    const int Z = 2 * z, li = blockIdx.y * TBY + (threadIdx.x >> 5), lj = blockIdx.x * TBX + (threadIdx.x & 31);
    double acc = 0.0;
    if (li < Z && lj < Z) {
        const size_t base = (size_t)n * N * N, c = (size_t)(xc[n] - z + li) * N + (yc[n] - z + lj);
        const size_t tb = (size_t)n * Z * Z, tc = (size_t)li * Z + lj;
        const real *X = jx + base, *Y = jy + base;
        real w[3][3];
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++) {
                // the ring around the zone, which no iteration writes, from phi
                const int ii = li + a - 1, jj = lj + b - 1;
                const bool ring = ii < 0 || ii >= Z || jj < 0 || jj >= Z;
                const size_t o = base + c + (size_t)(a - 1) * N + (b - 1);
                w[a][b] = ring ? phi[o] : ODD ? phin[o] : T[tb + (size_t)ii * Z + jj];
            }
        const real old = w[1][1];
        const real v = resh_update<real>(A, B, w, X[c], X[c + N], X[c - N], X[c + 1], X[c - 1], Y[c], Y[c + N],
                                         Y[c - N], Y[c + 1], Y[c - 1], old);
        if (ODD) T[tb + tc] = v;
        else phin[base + c] = v;
        phi[base + c] = old;
        acc = fabs((double)v - (double)old) * scale;
    }
    const double r = block_sum(acc);
    if (threadIdx.x == 0) part[((size_t)n * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = r;
}
// the last iterate back into phin for the cells with an odd iteration count
template <typename real>
__global__ void k_cell_last(real *__restrict__ phin, const real *__restrict__ T, const int *__restrict__ xc,
                            const int *__restrict__ yc, int N, int z, const int *__restrict__ iters) {
    const int n = blockIdx.z, Z = 2 * z;
    if (!(iters[n] & 1)) return;
    const int li = blockIdx.y * TBY + (threadIdx.x >> 5), lj = blockIdx.x * TBX + (threadIdx.x & 31);
    if (li < Z && lj < Z)
        phin[(size_t)n * N * N + (size_t)(xc[n] - z + li) * N + yc[n] - z + lj] =
            T[(size_t)n * Z * Z + (size_t)li * Z + lj];
}

// all cells active with ri = 0 and no iteration done ([3][ncells])
__global__ void k_cell_state(int *st, int ncells) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < 3 * ncells; k += gridDim.x * blockDim.x)
        st[k] = k < ncells ? 1 : 0;
}

// Convergence bookkeeping of the while loop at cell_phase_functions.cpp:475-574:
// after an iteration, the loop ends when rdev <= thr, or (ri > rimax) breaks.
// One warp per cell; rdev from the blocks' sums in a fixed order.
__global__ void k_cell_check(const double *__restrict__ part, int nblk, double thr, int rimax,
                             int *__restrict__ active, int *__restrict__ ri, int *__restrict__ iters,
                             unsigned *__restrict__ err) {
    const int n = blockIdx.x;
    if (!active[n]) return;
    double a = 0.0;
    for (int b = threadIdx.x; b < nblk; b += 32) a += part[(size_t)n * nblk + b];
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (threadIdx.x != 0) return;
    bool stop = false;
    if (ri[n] > rimax) { atomicOr(err, ERRBIT_RELAX); stop = true; }
    else ri[n]++;
    iters[n]++;
    if (a <= thr) stop = true;
    if (stop) active[n] = 0;
}

template <typename real>
__global__ void k_copy(real *__restrict__ dst, const real *__restrict__ src, size_t n) {
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x)
        dst[k] = src[k];
}

// ---------------------------------------------------------------------------
// ---- initial-condition generator (initialisation_code/prepare_initial_files.cpp:53-117)

// ini_phi (functions/initialisation_functions.cpp:116-160): N_ini cells on a
// ring of radius rcyst about the grid centre (one cell: at the centre), each a
// logistic profile 1/(1 + exp((dx r - R0)/wi)).  The float build computes the
// centre in double and stores it as float, r, the exponent and exp in float.
template <typename real>
__global__ void k_ini_phi(real *__restrict__ phi, int N, int N_ini, real dx, real R0, real wi, real rcyst) {
    const int n = blockIdx.z;
    const int i = blockIdx.y * blockDim.y + threadIdx.y, j = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N || j >= N) return;
    real xcen, ycen;
    if (N_ini > 1) {
        xcen = (real)((double)(N / 2) + (double)rcyst * cos((double)n * 2.0 * M_PI / (double)N_ini));
        ycen = (real)((double)(N / 2) + (double)rcyst * sin((double)n * 2.0 * M_PI / (double)N_ini));
    } else {
        xcen = (real)(N / 2);
        ycen = (real)(N / 2);
    }
    const real di = (real)i - xcen, dj = (real)j - ycen;
    const real e = exp((dx * sqrt(di * di + dj * dj) - R0) / wi);
    phi[(size_t)n * N * N + (size_t)i * N + j] = (real)(1.0 / (1.0 + (double)e));
}

// ini_ECM_lumen (initialisation_functions.cpp:72-110): the space the cells
// leave free, 1 - sum phi, is lumen inside the ring radius and ECM outside;
// zero where the cells fill the site.  Sites not assigned stay zero.
template <typename real>
__global__ void k_ini_lum_ecm(const real *__restrict__ phi, real *__restrict__ lum, real *__restrict__ ecm, int N,
                              int N_ini, real rcyst) {
    const int i = blockIdx.y * blockDim.y + threadIdx.y, j = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N || j >= N) return;
    const size_t k = (size_t)i * N + j, NN = (size_t)N * N;
    real all = (real)0.0;
    for (int n = 0; n < N_ini; n++) all += phi[(size_t)n * NN + k];
    real l = (real)0.0, e = (real)0.0;
    if (1.0 - (double)all > 0.0) {
        const int a = i - N / 2, b = j - N / 2;
        const double d = sqrt((double)(a * a + b * b));
        if (d < (double)rcyst) l = (real)(1.0 - (double)all);
        else e = (real)(1.0 - (double)all);
    }
    lum[k] = l;
    ecm[k] = e;
}

// The cortex density of a phase value (initialisation_functions.cpp:62-70 and
// update_rho_to_shape, cell_phase_functions.cpp:42-62), in double as both
// builds evaluate it: rho0 exp(-1/(4 h (1 - h) + tol) + 1/(1 + tol)),
// h = phi^2 (3 - 2 phi), and 0 below the floor rho0 exp(-1/(2 tol) + 1/(1 + tol)).
// set_everywhere: ini_rho assigns every site; update_rho_to_shape only sites
// with phi != 0 (then applies the floor to every site).
template <typename real>
__global__ void k_rho_shape(const real *__restrict__ phi, real *__restrict__ rho, size_t n, double rho0, double tol,
                            int set_everywhere) {
    // rho0 and tol are parameters of the build's precision
    rho0 = (double)(real)rho0;
    tol = (double)(real)tol;
    const double floor_v = rho0 * exp(-1.0 / (2.0 * tol) + 1.0 / (1.0 + tol));
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
        const real p = phi[k];
        const double f = (double)p;
        const double pp = (double)(p * p);     // phi*phi is a product in the build's precision there
        real r = rho[k];
        if (set_everywhere || p != (real)0.0)
            r = (real)(rho0 * exp(-1.0 / (4.0 * f * f * (3.0 - 2.0 * f) * (1.0 - pp * (3.0 - 2.0 * f)) + tol) +
                                  1.0 / (1.0 + tol)));
        if ((double)r < floor_v) r = (real)0.0;
        rho[k] = r;
    }
}

template <typename real> struct FFTX;
template <> struct FFTX<double> {
    static cufftResult exec(cufftHandle p, void *in, void *out, int dir) {
        return cufftExecZ2Z(p, (cufftDoubleComplex *)in, (cufftDoubleComplex *)out, dir);
    }
    static constexpr cufftType type = CUFFT_Z2Z;
};
template <> struct FFTX<float> {
    static cufftResult exec(cufftHandle p, void *in, void *out, int dir) {
        return cufftExecC2C(p, (cufftComplex *)in, (cufftComplex *)out, dir);
    }
    static constexpr cufftType type = CUFFT_C2C;
};

// the step's captured stretches (Plain::stretch)
struct PlainGraphs {
    cudaGraphExec_t exec[5] = {};
    long launches[5] = {};
    long steps = 0;            // steps taken: the first one runs eagerly
    bool failed = false;       // a refused capture: eager from then on
    int key = 0;
    void drop() {
        for (cudaGraphExec_t &e : exec) {
            if (e) cudaGraphExecDestroy(e);
            e = nullptr;
        }
    }
};

template <typename real>
struct Plain {
    typedef typename Cplx<real>::type cx;
    pfag_ctx *c;
    explicit Plain(pfag_ctx *ctx) : c(ctx) {}
    real *R(void *p) { return (real *)p; }
    dim3 zone_grid() { return grid2d(2 * c->zone, 2 * c->zone, c->Ntot); }
    dim3 interior_grid(int ncells) { return grid2d(c->N - 2, c->N - 2, ncells); }
    dim3 box_grid() { return grid2d(c->M, c->M, c->Ntot); }
    cx *fb(int k) { return (cx *)c->fftbuf + (size_t)k * c->Ntot * c->M * c->M; }

    int centres() {
        const int N = c->N;
        PFAG_CUDA_CHECK(cudaMemsetAsync(c->d_cacc, 0, sizeof(long long) * 3 * c->Ntot, c->stream));
        int nb = (int)std::min<size_t>(64, ((size_t)N * N + 255) / 256);
        k_centres_accum<real><<<dim3(nb, c->Ntot), 256, 0, c->stream>>>(R(c->phi), N, c->d_cacc);
        PFAG_LAUNCHED(c);
        k_centres_finalize<<<(c->Ntot + 127) / 128, 128, 0, c->stream>>>(c->d_cacc, c->Ntot, N, c->zone, c->d_xc,
                                                                           c->d_yc, c->d_err);
        PFAG_LAUNCHED(c);
        return PFAG_OK;
    }
    int maps() {
        void **m = c->maps;
        k_maps<real><<<zone_grid(), dim3(TBX, TBY), 0, c->stream>>>(
            R(c->phi), R(c->lum), R(c->ecm), c->d_xc, c->d_yc, c->dp, R(m[0]), R(m[1]), R(m[2]), R(m[3]), R(m[4]),
            R(m[5]));
        PFAG_LAUNCHED(c);
        return PFAG_OK;
    }
    int hfunc3d() {
        k_hfunc_zone<real><<<zone_grid(), dim3(TBX, TBY), 0, c->stream>>>(R(c->phi), R(c->hfunc), c->d_xc, c->d_yc,
                                                                           c->N, c->zone);
        PFAG_LAUNCHED(c);
        return PFAG_OK;
    }
    int hfunc2d() {
        k_hfunc_2d<real><<<592, 256, 0, c->stream>>>(R(c->lum), R(c->ecm), R(c->hlum), R(c->hecm), c->ng);
        PFAG_LAUNCHED(c);
        return PFAG_OK;
    }
    int bc_cells(void *t, int ncells) {
        k_bc_cells<real><<<dim3((4 * c->N + 255) / 256, ncells), 256, 0, c->stream>>>(R(t), c->N, ncells);
        PFAG_LAUNCHED(c);
        return PFAG_OK;
    }
    real c4() { return (real)(1.0 / c->dp.dx / c->dp.dx / 4.0); }
    int norm_grad() {
        k_norm_grad<real><<<interior_grid(c->Ntot), dim3(TBX, TBY), 0, c->stream>>>(R(c->phi), R(c->g), c->N, c4());
        PFAG_LAUNCHED(c);
        return bc_cells(c->g, c->Ntot);
    }
    int prod_norm_delta() {
        k_prod_norm_delta<real><<<zone_grid(), dim3(TBX, TBY), 0, c->stream>>>(
            R(c->g), R(c->phi), R(c->pnd), c->d_xc, c->d_yc, c->N, c->zone, (real)c->dp.sigma);
        PFAG_LAUNCHED(c);
        return PFAG_OK;
    }
    int psi() {
        k_psi<real><<<592, 256, 0, c->stream>>>(R(c->hfunc), R(c->psi), c->ng, c->Ntot);
        PFAG_LAUNCHED(c);
        return PFAG_OK;
    }
    int sum_s() {
        int nblk = RED_BLOCKS;
        if (c->serial_sums) {
            nblk = 1;
            k_serial_sum_cells<real><<<(c->Ntot + 63) / 64, 64, 0, c->stream>>>(R(c->hfunc), c->N, c->Ntot,
                                                                                c->dp.dx, c->d_part);
        } else {
            k_sum_cells<real><<<dim3(RED_BLOCKS, c->Ntot), RED_THREADS, 0, c->stream>>>(R(c->hfunc), c->ng,
                                                                                       c->dp.dx * c->dp.dx, c->d_part);
        }
        PFAG_LAUNCHED(c);
        k_sum_s_finalize<<<(c->Ntot + 127) / 128, 128, 0, c->stream>>>(c->d_part, nblk, c->Ntot, c->dp.alpha,
                                                                         c->dp.s0, c->d_s, c->d_f0);
        PFAG_LAUNCHED(c);
        return PFAG_OK;
    }
    int fft(cx *in, cx *out, int dir) {
        PFAG_CUFFT_CHECK(FFTX<real>::exec(c->plan, in, out, dir));
        c->launches += 2;   // cuFFT library launches (row and column passes)
        return PFAG_OK;
    }
    int cortices() {
        const int N = c->N, z = c->zone, M = c->M;
        cx *T = fb(0), *TR = fb(1), *Frho = fb(2), *Freact = fb(3), *Fxx = fb(4), *Fxy = fb(5), *Fyy = fb(6),
           *Fvx = fb(7), *Fvy = fb(8), *Frvx = fb(9), *Frvy = fb(10);
        dim3 bg = box_grid(), tb(TBX, TBY);
        cudaStream_t s = c->stream;
        k_box_load<real><<<bg, tb, 0, s>>>(R(c->rho), T, c->d_xc, c->d_yc, N, z, M); PFAG_LAUNCHED(c);
        PFAG_TRY(fft(T, Frho, CUFFT_FORWARD));
        k_box_deg_gen<real><<<bg, tb, 0, s>>>(R(c->maps[0]), R(c->rho), R(c->maps[1]), R(c->pnd), T, c->d_xc,
                                               c->d_yc, N, z, M);
        PFAG_LAUNCHED(c);
        PFAG_TRY(fft(T, Freact, CUFFT_FORWARD));
        k_pi<real><<<zone_grid(), tb, 0, s>>>(R(c->rho), R(c->g), R(c->phi), R(c->maps[2]), R(c->maps[3]),
                                              R(c->maps[5]), c->d_xc, c->d_yc, N, z, c4(), R(c->pixx), R(c->pixy),
                                              R(c->piyy));
        PFAG_LAUNCHED(c);
        k_box_load<real><<<bg, tb, 0, s>>>(R(c->pixx), T, c->d_xc, c->d_yc, N, z, M); PFAG_LAUNCHED(c);
        PFAG_TRY(fft(T, Fxx, CUFFT_FORWARD));
        k_box_load<real><<<bg, tb, 0, s>>>(R(c->pixy), T, c->d_xc, c->d_yc, N, z, M); PFAG_LAUNCHED(c);
        PFAG_TRY(fft(T, Fxy, CUFFT_FORWARD));
        k_box_load<real><<<bg, tb, 0, s>>>(R(c->piyy), T, c->d_xc, c->d_yc, N, z, M); PFAG_LAUNCHED(c);
        PFAG_TRY(fft(T, Fyy, CUFFT_FORWARD));
        k_velocity<real><<<bg, tb, 0, s>>>(Fxx, Fyy, Fxy, Fvx, Fvy, R(c->maps[4]), c->d_xc, c->d_yc, N, z, M,
                                           c->dp.kfac, (real)c->dp.friction);
        PFAG_LAUNCHED(c);
        PFAG_TRY(fft(Fvx, TR, CUFFT_INVERSE));
        k_load_rho_v<real><<<bg, tb, 0, s>>>(R(c->rho), TR, T, c->d_xc, c->d_yc, N, z, M,
                                             c->debug ? R(c->d_vx) : nullptr);
        PFAG_LAUNCHED(c);
        PFAG_TRY(fft(T, Frvx, CUFFT_FORWARD));
        PFAG_TRY(fft(Fvy, TR, CUFFT_INVERSE));
        k_load_rho_v<real><<<bg, tb, 0, s>>>(R(c->rho), TR, T, c->d_xc, c->d_yc, N, z, M,
                                             c->debug ? R(c->d_vy) : nullptr);
        PFAG_LAUNCHED(c);
        PFAG_TRY(fft(T, Frvy, CUFFT_FORWARD));
        k_update_fft_rho<real><<<bg, tb, 0, s>>>(Frho, Freact, Frvx, Frvy, M, (real)c->dp.dt, c->dp.kfac);
        PFAG_LAUNCHED(c);
        PFAG_TRY(fft(Frho, T, CUFFT_INVERSE));
        k_copy_to_rhon<real><<<bg, tb, 0, s>>>(T, R(c->rhon), c->d_xc, c->d_yc, N, z, M); PFAG_LAUNCHED(c);
        return bc_cells(c->rhon, c->Ntot);
    }
    int lum_ecm_update() {
        const int N = c->N;
        // sum_ecm = sum h(ECM) dx^2 over the full grid (FP64)
        if (c->serial_sums) {
            k_serial_sum_cells<real><<<1, 32, 0, c->stream>>>(R(c->hecm), N, 1, c->dp.dx, c->d_scal + 0);
            PFAG_LAUNCHED(c);
        } else {
            k_sum_cells<real><<<dim3(RED_BLOCKS, 1), RED_THREADS, 0, c->stream>>>(R(c->hecm), c->ng,
                                                                                 c->dp.dx * c->dp.dx, c->d_part);
            PFAG_LAUNCHED(c);
            k_sum_partials<<<1, 32, 0, c->stream>>>(c->d_part, RED_BLOCKS, c->d_scal + 0);
            PFAG_LAUNCHED(c);
        }
        k_lum_ecm_update<real><<<interior_grid(1), dim3(TBX, TBY), 0, c->stream>>>(
            R(c->lum), R(c->ecm), R(c->psi), R(c->hlum), R(c->hecm), R(c->lumn), R(c->ecmn), c->dp, c->d_scal + 0);
        PFAG_LAUNCHED(c);
        k_dirichlet<real><<<(4 * N + 255) / 256, 256, 0, c->stream>>>(R(c->lumn), N, (real)0.0, (real)0.0);
        PFAG_LAUNCHED(c);
        k_dirichlet<real><<<(4 * N + 255) / 256, 256, 0, c->stream>>>(R(c->ecmn), N, (real)1.0, (real)1.0);
        PFAG_LAUNCHED(c);
        return PFAG_OK;
    }
    // the lumen's (which 0) or the ECM's relaxation: normals and the loop's state
    // on the device (active, ri, iterations, passed rimax)
    int *lum_state() { return c->d_iflags + 8 * c->Ntot; }
    int lum_begin(int which) {
        const int N = c->N;
        void *f = which ? c->ecm : c->lum, *fn = which ? c->ecmn : c->lumn;
        k_norm_grad_2d<real><<<interior_grid(1), dim3(TBX, TBY), 0, c->stream>>>(R(f), R(c->ngl), N, c4());
        PFAG_LAUNCHED(c);
        PFAG_TRY(bc_cells(c->ngl, 1));
        // J_x, J_y: cell 0's slices of the normal arrays serve as scratch (:743)
        k_lum_normals<real><<<interior_grid(1), dim3(TBX, TBY), 0, c->stream>>>(
            R(fn), R(c->ngl), R(c->jx), R(c->jy), N, (real)(1.0 / (2.0 * c->dp.dx)));
        PFAG_LAUNCHED(c);
        PFAG_TRY(bc_cells(c->jx, 1));
        PFAG_TRY(bc_cells(c->jy, 1));
        k_lum_state<<<1, 32, 0, c->stream>>>(lum_state(), c->dp.rdev0_lum > c->dp.thr_lum ? 1 : 0);
        PFAG_LAUNCHED(c);
        return PFAG_OK;
    }
    // iterations it .. it + count - 1, then the state on its way to the host
    int lum_iters(int which, int it, int count) {
        const int N = c->N;
        void *f = which ? c->ecm : c->lum, *fn = which ? c->ecmn : c->lumn;
        const real side = which ? (real)1.0 : (real)0.0;
        const real A = (real)c->dp.A_resh, B = (real)c->dp.B_resh;
        const dim3 g((N + TBX - 1) / TBX, (N + TBY - 1) / TBY);
        real *T = R(c->lum_t);
        int *st = lum_state();
        for (int k = 0; k < count; k++, it++) {
            real *P = (it & 1) ? R(fn) : T, *Q = (it & 1) ? T : R(fn);
            k_lum_iter<real><<<g, 256, 0, c->stream>>>(P, Q, R(f), R(c->jx), R(c->jy), N, A, B, side,
                                                       c->dp.dx * c->dp.dx, st, c->part_z);
            PFAG_LAUNCHED(c);
            const double *part = c->part_z;
            int npart = (int)(g.x * g.y);
            if (c->serial_sums) {
                k_serial_absdiff<real><<<1, 32, 0, c->stream>>>(Q, R(f), N, c->dp.dx, st, c->d_scal + 1);
                PFAG_LAUNCHED(c);
                part = c->d_scal + 1;
                npart = 1;
            }
            k_lum_check<<<1, RED_THREADS, 0, c->stream>>>(part, npart, c->dp.thr_lum, c->p.rimax, st);
            PFAG_LAUNCHED(c);
        }
        PFAG_CUDA_CHECK(cudaMemcpyAsync(c->h_iflags + 8 * c->Ntot, st, 4 * sizeof(int), cudaMemcpyDeviceToHost,
                                        c->stream));
        return PFAG_OK;
    }
    // after the first LUM_AHEAD iterations: the host looks at the state, enqueues
    // more while the loop runs (iterations past its end do nothing)
    int lum_finish(int which, int *iters_out) {
        int *hst = c->h_iflags + 8 * c->Ntot;
        PFAG_CUDA_CHECK(cudaStreamSynchronize(c->stream));
        for (int it = LUM_AHEAD + 1; hst[0]; it += LUM_AHEAD) {
            PFAG_TRY(lum_iters(which, it, LUM_AHEAD));
            PFAG_CUDA_CHECK(cudaStreamSynchronize(c->stream));
        }
        if (hst[2] & 1) {
            k_lum_last<real><<<592, 256, 0, c->stream>>>(R(which ? c->ecmn : c->lumn), R(c->lum_t), c->ng, lum_state());
            PFAG_LAUNCHED(c);
        }
        if (hst[3]) c->stats.relax_failures++;
        if (iters_out) *iters_out = hst[1];
        return PFAG_OK;
    }
    int reshape_lum(int which, int *iters_out) {
        PFAG_TRY(lum_begin(which));
        PFAG_TRY(lum_iters(which, 1, LUM_AHEAD));
        return lum_finish(which, iters_out);
    }
    int normals() {
        k_normals<real><<<interior_grid(c->Ntot), dim3(TBX, TBY), 0, c->stream>>>(
            R(c->phi), R(c->g), R(c->jx), R(c->jy), c->N, (real)(1.0 / (2.0 * c->dp.dx)));
        PFAG_LAUNCHED(c);
        PFAG_TRY(bc_cells(c->jx, c->Ntot));
        return bc_cells(c->jy, c->Ntot);
    }
    int update_cells() {
        k_update_cells<real><<<zone_grid(), dim3(TBX, TBY), 0, c->stream>>>(
            R(c->phi), R(c->phin), R(c->g), R(c->rho), R(c->hfunc), c->d_f0, R(c->psi), c->d_xc, c->d_yc,
            R(c->hlum), R(c->hecm), c->dp);
        PFAG_LAUNCHED(c);
        return bc_cells(c->phin, c->Ntot);
    }
    static constexpr int CELL_AHEAD = 8, LUM_AHEAD = 2;
    int cell_check(int nblk, bool odd, int *active, int *ri, int *iters) {
        const double *part = c->part_z;
        if (c->serial_sums) {
            const real *Q = odd ? R(c->cell_t) : R(c->phin);
            k_serial_cell_rdev<real><<<(c->Ntot + 63) / 64, 64, 0, c->stream>>>(
                Q, R(c->phi), odd, c->d_xc, c->d_yc, c->N, c->zone, c->Ntot, c->dp.dx, (double)c->dp.Ncur, active,
                c->d_part);
            PFAG_LAUNCHED(c);
            part = c->d_part;
            nblk = 1;
        }
        k_cell_check<<<c->Ntot, 32, 0, c->stream>>>(part, nblk, c->dp.thr_cells, c->p.rimax, active, ri, iters,
                                                    c->d_err);
        PFAG_LAUNCHED(c);
        return PFAG_OK;
    }
    int cells_begin() {
        k_cell_state<<<4, 256, 0, c->stream>>>(c->d_iflags, c->Ntot);
        PFAG_LAUNCHED(c);
        return PFAG_OK;
    }
    // CELL_AHEAD iterations, then the flags on their way to the host: a look costs
    // a copy and a wait, an iteration of stopped cells two launches that return
    // (7 cells of 130 x 130, 17 iterations a step, double: 1255 us a step with five
    // launches and a look per iteration, 693 so)
    int cells_iters() {
        const int Nt = c->Ntot;
        int *active = c->d_iflags, *ri = active + Nt, *iters = active + 2 * Nt;
        const real A = (real)c->dp.A_resh, B = (real)c->dp.B_resh;
        const double scale = c->dp.dx * c->dp.dx / (double)c->dp.Ncur;
        const dim3 g = zone_grid();
        const int nblk = (int)(g.x * g.y);
        real *T = R(c->cell_t);
        for (int k = 0; k < CELL_AHEAD; k += 2) {
            k_cell_iter<real, true><<<g, 256, 0, c->stream>>>(R(c->phi), R(c->phin), T, R(c->jx), R(c->jy), c->d_xc,
                                                             c->d_yc, c->N, c->zone, A, B, scale, active, c->part_z);
            PFAG_LAUNCHED(c);
            PFAG_TRY(cell_check(nblk, true, active, ri, iters));
            k_cell_iter<real, false><<<g, 256, 0, c->stream>>>(R(c->phi), R(c->phin), T, R(c->jx), R(c->jy), c->d_xc,
                                                              c->d_yc, c->N, c->zone, A, B, scale, active, c->part_z);
            PFAG_LAUNCHED(c);
            PFAG_TRY(cell_check(nblk, false, active, ri, iters));
        }
        PFAG_CUDA_CHECK(cudaMemcpyAsync(c->h_iflags, c->d_iflags, sizeof(int) * 2 * Nt, cudaMemcpyDeviceToHost,
                                        c->stream));
        return PFAG_OK;
    }
    int cells_last() {
        k_cell_last<real><<<zone_grid(), 256, 0, c->stream>>>(R(c->phin), R(c->cell_t), c->d_xc, c->d_yc, c->N, c->zone,
                                                              c->d_iflags + 2 * c->Ntot);
        PFAG_LAUNCHED(c);
        return PFAG_OK;
    }
    // waits for the flags; whether some cell still iterates
    int cells_look(bool *any) {
        PFAG_CUDA_CHECK(cudaStreamSynchronize(c->stream));
        *any = false;
        for (int n = 0; n < c->Ntot; n++) *any = *any || c->h_iflags[n];
        return PFAG_OK;
    }
    int reshape_cells() {
        PFAG_TRY(cells_begin());
        for (bool any = true; any;) {
            PFAG_TRY(cells_iters());
            PFAG_TRY(cells_look(&any));
        }
        PFAG_TRY(cells_last());
        return cells_stats();
    }
    int cells_stats() {
        const int Nt = c->Ntot;
        int mx = 0, sm = 0;
        for (int n = 0; n < Nt; n++) {
            // the loop body increments ri once per iteration that does not break
            int it = c->h_iflags[Nt + n];
            c->h_iflags[4 * Nt + n] = it;   // per-cell counts, read by pfag_get_cell_iters
            mx = std::max(mx, it);
            sm += it;
        }
        c->stats.cell_iters_max = mx;
        c->stats.cell_iters_sum = sm;
        return PFAG_OK;
    }
    int copy_back() {
        k_copy<real><<<1184, 256, 0, c->stream>>>(R(c->rho), R(c->rhon), c->nc); PFAG_LAUNCHED(c);
        k_copy<real><<<592, 256, 0, c->stream>>>(R(c->ecm), R(c->ecmn), c->ng); PFAG_LAUNCHED(c);
        k_copy<real><<<592, 256, 0, c->stream>>>(R(c->lum), R(c->lumn), c->ng); PFAG_LAUNCHED(c);
        return PFAG_OK;
    }
    int check_zone() {
        // the reference reads xcenters on the host here (acc update host); so do we
        PFAG_TRY(pfag_check_device_error(c));
        return PFAG_OK;
    }
    // prepare_initial_files.cpp:53-117: the initial fields (when make_fields),
    // then centres, phin <- phi, |grad phi| and normals, the cells' reshaping,
    // rho fitted to the reshaped cells, the lumen/ECM update and their
    // reshaping.  The reference reads hfunc_lum, hfunc_ECM and psi there before
    // anything writes them (fresh, zero-filled allocations); they are zeroed.
    int generate(double rho0, double tol, int make_fields) {
        const int N = c->N, Nt = c->Ntot;
        cudaStream_t s = c->stream;
        PFAG_CUDA_CHECK(cudaMemsetAsync(c->d_err, 0, sizeof(unsigned), s));
        const real rcyst = (real)((double)Nt * 0.9 * c->p.R / c->p.dx / M_PI);
        if (make_fields) {
            const dim3 tb(TBX, TBY), gb((N + TBX - 1) / TBX, (N + TBY - 1) / TBY, Nt);
            PFAG_CUDA_CHECK(cudaMemsetAsync(c->lum, 0, c->ng * c->rsz, s));
            PFAG_CUDA_CHECK(cudaMemsetAsync(c->ecm, 0, c->ng * c->rsz, s));
            k_ini_phi<real><<<gb, tb, 0, s>>>(R(c->phi), N, Nt, (real)c->p.dx, (real)c->p.R, (real)c->p.wi, rcyst);
            PFAG_LAUNCHED(c);
            k_ini_lum_ecm<real><<<dim3(gb.x, gb.y), tb, 0, s>>>(R(c->phi), R(c->lum), R(c->ecm), N, Nt, rcyst);
            PFAG_LAUNCHED(c);
            k_rho_shape<real><<<1184, 256, 0, s>>>(R(c->phi), R(c->rho), c->nc, rho0, tol, 1);
            PFAG_LAUNCHED(c);
        }
        PFAG_CUDA_CHECK(cudaMemsetAsync(c->hfunc, 0, c->nc * c->rsz, s));
        PFAG_CUDA_CHECK(cudaMemsetAsync(c->psi, 0, c->ng * c->rsz, s));
        PFAG_CUDA_CHECK(cudaMemsetAsync(c->hlum, 0, c->ng * c->rsz, s));
        PFAG_CUDA_CHECK(cudaMemsetAsync(c->hecm, 0, c->ng * c->rsz, s));
        PFAG_TRY(centres());
        PFAG_TRY(check_zone());
        k_copy<real><<<1184, 256, 0, s>>>(R(c->phin), R(c->phi), c->nc); PFAG_LAUNCHED(c);
        PFAG_TRY(norm_grad());
        PFAG_TRY(normals());
        PFAG_TRY(reshape_cells());
        k_rho_shape<real><<<1184, 256, 0, s>>>(R(c->phi), R(c->rho), c->nc, rho0, tol, 0);
        PFAG_LAUNCHED(c);
        PFAG_TRY(lum_ecm_update());
        PFAG_TRY(reshape_lum(0, &c->stats.lum_iters));
        PFAG_TRY(reshape_lum(1, &c->stats.ecm_iters));
        PFAG_CUDA_CHECK(cudaStreamSynchronize(s));
        return pfag_check_device_error(c);
    }
    // One stretch of the step without a look of the host: enqueued by f, and from
    // the second step on replayed as a CUDA graph (about 100 launches of a step
    // in five graphs: 7 cells of 130 x 130, 693 us a step with single launches,
    // 474 so).  Profiling and PFAG_NO_GRAPH keep the single launches.
    template <typename Fn> int stretch(int k, Fn f) {
        PlainGraphs *pg = (PlainGraphs *)c->plain_graphs;
        if (!pg || pg->steps < 1 || pg->failed || pfag_prof_on(c) || std::getenv("PFAG_NO_GRAPH")) return f();
        if (!pg->exec[k]) {
            const long l0 = c->launches;
            pg->failed = true;
            if (cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
                const int rc = f();
                cudaGraph_t g = nullptr;
                const cudaError_t e = cudaStreamEndCapture(c->stream, &g);
                if (rc == PFAG_OK && e == cudaSuccess && g && cudaGraphInstantiate(&pg->exec[k], g, 0) == cudaSuccess) {
                    pg->failed = false;
                    pg->launches[k] = c->launches - l0;
                } else {
                    pg->exec[k] = nullptr;
                }
                if (g) cudaGraphDestroy(g);
            }
            c->launches = l0;
            (void)cudaGetLastError();
            if (pg->failed) return f();
        }
        PFAG_CUDA_CHECK(cudaGraphLaunch(pg->exec[k], c->stream));
        c->launches += pg->launches[k];
        return PFAG_OK;
    }
    int step(int it) {
        (void)it;
        PlainGraphs *pg = (PlainGraphs *)c->plain_graphs;
        // the captured launches depend on these two switches
        const int key = (c->serial_sums ? 1 : 0) | (c->debug ? 2 : 0);
        if (pg && pg->key != key) {
            pg->drop();
            pg->key = key;
        }
        PFAG_TRY(centres());
        PFAG_TRY(check_zone());
        PFAG_TRY(stretch(0, [&] {
            PFAG_TRY(maps());
            PFAG_TRY(hfunc3d());
            PFAG_TRY(hfunc2d());
            PFAG_TRY(norm_grad());
            PFAG_TRY(prod_norm_delta());
            PFAG_TRY(psi());
            PFAG_TRY(sum_s());
            PFAG_TRY(cortices());
            PFAG_TRY(lum_ecm_update());
            PFAG_TRY(lum_begin(0));
            return lum_iters(0, 1, LUM_AHEAD);
        }));
        PFAG_TRY(lum_finish(0, &c->stats.lum_iters));
        PFAG_TRY(stretch(1, [&] {
            PFAG_TRY(lum_begin(1));
            return lum_iters(1, 1, LUM_AHEAD);
        }));
        PFAG_TRY(lum_finish(1, &c->stats.ecm_iters));
        PFAG_TRY(stretch(2, [&] {
            PFAG_TRY(normals());
            PFAG_TRY(update_cells());
            PFAG_TRY(cells_begin());
            return cells_iters();
        }));
        bool any = false;
        PFAG_TRY(cells_look(&any));
        while (any) {
            PFAG_TRY(stretch(3, [&] { return cells_iters(); }));
            PFAG_TRY(cells_look(&any));
        }
        PFAG_TRY(stretch(4, [&] {
            PFAG_TRY(cells_last());
            return copy_back();
        }));
        if (pg) pg->steps++;
        return cells_stats();
    }
};

}  // namespace

int pfag_plain_alloc(pfag_ctx *c) {
    const size_t rs = c->rsz, nc = c->nc, ng = c->ng;
    PFAG_CUDA_CHECK(cudaMalloc(&c->g, nc * rs));
    PFAG_CUDA_CHECK(cudaMalloc(&c->pnd, nc * rs));
    PFAG_CUDA_CHECK(cudaMalloc(&c->jx, nc * rs));
    PFAG_CUDA_CHECK(cudaMalloc(&c->jy, nc * rs));
    PFAG_CUDA_CHECK(cudaMalloc(&c->ngl, ng * rs));
    const size_t Z = 2 * (size_t)c->zone;
    PFAG_CUDA_CHECK(cudaMalloc(&c->cell_t, c->Ntot * Z * Z * rs));
    PFAG_CUDA_CHECK(cudaMalloc(&c->lum_t, ng * rs));
    const size_t zb = c->Ntot * ((Z + TBX - 1) / TBX) * ((Z + TBY - 1) / TBY);
    const size_t lb = (size_t)((c->N + TBX - 1) / TBX) * ((c->N + TBY - 1) / TBY);
    PFAG_CUDA_CHECK(cudaMalloc(&c->part_z, std::max(zb, lb) * sizeof(double)));
    for (int k = 0; k < 6; k++) PFAG_CUDA_CHECK(cudaMalloc(&c->maps[k], nc * rs));
    PFAG_CUDA_CHECK(cudaMalloc(&c->pixx, nc * rs));
    PFAG_CUDA_CHECK(cudaMalloc(&c->pixy, nc * rs));
    PFAG_CUDA_CHECK(cudaMalloc(&c->piyy, nc * rs));
    PFAG_CUDA_CHECK(cudaMemset(c->g, 0, nc * rs));
    PFAG_CUDA_CHECK(cudaMemset(c->jx, 0, nc * rs));
    PFAG_CUDA_CHECK(cudaMemset(c->jy, 0, nc * rs));
    const size_t mm = (size_t)c->M * c->M;
    PFAG_CUDA_CHECK(cudaMalloc(&c->fftbuf, 11 * (size_t)c->Ntot * mm * 2 * rs));
    int dims[2] = {c->M, c->M};
    PFAG_CUFFT_CHECK(cufftPlanMany(&c->plan, 2, dims, nullptr, 1, (int)mm, nullptr, 1, (int)mm,
                                   c->prec == 64 ? CUFFT_Z2Z : CUFFT_C2C, c->Ntot));
    PFAG_CUFFT_CHECK(cufftSetStream(c->plan, c->stream));
    c->plan_ok = true;
    c->plain_graphs = new PlainGraphs();
    return PFAG_OK;
}

void pfag_plain_free(pfag_ctx *c) {
    if (PlainGraphs *pg = (PlainGraphs *)c->plain_graphs) {
        pg->drop();
        delete pg;
        c->plain_graphs = nullptr;
    }
    void *bufs[] = {c->g, c->pnd, c->jx, c->jy, c->ngl, c->pixx, c->pixy, c->piyy, c->fftbuf, c->cell_t, c->lum_t,
                    c->part_z};
    for (void *b : bufs) if (b) cudaFree(b);
    for (int k = 0; k < 6; k++) if (c->maps[k]) cudaFree(c->maps[k]);
    if (c->plan_ok) cufftDestroy(c->plan);
    c->plan_ok = false;
}

int pfag_plain_step(pfag_ctx *c, int it, bool) {
    return c->prec == 64 ? Plain<double>(c).step(it) : Plain<float>(c).step(it);
}

int pfag_plain_generate(pfag_ctx *c, double rho0, double tol, int make_fields) {
    return c->prec == 64 ? Plain<double>(c).generate(rho0, tol, make_fields)
                         : Plain<float>(c).generate(rho0, tol, make_fields);
}

// Per-function entry points (the drop-in layer's targets).
#define PLAIN_DISPATCH(ctx, call) \
    ((ctx)->prec == 64 ? Plain<double>(ctx).call : Plain<float>(ctx).call)

int pfag_plain_fn(pfag_ctx *c, const char *which, int arg) {
    std::string w(which);
    if (w == "centres") { PFAG_TRY(PLAIN_DISPATCH(c, centres())); return pfag_check_device_error(c); }
    if (w == "maps") return PLAIN_DISPATCH(c, maps());
    if (w == "hfunc3d") return PLAIN_DISPATCH(c, hfunc3d());
    if (w == "hfunc2d") return PLAIN_DISPATCH(c, hfunc2d());
    if (w == "norm_grad") return PLAIN_DISPATCH(c, norm_grad());
    if (w == "pnd") return PLAIN_DISPATCH(c, prod_norm_delta());
    if (w == "psi") return PLAIN_DISPATCH(c, psi());
    if (w == "sum_s") return PLAIN_DISPATCH(c, sum_s());
    if (w == "cortices") return PLAIN_DISPATCH(c, cortices());
    if (w == "lum_ecm_update") return PLAIN_DISPATCH(c, lum_ecm_update());
    if (w == "reshape_lum") return PLAIN_DISPATCH(c, reshape_lum(arg, arg ? &c->stats.ecm_iters : &c->stats.lum_iters));
    if (w == "normals") return PLAIN_DISPATCH(c, normals());
    if (w == "update_cells") return PLAIN_DISPATCH(c, update_cells());
    if (w == "reshape_cells") return PLAIN_DISPATCH(c, reshape_cells());
    if (w == "copy_back") return PLAIN_DISPATCH(c, copy_back());
    pfag_set_error("unknown plain function %s", which);
    return PFAG_E_ARG;
}
