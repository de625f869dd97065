// LDA exchange-correlation on a quadrature grid, replacing the reference's per-element
// adaptive quadrature (kohnsham/integration.py:7-61):
//   k_basis_on_grid  Basis.value / PrimitiveBasis.value (objects/basis_function.py,
//                    objects/primitive_basis_function.py:44-60) of every function at every
//                    grid point, one thread per (point, shell): the contracted radial
//                    factor sum_k coef_k exp(-alpha_k r^2) once per shell, then one product
//                    per Cartesian component (s; x,y,z; xx,yy,zz,xy,xz,yz)
//   k_lda            per point: Slater exchange (kohnsham/exchange/slater_exchange.py) and
//                    Vosko-Wilk-Nusair correlation (kohnsham/correlation/local_density.py)
//                    energy density and potential, times the quadrature weight
//   k_xc_density, k_xc_matrix, k_xc_sum   a whole XC build for one density: rho =
//                    diag(Phi P Phi^T) with the functionals at its end, V = Phi^T diag(w v) Phi
//                    over its lower triangle, and the sums of the blocks' parts in a fixed order
#include <cuda_runtime.h>
#include "gs_args.h"

namespace {

constexpr int kThreads = 256;
constexpr double kRhoFloor = 1e-300;

__global__ void __launch_bounds__(kThreads)
k_basis_on_grid(const double* __restrict__ centre, const int* __restrict__ l,
                const int* __restrict__ prim_off, const double* __restrict__ expo,
                const double* __restrict__ coef, const double* __restrict__ comp_scale,
                const int* __restrict__ func_off, int nshell, int nbf, long long npts,
                const double* __restrict__ pts, double* __restrict__ phi) {
    const long long total = npts * nshell;
    for (long long q = (long long)blockIdx.x * kThreads + threadIdx.x; q < total;
         q += (long long)gridDim.x * kThreads) {
        const long long g = q / nshell;
        const int s = (int)(q - g * nshell);
        const double dx = pts[3 * g] - centre[3 * s];
        const double dy = pts[3 * g + 1] - centre[3 * s + 1];
        const double dz = pts[3 * g + 2] - centre[3 * s + 2];
        const double r2 = dx * dx + dy * dy + dz * dz;
        double rad = 0.0;
        for (int k = prim_off[s]; k < prim_off[s + 1]; ++k) rad += coef[k] * exp(-expo[k] * r2);
        const double* cs = comp_scale + 6 * s;
        double* out = phi + g * nbf + func_off[s];
        const int L = l[s];
        if (L == 0) {
            out[0] = cs[0] * rad;
        } else if (L == 1) {
            out[0] = cs[0] * dx * rad;
            out[1] = cs[1] * dy * rad;
            out[2] = cs[2] * dz * rad;
        } else {
            out[0] = cs[0] * dx * dx * rad;
            out[1] = cs[1] * dy * dy * rad;
            out[2] = cs[2] * dz * dz * rad;
            out[3] = cs[3] * dx * dy * rad;
            out[4] = cs[4] * dx * dz * rad;
            out[5] = cs[5] * dy * dz * rad;
        }
    }
}

struct LdaParams {
    double slater_alpha;       // 0: no exchange
    int vwn;                   // 0: no correlation
    double a, x0, b, c;        // VWN fit (a in Rydberg)
};

// Energy per electron and potential of the selected functionals at density rho > 0.
__device__ __forceinline__ void lda_point(double rho, const LdaParams& p, double& eps, double& v) {
    eps = 0.0;
    v = 0.0;
    const double third = 1.0 / 3.0;
    if (p.slater_alpha != 0.0) {
        const double k = p.slater_alpha * cbrt(3.0 / 3.14159265358979323846) * cbrt(rho);
        eps += -(9.0 / 8.0) * k;
        v += -(3.0 / 2.0) * k;
    }
    if (p.vwn) {
        const double a = p.a / 2.0;   // Rydberg to Hartree
        const double x = sqrt(cbrt(3.0 / (4.0 * 3.14159265358979323846 * rho)));
        const double xx = x * x + p.b * x + p.c;
        const double xx0 = p.x0 * p.x0 + p.b * p.x0 + p.c;
        const double q = sqrt(4.0 * p.c - p.b * p.b);
        const double at = atan(q / (2.0 * x + p.b));
        const double dx0 = x - p.x0;
        const double e = a * (log(x * x / xx) + (2.0 * p.b / q) * at -
                              (p.b * p.x0 / xx0) *
                                  (log(dx0 * dx0 / xx) + (2.0 * (p.b + 2.0 * p.x0) / q) * at));
        eps += e;
        v += e - (a * third) * ((p.c * dx0 - p.b * p.x0 * x) / (dx0 * xx));
    }
}

__global__ void __launch_bounds__(kThreads)
k_lda(long long npts, const double* __restrict__ rho, const double* __restrict__ w, LdaParams p,
      double* __restrict__ wv, double* __restrict__ we) {
    for (long long g = (long long)blockIdx.x * kThreads + threadIdx.x; g < npts;
         g += (long long)gridDim.x * kThreads) {
        const double r = rho[g];
        double eps = 0.0, v = 0.0;
        // zero density contributes nothing (the reference returns 0 there); so do a
        // rounding-negative density of a positive semidefinite P and a subnormal one,
        // whose Wigner-Seitz radius 3 / (4 pi rho) would overflow
        if (r > kRhoFloor) lda_point(r, p, eps, v);
        wv[g] = w[g] * v;
        we[g] = w[g] * r * eps;
    }
}

// ---------------------------------------------------------------------- one XC build
// rho and V are contractions of the same matrix with itself, so both need only a triangle:
// rho_g = sum_i phi_gi (sum_{c <= i} Q_ic phi_gc) with Q_ic = P_ic + P_ci below the diagonal,
// and V's lower triangle, N (N + 1) / 2 multiply-adds a point each, half of what two GEMMs
// take.  Both are bound by the FP64 pipe (64 cycles a warp-wide multiply-add on each of an
// SM's four schedulers); one or two warps a scheduler with eight or sixteen independent
// chains fill it, and shared memory, at two to twenty cycles a multiply-add of that, is no
// limit.  129,600 points, 76 functions: 1.54 ms a build, of which the triangles' multiply-adds
// alone are 1.2 ms; with GEMMs 5.8 ms (0.30 and 0.81 TFLOP/s) and 0.3 ms of elementwise passes.
constexpr int kXcPoints = 32;              // points of a density block, one a lane
constexpr int kXcWarps = 4;
constexpr int kXcCols = 8;                 // columns of Q a warp takes at a time
constexpr int kXcStage = 32;               // points of a staged tile of the matrix kernel

__host__ __device__ inline int xc_pad(int n) { return (n + kXcCols - 1) / kXcCols * kXcCols; }

// Q (n rows of xc_pad(n) columns): the folded lower triangle of P, zero elsewhere.
__global__ void k_xc_fold(int n, const double* __restrict__ P, double* __restrict__ Q) {
    const int np = xc_pad(n);
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= n * np) return;
    const int i = x / np, c = x - i * np;
    Q[x] = c == i ? P[i * n + i] : c < i ? P[i * n + c] + P[c * n + i] : 0.0;
}

// Block: kXcPoints points, rows of Phi in shared memory at an odd pitch (a lane reads its own
// point's row: no bank conflicts).  Warp w takes column strips dealt in a zigzag (strip s
// needs the rows from 8 s on), eight accumulators a lane; the warps' parts of rho are added
// in warp order by the first warp, which evaluates the functionals and the block's energy.
__global__ void __launch_bounds__(32 * kXcWarps)
k_xc_density(long long npts, int n, const double* __restrict__ phi, const double* __restrict__ Q,
             const double* __restrict__ w, LdaParams p, double* __restrict__ wv,
             double* __restrict__ epart) {
    extern __shared__ __align__(16) double sm[];
    const int pitch = n | 1, np = xc_pad(n);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long g0 = (long long)blockIdx.x * kXcPoints;
    const int have = (int)(npts - g0 < kXcPoints ? npts - g0 : kXcPoints);
    double* part = sm + kXcPoints * pitch;
    for (int x = threadIdx.x; x < kXcPoints * n; x += 32 * kXcWarps) {
        const int g = x / n, i = x - g * n;
        sm[g * pitch + i] = g < have ? phi[g0 * n + x] : 0.0;
    }
    __syncthreads();
    const double* row = sm + lane * pitch;
    double rho = 0.0;
    const int strips = np / kXcCols;
    for (int k = 0; k * kXcWarps < strips; ++k) {
        const int s = k * kXcWarps + ((k & 1) ? kXcWarps - 1 - warp : warp);
        if (s >= strips) continue;
        const int c0 = s * kXcCols;
        double t[kXcCols];
#pragma unroll
        for (int c = 0; c < kXcCols; ++c) t[c] = 0.0;
        // rows c0.. of the strip; its first eight hold the diagonal, their upper part zeros
#pragma unroll 4
        for (int i = c0; i < n; ++i) {
            const double2* q = reinterpret_cast<const double2*>(Q + (size_t)i * np + c0);
            const double f = row[i];
#pragma unroll
            for (int c = 0; c < kXcCols / 2; ++c) {
                const double2 v = __ldg(q + c);
                t[2 * c] = fma(f, v.x, t[2 * c]);
                t[2 * c + 1] = fma(f, v.y, t[2 * c + 1]);
            }
        }
#pragma unroll
        for (int c = 0; c < kXcCols; ++c)
            if (c0 + c < n) rho = fma(t[c], row[c0 + c], rho);
    }
    part[warp * kXcPoints + lane] = rho;
    __syncthreads();
    if (warp != 0) return;
    double r = 0.0;
#pragma unroll
    for (int k = 0; k < kXcWarps; ++k) r += part[k * kXcPoints + lane];
    double e = 0.0;
    if (lane < have) {
        double eps = 0.0, v = 0.0;
        if (r > kRhoFloor) lda_point(r, p, eps, v);
        wv[g0 + lane] = w[g0 + lane] * v;
        e = w[g0 + lane] * r * eps;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if (lane == 0) epart[blockIdx.x] = e;
}

// Micro-tile q of V's lower triangle in 4 x 4 blocks: rows 4 r.., columns 4 c.., c <= r.
__device__ __forceinline__ void xc_tile(int q, int& r, int& c) {
    r = (int)((sqrtf(8.0f * (float)q + 1.0f) - 1.0f) * 0.5f);
    while (r * (r + 1) / 2 > q) --r;
    while ((r + 1) * (r + 2) / 2 <= q) ++r;
    c = q - r * (r + 1) / 2;
}

// Block (x, y): points of part x, micro-tiles y T.. (one a thread, 16 accumulators).  Tiles
// of kXcStage points are staged twice, plain and times w v; rows are padded to whole
// micro-tiles with zeros.
__global__ void __launch_bounds__(256)
k_xc_matrix(long long npts, int n, int ntile, long long per, const double* __restrict__ phi,
            const double* __restrict__ wv, double* __restrict__ part) {
    extern __shared__ __align__(16) double sm[];
    const int m4 = (n + 3) / 4 * 4;
    double* A = sm;
    double* B = sm + kXcStage * m4;
    const int q = blockIdx.y * blockDim.x + threadIdx.x;
    int r = 0, c = 0;
    if (q < ntile) xc_tile(q, r, c);
    double acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0;
    const long long lo = (long long)blockIdx.x * per;
    const long long hi = lo + per < npts ? lo + per : npts;
    for (long long g0 = lo; g0 < hi; g0 += kXcStage) {
        const int have = (int)(hi - g0 < kXcStage ? hi - g0 : kXcStage);
        __syncthreads();
        for (int x = threadIdx.x; x < kXcStage * m4; x += blockDim.x) {
            const int g = x / m4, i = x - g * m4;
            const double f = g < have && i < n ? phi[(g0 + g) * n + i] : 0.0;
            A[x] = f;
            B[x] = g < have ? f * wv[g0 + g] : 0.0;
        }
        __syncthreads();
        if (q < ntile) {
#pragma unroll 2
            for (int g = 0; g < kXcStage; ++g) {
                const double2* a = reinterpret_cast<const double2*>(A + g * m4 + 4 * r);
                const double2* b = reinterpret_cast<const double2*>(B + g * m4 + 4 * c);
                const double2 a0 = a[0], a1 = a[1], b0 = b[0], b1 = b[1];
                const double av[4] = {a0.x, a0.y, a1.x, a1.y}, bv[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = fma(av[i], bv[j], acc[i][j]);
            }
        }
    }
    if (q >= ntile) return;
    double2* o = reinterpret_cast<double2*>(part + ((size_t)blockIdx.x * ntile + q) * 16);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        o[2 * i] = make_double2(acc[i][0], acc[i][1]);
        o[2 * i + 1] = make_double2(acc[i][2], acc[i][3]);
    }
}

// V from the parts, in a fixed order, both triangles; the last block adds the energies.
__global__ void __launch_bounds__(kThreads)
k_xc_sum(int n, int ntile, int nparts, const double* __restrict__ part, int neparts,
         const double* __restrict__ epart, double* __restrict__ V, double* __restrict__ E) {
    if (blockIdx.x == gridDim.x - 1) {
        __shared__ double s[kThreads];
        double e = 0.0;
        for (int k = threadIdx.x; k < neparts; k += kThreads) e += epart[k];
        s[threadIdx.x] = e;
        __syncthreads();
        for (int o = kThreads / 2; o > 0; o >>= 1) {
            if ((int)threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0) *E = s[0];
        return;
    }
    const int x = blockIdx.x * kThreads + threadIdx.x;
    if (x >= ntile * 16) return;
    int r, c;
    xc_tile(x / 16, r, c);
    const int i = 4 * r + (x & 15) / 4, j = 4 * c + (x & 3);
    // eight sums, then theirs in pairs: the parts' own errors average out, so the longest chain of
    // additions here sets V's.  Against quadruple precision (64,800 points, 7 to 26 functions) V is
    // off by 0.7 to 3.0e-16 of its norm, with one chain 1.7 to 10e-16, through cuBLAS GEMMs 2.4 to
    // 8.2e-16; the build of 129,600 points and 76 functions stays at 1.54 ms
    double s[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = 0.0;
    const size_t step = (size_t)ntile * 16;
    const double* from = part + x;
    int k = 0;
    for (; k + 8 <= nparts; k += 8, from += 8 * step)
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i] += from[i * step];
#pragma unroll
    for (int i = 0; i < 7; ++i)
        if (k + i < nparts) s[i] += from[i * step];
    const double v = ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
    if (i < n && j <= i) {
        V[(size_t)i * n + j] = v;
        V[(size_t)j * n + i] = v;
    }
}

// Shapes of an XC build.
struct XcPlan {
    int ntile, threads, ny, nx, nep;
    long long per;
    size_t density_smem, matrix_smem, bytes;
};
XcPlan xc_plan(long long npts, int n) {
    XcPlan p;
    const int m = (n + 3) / 4;
    p.ntile = m * (m + 1) / 2;
    p.ny = (p.ntile + 255) / 256;
    p.threads = ((p.ntile + p.ny - 1) / p.ny + 31) / 32 * 32;
    // two blocks an SM over all the parts of the points; a part is whole staged tiles
    const long long want = (2LL * gs::sm_count() + p.ny - 1) / p.ny;
    p.per = ((npts + want - 1) / want + kXcStage - 1) / kXcStage * kXcStage;
    p.nx = (int)((npts + p.per - 1) / p.per);
    p.nep = (int)((npts + kXcPoints - 1) / kXcPoints);
    p.density_smem = ((size_t)kXcPoints * (n | 1) + kXcWarps * kXcPoints) * sizeof(double);
    p.matrix_smem = 2 * (size_t)kXcStage * 4 * m * sizeof(double);
    p.bytes = ((size_t)n * xc_pad(n) + npts + p.nep + (size_t)p.nx * p.ntile * 16 + 8) *
              sizeof(double);
    return p;
}
// functions whose tiles fit a block's shared memory
constexpr int kXcMaxFunctions = 440;

unsigned grid_for(long long work) {
    long long b = (work + kThreads - 1) / kThreads;
    const long long cap = 16LL * gs::sm_count();   // grid-stride beyond 16 blocks per SM
    return (unsigned)(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace

extern "C" {

int gs_basis_on_grid(const double* centre, const int* l, const int* prim_off, const double* expo,
                     const double* coef, const double* comp_scale, const int* func_off,
                     int nshell, int nbf, long long npts, const double* points, double* phi,
                     void* stream) {
    if (nshell < 0 || nbf < 0 || npts < 0) return GS_ERR_ARG;
    if (nshell == 0 || npts == 0) return GS_OK;
    if (!centre || !l || !prim_off || !expo || !coef || !comp_scale || !func_off || !points ||
        !phi)
        return GS_ERR_ARG;
    k_basis_on_grid<<<grid_for(npts * nshell), kThreads, 0, (cudaStream_t)stream>>>(
        centre, l, prim_off, expo, coef, comp_scale, func_off, nshell, nbf, npts, points, phi);
    return cudaGetLastError() == cudaSuccess ? GS_OK : GS_ERR_CUDA;
}

int gs_lda_xc(long long npts, const double* rho, const double* weights, double slater_alpha,
              int vwn, double vwn_a, double vwn_x0, double vwn_b, double vwn_c,
              double* weighted_potential, double* weighted_energy, void* stream) {
    if (npts < 0) return GS_ERR_ARG;
    if (npts == 0) return GS_OK;
    if (!rho || !weights || !weighted_potential || !weighted_energy) return GS_ERR_ARG;
    if (vwn && !(4.0 * vwn_c - vwn_b * vwn_b > 0.0)) return GS_ERR_ARG;
    LdaParams p{slater_alpha, vwn, vwn_a, vwn_x0, vwn_b, vwn_c};
    k_lda<<<grid_for(npts), kThreads, 0, (cudaStream_t)stream>>>(npts, rho, weights, p,
                                                                 weighted_potential,
                                                                 weighted_energy);
    return cudaGetLastError() == cudaSuccess ? GS_OK : GS_ERR_CUDA;
}

int gs_xc_lda_max_functions(void) { return kXcMaxFunctions; }

long long gs_xc_lda_workspace(long long npts, int nbf) {
    if (npts <= 0 || nbf <= 0 || nbf > kXcMaxFunctions) return 0;
    return (long long)xc_plan(npts, nbf).bytes;
}

int gs_xc_lda(long long npts, int nbf, const double* phi, const double* density,
              const double* weights, double slater_alpha, int vwn, double vwn_a, double vwn_x0,
              double vwn_b, double vwn_c, double* matrix, double* energy, void* workspace,
              long long ws_bytes, void* stream) {
    if (npts <= 0 || npts >= (1LL << 31) * kXcPoints || nbf <= 0 || !phi || !density || !weights ||
        !matrix || !energy || !workspace)
        return GS_ERR_ARG;
    if (nbf > kXcMaxFunctions) return GS_ERR_LIMIT;
    if (vwn && !(4.0 * vwn_c - vwn_b * vwn_b > 0.0)) return GS_ERR_ARG;
    const XcPlan p = xc_plan(npts, nbf);
    if (ws_bytes < (long long)p.bytes || ((size_t)workspace & 15)) return GS_ERR_NOMEM;
    cudaStream_t st = (cudaStream_t)stream;
    double* Q = (double*)workspace;                        // n xc_pad(n), a multiple of eight
    double* part = Q + (size_t)nbf * xc_pad(nbf);          // nx ntile 16
    double* wv = part + (size_t)p.nx * p.ntile * 16;
    double* epart = wv + npts;
    if (cudaFuncSetAttribute(k_xc_density, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             227 * 1024) != cudaSuccess ||
        cudaFuncSetAttribute(k_xc_matrix, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             227 * 1024) != cudaSuccess)
        return GS_ERR_CUDA;
    const int fold = nbf * xc_pad(nbf);
    k_xc_fold<<<(fold + kThreads - 1) / kThreads, kThreads, 0, st>>>(nbf, density, Q);
    k_xc_density<<<p.nep, 32 * kXcWarps, p.density_smem, st>>>(
        npts, nbf, phi, Q, weights, LdaParams{slater_alpha, vwn, vwn_a, vwn_x0, vwn_b, vwn_c}, wv,
        epart);
    k_xc_matrix<<<dim3(p.nx, p.ny), p.threads, p.matrix_smem, st>>>(npts, nbf, p.ntile, p.per, phi,
                                                                   wv, part);
    k_xc_sum<<<(p.ntile * 16 + kThreads - 1) / kThreads + 1, kThreads, 0, st>>>(
        nbf, p.ntile, p.nx, part, p.nep, epart, matrix, energy);
    return cudaGetLastError() == cudaSuccess ? GS_OK : GS_ERR_CUDA;
}

}  // extern "C"
