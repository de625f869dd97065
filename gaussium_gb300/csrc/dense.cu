// Dense N^4 ERI tensor from the unique shell-quartet blocks: the 8-fold expansion of the
// reference's create_repulsion_matrix (matrixelements/electron_repulsion_matrix.py:43-45,
// which fills repulsion[i,j,k,l] and its seven images for every canonical key).
//
// One warp per unique shell quartet (A B | C D): its lanes stride over the block's
// n_A n_B n_C n_D elements (row-major, as the class kernels write them at offset[q]) and
// store each value at its eight index images.  Where shells repeat (A = B, C = D, or
// AB = CD) a block holds an index orbit more than once, with values equal only to
// rounding (they come from different recursion paths); there only the element with
// a >= b, c >= d and (a, b) >= (c, d) writes, so every orbit has one writer and the tensor
// has the reference's exact 8-fold symmetry.  HBM-bound: every element written once or
// more, 8 bytes each.
#include <cuda_runtime.h>
#include "gs_args.h"

namespace {

constexpr int kWarps = 8;

__device__ __forceinline__ int ncart(int l) { return (l + 1) * (l + 2) / 2; }

__global__ void __launch_bounds__(32 * kWarps)
k_dense_expand(long long nq, const int4* __restrict__ quartets,
               const long long* __restrict__ offsets, const double* __restrict__ vals,
               const int* __restrict__ l, const int* __restrict__ func_off, long long n,
               double* __restrict__ out) {
    const long long q = (long long)blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (q >= nq) return;
    const int lane = threadIdx.x & 31;
    const int4 s = quartets[q];
    const int nb = ncart(l[s.y]), nc = ncart(l[s.z]), nd = ncart(l[s.w]);
    const int size = ncart(l[s.x]) * nb * nc * nd;
    const long long fa = func_off[s.x], fb = func_off[s.y], fc = func_off[s.z], fd = func_off[s.w];
    const double* v = vals + offsets[q];
    for (int e = lane; e < size; e += 32) {
        const int id = e % nd, ic = (e / nd) % nc, ib = (e / (nd * nc)) % nb, ia = e / (nd * nc * nb);
        const long long a = fa + ia, b = fb + ib, c = fc + ic, d = fd + id;
        if ((s.x == s.y && a < b) || (s.z == s.w && c < d) ||
            (s.x == s.z && s.y == s.w && (a < c || (a == c && b < d))))
            continue;                              // another element of the orbit writes
        const double x = v[e];
        out[((a * n + b) * n + c) * n + d] = x;
        out[((b * n + a) * n + c) * n + d] = x;
        out[((a * n + b) * n + d) * n + c] = x;
        out[((b * n + a) * n + d) * n + c] = x;
        out[((c * n + d) * n + a) * n + b] = x;
        out[((d * n + c) * n + a) * n + b] = x;
        out[((c * n + d) * n + b) * n + a] = x;
        out[((d * n + c) * n + b) * n + a] = x;
    }
}

// Unique quartets as products of ranges of a pair list: range r holds the quartets (bra pair
// b, ket pair k) with b in [bra, bra + nbra) and k in [ket, ket + nket), or, for nket = 0, the
// pairs k <= b of [bra, bra + nbra) with themselves.  Its quartets are numbers first[r] ..
// first[r + 1]; their blocks have size[r] elements from base[r] on.
struct QuartetRange {
    long long first, base;
    int bra, nbra, ket, nket, size, pad;
};

__global__ void __launch_bounds__(256)
k_product_tasks(long long n, int nranges, const QuartetRange* __restrict__ ranges,
                const int2* __restrict__ pair_shells, int* __restrict__ tasks,
                int4* __restrict__ quartets, long long* __restrict__ offsets) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    int lo = 0, hi = nranges - 1;                  // the last range that starts at or before t
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (ranges[mid].first <= t) lo = mid; else hi = mid - 1;
    }
    const QuartetRange r = ranges[lo];
    const long long x = t - r.first;
    int b, k;
    if (r.nket > 0) {
        b = r.bra + (int)(x / r.nket);
        k = r.ket + (int)(x % r.nket);
    } else {                                       // row i of the triangle holds i + 1 pairs
        long long i = (long long)((sqrt(8.0 * (double)x + 1.0) - 1.0) * 0.5);
        while (i * (i + 1) / 2 > x) --i;
        while ((i + 1) * (i + 2) / 2 <= x) ++i;
        b = r.bra + (int)i;
        k = r.bra + (int)(x - i * (i + 1) / 2);
    }
    const long long off = r.base + x * r.size;
    int* w = tasks + 6 * t;                        // WriteTask: bra, ket, code, pad, offset
    w[0] = b;
    w[1] = k;
    w[2] = 0;
    w[3] = 0;
    *reinterpret_cast<long long*>(w + 4) = off;
    const int2 B = pair_shells[b], K = pair_shells[k];
    quartets[t] = make_int4(B.x, B.y, K.x, K.y);
    offsets[t] = off;
}

}  // namespace

extern "C" {

int gs_product_tasks(long long n, int nranges, const void* ranges, const int* pair_shells,
                     void* tasks, int* quartets, long long* offsets, void* stream) {
    if (n < 0 || nranges < 0 ||
        (n > 0 && (nranges == 0 || !ranges || !pair_shells || !tasks || !quartets || !offsets)))
        return GS_ERR_ARG;
    if (n == 0) return GS_OK;
    const long long blocks = (n + 255) / 256;
    if (blocks > 0x7fffffffLL) return GS_ERR_ARG;
    k_product_tasks<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(
        n, nranges, (const QuartetRange*)ranges, (const int2*)pair_shells, (int*)tasks,
        (int4*)quartets, offsets);
    return cudaGetLastError() == cudaSuccess ? GS_OK : GS_ERR_CUDA;
}

int gs_dense_expand(long long nq, const int* quartets, const long long* offsets,
                    const double* vals, const int* l, const int* func_off, int n, double* out,
                    void* stream) {
    if (nq < 0 || n < 0) return GS_ERR_ARG;
    if (nq == 0) return GS_OK;
    if (!quartets || !offsets || !vals || !l || !func_off || !out) return GS_ERR_ARG;
    const long long blocks = (nq + kWarps - 1) / kWarps;
    if (blocks > 0x7fffffffLL) return GS_ERR_ARG;
    k_dense_expand<<<(unsigned)blocks, 32 * kWarps, 0, (cudaStream_t)stream>>>(
        nq, (const int4*)quartets, offsets, vals, l, func_off, (long long)n, out);
    return cudaGetLastError() == cudaSuccess ? GS_OK : GS_ERR_CUDA;
}

}  // extern "C"
