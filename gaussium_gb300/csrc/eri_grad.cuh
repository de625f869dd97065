// K6 fused ERI adjoint: one warp per unique shell quartet evaluates the derivative
// integrals of all three independent centres from one VRR pass per primitive quartet
// (four weighted contraction sets: 1, 2 alpha, 2 beta, 2 gamma), forms the raised and
// lowered blocks by HRR in shared memory, contracts them with the RHF density weights
//   Gamma_abcd = w (1/2 P_ab P_cd - 1/8 (P_ac P_bd + P_ad P_bc))   (w = orbit size)
// and adds dE/dR of the four centres to the per-atom gradient (D by translational
// invariance).  Programs come from gen_grad.py (GradProg<...>).
#pragma once
#include "eri_wide.cuh"

namespace gs {

template <int LA, int LB, int LC, int LD> struct GradProg;
template <int LA, int LB, int LC, int LD> struct GradThread;

struct GradArgs {
    const PairRec* pairs;
    const PrimRec<double>* prims;   // pad holds the first shell's exponent
    const double* comp_scale;
    const int* func_off;
    const int* shell_atom;
    const int2* tasks;
    int ntask;
    int nbf;
    const double* P;
    double* grad;
    int natom;
    // FP32 evaluation (thread and split forms): recursion and accumulation in FP32 from the
    // FP32 records (pad0 holds the first shell's exponent), HRR and contraction in FP64
    const PrimRec<float>* prims32;
    bool fp32;
    // density-weighted screening: a quartet is evaluated when its Schwarz bound times the
    // largest |P| of its six shell blocks (shell_dmax, nshell x nshell) is at least
    // screen_thr and lies in [prec_lo, prec_hi); screen_thr <= 0 evaluates every quartet
    const double* shell_dmax;
    int nshell;
    double screen_thr, prec_lo, prec_hi;
    int per;                        // tasks a warp of the warp form takes
    const int* ntask_dev;           // if set, the task count (thread and split forms; ntask: bound)
};

__device__ __forceinline__ bool grad_keep(const GradArgs& a, const PairRec& B, const PairRec& K) {
    if (a.screen_thr <= 0.0) return true;
    const int ns = a.nshell;
    const double* d = a.shell_dmax;
    double dm = d[B.sa * ns + B.sb];
    dm = max_nonneg(dm, d[K.sa * ns + K.sb]);
    dm = max_nonneg(dm, d[B.sa * ns + K.sa]);
    dm = max_nonneg(dm, d[B.sa * ns + K.sb]);
    dm = max_nonneg(dm, d[B.sb * ns + K.sa]);
    dm = max_nonneg(dm, d[B.sb * ns + K.sb]);
    const double est = widen(B.qmax) * widen(K.qmax) * dm;
    return !(est < a.screen_thr || est < a.prec_lo || est >= a.prec_hi);
}

__device__ __forceinline__ double prim_expo(const PrimRec<double>& r) { return r.pad; }
__device__ __forceinline__ float prim_expo(const PrimRec<float>& r) { return r.pad0; }

constexpr int kGradWarps = 2;        // warps per block, unless the class's buffer is too large
constexpr int kNCoefG = 36;
// classes with more contracted accumulators than this per warp (3 per lane... 24 per lane)
// keep them in shared memory at their HRR positions instead of in registers
constexpr int kGradRegAcc = 32 * 24;

// Per-warp shared memory of one class: the VRR buffers (coefficients, Boys values, node
// slots) and, in the shared-accumulator form, the accumulators [0, NACC) ahead of them;
// the HRR reuses the whole buffer afterwards.
template <int LA, int LB, int LC, int LD> struct GradLayout {
    using W = GradProg<LA, LB, LC, LD>;
    static constexpr bool SMEM_ACC = W::NACC > kGradRegAcc;
    static constexpr int ACC = SMEM_ACC ? W::NACC : 0;
    static constexpr int SC = kSetupBatch * kNCoefG;
    static constexpr int SF = kSetupBatch * (W::L + 1);
    static constexpr int VRR = ACC + SC + SF + W::NVSLOT;
    // several quartets a warp: the set-up buffers outlive a quartet's HRR, which takes the
    // node buffer's place
    static constexpr int MANY = SC + SF + (W::NVSLOT > W::HSIZE ? W::NVSLOT : W::HSIZE);
    static constexpr int WARP = !SMEM_ACC ? MANY : VRR > W::HSIZE ? VRR : W::HSIZE;
    // two warps per block while they fit the 227 KB a block may use, else one
    static constexpr int WARPS = (size_t)WARP * sizeof(double) * kGradWarps <= 227 * 1024 ? kGradWarps : 1;
    static constexpr size_t BYTES = (size_t)WARP * sizeof(double) * WARPS;
    static_assert((size_t)WARP * sizeof(double) <= 227 * 1024, "gradient class buffer exceeds shared memory");
};

// VRR of the set-up primitive quartets j0 .. j0 + nb and their weighted accumulation: target
// lane + 32 k is added to acc[k] (slot | kind << 16 in ent[k], kind 255: none), or to the
// shared accumulators at their HRR positions, which fill [0, NACC).
template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ void grad_items(const double* __restrict__ sC,
                                           const double* __restrict__ sF, double* node, int j0,
                                           int nb, int lane, double* acc, const unsigned* ent,
                                           double* shared_acc) {
    using W = GradProg<LA, LB, LC, LD>;
    using Lay = GradLayout<LA, LB, LC, LD>;
    constexpr int L = W::L;
    constexpr int NACCW = Lay::SMEM_ACC ? 1 : (W::NACC + 31) / 32;
    const uint4* __restrict__ vrec = W::vrec();
    const int* __restrict__ vseg = W::vseg();
    for (int j = j0; j < j0 + nb; ++j) {
        const double* __restrict__ c = sC + j * kNCoefG;
        if (lane <= L) node[lane] = sF[j * (L + 1) + lane];
        __syncwarp();
        for (int s = 0; s < W::NVSEG; ++s) {
            const int noff = __ldg(vseg + 4 * s), cnt = __ldg(vseg + 4 * s + 1);
            const int nt = __ldg(vseg + 4 * s + 2), sync = __ldg(vseg + 4 * s + 3);
            if (sync && s > 0) __syncwarp();
            int n = lane;
            uint4 ra = make_uint4(0, 0, 0, 0), rb = ra;
            if (n < cnt) {
                ra = __ldg(vrec + 2 * (noff + n));
                rb = __ldg(vrec + 2 * (noff + n) + 1);
            }
            for (; n < cnt; n += 32) {
                const uint4 x = ra, y = rb;
                if (n + 32 < cnt) {
                    ra = __ldg(vrec + 2 * (noff + n + 32));
                    rb = __ldg(vrec + 2 * (noff + n + 32) + 1);
                }
                double r = gs_mul(c[x.y >> 16], node[x.y & 0xffff]);
                r = fma(c[x.z >> 16], node[x.z & 0xffff], r);
                if (nt > 2) r = fma(c[x.w >> 16], node[x.w & 0xffff], r);
                if (nt > 3) r = fma(c[y.x >> 16], node[y.x & 0xffff], r);
                if (nt > 4) r = fma(c[y.y >> 16], node[y.y & 0xffff], r);
                node[x.x & 0xffff] = r;
            }
        }
        __syncwarp();
        if constexpr (Lay::SMEM_ACC) {
            for (int q = lane; q < W::NACC; q += 32) {
                const unsigned e = __ldg(W::acc() + q);
                const int kind = (int)(e >> 16);
                const double w = kind == 0 ? 1.0 : c[31 + kind];
                const int pos = __ldg(W::accpos() + q);
                shared_acc[pos] = fma(w, node[e & 0xffff], shared_acc[pos]);
            }
        } else {
#pragma unroll
            for (int k = 0; k < NACCW; ++k) {
                const unsigned kind = ent[k] >> 16;
                if (kind != 255u) {
                    const double w = kind == 0 ? 1.0 : c[31 + kind];
                    acc[k] = fma(w, node[ent[k] & 0xffff], acc[k]);
                }
            }
        }
        __syncwarp();
    }
}

// Set-up of the primitive quartet (P, Q) into slot x of a round.
template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ void grad_setup_slot(const PrimRec<double>& P, const PrimRec<double>& Q,
                                                double* __restrict__ sC, double* __restrict__ sF,
                                                int x) {
    constexpr int L = GradProg<LA, LB, LC, LD>::L;
    double* c = sC + x * kNCoefG;
    wide_setup_m<L, double>(P, Q, c, sF + x * (L + 1));
    c[32] = twice(P.pad);               // 2 alpha (first bra shell)
    c[33] = twice(P.p - P.pad);         // 2 beta
    c[34] = twice(Q.pad);               // 2 gamma (first ket shell)
    c[35] = 5.0 * c[28];                // 5/(2(p+q)), raised (dd|..) classes
}

// HRR of the accumulators at H, contraction with the density weights and the atomic adds.
// The raised and lowered slots of every (element, centre, direction) come from the class's
// table (gen_grad.contraction_table): worked out in the kernel they were 90,000 instructions
// for one (dd|dd) quartet.  The nine sums over the lanes are reduced by halves (14 FP64
// additions instead of 45), which leaves each in its own lanes for the atomics.
template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ void grad_tail(const GradArgs& a, const int2& task, const PairRec& B,
                                          const PairRec& K, double* H, int lane) {
    using W = GradProg<LA, LB, LC, LD>;
    const unsigned int* __restrict__ hop = W::hop();
    const int* __restrict__ hlev = W::hlev();
    const double dv0 = B.ABx, dv1 = B.ABy, dv2 = B.ABz, dv3 = K.ABx, dv4 = K.ABy, dv5 = K.ABz;
    for (int lv = 0; lv < W::NHLEV; ++lv) {
        const int e1 = __ldg(hlev + lv + 1);
        for (int e = __ldg(hlev + lv) + lane; e < e1; e += 32) {
            const unsigned int u = __ldg(hop + 2 * e), v = __ldg(hop + 2 * e + 1);
            const int d = v >> 16;
            const double dv = d == 0 ? dv0 : d == 1 ? dv1 : d == 2 ? dv2 : d == 3 ? dv3 : d == 4 ? dv4 : dv5;
            H[u & 0xffff] = fma(dv, H[v & 0xffff], H[u >> 16]);
        }
        __syncwarp();
    }
    constexpr int NB = (LB + 1) * (LB + 2) / 2, NC = (LC + 1) * (LC + 2) / 2;
    constexpr int ND = (LD + 1) * (LD + 2) / 2, NBLK = (LA + 1) * (LA + 2) / 2 * NB * NC * ND;
    const int fa = a.func_off[B.sa], fb = a.func_off[B.sb];
    const int fc = a.func_off[K.sa], fd = a.func_off[K.sb];
    const int halves = (B.sa == B.sb) + (K.sa == K.sb) + (task.x == task.y);
    const double w8 = halves == 0 ? 1.0 : halves == 1 ? 0.5 : halves == 2 ? 0.25 : 0.125;
    const int nbf = a.nbf;
    const double* __restrict__ Pm = a.P;
    const double* __restrict__ cs = a.comp_scale;
    const unsigned* __restrict__ con = W::con();
    double g[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) g[k] = 0.0;
    for (int e = lane; e < NBLK; e += 32) {
        const int ia = e / (NB * NC * ND), ib = e / (NC * ND) % NB, ic = e / ND % NC, id = e % ND;
        const int pa = fa + ia, pb = fb + ib, pc = fc + ic, pd = fd + id;
        // w (P_ab P_cd / 2 - (P_ac P_bd + P_ad P_bc) / 8), w8 = w / 8
        const double x = fma(Pm[pa * nbf + pc], Pm[pb * nbf + pd],
                             gs_mul(Pm[pa * nbf + pd], Pm[pb * nbf + pc]));
        const double gam = gs_mul(w8, fma(twice(twice(Pm[pa * nbf + pb])), Pm[pc * nbf + pd], -x));
        // the HRR blocks are unscaled: the element carries the component scales of all four
        // functions (not 1 for the xy, xz, yz components of a d shell)
        const double s = gs_mul(gs_mul(gam, cs[6 * B.sa + ia]),
                                gs_mul(gs_mul(cs[6 * B.sb + ib], cs[6 * K.sa + ic]),
                                       cs[6 * K.sb + id]));
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const unsigned u = __ldg(con + k * NBLK + e);
            const unsigned dn = (u >> 16) & 0x7fffu;
            double v = H[u & 0xffffu];
            if (dn != 0x7fffu) v = fma(u >> 31 ? -2.0 : -1.0, H[dn], v);
            g[k] = fma(s, v, g[k]);
        }
    }
    constexpr unsigned ALL = 0xffffffffu;
    double last = g[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) last = gs_add(__shfl_xor_sync(ALL, last, o), last);
#pragma unroll
    for (int o = 16, n = 4; n > 0; o >>= 1, n >>= 1) {
        const bool hi = lane & o;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const double send = hi ? g[i] : g[i + n], keep = hi ? g[i + n] : g[i];
            g[i] = gs_add(__shfl_xor_sync(ALL, send, o), keep);
        }
    }
    double v = g[0];
    v = gs_add(__shfl_xor_sync(ALL, v, 2), v);
    v = gs_add(__shfl_xor_sync(ALL, v, 1), v);
    // lanes 4 k (k < 8) hold component k's sum, lane 1 the last
    const int k = lane == 1 ? 8 : lane >> 2;
    if (lane == 1) v = last;
    if (lane == 1 || (lane & 3) == 0) {
        const int cen = k / 3, x = k - 3 * cen;
        const int shell = cen == 0 ? B.sa : cen == 1 ? B.sb : K.sa;
        atomicAdd(a.grad + 3 * a.shell_atom[shell] + x, v);
        atomicAdd(a.grad + 3 * a.shell_atom[K.sb] + x, -v);
    }
}

// a.per consecutive tasks a warp (one for the classes with shared accumulators), their
// primitive quartets set up together as in wide_many.
template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(32 * kGradWarps) k_eri_grad(const GradArgs a) {
    using W = GradProg<LA, LB, LC, LD>;
    using Lay = GradLayout<LA, LB, LC, LD>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* sm = reinterpret_cast<double*>(smem_raw) + (size_t)warp * Lay::WARP;
    double* sC = sm + Lay::ACC;
    double* sF = sC + Lay::SC;
    double* node = sF + Lay::SF;
    if constexpr (Lay::SMEM_ACC) {
        const int t = blockIdx.x * Lay::WARPS + warp;
        if (t >= a.ntask) return;
        const int2 task = a.tasks[t];
        const PairRec B = a.pairs[task.x];
        const PairRec K = a.pairs[task.y];
        if (!grad_keep(a, B, K)) return;               // warp-uniform
        for (int q = lane; q < W::NACC; q += 32) sm[q] = 0.0;
        const int nK = K.nprim, ntot = B.nprim * nK;
        for (int base = 0; base < ntot; base += kSetupBatch) {
            const int i = base + lane;
            if (lane < kSetupBatch && i < ntot)
                grad_setup_slot<LA, LB, LC, LD>(a.prims[B.prim_off + i / nK],
                                                a.prims[K.prim_off + i % nK], sC, sF, lane);
            __syncwarp();
            grad_items<LA, LB, LC, LD>(sC, sF, node, 0, min(kSetupBatch, ntot - base), lane,
                                       nullptr, nullptr, sm);
        }
        grad_tail<LA, LB, LC, LD>(a, task, B, K, sm, lane);
    } else {
        constexpr int NACCW = (W::NACC + 31) / 32;
        constexpr unsigned ALL = 0xffffffffu;
        const int per = a.per;
        const int t0 = (blockIdx.x * Lay::WARPS + warp) * per;
        const int nq = min(per, a.ntask - t0);
        if (nq <= 0) return;
        int w = 0, bo = 0, ko = 0, kn = 1;
        if (lane < nq) {
            const int2 task = a.tasks[t0 + lane];
            const PairRec& B = a.pairs[task.x];
            const PairRec& K = a.pairs[task.y];
            bo = B.prim_off;
            ko = K.prim_off;
            kn = K.nprim;
            w = grad_keep(a, B, K) ? B.nprim * kn : 0;
        }
        int end = w;
#pragma unroll
        for (int o = 1; o < kManyTasks; o <<= 1) {
            const int y = __shfl_up_sync(ALL, end, o);
            if (lane >= o) end += y;
        }
        const int total = __shfl_sync(ALL, end, kManyTasks - 1);
        double acc[NACCW];
        unsigned ent[NACCW];
#pragma unroll
        for (int k = 0; k < NACCW; ++k) {
            acc[k] = 0.0;
            const int q = lane + 32 * k;
            ent[k] = q < W::NACC ? __ldg(W::acc() + q) : 255u << 16;
        }
        int q = 0, left = __shfl_sync(ALL, w, 0);
        auto close = [&]() {                             // ends quartet q, moves to the next
            if (__shfl_sync(ALL, w, q) > 0) {
#pragma unroll
                for (int k = 0; k < NACCW; ++k) {
                    const int t = lane + 32 * k;
                    if (t < W::NACC) node[__ldg(W::accpos() + t)] = acc[k];
                    acc[k] = 0.0;
                }
                __syncwarp();
                const int2 task = a.tasks[t0 + q];
                const PairRec B = a.pairs[task.x];
                const PairRec K = a.pairs[task.y];
                grad_tail<LA, LB, LC, LD>(a, task, B, K, node, lane);
                __syncwarp();
            }
            ++q;
            left = __shfl_sync(ALL, w, q & 31);
        };
        for (int base = 0; base < total; base += kSetupBatch) {
            const int x = base + lane;
            int mine = 0;
#pragma unroll
            for (int k = 0; k < kManyTasks - 1; ++k) mine += __shfl_sync(ALL, end, k) <= x;
            const int start = __shfl_sync(ALL, end - w, mine), nK = __shfl_sync(ALL, kn, mine);
            const int po = __shfl_sync(ALL, bo, mine), qo = __shfl_sync(ALL, ko, mine);
            if (lane < kSetupBatch && x < total) {
                const int i = x - start, j = i / nK;
                grad_setup_slot<LA, LB, LC, LD>(a.prims[po + j], a.prims[qo + i - j * nK], sC, sF,
                                                lane);
            }
            __syncwarp();
            const int nb = min(kSetupBatch, total - base);
            for (int j = 0; j < nb;) {
                while (left == 0) close();
                const int run = min(left, nb - j);
                grad_items<LA, LB, LC, LD>(sC, sF, node, j, run, lane, acc, ent, nullptr);
                j += run;
                left -= run;
            }
        }
        while (q < nq) close();
    }
}

// Thread-per-quartet form for the small classes (generated straight-line code, csrc
// gen_grad.py emit_grad_thread): each thread runs the same VRR, accumulation, HRR and
// density contraction as the warp form for its own quartet, with node values and
// accumulators in registers.  Gradient contributions are summed per block in shared
// memory (3 natom doubles) before one global atomic per atom coordinate.
constexpr int kGradThreads = 128;
constexpr int kGradSmemAtoms = 2048;

// HRR, contraction with the RHF weights and the atomic adds of one quartet whose weighted
// contraction sets are in H[0 .. NACC).  With warp_sum, lanes of a full warp whose quartets
// share an atom at a centre sum first and one lane adds (every lane of the warp must call
// it); without, each caller adds its own (a single lane may call it).
template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ void grad_finish(const GradArgs& a, const int2 task, const PairRec& B,
                                            const PairRec& K, double* H, double* dst,
                                            bool warp_sum) {
    using W = GradThread<LA, LB, LC, LD>;
    constexpr int NA = (LA + 1) * (LA + 2) / 2, NB = (LB + 1) * (LB + 2) / 2;
    constexpr int NC = (LC + 1) * (LC + 2) / 2, ND = (LD + 1) * (LD + 2) / 2;
    const double dv[6] = {B.ABx, B.ABy, B.ABz, K.ABx, K.ABy, K.ABz};
    W::hrr(H, dv);
    const int fa = a.func_off[B.sa], fb = a.func_off[B.sb];
    const int fc = a.func_off[K.sa], fd = a.func_off[K.sb];
    const int nbf = a.nbf;
    const double* Pm = a.P;
    double pab[NA * NB], pcd[NC * ND], pac[NA * NC], pbd[NB * ND], pad[NA * ND], pbc[NB * NC];
#pragma unroll
    for (int i = 0; i < NA; ++i) {
#pragma unroll
        for (int j = 0; j < NB; ++j) pab[i * NB + j] = Pm[(fa + i) * nbf + fb + j];
#pragma unroll
        for (int j = 0; j < NC; ++j) pac[i * NC + j] = Pm[(fa + i) * nbf + fc + j];
#pragma unroll
        for (int j = 0; j < ND; ++j) pad[i * ND + j] = Pm[(fa + i) * nbf + fd + j];
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) {
#pragma unroll
        for (int j = 0; j < ND; ++j) pbd[i * ND + j] = Pm[(fb + i) * nbf + fd + j];
#pragma unroll
        for (int j = 0; j < NC; ++j) pbc[i * NC + j] = Pm[(fb + i) * nbf + fc + j];
    }
#pragma unroll
    for (int i = 0; i < NC; ++i)
#pragma unroll
        for (int j = 0; j < ND; ++j) pcd[i * ND + j] = Pm[(fc + i) * nbf + fd + j];
    double cs0[NA], cs1[NB], cs2[NC], cs3[ND];
#pragma unroll
    for (int i = 0; i < NA; ++i) cs0[i] = a.comp_scale[6 * B.sa + i];
#pragma unroll
    for (int i = 0; i < NB; ++i) cs1[i] = a.comp_scale[6 * B.sb + i];
#pragma unroll
    for (int i = 0; i < NC; ++i) cs2[i] = a.comp_scale[6 * K.sa + i];
#pragma unroll
    for (int i = 0; i < ND; ++i) cs3[i] = a.comp_scale[6 * K.sb + i];
    double w = 8.0;
    if (B.sa == B.sb) w *= 0.5;
    if (K.sa == K.sb) w *= 0.5;
    if (task.x == task.y) w *= 0.5;
    double g[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) g[k] = 0.0;
    W::contract(H, w, pab, pcd, pac, pbd, pad, pbc, cs0, cs1, cs2, cs3, g);
    const int at[4] = {a.shell_atom[B.sa], a.shell_atom[B.sb], a.shell_atom[K.sa],
                       a.shell_atom[K.sb]};
    // per-centre contributions (D by translational invariance); when the whole warp is
    // active and every lane has the same atom at a centre (neighbouring tasks usually
    // share their bra pair), the warp sums first and one lane adds
    double gc[4][3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        gc[0][x] = g[x];
        gc[1][x] = g[3 + x];
        gc[2][x] = g[6 + x];
        gc[3][x] = -(g[x] + g[3 + x] + g[6 + x]);
    }
    const unsigned act = warp_sum ? __activemask() : 0u;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int cen = 0; cen < 4; ++cen) {
        const bool uniform = warp_sum && act == 0xffffffffu &&
                             __all_sync(act, at[cen] == __shfl_sync(act, at[cen], 0));
        if (uniform) {
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                double v = gc[cen][x];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(act, v, o);
                if (lane == 0) atomicAdd(dst + 3 * at[cen] + x, v);
            }
        } else {
#pragma unroll
            for (int x = 0; x < 3; ++x) atomicAdd(dst + 3 * at[cen] + x, gc[cen][x]);
        }
    }
}

// Weighted contraction sets of primitive quartets start, start + stride, ... of the quartet
// into H[0 .. NACC), the recursion in T.
template <int LA, int LB, int LC, int LD, typename T>
__device__ __forceinline__ void grad_accumulate(const GradArgs& a, const PairRec& B,
                                                const PairRec& K, double* H, int start,
                                                int stride) {
    using W = GradThread<LA, LB, LC, LD>;
    constexpr int L = W::L;
    const PrimRec<T>* __restrict__ prims;
    if constexpr (sizeof(T) == 8) prims = a.prims;
    else prims = a.prims32;
    T acc[W::NACC];
#pragma unroll
    for (int k = 0; k < W::NACC; ++k) acc[k] = T(0);
    const int nK = K.nprim, ntot = B.nprim * nK;
    for (int i = start; i < ntot; i += stride) {
        const PrimRec<T> P = prims[B.prim_off + i / nK];
        const PrimRec<T> Q = prims[K.prim_off + i % nK];
        T c[kNCoefG], n[W::NVSLOT];
        wide_setup_m<L, T>(P, Q, c, n);
        const T ea = prim_expo(P);
        c[32] = T(2) * ea;                  // 2 alpha (first bra shell)
        c[33] = T(2) * (P.p - ea);          // 2 beta
        c[34] = T(2) * prim_expo(Q);        // 2 gamma (first ket shell)
        c[35] = T(5) * c[28];               // 5/(2(p+q)), raised (dd|..) classes
        W::template prim<T>(c, n, acc);
    }
#pragma unroll
    for (int k = 0; k < W::NACC; ++k) H[k] = (double)acc[k];
}

// Copies of the block's gradient sums: two a warp, by the lanes' parity, while they are small
// (a shared FP64 addition is a compare-and-swap loop, and lanes that share an atom repeat it).
constexpr int kGradCopies = 2 * kGradThreads / 32;
__host__ __device__ inline int grad_copies(int natom) {
    return natom <= kGradSmemAtoms / kGradCopies ? kGradCopies : 1;
}

template <int LA, int LB, int LC, int LD, typename T>
__global__ void __launch_bounds__(kGradThreads) k_eri_grad_thread(const GradArgs a) {
    using W = GradThread<LA, LB, LC, LD>;
    extern __shared__ double sg[];
    const int ntask = a.ntask_dev ? *a.ntask_dev : a.ntask;
    if (blockIdx.x * blockDim.x >= ntask) return;          // block-uniform
    const bool shared_sum = a.natom > 0 && a.natom <= kGradSmemAtoms;
    const int copies = grad_copies(a.natom), n3 = 3 * a.natom;
    if (shared_sum) {
        for (int i = threadIdx.x; i < copies * n3; i += blockDim.x) sg[i] = 0.0;
        __syncthreads();
    }
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < ntask) {
        const int2 task = a.tasks[t];
        const PairRec B = a.pairs[task.x];
        const PairRec K = a.pairs[task.y];
        if (grad_keep(a, B, K)) {
            double H[W::HSIZE];
            grad_accumulate<LA, LB, LC, LD, T>(a, B, K, H, 0, 1);
            const int copy = copies > 1 ? 2 * (threadIdx.x >> 5) + (threadIdx.x & 1) : 0;
            grad_finish<LA, LB, LC, LD>(a, task, B, K, H, shared_sum ? sg + copy * n3 : a.grad,
                                        true);
        }
    }
    if (shared_sum) {
        __syncthreads();
        for (int i = threadIdx.x; i < n3; i += blockDim.x) {
            double v = sg[i];
            for (int c = 1; c < copies; ++c) v += sg[c * n3 + i];
            if (v != 0.0) atomicAdd(a.grad + i, v);
        }
    }
}

template <int LA, int LB, int LC, int LD, typename T>
int launch_grad_thread_t(const GradArgs& a, cudaStream_t st) {
    const size_t sh = (a.natom > 0 && a.natom <= kGradSmemAtoms)
                          ? 3 * sizeof(double) * a.natom * grad_copies(a.natom) : 0;
    if (set_smem<k_eri_grad_thread<LA, LB, LC, LD, T>>(3 * sizeof(double) * kGradSmemAtoms))
        return GS_ERR_CUDA;
    k_eri_grad_thread<LA, LB, LC, LD, T><<<(a.ntask + kGradThreads - 1) / kGradThreads,
                                           kGradThreads, sh, st>>>(a);
    return cudaGetLastError() == cudaSuccess ? 0 : GS_ERR_CUDA;
}

template <int LA, int LB, int LC, int LD>
int launch_grad_thread(const GradArgs& a, cudaStream_t st) {
    if (a.ntask <= 0) return 0;
    return a.fp32 ? launch_grad_thread_t<LA, LB, LC, LD, float>(a, st)
                  : launch_grad_thread_t<LA, LB, LC, LD, double>(a, st);
}

// Split form of the thread kernel, for quartets with many primitive quartets (the heavy
// prefix of a class's task list, sorted by descending primitive work): one warp per
// quartet, its lanes taking the primitive quartets 32 apart with the same generated code,
// a butterfly sum of the weighted contraction sets, then lane 0 finishes the quartet.
constexpr int kGradSplitWarps = 4;

template <int LA, int LB, int LC, int LD, typename T>
__global__ void __launch_bounds__(32 * kGradSplitWarps) k_eri_grad_split(const GradArgs a) {
    using W = GradThread<LA, LB, LC, LD>;
    const int lane = threadIdx.x & 31;
    const int t = blockIdx.x * kGradSplitWarps + (threadIdx.x >> 5);
    if (t >= (a.ntask_dev ? *a.ntask_dev : a.ntask)) return;       // warp-uniform
    const int2 task = a.tasks[t];
    const PairRec B = a.pairs[task.x];
    const PairRec K = a.pairs[task.y];
    if (!grad_keep(a, B, K)) return;               // warp-uniform
    double H[W::HSIZE];
    grad_accumulate<LA, LB, LC, LD, T>(a, B, K, H, lane, 32);
#pragma unroll
    for (int k = 0; k < W::NACC; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) H[k] = gs_add(__shfl_xor_sync(0xffffffffu, H[k], o), H[k]);
    if (lane == 0) grad_finish<LA, LB, LC, LD>(a, task, B, K, H, a.grad, false);
}

template <int LA, int LB, int LC, int LD>
int launch_grad_split(const GradArgs& a, cudaStream_t st) {
    if (a.ntask <= 0) return 0;
    const int grid = (a.ntask + kGradSplitWarps - 1) / kGradSplitWarps;
    if (a.fp32)
        k_eri_grad_split<LA, LB, LC, LD, float><<<grid, 32 * kGradSplitWarps, 0, st>>>(a);
    else
        k_eri_grad_split<LA, LB, LC, LD, double><<<grid, 32 * kGradSplitWarps, 0, st>>>(a);
    return cudaGetLastError() == cudaSuccess ? 0 : GS_ERR_CUDA;
}

template <int LA, int LB, int LC, int LD>
int launch_grad(const GradArgs& a, cudaStream_t st) {
    if (a.ntask <= 0) return 0;
    using Lay = GradLayout<LA, LB, LC, LD>;
    auto k = k_eri_grad<LA, LB, LC, LD>;
    if (set_smem<k_eri_grad<LA, LB, LC, LD>>(Lay::BYTES)) return GS_ERR_CUDA;
    GradArgs b = a;
    if (Lay::SMEM_ACC || b.per < 1) b.per = 1;
    const int tasks = b.per * Lay::WARPS;
    k<<<(b.ntask + tasks - 1) / tasks, 32 * Lay::WARPS, Lay::BYTES, st>>>(b);
    return cudaGetLastError() == cudaSuccess ? 0 : GS_ERR_CUDA;
}

}  // namespace gs
