// Kernel table of one (ndim, p, tile) instantiation and the element-local
// set-up kernels. Instantiated in spdk_select_*.cu so the (ndim, p) variants
// compile in parallel.
#pragma once
#include <cuda_runtime.h>

#include <cmath>

#include "spdk_fallback.cuh"
#include "spdk_kernels.cuh"
#include "spdk_viscous.cuh"

namespace spdk {

// ---------------------------------------------------------------------------
// element-local set-up kernels
// ---------------------------------------------------------------------------
// U_sp = conservatives(cv_to_sp(W_cv)) and dt(W_cv): the constructor tail
// (src/hydro_ader.hpp:205-208)
template <typename R, int D, int P>
__global__ void __launch_bounds__(kThreads) init_state_kernel(DevGrid G, DevMatsT<R> M, const R* __restrict__ wcv,
                                                             R* __restrict__ u,
                                                             unsigned long long* dtmin) {
    using S = Shape<D, P>;
    constexpr int V = S::V, NPT = S::NPT;
    __shared__ R b0[V * NPT], b1[V * NPT];
    const long long ge = blockIdx.x;
    for (int q = threadIdx.x; q < V * NPT; q += blockDim.x) b0[q] = wcv[ge * V * NPT + q];
    __syncthreads();
    double dtl = 1.7976931348623157e308;
    for (int q = threadIdx.x; q < NPT; q += blockDim.x) {
        R w[V];
        for (int v = 0; v < V; v++) w[v] = b0[v * NPT + q];
        dtl = smin(dtl, point_dt<D>(G, w, S::n));
    }
    R* bufs[2] = {b1, b0};
    const R* src = b0;
    for (int d = 0; d < D; d++) {
        R* dst = bufs[d % 2];
        sweep_smem<D, P, R>(src, dst, M.cv_to_sp, d, V * NPT);
        __syncthreads();
        src = dst;
    }
    for (int q = threadIdx.x; q < NPT; q += blockDim.x) {
        R w[V], uu[V];
        for (int v = 0; v < V; v++) w[v] = src[v * NPT + q];
        conservatives<D>(w, uu, (R)G.gm);
        for (int v = 0; v < V; v++) u[ge * V * NPT + v * NPT + q] = uu[v];
    }
    block_min_dt(dtl, dtmin);
}

// W_cv = sp_to_cv(primitives(U_sp)) and dt, for a state written by the host
template <typename R, int D, int P>
__global__ void __launch_bounds__(kThreads) derive_kernel(DevGrid G, DevMatsT<R> M, const R* __restrict__ u,
                                                         R* __restrict__ wcv, unsigned long long* dtmin) {
    using S = Shape<D, P>;
    constexpr int V = S::V, NPT = S::NPT;
    __shared__ R b0[V * NPT], b1[V * NPT];
    const long long ge = blockIdx.x;
    for (int q = threadIdx.x; q < NPT; q += blockDim.x) {
        R uu[V], w[V];
        for (int v = 0; v < V; v++) uu[v] = u[ge * V * NPT + v * NPT + q];
        primitives<D>(uu, w, (R)G.gm);
        for (int v = 0; v < V; v++) b0[v * NPT + q] = w[v];
    }
    __syncthreads();
    R* bufs[2] = {b1, b0};
    const R* src = b0;
    for (int d = 0; d < D; d++) {
        R* dst = bufs[d % 2];
        sweep_smem<D, P, R>(src, dst, M.sp_to_cv, d, V * NPT);
        __syncthreads();
        src = dst;
    }
    double dtl = 1.7976931348623157e308;
    for (int q = threadIdx.x; q < NPT; q += blockDim.x) {
        R w[V];
        for (int v = 0; v < V; v++) {
            w[v] = src[v * NPT + q];
            wcv[ge * V * NPT + v * NPT + q] = w[v];
        }
        dtl = smin(dtl, point_dt<D>(G, w, S::n));
    }
    block_min_dt(dtl, dtmin);
}

// next dt <- reduced minimum, capped by the viscous diffusion limit when
// cap > 0 (src/hydro.cpp:245-254: every point's candidate is min(dt, cap),
// so the minimum over points is min(reduced, cap)); re-arm the reduction
static __global__ void advance_dt_kernel(double* dt, unsigned long long* dtmin, double cap) {
    pdl_wait();
    const double v = __longlong_as_double((long long)*dtmin);
    *dt = (cap > 0.0 && !(v < cap)) ? cap : v;
    *dtmin = 0x7FEFFFFFFFFFFFFFULL;
}

// The device-resident time loop's step end (src/hydro_ader.hpp:234-261):
// t += dt of the step, next dt from the reduction (viscous cap as above),
// dt clamped to the next output time, and the gate closed once t >= t_end.
// tb = {t, t_output, steps, t_end, dt_output (<= 0: no outputs)}; the same
// FP64 operations as the host loop, so the dt sequence is identical.
static __global__ void evolve_advance_kernel(double* dt, unsigned long long* dtmin, double cap, double* tb,
                                             int* gate) {
    pdl_wait();
    if (*gate) return;
    const double used = *dt;
    const double v = __longlong_as_double((long long)*dtmin);
    double next = (cap > 0.0 && !(v < cap)) ? cap : v;
    *dtmin = 0x7FEFFFFFFFFFFFFFULL;
    const double t = tb[0] + used;
    double t_output = tb[1];
    if (tb[4] > 0) {
        if (t >= t_output) t_output = t + tb[4];
        if (t + next > t_output) next = t_output - t;
    }
    *dt = next;
    tb[0] = t;
    tb[1] = t_output;
    tb[2] += 1.0;
    if (!(t < tb[3])) *gate = 1;
}

constexpr unsigned kSMs = 148;

// ---------------------------------------------------------------------------
// kernel table of one (R, D, P, tile) instantiation
// ---------------------------------------------------------------------------
template <typename R>
struct KernelSetT {
    void (*predict)(DevGrid, DevMatsT<R>, PicardArgsT<R>) = nullptr;
    void (*correct)(DevGrid, DevMatsT<R>, PicardArgsT<R>) = nullptr;
    void (*flux)(DevGrid, DevMatsT<R>, PicardArgsT<R>) = nullptr;
    // correctors of the same tile (null: `correct`): of an ADER step and of an
    // SSP-RK stage on at most few_blocks blocks, and of an SSP-RK stage on more
    void (*correct_few)(DevGrid, DevMatsT<R>, PicardArgsT<R>) = nullptr;
    void (*correct_rk_few)(DevGrid, DevMatsT<R>, PicardArgsT<R>) = nullptr;
    void (*correct_rk)(DevGrid, DevMatsT<R>, PicardArgsT<R>) = nullptr;
    unsigned few_blocks = 0;
    // passes on small tiles (3D: blocks compiled for one per SM), for at most
    // small_blocks of them (null: none);
    // [predict, corrector of an ADER step, of an SSP-RK stage]
    void (*small[3])(DevGrid, DevMatsT<R>, PicardArgsT<R>) = {nullptr, nullptr, nullptr};
    size_t small_smem[3] = {0, 0, 0};
    int small_threads = 0, small_tile[3] = {1, 1, 1};
    unsigned small_blocks = 0;
    // the corrector on state buffers that start on no 16-byte boundary (null:
    // `correct` takes them if n is odd, and nothing does if n is even)
    void (*correct_any)(DevGrid, DevMatsT<R>, PicardArgsT<R>) = nullptr;
    void (*detect)(DevGrid, DetectArgs) = nullptr;
    void (*blend)(DevGrid, DevMatsT<R>, BlendArgsT<R>) = nullptr;
    void (*update)(DevGrid, DevMatsT<R>, FallbackArgsT<R>) = nullptr;
    void (*init)(DevGrid, DevMatsT<R>, const R*, R*, unsigned long long*) = nullptr;
    void (*derive)(DevGrid, DevMatsT<R>, const R*, R*, unsigned long long*) = nullptr;
    void (*visc)(DevGrid, DevMatsT<R>, ViscArgsT<R>) = nullptr;
    size_t picard_smem[3] = {0, 0, 0}, blend_smem = 0, update_smem = 0;  // predict, correct, flux
    int picard_threads = kThreads;
    // elements of a Picard pass's block: a tile (2D, may hang over the
    // domain's edge) or consecutive ones (3D)
    int picard_tile[3] = {1, 1, 1}, picard_elems = 0;
    int tile[3] = {1, 1, 1};         // elements of a detect block
    int blend_tile[3] = {1, 1, 1};   // elements of a blend block
    int update_elems = 1;            // consecutive elements of an update block
    int visc_epb = 1;  // elements per block of the viscous face kernel
};
using KernelSet = KernelSetT<double>;

template <typename R, int D, int P, int TX, int TY, int TZ, bool VISC = false>
KernelSetT<R> make_set() {
    KernelSetT<R> k;
    constexpr int PX = D == 2 ? kLineTX<P> : 1, PY = D == 2 ? kLineTY<P> : 1;
    k.predict = picard_kernel<R, D, P, PX, PY, kPredict, VISC>;
    k.correct = picard_kernel<R, D, P, PX, PY, kCorrect, VISC>;
    k.flux = picard_kernel<R, D, P, PX, PY, kFlux, VISC>;
    if constexpr (D == 2) {
        constexpr bool f64 = sizeof(R) == 8;
        if constexpr (f64 && !VISC) {
            constexpr int few = P <= 4 ? 2 : 1;
            k.correct_few = picard2d_kernel<R, P, PX, PY, kCorrect, false, false, few>;
            k.correct_rk_few = picard2d_kernel<R, P, PX, PY, kCorrect, false, true, few>;
            k.few_blocks = P <= 4 ? 2 * kSMs : 128;
        }
        if constexpr (f64) k.correct_rk = picard2d_kernel<R, P, PX, PY, kCorrect, VISC, true, picard_blocks<R, 2, P, kCorrect, VISC>()>;
        if constexpr (P > 4 || (!f64 && (P == 2 || P == 3))) {
            constexpr int SX = P > 4 ? 2 : 4, SY = 2, blocks = P > 4 ? 1 : 4;
            k.small[0] = picard2d_kernel<R, P, SX, SY, kPredict, VISC, false, blocks>;
            k.small[1] = picard2d_kernel<R, P, SX, SY, kCorrect, VISC, false, blocks>;
            k.small[2] = picard2d_kernel<R, P, SX, SY, kCorrect, VISC, f64, blocks>;
            k.small_smem[0] = Line2<R, P, SX, SY, kPredict>::bytes;
            k.small_smem[1] = k.small_smem[2] = Line2<R, P, SX, SY, kCorrect>::bytes;
            k.small_threads = Line2<R, P, SX, SY, kPredict>::threads;
            k.small_tile[0] = SX;
            k.small_tile[1] = SY;
            k.small_blocks = P > 4 ? 64 : 512;
        }
    }
    if constexpr (D == 3 && sizeof(R) == 8 && P % 2 == 1 && !VISC) k.correct_any = correct_any_kernel<R, P>;
    k.picard_threads = picard_threads<R, D, P, PX, PY>();
    k.picard_tile[0] = PX;
    k.picard_tile[1] = PY;
    if constexpr (D == 3) {
        using L3 = Line3<R, P, kFlux>;
        k.picard_elems = L3::EB;
        if constexpr (P == 5 || (P == 4 && sizeof(R) == 4)) {
            static_assert(L3::EB == 1, "blocks of one element, as tile_blocks counts them");
            k.small[0] = picard3d_kernel<R, P, kPredict, VISC>;
            k.small[1] = k.small[2] = picard3d_kernel<R, P, kCorrect, VISC>;
            k.small_smem[0] = Line3<R, P, kPredict>::bytes;
            k.small_smem[1] = k.small_smem[2] = Line3<R, P, kCorrect>::bytes;
            k.small_threads = L3::threads;
            k.small_blocks = kSMs;
        }
    }
    k.detect = fv_detect_kernel<R, D, P, TX, TY, TZ>;
    using BT = BlendTile<D, P>;
    k.blend = fv_blend_kernel<R, D, P, BT::X, BT::Y, BT::Z>;
    k.blend_smem = BlendSmem<R, D, P, BT::X, BT::Y, BT::Z>::bytes;
    k.blend_tile[0] = BT::X;
    k.blend_tile[1] = BT::Y;
    k.blend_tile[2] = BT::Z;
    k.update = fv_update_kernel<R, D, P>;
    k.update_elems = UpdateBlock<D, P>::NE;
    k.init = init_state_kernel<R, D, P>;
    k.derive = derive_kernel<R, D, P>;
    k.visc = visc_face_kernel<R, D, P>;
    k.visc_epb = ViscShape<R, D, P>::EPB;
    k.picard_smem[kPredict] = picard_smem_bytes<R, D, P, PX, PY, kPredict>();
    k.picard_smem[kCorrect] = picard_smem_bytes<R, D, P, PX, PY, kCorrect>();
    k.picard_smem[kFlux] = picard_smem_bytes<R, D, P, PX, PY, kFlux>();
    k.update_smem = UpdateSmem<R, D, P>::bytes;
    k.tile[0] = TX;
    k.tile[1] = TY;
    k.tile[2] = TZ;
    return k;
}

// blocks of a blend launch at most (two to four per SM are resident and
// share out the listed tiles, the others find the list done)
constexpr unsigned kBlendGrid = 8 * kSMs;

// blocks of tiles that cover the domain
inline unsigned tile_blocks(int D, const int N[3], const int tile[3]) {
    long long b = 1;
    for (int d = 0; d < D; d++) b *= (N[d] + tile[d] - 1) / tile[d];
    return (unsigned)b;
}

// the launch of a Picard pass of nt slices
template <typename R>
struct PicardLaunch {
    void (*kernel)(DevGrid, DevMatsT<R>, PicardArgsT<R>);
    unsigned blocks, threads;
    size_t smem;
};
// Which kernel a pass takes. Small tiles (2 x 2 elements above p = 4): a grid of
// few blocks is a chain of latencies that grows with the elements of a block;
// 16^2 steps without the fallback on 4 x 2 / 2 x 2 tiles: p=5 FP64 154 / 137 us,
// p=7 FP64 362 / 317 us, p=5 FP32 97 / 74 us; beyond 64 blocks the device no longer
// gives each an SM of its own (24^2, 144 blocks: p=5 FP64 186 / 214 us). In FP32 at
// p = 2 and 3, whose blocks are shortest, 4 x 2 tiles up to 512 blocks (64^2 on 4 x 4 /
// 4 x 2: p=2 33 / 28.5 us, RK3 34 / 30.5 us, p=3 50 / 43.5 us; 768 blocks, 96 x 64: p=3 56 / 61 us).
// In 3D at p = 5 (FP32 also p = 4) the same blocks of one element compiled for one per
// SM, while there are no more (4^3: p=5 FP64 226 / 200 us, FP32 129 / 112 us, p=4 FP32
// 112 / 85 us; 6^3, 216 blocks: p=5 FP64 360 / 513 us).
// Few blocks: a corrector compiled for two blocks per SM (above p = 4: one), without
// spills (32^2 p=3 FP64, 8 steps: 272 -> 262 us; 32^2 p=5 RK3 42.5 -> 41 us), up to
// what is resident at once; from there the other one's occupancy counts (68 x 72
// and 80^2, p=3 RK3: 47 / 59 us and 47 / 65 us).
template <typename R>
PicardLaunch<R> picard_launch(const KernelSetT<R>& k, int mode, int D, const int N[3], int nt) {
    if (k.small[0] && mode != kFlux) {
        const unsigned b = tile_blocks(D, N, k.small_tile);
        const int i = mode == kPredict ? 0 : (nt > 1 ? 1 : 2);
        if (b <= k.small_blocks) return {k.small[i], b, (unsigned)k.small_threads, k.small_smem[i]};
    }
    const long long E = (long long)N[0] * N[1] * N[2];
    const unsigned b = k.picard_elems ? (unsigned)((E + k.picard_elems - 1) / k.picard_elems)
                                      : tile_blocks(D, N, k.picard_tile);
    auto kernel = mode == kPredict ? k.predict : (mode == kFlux ? k.flux : k.correct);
    if (mode == kCorrect) {
        if (b <= k.few_blocks) kernel = nt > 1 ? k.correct_few : k.correct_rk_few;
        else if (nt == 1 && k.correct_rk) kernel = k.correct_rk;
    }
    return {kernel, b, (unsigned)k.picard_threads, k.picard_smem[mode]};
}

// element widths, their reciprocals and powers of two (G.N, D and the box
// lengths given), and whether every derivative coefficient is zero or far
// from under- and overflow (div_const)
inline void set_spacing(DevGrid& G, int D, const double h[3], const double* dfp_to_sp, int coefs) {
    G.uniform_pow2 = 1;
    G.safe_div = 1;
    for (int d = 0; d < 3; d++) {
        G.h[d] = h[d];
        int ex = 0;
        const double m = std::frexp(h[d], &ex);
        G.pow2[d] = m == 0.5 ? 1 : 0;
        G.rh[d] = G.pow2[d] ? std::ldexp(1.0, 1 - ex) : 0.0;
        G.ih[d] = 1.0 / h[d];
        G.ihl[d] = std::fma(-h[d], G.ih[d], 1.0) * G.ih[d];
        if (d < D && (!G.pow2[d] || h[d] != h[0])) G.uniform_pow2 = 0;
        if (d < D && !(h[d] > 1e-30 && h[d] < 1e30)) G.safe_div = 0;
    }
    for (int q = 0; q < coefs; q++) {
        const double a = std::fabs(dfp_to_sp[q]);
        if (a != 0.0 && !(a > 1e-30 && a < 1e30)) G.safe_div = 0;
    }
}

// 2D: the detect tile (its blocks may hang over the domain) is 4 x 4 elements
// up to p = 4 and 2 x 2 above. At p = 4 a 4 x 4 tile gives a thread two sub-cells,
// so there too it is 2 x 2 as long as each of those has an SM of its own (6^2 FP32
// steps 204 -> 176 us, 24^2 FP64 310 -> 295 us; up to p = 3 the two are within 3 %)
template <typename R, int P, bool VISC>
bool pick2_t(const int N[3], KernelSetT<R>* k) {
    const int small[3] = {2, 2, 1};
    if constexpr (P < 4) *k = make_set<R, 2, P, 4, 4, 1, VISC>();
    else if constexpr (P > 4) *k = make_set<R, 2, P, 2, 2, 1, VISC>();
    else if (tile_blocks(2, N, small) <= kSMs) *k = make_set<R, 2, P, 2, 2, 1, VISC>();
    else *k = make_set<R, 2, P, 4, 4, 1, VISC>();
    return true;
}
template <typename R, int P>
bool pick2(const int N[3], KernelSetT<R>* k, bool visc) {
    return visc ? pick2_t<R, P, true>(N, k) : pick2_t<R, P, false>(N, k);
}
// 3D: 2x2x1 elements up to p = 3 (one element's (p+1)^3 points would leave
// most of the block idle), one above
template <typename R, int P>
bool pick3(KernelSetT<R>* k, bool visc) {
    constexpr int T = P <= 3 ? 2 : 1;
    *k = visc ? make_set<R, 3, P, T, T, 1, true>() : make_set<R, 3, P, T, T, 1>();
    return true;
}

// per-translation-unit selectors (spdk_select_*.cu): the FP64 units are
// compiled without FMA contraction (reference rounding), the FP32 units with it
bool select_2d_low(int p, const int N[3], KernelSetT<double>* k, bool visc);   // p = 1..3
bool select_2d_high(int p, const int N[3], KernelSetT<double>* k, bool visc);  // p = 4..7
bool select_3d(int p, KernelSetT<double>* k, bool visc);                       // p = 1..5
bool select_f32_2d(int p, const int N[3], KernelSetT<float>* k, bool visc);    // p = 1..7
bool select_f32_3d(int p, KernelSetT<float>* k, bool visc);                    // p = 1..5

inline bool select_kernels(int D, int p, const int N[3], KernelSetT<double>* k, bool visc = false) {
    if (D == 2) return p <= 3 ? select_2d_low(p, N, k, visc) : select_2d_high(p, N, k, visc);
    if (D == 3) return select_3d(p, k, visc);
    return false;
}
inline bool select_kernels(int D, int p, const int N[3], KernelSetT<float>* k, bool visc = false) {
    if (D == 2) return select_f32_2d(p, N, k, visc);
    if (D == 3) return select_f32_3d(p, k, visc);
    return false;
}

}  // namespace spdk
