// Fused device kernels of the spd_K B200 hydro step.
//
// State layout (device, arithmetic type R = double or float, no ghost elements):
//   U, U_cv          [element][var][point]            V = D+2 slots
//   U_ader (A and B) [slice][element][var][point]     ping-pong per Picard pass
//   FF_d             [slice][element][var][face point] FV face fluxes of direction d,
//                                                      laid out like the element's
//                                                      d-flux points (n_f per line)
//   RP_old, RP_new   [element][point] double2          (rho, p) of the FV candidate
//   T, theta         [element][point] uint8            trouble flag / theta*8
// element = (k*Ny + j)*Nx + i, point = (kk*n + jj)*n + ii.
//
// Boundary conditions are applied by index mapping instead of ghost storage:
// an SD face on the domain edge pairs the element's own interface state with
// its periodic partner, a copy (gradfree) or a mirror (reflective); FV ghost
// cells are images of active cells (spdk::fv_image).
#pragma once
#include <cuda_runtime.h>

#include "spdk_physics.cuh"

namespace spdk {

constexpr int kThreads = 256;
constexpr int kMaxNd = 8;    // n = p+1 <= 8
constexpr int kMaxNfd = 9;

// Transform matrices in the arithmetic type R, passed by value (kernel
// parameter space). R = double is the plain form; R = float the precision form.
template <typename R>
struct DevMatsT {
    R sp_to_fp[kMaxNfd * kMaxNd];   // [nf][n]
    R dfp_to_sp[kMaxNd * kMaxNfd];  // [n][nf]
    R sp_to_cv[kMaxNd * kMaxNd];    // [n][n]
    R cv_to_sp[kMaxNd * kMaxNd];
    R invader[kMaxNd * kMaxNd];     // [nt][nt]
    R wt[kMaxNd];
    R pred[kMaxNd * kMaxNd];        // invader(t,l) w_l (precision form)
};
using DevMats = DevMatsT<double>;

// a width of the sub-cell grid, its reciprocal rounded to nearest, and what
// that lacks of 1/h (div_const)
struct __align__(16) Width {
    double h, ih, ihl, pad;
};

struct DevGrid {
    int N[3];
    int bc[3];
    double h[3], rh[3];
    double ih[3], ihl[3];  // 1/h rounded to nearest, and what it lacks of 1/h
    int safe_div;          // the derivative coefficients allow divisions by h from ih, ihl (div_const)
    int pow2[3];
    int uniform_pow2;  // all active h equal and a power of two
    double gm, cfl;
    double g[3];
    int grav;
    int nt;
    long long E;
    const double* fvf[3];  // FV faces in frame indexing (active cell a has faces a+2, a+3)
    const double* fvc[3];  // FV centres in frame indexing
    const Width* fw[3];    // widths of the sub-cells (faces i, i+1), frame indexing
    const Width* fd[3];    // distances of the centres i, i+1
    int* status;           // device-detected faults (kStatus* bits)
    // fallback settings
    double nad_tol;
    int nad_delta, nad_moore, use_sed, blending;
    // viscous terms (hydro/nu > 0; src/hydro.cpp:420-572)
    double nu, beta;
    // learned indicator: per element, set when NAD/SED/PAD flags any of its
    // sub-cells in any slice of the step (NULL: not recorded), and the
    // a-priori prediction that counts all its sub-cells troubled (NULL: off)
    uint8_t* elem_trouble;
    const uint8_t* elem_pred;
    // device-resident time loop (spdk_hydro_evolve): set once t reaches
    // t_end; every kernel of a step launched after that returns at once
    // (NULL: never)
    const int* gate;
};

__device__ __forceinline__ bool gate_closed(const DevGrid& G) { return G.gate && *G.gate; }

// Programmatic dependent launch: a step's kernels are launched with
// programmatic stream serialization, so a kernel may be scheduled while its
// predecessor drains; it waits here, before touching any memory, until the
// predecessor has completed and its writes are visible (a no-op for a
// normal launch). Letting the successor's blocks be scheduled early
// (griddepcontrol.launch_dependents) was slower: 32^2 steps without the
// fallback 34.2 -> 36.6 us, 96x120 RK3 steps 122 -> 133 us
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

enum { kPredict = 0, kCorrect = 1, kFlux = 2 };

template <typename R>
struct PicardArgsT {
    const R* ua_in;        // [slice][E][V][NPT], or U when in_slices == 1
    int in_slices;         // 1: every slice equals U (first Picard pass / RK stage)
    const R* u;            // U_sp
    R* ua_out;             // kPredict output
    R* u_out;              // kCorrect output (may alias u: element-local)
    const R* u0;           // RK step-start state
    double rk_a;           // RK convex weight (0: none)
    R* ff[3];              // kFlux: FV face fluxes, all slices
    R* ucv;                // kFlux: U_cv = sp_to_cv(U)
    double2* rp_old;       // kFlux: slice-0 candidate (rho, p) of U_old, FP64
    double2* rp_new;       // kFlux: slice-0 candidate (rho, p) of U_new, FP64
    uint8_t* labels;       // kFlux: per-element trouble labels, cleared for the detections (nullable)
    R* wcv;                // kCorrect: W_cv output (nullable)
    unsigned long long* dtmin;  // kCorrect: next-dt reduction
    int final_stage;       // kCorrect: compute W_cv and dt
    const double* dt;      // device dt of this step
    const R* vg[3];        // viscous face fluxes of this pass's input (NULL: inviscid)
};
using PicardArgs = PicardArgsT<double>;

template <int D, int P>
struct Shape {
    static constexpr int n = P + 1;
    static constexpr int nf = P + 2;
    static constexpr int V = D + 2;
    static constexpr int NPT = D == 2 ? n * n : n * n * n;
    static constexpr int NTP = NPT / n;    // points across one direction
    static constexpr int NFP = NTP * nf;   // flux points per direction
};

// stride of a staged element of the 2D Picard pass: whole 16-byte units (it is
// a bulk copy's destination), not a multiple of 32 banks
template <int D, int P, typename R = double>
struct PicardPad {
    static constexpr int V = D + 2;
    static constexpr int NPT = D == 2 ? (P + 1) * (P + 1) : (P + 1) * (P + 1) * (P + 1);
    static constexpr int Q = 16 / (int)sizeof(R);                   // elements per 16 bytes
    static constexpr int WORDS = (int)sizeof(R) / 4;                 // 4-byte banks per element
    static constexpr int SS0 = (V * NPT + Q - 1) / Q * Q;
    static constexpr int SS = SS0 + ((SS0 * WORDS) % 32 == 0 ? Q : 0);
};

// coordinates of a point index
template <int n>
__device__ __forceinline__ void pt_coords(int pt, int c[3]) {
    c[0] = pt % n;
    c[1] = (pt / n) % n;
    c[2] = pt / (n * n);
}
template <int n>
__device__ __forceinline__ int pt_index(const int c[3]) {
    return c[0] + n * (c[1] + n * c[2]);
}
// flux-point index of direction d: extent nf along d, n along the others
template <int n, int nf>
__device__ __forceinline__ int fp_index(int d, const int c[3]) {
    if (d == 0) return c[0] + nf * (c[1] + n * c[2]);
    if (d == 1) return c[0] + n * (c[1] + nf * c[2]);
    return c[0] + n * (c[1] + n * c[2]);
}
// transverse point tp of direction d -> coordinates (coordinate d untouched)
template <int D, int n>
__device__ __forceinline__ void tp_coords(int d, int tp, int c[3]) {
    const int a = tp % n, b = tp / n;
    if (d == 0) { c[1] = a; c[2] = D == 3 ? b : 0; }
    else if (d == 1) { c[0] = a; c[2] = D == 3 ? b : 0; }
    else { c[0] = a; c[1] = b; }
}

// Tile of TX x TY x TZ elements plus its face halo (no edges or corners).
template <int D, int TX, int TY, int TZ>
struct Tile {
    static constexpr int NE = TX * TY * TZ;
    static constexpr int HX = TY * TZ, HY = TX * TZ, HZ = TX * TY;
    static constexpr int NS = NE + 2 * HX + 2 * HY + (D == 3 ? 2 * HZ : 0);
    // slot of tile-local element coordinates (at most one outside the tile)
    __device__ static int slot(int lx, int ly, int lz) {
        if (lx < 0 || lx >= TX) return NE + (lx < 0 ? 0 : HX) + ly + TY * lz;
        if (ly < 0 || ly >= TY) return NE + 2 * HX + (ly < 0 ? 0 : HY) + lx + TX * lz;
        if (lz < 0 || lz >= TZ) return NE + 2 * HX + 2 * HY + (lz < 0 ? 0 : HZ) + lx + TX * ly;
        return lx + TX * (ly + TY * lz);
    }
    // local coordinates of a slot
    __device__ static void coords(int s, int l[3]) {
        if (s < NE) {
            l[0] = s % TX; l[1] = (s / TX) % TY; l[2] = s / (TX * TY);
            return;
        }
        int r = s - NE;
        if (r < 2 * HX) {
            const int side = r / HX, q = r % HX;
            l[0] = side ? TX : -1; l[1] = q % TY; l[2] = q / TY;
            return;
        }
        r -= 2 * HX;
        if (r < 2 * HY) {
            const int side = r / HY, q = r % HY;
            l[1] = side ? TY : -1; l[0] = q % TX; l[2] = q / TX;
            return;
        }
        r -= 2 * HY;
        const int side = r / HZ, q = r % HZ;
        l[2] = side ? TZ : -1; l[0] = q % TX; l[1] = q / TX;
    }
};

// dt candidate of one W_cv point (src/hydro.cpp:222-254, inviscid), always
// evaluated in FP64
template <int D, typename R>
__device__ __forceinline__ double point_dt(const DevGrid& G, const R* wr, int n) {
    double w[D + 2];
#pragma unroll
    for (int v = 0; v < D + 2; v++) w[v] = (double)wr[v];
    const double cs = sound_speed(w[0], w[D + 1], G.gm);
    double cmax = 0, dxmin = 1;
#pragma unroll
    for (int d = 0; d < D; d++) {
        cmax += (fabs(w[1 + d]) + cs);
        dxmin = smin(dxmin, G.h[d]);
    }
    return G.cfl * dxmin / cmax / n;
}

// block-wide min of positive doubles, then one atomic per block (the order
// of a min never changes its value)
__device__ __forceinline__ void block_min_dt(double v, unsigned long long* out) {
    __shared__ double red[32];
    for (int o = 16; o > 0; o >>= 1) v = smin(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) red[w] = v;
    __syncthreads();
    if (w == 0) {
        v = l < (int)(blockDim.x >> 5) ? red[l] : 1.7976931348623157e308;
        for (int o = 16; o > 0; o >>= 1) v = smin(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (l == 0) atomicMin(out, (unsigned long long)__double_as_longlong(v));
    }
}

// One directional sweep of element-local arrays in shared memory
// (src/transforms.cpp:120-147): out(c) = sum_l in(c with c_d = l) * M(c_d, l)
template <int D, int P, typename R>
__device__ __forceinline__ void sweep_smem(const R* in, R* out, const R* M, int d, int count) {
    using S = Shape<D, P>;
    constexpr int n = S::n;
    for (int q = threadIdx.x; q < count; q += blockDim.x) {
        const int pt = q % S::NPT, base = q - pt;
        int c[3];
        pt_coords<n>(pt, c);
        const int id = c[d];
        R u = 0;
#pragma unroll
        for (int l = 0; l < n; l++) {
            c[d] = l;
            u += in[base + pt_index<n>(c)] * M[id * n + l];
        }
        out[q] = u;
    }
}

// x / h for a step-constant h from its correctly rounded reciprocal y and
// y's own remainder: q is a faithful quotient, and the exact remainder
// x - h q times y rounds it correctly (Markstein's theorem for a quotient
// with a fused multiply-add), for x = 0 or x far from under- and overflow
__device__ __forceinline__ double div_const(double x, double h, double y, double yl) {
    const double q = __fma_rn(x, y, __dmul_rn(x, yl));
    return __fma_rn(__fma_rn(-h, q, x), y, q);
}
// whether a flux value's products with the derivative coefficients lie in
// that range: zero, or an exponent within 700 of 1's
__device__ __forceinline__ bool div_range(double x) {
    const unsigned e = (unsigned)__double2hiint(x) & 0x7ff00000u;
    return (e - ((1023u - 700u) << 20)) < (1400u << 20) || x == 0.0;
}
__device__ __forceinline__ bool div_range(float) { return true; }

// x / h for a width of the sub-cell grid: the division's own bits in FP64 (-0 may
// come out as +0, a sign that no state, flag or dt depends on), a product with the
// reciprocal in FP32
__device__ __forceinline__ double div_width(const DevGrid& G, double x, const Width& w) {
    double q = div_const(x, w.h, w.ih, w.ihl);
    if (!div_range(x) || !G.safe_div) q = x / w.h;
    return q;
}
__device__ __forceinline__ float div_width(const DevGrid&, float x, const Width& w) { return x * (float)w.ih; }

// Sub-cell candidate of the FV update (src/transforms.cpp:483-543 with
// update=0): U_new = U_old - (w_t dt) sum_d (F_{+} - F_{-}) / h_d for the
// cell at point pt of the element at eg; f[d]: the element's face fluxes of
// direction d and slice t.
template <int D, int P, typename R>
__device__ __forceinline__ void fv_candidate(const DevGrid& G, const R* const (&f)[D], const int eg[3], int pt,
                                             const R* uold, R wdt, R* unew) {
    using S = Shape<D, P>;
    constexpr int n = S::n, nf = S::nf, V = S::V;
    int c[3];
    pt_coords<n>(pt, c);
    Width hd[D];
    int fl[3], fr[3];
#pragma unroll
    for (int d = 0; d < D; d++) {
        hd[d] = G.fw[d][eg[d] * n + c[d] + 2];
        int cc[3] = {c[0], c[1], c[2]};
        fl[d] = fp_index<n, nf>(d, cc);
        cc[d] = c[d] + 1;
        fr[d] = fp_index<n, nf>(d, cc);
    }
#pragma unroll
    for (int v = 0; v < V; v++) {
        R F = 0;
#pragma unroll
        for (int d = 0; d < D; d++)
            F += div_width(G, f[d][v * S::NFP + fr[d]] - f[d][v * S::NFP + fl[d]], hd[d]);
        if (G.grav) {
            R s = 0;
            if (v >= 1 && v <= D) s = uold[0] * (R)G.g[v - 1];
            else if (v == D + 1) {
                s = uold[1] * (R)G.g[0] + uold[2] * (R)G.g[1];
                if (D == 3) s = s + uold[3] * (R)G.g[2];
            }
            if (v != 0) F -= s;
        }
        unew[v] = uold[v] - wdt * F;
    }
}
// its element's position
__device__ __forceinline__ void elem_pos(const DevGrid& G, int ge, int eg[3]) {
    eg[0] = ge % G.N[0];
    eg[1] = (ge / G.N[0]) % G.N[1];
    eg[2] = ge / (G.N[0] * G.N[1]);
}
// the face-flux blocks of element ge and slice t
template <int D, int P, typename R>
__device__ __forceinline__ void face_blocks(const DevGrid& G, const R* const* ff, int t, int ge, const R* (&f)[D]) {
#pragma unroll
    for (int d = 0; d < D; d++) f[d] = ff[d] + ((long long)t * G.E + ge) * (D + 2) * Shape<D, P>::NFP;
}

// (rho, p) of a conserved state with the pressure recovered in FP64
// (src/hydro.cpp:95-106); for R = double these are primitives()'s operations
template <int D, typename R>
__device__ __forceinline__ double2 rho_p_fp64(const R* u, double gm) {
    const double r = (double)u[0];
    if constexpr (sizeof(R) == 4) {
        double m2 = 0;
#pragma unroll
        for (int d = 1; d <= D; d++) m2 += (double)u[d] * (double)u[d];
        return make_double2(r, ((double)u[D + 1] - 0.5 * m2 * rcp_fp64(u[0])) * (gm - 1.));
    }
    double ek = 0;
#pragma unroll
    for (int d = 1; d <= D; d++) {
        const double v = (double)u[d] / r;
        ek += v * (double)u[d];
    }
    return make_double2(r, ((double)u[D + 1] - 0.5 * ek) * (gm - 1.));
}

// ---------------------------------------------------------------------------
// Bulk asynchronous copies (TMA engine, 1-D cp.async.bulk) into shared memory
// completing on an mbarrier. Every wait is bounded: on time-out the kernel
// records kStatusStagingTimeout in *status and carries on, so a lost copy
// can never hang the device; the host turns the flag into an error.
// ---------------------------------------------------------------------------
constexpr int kStatusStagingTimeout = 1;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// bounded wait on one mbarrier phase; false (and the status flag) on time-out
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, int* status) {
    for (int i = 0; i < (1 << 20); i++)
        if (mbar_try_wait(bar, parity)) return true;
    if (status) atomicOr(status, kStatusStagingTimeout);
    return false;
}

}  // namespace spdk

#include "spdk_picard2d.cuh"
#include "spdk_picard3d.cuh"

namespace spdk {

// threads and resident blocks of a pass
template <typename R, int D, int P, int TX, int TY>
constexpr int picard_threads() {
    if constexpr (D == 2) return Line2<R, P, TX, TY, kFlux>::threads;
    else return Line3<R, P, kFlux>::threads;
}
template <typename R, int D, int P, int MODE, bool VISC = false>
constexpr int picard_blocks() {
    if constexpr (D == 2) return VISC ? kLineBlocksPerSMVisc<R, P, MODE> : kLineBlocksPerSM<R, P, MODE>;
    else return kLine3BlocksPerSM<R, P, MODE>;
}

// VISC: instantiation that adds the viscous interface fluxes (hydro/nu > 0);
// the inviscid kernels carry none of that code. (TX, TY: tile of the 2D pass)
template <typename R, int D, int P, int TX, int TY, int MODE, bool VISC = false>
__global__ void __launch_bounds__(picard_threads<R, D, P, TX, TY>(), picard_blocks<R, D, P, MODE, VISC>())
    picard_kernel(DevGrid G, DevMatsT<R> M, PicardArgsT<R> A) {
    pdl_wait();
    if (gate_closed(G)) return;
    if constexpr (D == 2) picard2d_body<R, P, TX, TY, MODE, VISC>(G, M, A, blockIdx.x);
    else picard3d_body<R, P, MODE, VISC>(G, M, A, blockIdx.x);
}

// The 2D pass with a tile, a direction form (RT) and registers of its own
template <typename R, int P, int TX, int TY, int MODE, bool VISC, bool RT, int BLOCKS>
__global__ void __launch_bounds__(Line2<R, P, TX, TY, MODE>::threads, BLOCKS)
    picard2d_kernel(DevGrid G, DevMatsT<R> M, PicardArgsT<R> A) {
    pdl_wait();
    if (gate_closed(G)) return;
    picard2d_body<R, P, TX, TY, MODE, VISC, RT>(G, M, A, blockIdx.x);
}

// The 3D pass with all the registers of one block per SM, for launches of at most
// that many
template <typename R, int P, int MODE, bool VISC>
__global__ void __launch_bounds__(Line3<R, P, MODE>::threads, 1)
    picard3d_kernel(DevGrid G, DevMatsT<R> M, PicardArgsT<R> A) {
    pdl_wait();
    if (gate_closed(G)) return;
    picard3d_body<R, P, MODE, VISC>(G, M, A, blockIdx.x);
}

// The 3D corrector on a caller's buffers that start on no 16-byte boundary
template <typename R, int P>
__global__ void __launch_bounds__(picard_threads<R, 3, P, 1, 1>(), picard_blocks<R, 3, P, kCorrect>())
    correct_any_kernel(DevGrid G, DevMatsT<R> M, PicardArgsT<R> A) {
    pdl_wait();
    if (gate_closed(G)) return;
    picard3d_body<R, P, kCorrect, false, true>(G, M, A, blockIdx.x);
}

template <typename R, int D, int P, int TX, int TY, int MODE>
constexpr size_t picard_smem_bytes() {
    if constexpr (D == 2) return Line2<R, P, TX, TY, MODE>::bytes;
    else return Line3<R, P, MODE>::bytes;
}

}  // namespace spdk
