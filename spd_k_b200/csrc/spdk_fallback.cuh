// A-posteriori fallback of the spd_K B200 hydro step: NAD/SED/PAD trouble
// detection, theta blending and the MUSCL-Hancock/HLLC fallback flux on the
// FV sub-grid (the p+1 Gauss-point cells of every element), one time slice
// at a time (src/hydro_ader.hpp:500-575).
//
// The reference keeps the sub-grid in separate ghost-framed arrays; here the
// sub-cells stay inside their elements ([element][point] order) and the two
// ghost layers are evaluated through spdk::fv_image, which reproduces the
// reference's x-then-y-then-z ghost fill (corner ghosts included).
#pragma once
#include <cuda_runtime.h>

#include "spdk_kernels.cuh"

namespace spdk {

// The blend tiles that have trouble within three cells, collected by the
// detection and emptied again by the blend (marks) and the update (count)
struct BlendList {
    int* mark;   // [tile] 1: listed
    int* tiles;  // block numbers of the listed tiles
    int* count;
    int first;   // block number of tile 0 (a batch lists its members' tiles together)
};

// Blended fluxes of one slice (blend kernel): the SD face fluxes of the faces
// that the troubles reach are replaced in place
template <typename R>
struct BlendArgsT {
    const R* ucv;             // U_cv at the start of slice t [E][V][NPT]
    R* ff[3];                 // FV face fluxes of each direction, all slices
    const uint8_t* trouble;   // [E][NPT]
    uint8_t* theta;           // [E][NPT], theta * 8 (zero on entry where no trouble is near)
    BlendList list;           // tiles with trouble near
    int t;                    // slice
    const double* dt;
};

template <typename R>
struct FallbackArgsT {
    const R* ucv_in;        // U_cv at the start of slice t [E][V][NPT]
    R* ucv_out;             // U_cv after slice t
    R* ff[3];               // FV face fluxes of each direction, all slices
    double2* rp_old_next;   // (rho, p) of U_old / U_new candidates of slice t+1
    double2* rp_new_next;
    int t;                  // slice
    int last;               // last slice of the stage: U_sp = cv_to_sp(U_cv)
    R* u;                   // U_sp (written on the last slice)
    const R* u0;            // RK step-start state
    double rk_a;
    int final_stage;        // compute W_cv and the next dt
    R* wcv;
    unsigned long long* dtmin;
    const double* dt;
    int* blend_count;       // emptied for the next slice's detection
    // learned indicator (nullable): after the final stage, the element means
    // of (rho, p) and the nodal part of each feature row (row length n_in)
    // of the new state, for the next step's a-priori flags
    uint16_t* feat;
    float2* means;
    int n_in;
};

// what a detect launch reads and writes
struct DetectArgs {
    const double2* rpo;  // (rho, p) of the U_old / U_new candidates
    const double2* rpn;
    uint8_t* T;          // troubles
    uint8_t* theta;      // cleared for the blend kernel
    BlendList list;      // blend tiles the troubles reach
};

// Cell numbers of a tile and its halo: the number of cell (x, y, z) of the
// frame that begins H cells outside the tile is x0[x] + x1[y] + x2[z], each
// part from the cell's image in that direction; a part is kNoCell where there
// is none (outside the domain and its `layers` ghost layers), and flip[d]
// marks reflective images. Formed once per block, so that a staged cell costs
// two or three shared loads instead of the image arithmetic. Cell numbers fit
// 32 bits: the smallest state with the fallback (2D, FP32, SSP-RK1) takes 146
// bytes a cell, 313 GB for 2^31 of them.
constexpr int kNoCell = -1;
__host__ __device__ constexpr int cell_number(int x, int y, int z) {
    return (x | y | z) < 0 ? kNoCell : x + y + z;  // a part that is missing outweighs any sum of the others
}
static_assert(cell_number(kNoCell, 1 << 30, 0) < 0 && cell_number(1 << 30, kNoCell, 0) < 0 &&
              cell_number(1 << 29, 1 << 29, kNoCell) < 0, "no image whatever the other parts");
static_assert(cell_number(5, 1 << 29, 1 << 30) == 5 + (1 << 29) + (1 << 30), "large cell numbers");
template <int D, int P, int TX, int TY, int TZ, int H>
struct CellMap {
    static constexpr int n = P + 1;
    static constexpr int Lx = TX * n + 2 * H, Ly = TY * n + 2 * H, Lz = D == 3 ? TZ * n + 2 * H : 1;
    int x0[Lx], x1[Ly], x2[Lz];
    uint8_t flip[Lx + Ly + Lz];
    __device__ __forceinline__ void fill(const DevGrid& G, const int o[3], int layers) {
        constexpr int NPT = Shape<D, P>::NPT;
        for (int q = threadIdx.x; q < Lx + Ly + (D == 3 ? Lz : 0); q += blockDim.x) {
            const int d = q < Lx ? 0 : (q < Lx + Ly ? 1 : 2);
            const int i = q - (d == 0 ? 0 : (d == 1 ? Lx : Lx + Ly));
            const int a = o[d] - H + i, na = G.N[d] * n;
            const int g = G.bc[d] == kPeriodic ? layers : (layers < 2 ? layers : 2);
            int part = kNoCell;
            bool f = false;
            if (a >= -g && a < na + g) {
                const int m = fv_image(a, na, G.bc[d], &f), e = m / n, c = m - e * n;
                if (d == 0) part = e * NPT + c;
                else if (d == 1) part = e * G.N[0] * NPT + c * n;
                else part = e * G.N[0] * G.N[1] * NPT + c * n * n;
            }
            (d == 0 ? x0 : (d == 1 ? x1 : x2))[i] = part;
            flip[q] = f;
        }
        if (D == 2 && threadIdx.x == 0) x2[0] = 0;
    }
    // cell number, negative where the cell has no image
    __device__ __forceinline__ int cell(int x, int y, int z) const {
        return cell_number(x0[x], x1[y], D == 3 ? x2[z] : 0);
    }
};

// a cell of the domain (tiles at the high edges may hang over it)
template <int D, int P>
__device__ __forceinline__ bool in_domain(const DevGrid& G, const int a[3]) {
    bool in = true;
#pragma unroll
    for (int d = 0; d < D; d++) in &= a[d] < G.N[d] * (P + 1);
    return in;
}
// a cell of the domain or of its first `layers` ghost layers (the ghost frame
// of a non-periodic edge is two layers deep)
template <int D, int P>
__device__ __forceinline__ bool has_image(const DevGrid& G, const int a[3], int layers) {
    bool in = true;
#pragma unroll
    for (int d = 0; d < D; d++) {
        const int g = G.bc[d] == kPeriodic ? layers : (layers < 2 ? layers : 2);
        in &= a[d] >= -g && a[d] < G.N[d] * (P + 1) + g;
    }
    return in;
}

__device__ __forceinline__ double rp_var(const double2 v, int k) { return k == 0 ? v.x : v.y; }

// elements of a blend block: 64 to 144 sub-cells in 2D and 16 to 216 in 3D, so
// that nearly every one of the block's phases takes its 256 threads one round: a
// tile's time is a chain of their latencies (4 x 4 elements at p = 3 took twice
// as long)
template <int D, int P>
struct BlendTile {
    static constexpr int X = D == 2 ? (P <= 3 ? 4 : 2) : (P <= 3 ? 2 : 1);
    static constexpr int Y = D == 2 ? (P <= 2 ? 4 : (P <= 5 ? 2 : 1)) : 1;
    static constexpr int Z = 1;
};

// ---------------------------------------------------------------------------
// Trouble detection of every active sub-cell (src/trouble_detection.cpp:35-290
// with limit mask rho|p, src/hydro_ader.hpp:522-524).
//
// The SED relaxation can only clear a flag NAD raised (relax_NAD keeps a
// flag iff alpha < 1), so the division-heavy smooth-extrema indicator is
// evaluated only at cells NAD flagged; the result is identical to computing
// it everywhere. W_old (rho, p) of the tile + 1 halo is staged in shared
// memory for the NAD box.
// ---------------------------------------------------------------------------
// FV axes of the smooth-extrema indicator: active cells and the ghost-framed
// centre / face coordinates of each direction
struct SedGeom {
    int nd[3];
    const double* C[3];
    const double* Fc[3];
};

template <int D, int P>
__device__ __forceinline__ SedGeom sed_geom(const DevGrid& G) {
    SedGeom S;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        S.nd[d] = G.N[d] * (P + 1);
        S.C[d] = G.fvc[d];
        S.Fc[d] = G.fvf[d];
    }
    return S;
}

// rpv(b, k): variable k (rho, p) of the candidate at FV coordinate b, which
// lies at most two cells outside the active cells.
// The smooth-extrema alpha of position a in direction d (0 outside the
// active cells, where the reference never computes it).
template <typename RPV>
__device__ __forceinline__ double sed_al(const SedGeom& S, const RPV& rpv, const int a[3], int d, int k) {
    const int ad = a[d];
    if (ad < 0 || ad >= S.nd[d]) return 0.0;
    const double* C = S.C[d];
    const double* Fc = S.Fc[d];
    int b[3] = {a[0], a[1], a[2]};
    double Wv[5];
#pragma unroll
    for (int off = -2; off <= 2; off++) {
        b[d] = ad + off;
        Wv[off + 2] = rpv(b, k);
    }
    const int l = ad + 2;
    const double h = (C[l + 1] - C[l - 1]);
    const double hp = (C[l + 2] - C[l]);
    const double hm = (C[l] - C[l - 2]);
    const double u = Wv[2];
    const double du = (Wv[3] - Wv[1]) / h;
    const double dup = (Wv[4] - u) / hp;
    const double dum = (u - Wv[0]) / hm;
    const double d2u = (dup - dum) / (C[l + 1] - C[l - 1]);
    const double dv = 0.5 * d2u * (Fc[l + 1] - Fc[l]);
    return sed_alpha(dv, dum, du, dup);
}

// min of the alphas of the cell and its two neighbours in direction d
template <typename RPV>
__device__ __forceinline__ double sed_component(const SedGeom& S, const RPV& rpv, const int a[3], int d, int k) {
    double al[3];
#pragma unroll
    for (int s = -1; s <= 1; s++) {
        int b[3] = {a[0], a[1], a[2]};
        b[d] += s;
        al[s + 1] = sed_al(S, rpv, b, d, k);
    }
    return smin(smin(al[0], al[1]), al[2]);
}

// min over the directions of the SED alpha of 2D cell (ax, ay), variable k,
// from candidates staged on the tile + 3 halo (Rn, row length E3x, origin
// ox - 3, oy - 3). Not inlined: the rare flagged cells pay for its registers
// in its own frame, and the NAD pass of every cell keeps to its cap.
static __device__ __noinline__ double sed_alpha_staged_2d(const SedGeom S, const double2* Rn, int E3x, int ox, int oy,
                                                         int ax, int ay, int k) {
    auto staged = [&](const int b[3], int kk) { return rp_var(Rn[(b[0] - ox + 3) + E3x * (b[1] - oy + 3)], kk); };
    const int a[3] = {ax, ay, 0};
    const double m0 = sed_component(S, staged, a, 0, k);
    return smin(m0, sed_component(S, staged, a, 1, k));
}

// the same for a 3D cell, candidates staged on the tile + 3 halo (rows of
// E3x, planes of E3x * E3y, origin o - 3)
static __device__ __noinline__ double sed_alpha_staged_3d(const SedGeom S, const double2* Rn, int E3x, int E3y,
                                                         const int o[3], const int a[3], int k) {
    auto staged = [&](const int b[3], int kk) {
        return rp_var(Rn[(b[0] - o[0] + 3) + E3x * ((b[1] - o[1] + 3) + E3y * (b[2] - o[2] + 3))], kk);
    };
    const double m0 = sed_component(S, staged, a, 0, k);
    const double m1 = smin(m0, sed_component(S, staged, a, 1, k));
    return smin(m1, sed_component(S, staged, a, 2, k));
}

// every alpha of variable k that the cells of a 3D tile (Bx x By x Bz from
// o) take along each direction d: the tile extended by one cell along d
// only, Al = [d = 0: (Bx + 2) By Bz][d = 1: Bx (By + 2) Bz][d = 2: Bx By
// (Bz + 2)], each x-fastest; candidates staged on the tile + 3 halo
static __device__ __noinline__ void sed_al_tile_3d(const SedGeom S, const double2* Rn, int E3x, int E3y,
                                                   const int o[3], int Bx, int By, int Bz, int k, double* Al) {
    auto staged = [&](const int b[3], int kk) {
        return rp_var(Rn[(b[0] - o[0] + 3) + E3x * ((b[1] - o[1] + 3) + E3y * (b[2] - o[2] + 3))], kk);
    };
    const int n0 = (Bx + 2) * By * Bz, n1 = Bx * (By + 2) * Bz, n2 = Bx * By * (Bz + 2);
    for (int w = threadIdx.x; w < n0 + n1 + n2; w += blockDim.x) {
        const int d = w < n0 ? 0 : (w < n0 + n1 ? 1 : 2);
        const int r = w - (d == 0 ? 0 : (d == 1 ? n0 : n0 + n1));
        const int ex = Bx + 2 * (d == 0), ey = By + 2 * (d == 1);
        const int a[3] = {o[0] + r % ex - (d == 0), o[1] + (r / ex) % ey - (d == 1), o[2] + r / (ex * ey) - (d == 2)};
        Al[w] = sed_al(S, staged, a, d, k);
    }
}

// every alpha of the 2D tile + 1 halo (E1x x E1y positions from ox - 1,
// oy - 1) of the variables in kmask, by the whole block: Al[(k * 2 + d) *
// E1x * E1y + position]; for blocks with many flagged cells, whose
// neighbours would otherwise evaluate the same positions again
static __device__ __noinline__ void sed_al_tile_2d(const SedGeom S, const double2* Rn, int E3x, int E1x, int E1y,
                                                   int ox, int oy, unsigned kmask, double* Al) {
    auto staged = [&](const int b[3], int kk) { return rp_var(Rn[(b[0] - ox + 3) + E3x * (b[1] - oy + 3)], kk); };
    const int np = E1x * E1y;
    for (int w = threadIdx.x; w < 4 * np; w += blockDim.x) {
        const int pos = w % np, kd = w / np, k = kd >> 1, d = kd & 1;
        if (!((kmask >> k) & 1u)) continue;
        const int a[3] = {ox - 1 + pos % E1x, oy - 1 + pos / E1x, 0};
        Al[w] = sed_al(S, staged, a, d, k);
    }
}

// R names the form (double: plain, float: precision) that launches the
// kernel; the detector computes in FP64 in both, and a separate
// instantiation per form keeps each form's compile flags on its own copy.
//
// Each thread loads its cells' candidates before it stages the tile's W_old,
// so a block waits for one memory round trip, not two. Cell numbers come from
// per-direction tables (CellMap), and a thread's cells are in memory order, so
// the flags leave in whole sectors. In 2D the kernel is
// compiled for 4 resident blocks (64 registers, the NAD pass unspilled;
// measured on B200: 38.6 us against 43.2 us at 6 blocks with spills); in
// 3D for 3 (80 registers, 20-50 bytes of spills; 90 registers and 2
// blocks uncapped: KH 16^3 p=5 FP64 step 11.40 -> 11.28 ms at 3).
template <int D>
constexpr int kDetectBlocksPerSM = D == 2 ? 4 : 3;
// flagged threads of a block above which it evaluates every alpha of its
// tile once instead of each flagged cell evaluating its own six
constexpr int kSedTileThreshold = 24;

template <typename R, int D, int P, int TX, int TY, int TZ>
__device__ __forceinline__ void fv_detect_kernel_body(const DevGrid& G, const DetectArgs& A, long long bidx) {
    constexpr int n = P + 1;
    constexpr int NPT = Shape<D, P>::NPT;
    constexpr int NE = TX * TY * TZ;
    constexpr int Bx = TX * n, By = TY * n, Bz = D == 3 ? TZ * n : 1;
    constexpr int E1x = Bx + 2, E1y = By + 2, E1z = D == 3 ? Bz + 2 : 1;
    constexpr int NC = Bx * By * Bz;
    constexpr int CPT = (NC + kThreads - 1) / kThreads;  // cells per thread
    static_assert(CPT <= 16, "NAD flag bits");
    constexpr int E3x = Bx + 6, E3y = By + 6, E3z = D == 3 ? Bz + 6 : 1;
    // (a flagged cell would otherwise read its 45 candidates per variable from global memory)
    static_assert(D == 2 || (size_t)(E3x * E3y * E3z + E1x * E1y * E1z) * sizeof(double2) <= 46 * 1024,
                  "the candidates on the tile + 3 halo fit the static shared memory beside W_old's tile + 1 halo");
    const double2* __restrict__ rpo = A.rpo;
    const double2* __restrict__ rpn = A.rpn;
    __shared__ int el_any[NE];
    for (int e = threadIdx.x; e < NE; e += blockDim.x) el_any[e] = 0;
    __shared__ double2 Ro[E1x * E1y * E1z];
    __shared__ double2 Rn[E3x * E3y * E3z];
    __shared__ double Al[D == 2 ? 4 * E1x * E1y : 1];
    __shared__ CellMap<D, P, TX, TY, TZ, 3> map;
    const int dz = D == 3 ? 1 : 0;
    int o[3];
    {
        int b = bidx;
        const int tx = (G.N[0] + TX - 1) / TX, ty = (G.N[1] + TY - 1) / TY;
        o[0] = (b % tx) * Bx;
        b /= tx;
        o[1] = (b % ty) * By;
        b /= ty;
        o[2] = D == 3 ? b * Bz : 0;
    }
    map.fill(G, o, 3);
    __syncthreads();
    // this thread's cells, in memory order: element q / NPT, point q % NPT;
    // cells of a tile that hangs over the domain: bit r is clear
    auto place = [&](int q, int l[3]) {
        const int el = q / NPT, pt = q % NPT;
        l[0] = (el % TX) * n + pt % n;
        l[1] = ((el / TX) % TY) * n + (pt / n) % n;
        l[2] = D == 3 ? (el / (TX * TY)) * n + pt / (n * n) : 0;
    };
    unsigned mine = 0;
    double2 here_new[CPT];
#pragma unroll
    for (int r = 0; r < CPT; r++) {
        const int q = threadIdx.x + r * kThreads;
        here_new[r] = make_double2(1.0, 1.0);
        if (NC % kThreads == 0 || q < NC) {
            int l[3];
            place(q, l);
            int a[3] = {o[0] + l[0], o[1] + l[1], o[2] + l[2]};
            if (in_domain<D, P>(G, a)) {
                mine |= 1u << r;
                here_new[r] = rpn[map.cell(l[0] + 3, l[1] + 3, l[2] + 3 * dz)];
            }
        }
    }
    for (int q = threadIdx.x; q < E1x * E1y * E1z; q += blockDim.x) {
        const int id = map.cell(q % E1x + 2, (q / E1x) % E1y + 2, q / (E1x * E1y) + 2 * dz);
        Ro[q] = id >= 0 ? rpo[id] : make_double2(1.0, 1.0);
    }
    __syncthreads();
    // NAD flags of this thread's cells: bit 2r + k for variable k of cell r
    unsigned nad = 0;
#pragma unroll
    for (int r = 0; r < CPT; r++) {
        const int q = threadIdx.x + r * kThreads;
        if (!((mine >> r) & 1u)) continue;
        int l[3];
        place(q, l);
        const int sc = (l[0] + 1) + E1x * ((l[1] + 1) + E1y * (l[2] + dz));
        // extrema of both variables over the box (or the cross)
        double2 mx = Ro[sc], mn = mx;
        auto take = [&](const double2 u) {
            mx.x = smax(mx.x, u.x);
            mn.x = smin(mn.x, u.x);
            mx.y = smax(mx.y, u.y);
            mn.y = smin(mn.y, u.y);
        };
        if (G.nad_moore) {
            for (int ok = -dz; ok <= dz; ok++)
#pragma unroll
                for (int oj = -1; oj <= 1; oj++)
#pragma unroll
                    for (int oi = -1; oi <= 1; oi++) take(Ro[sc + oi + E1x * (oj + E1y * ok)]);
        } else {
#pragma unroll
            for (int d = 0; d < D; d++) {
                const int st = d == 0 ? 1 : (d == 1 ? E1x : E1x * E1y);
                const double2 uL = Ro[sc - st], uR = Ro[sc + st];
                mx = make_double2(smax(smax(uL.x, mx.x), uR.x), smax(smax(uL.y, mx.y), uR.y));
                mn = make_double2(smin(smin(uL.x, mn.x), uR.x), smin(smin(uL.y, mn.y), uR.y));
            }
        }
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const double un = rp_var(here_new[r], k);
            double hi = rp_var(mx, k), lo = rp_var(mn, k);
            if (G.nad_delta) {
                const double eps = G.nad_tol * (hi - lo);
                lo -= eps;
                hi += eps;
            } else {
                lo -= fabs(lo) * G.nad_tol;
                hi += fabs(hi) * G.nad_tol;
            }
            if (un > hi || un < lo) nad |= 1u << (2 * r + k);
        }
    }
    // SED relaxation of the NAD flags (it can only clear one). The block stages
    // the candidates of the tile + 3 halo once when any of its cells needs it, so
    // a flagged cell reads its stencils from shared memory instead of a chain of
    // global loads.
    const int nflag = G.use_sed ? __syncthreads_count(nad != 0) : 0;
    if (nflag) {
        for (int q = threadIdx.x; q < E3x * E3y * E3z; q += blockDim.x) {
            // (three cells outside a non-periodic boundary: never read)
            const int id = map.cell(q % E3x, (q / E3x) % E3y, q / (E3x * E3y));
            Rn[q] = id >= 0 ? rpn[id] : make_double2(0.0, 0.0);
        }
        __syncthreads();
        const SedGeom SG = sed_geom<D, P>(G);
        const bool tile = D == 2 && nflag > kSedTileThreshold;
        const bool tile3 = D == 3 && nflag > kSedTileThreshold;
        if (tile3) {
            if constexpr (D == 3) {
                // many flagged cells: every alpha of the tile once per
                // variable, in the W_old tile's storage (free after NAD),
                // then each flagged cell takes the min of its own and its
                // neighbours' along each direction, in sed_component's order
                constexpr int n0 = (Bx + 2) * By * Bz, n1 = Bx * (By + 2) * Bz, n2 = Bx * By * (Bz + 2);
                static_assert((size_t)(n0 + n1 + n2) * sizeof(double) <= sizeof(Ro), "alphas fit the W_old tile");
                double* Al3 = reinterpret_cast<double*>(Ro);
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    if (!__syncthreads_or(nad & (k == 0 ? 0x55555555u : 0xAAAAAAAAu))) continue;
                    sed_al_tile_3d(SG, Rn, E3x, E3y, o, Bx, By, Bz, k, Al3);
                    __syncthreads();
#pragma unroll
                    for (int r = 0; r < CPT; r++) {
                        if (!(nad & (1u << (2 * r + k)))) continue;
                        int l[3];
                        place(threadIdx.x + r * kThreads, l);
                        const int x = l[0], y = l[1], z = l[2];
                        double alpha = 1;
#pragma unroll
                        for (int d = 0; d < 3; d++) {
                            double al[3];
#pragma unroll
                            for (int sft = -1; sft <= 1; sft++) {
                                const int i = d == 0 ? (x + 1 + sft) + (Bx + 2) * (y + By * z)
                                                     : (d == 1 ? n0 + x + Bx * ((y + 1 + sft) + (By + 2) * z)
                                                               : n0 + n1 + x + Bx * (y + By * (z + 1 + sft)));
                                al[sft + 1] = Al3[i];
                            }
                            const double m3 = smin(smin(al[0], al[1]), al[2]);
                            alpha = d == 0 ? m3 : smin(alpha, m3);
                        }
                        if (!(alpha < 1)) nad &= ~(1u << (2 * r + k));
                    }
                    __syncthreads();
                }
            }
        } else {
            if (tile) {
                const unsigned kmask = (__syncthreads_or(nad & 0x55555555u) ? 1u : 0u) |
                                       (__syncthreads_or(nad & 0xAAAAAAAAu) ? 2u : 0u);
                sed_al_tile_2d(SG, Rn, E3x, E1x, E1y, o[0], o[1], kmask, Al);
                __syncthreads();
            }
#pragma unroll
            for (int r = 0; r < CPT; r++) {
                if (!(nad & (3u << (2 * r)))) continue;
                int l[3];
                place(threadIdx.x + r * kThreads, l);
                int a[3] = {o[0] + l[0], o[1] + l[1], o[2] + l[2]};
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    if (!(nad & (1u << (2 * r + k)))) continue;
                    double alpha = 1;
                    if (tile) {
                        // the alphas of the cell and its neighbours, in the
                        // order sed_component takes them
                        const int x = a[0] - o[0] + 1, y = a[1] - o[1] + 1;
                        const double* A0 = Al + (k * 2 + 0) * E1x * E1y;
                        const double* A1 = Al + (k * 2 + 1) * E1x * E1y;
                        const double m0 = smin(smin(A0[(x - 1) + E1x * y], A0[x + E1x * y]), A0[(x + 1) + E1x * y]);
                        const double m1 = smin(smin(A1[x + E1x * (y - 1)], A1[x + E1x * y]), A1[x + E1x * (y + 1)]);
                        alpha = smin(m0, m1);
                    } else if (D == 2) {
                        alpha = sed_alpha_staged_2d(SG, Rn, E3x, o[0], o[1], a[0], a[1], k);
                    } else {
                        alpha = sed_alpha_staged_3d(SG, Rn, E3x, E3y, o, a, k);
                    }
                    if (!(alpha < 1)) nad &= ~(1u << (2 * r + k));
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < CPT; r++) {
        const int q = threadIdx.x + r * kThreads;
        if (!((mine >> r) & 1u)) continue;
        int l[3];
        place(q, l);
        const int cid = map.cell(l[0] + 3, l[1] + 3, l[2] + 3 * dz);
        bool tr = (nad >> (2 * r)) & 3u;
        const double rho = here_new[r].x, p = here_new[r].y;
        if (rho < kRhoMin || rho > kRhoMax) tr = true;
        if (p < kPMin || p > kPMax) tr = true;
        const int el = cid / NPT;
        if (G.elem_trouble && tr) G.elem_trouble[el] = 1;  // a-posteriori label
        if (G.elem_pred && G.elem_pred[el]) tr = true;     // a-priori prediction
        A.T[cid] = tr ? 1 : 0;
        A.theta[cid] = 0;
        if (tr) el_any[q / NPT] = 1;
    }
    __syncthreads();
    // list the blend tiles within three cells (K elements) of a troubled element
    using BT = BlendTile<D, P>;
    constexpr int K = (3 + n - 1) / n;
    constexpr int Rx = 2 * K + 1, Ry = Rx, Rz = D == 3 ? Rx : 1;
    const int nbx = (G.N[0] + BT::X - 1) / BT::X, nby = (G.N[1] + BT::Y - 1) / BT::Y;
    for (int w = threadIdx.x; w < NE * Rx * Ry * Rz; w += blockDim.x) {
        const int e = w / (Rx * Ry * Rz), r = w % (Rx * Ry * Rz);
        if (!el_any[e]) continue;
        int g[3] = {o[0] / n + e % TX + r % Rx - K, o[1] / n + (e / TX) % TY + (r / Rx) % Ry - K,
                    D == 3 ? o[2] / n + e / (TX * TY) + r / (Rx * Ry) - K : 0};
        bool in = true;
#pragma unroll
        for (int d = 0; d < D; d++) {
            if (g[d] >= 0 && g[d] < G.N[d]) continue;
            // ghosts of a non-periodic edge are images of the edge's own cells
            if (G.bc[d] != kPeriodic) in = false;
            else g[d] = (g[d] + K * G.N[d]) % G.N[d];
        }
        if (!in) continue;
        const int tile = g[0] / BT::X + nbx * (g[1] / BT::Y + nby * (g[2] / BT::Z));
        if (!*(volatile int*)&A.list.mark[tile] && atomicExch(&A.list.mark[tile], 1) == 0)
            A.list.tiles[atomicAdd(A.list.count, 1)] = A.list.first + tile;
    }
}

template <typename R, int D, int P, int TX, int TY, int TZ>
__global__ void __launch_bounds__(kThreads, kDetectBlocksPerSM<D>) fv_detect_kernel(DevGrid G, DetectArgs A) {
    pdl_wait();
    if (gate_closed(G)) return;
    fv_detect_kernel_body<R, D, P, TX, TY, TZ>(G, A, blockIdx.x);
}

// ---------------------------------------------------------------------------
// theta = max over the Moore box of w(#offsets) * trouble, plus the 0.25 ring
// (src/trouble_detection.cpp:191-242; theta_from_troubles without blending),
// evaluated by the blend kernel on its tile + 1 halo from the troubles on
// the tile + 3 halo, in eighths: w * 8 = 8, 6, 4, 3 and the ring 2 (all
// exact, as is theta * 8 of the reference's float weights).
//
// A ghost cell's theta is the theta of its image (the reference fills the
// ghosts of theta after computing it on the active cells). Outside a
// periodic boundary that equals the theta evaluated in place, since the
// troubles around it are periodic images too; outside a reflective or
// zero-gradient boundary the image (one or two cells inside) lies in the
// same tile and its value is used. The tile's own cells are written to
// `theta_out` (the THETA field).
// ---------------------------------------------------------------------------
template <int D, int P, int TX, int TY, int TZ>
struct ThetaTile {
    static constexpr int n = P + 1;
    static constexpr int Bx = TX * n, By = TY * n, Bz = D == 3 ? TZ * n : 1;
    static constexpr int E3x = Bx + 6, E3y = By + 6, E3z = D == 3 ? Bz + 6 : 1;
    static constexpr int E2x = Bx + 4, E2y = By + 4, E2z = D == 3 ? Bz + 4 : 1;
    static constexpr int E1x = Bx + 2, E1y = By + 2, E1z = D == 3 ? Bz + 2 : 1;
    static constexpr int n3 = E3x * E3y * E3z, n2 = E2x * E2y * E2z, n1 = E1x * E1y * E1z;
    static constexpr size_t scratch = (size_t)n3 + n2;  // bytes of T3 + Th2
};

// called by every thread of the block; `scratch` holds ThetaTile::scratch
// bytes; th (tile + 1 halo) is complete after the caller's next barrier.
// theta_out of the tile's cells was cleared by the detection.
template <int D, int P, int TX, int TY, int TZ>
__device__ __forceinline__ void theta_on_tile(const DevGrid& G, const CellMap<D, P, TX, TY, TZ, 3>& map,
                                              const uint8_t* __restrict__ T, const int o[3], uint8_t* scratch, uint8_t* th, uint8_t* __restrict__ theta_out) {
    using TT = ThetaTile<D, P, TX, TY, TZ>;
    constexpr int n = P + 1;
    const int dz = D == 3 ? 1 : 0;
    uint8_t* T3 = scratch;
    uint8_t* Th2 = scratch + TT::n3;
    for (int q = threadIdx.x; q < TT::n3; q += blockDim.x) {
        // a cell three layers outside a non-periodic boundary has no image
        // (the ghost frame is two layers deep) and feeds no theta below:
        // the theta of a ghost cell there is its image's
        const int id = map.cell(q % TT::E3x, (q / TT::E3x) % TT::E3y, q / (TT::E3x * TT::E3y));
        T3[q] = id >= 0 ? T[id] : (uint8_t)0;
    }
    __syncthreads();
    if (G.blending) {
        for (int q = threadIdx.x; q < TT::n2; q += blockDim.x) {
            const int x = q % TT::E2x + 1, y = (q / TT::E2x) % TT::E2y + 1, z = q / (TT::E2x * TT::E2y) + dz;
            int m = 0;
            for (int ok = -dz; ok <= dz; ok++)
#pragma unroll
                for (int oj = -1; oj <= 1; oj++)
#pragma unroll
                    for (int oi = -1; oi <= 1; oi++) {
                        const int n0 = (oi != 0) + (oj != 0) + (ok != 0);
                        const int w8 = n0 == 0 ? 8 : (n0 == 1 ? 6 : (n0 == 2 ? 4 : 3));
                        if (T3[(x + oi) + TT::E3x * ((y + oj) + TT::E3y * (z + ok))]) m = m < w8 ? w8 : m;
                    }
            Th2[q] = (uint8_t)m;
        }
        __syncthreads();
    }
    for (int q = threadIdx.x; q < TT::n1; q += blockDim.x) {
        const int l0[3] = {q % TT::E1x, (q / TT::E1x) % TT::E1y, q / (TT::E1x * TT::E1y)};
        int l[3] = {l0[0], l0[1], l0[2]};
        int ga[3] = {o[0] + l0[0] - 1, o[1] + l0[1] - 1, o[2] + l0[2] - dz};
        if (!has_image<D, P>(G, ga, 1)) {
            th[q] = 0;
            continue;
        }
#pragma unroll
        for (int d = 0; d < D; d++) {
            const int na = G.N[d] * n;
            if ((ga[d] < 0 || ga[d] >= na) && G.bc[d] != kPeriodic) {
                bool f = false;
                l[d] = fv_image(ga[d], na, G.bc[d], &f) - o[d] + 1;
            }
        }
        int t8;
        if (G.blending) {
            const int x = l[0] + 1, y = l[1] + 1, z = l[2] + dz;
            const int c = Th2[x + TT::E2x * (y + TT::E2y * z)];
            int ring = 0;
            for (int ok = -dz; ok <= dz; ok++)
#pragma unroll
                for (int oj = -1; oj <= 1; oj++)
#pragma unroll
                    for (int oi = -1; oi <= 1; oi++)
                        if (Th2[(x + oi) + TT::E2x * ((y + oj) + TT::E2y * (z + ok))]) ring = 2;
            t8 = c < ring ? ring : c;
        } else {
            t8 = T3[(l[0] + 2) + TT::E3x * ((l[1] + 2) + TT::E3y * (l[2] + 2 * dz))] ? 8 : 0;
        }
        th[q] = (uint8_t)t8;
        const bool inner = l0[0] >= 1 && l0[0] <= TT::Bx && l0[1] >= 1 && l0[1] <= TT::By &&
                           (D == 2 || (l0[2] >= 1 && l0[2] <= TT::Bz));
        if (inner && in_domain<D, P>(G, ga)) theta_out[map.cell(l0[0] + 2, l0[1] + 2, l0[2] + 2 * dz)] = (uint8_t)t8;
    }
}

// Limited slopes of W_old along every direction and the Hancock time
// derivative of cell fa (frame indices), from W_old around it
// (src/hydro.cpp:622-681); Wc(oi, oj, ok) gives W_old of neighbouring cells
template <int D, typename R, typename WF>
__device__ __forceinline__ void muscl_slopes(const DevGrid& G, const int fa[3], WF Wc, R (*dW)[D + 2], R* dwt) {
    constexpr int V = D + 2;
    R w[V];
    const R* wc = Wc(0, 0, 0);
#pragma unroll
    for (int v = 0; v < V; v++) w[v] = wc[v];
#pragma unroll
    for (int d = 0; d < D; d++) {
        const R* wm = Wc(d == 0 ? -1 : 0, d == 1 ? -1 : 0, d == 2 ? -1 : 0);
        const R* wp = Wc(d == 0 ? 1 : 0, d == 1 ? 1 : 0, d == 2 ? 1 : 0);
        const Width dp = G.fd[d][fa[d]], dm = G.fd[d][fa[d] - 1];
        const R h = (R)G.fw[d][fa[d]].h;
#pragma unroll
        for (int v = 0; v < V; v++)
            dW[d][v] = minmod(div_width(G, wp[v] - w[v], dp), div_width(G, w[v] - wm[v], dm), h);
    }
    hancock<D>(w, dwt, dW, (R)G.gm);
}

// ---------------------------------------------------------------------------
// Blend kernel of slice t: fluxes of the faces with theta > 0
// (src/hydro.cpp:683-788) written over the SD face fluxes, each element's own
// copy of an interface.
//
// The launch's blocks share out the tiles that the detection listed (those
// with trouble within three cells). W_old is formed once on the tile + 2 halo, the slopes of a cell once for all its faces (they were formed
// by every face for both of its cells: 4 times a cell in 2D, 6 in 3D, with
// the divisions that dominate them in FP64), and each face takes one HLLC
// solve. Measured per launch: 64^2 p=3 FP64 26 us beside a 12 us update (one
// kernel for both: 107 us); KH 16^3 p=5 FP64, where every tile blends, 572 + 96
// us (997 us). Bounded by the latency of its chain of phases: it is separate from
// the update, whose blocks would otherwise all reserve the shared memory and
// wait for the few that blend.
// ---------------------------------------------------------------------------
template <typename R, int D, int P, int TX, int TY, int TZ>
struct BlendSmem {
    static constexpr int n = P + 1, V = D + 2;
    static constexpr int Bx = TX * n, By = TY * n, Bz = D == 3 ? TZ * n : 1;
    static constexpr int E1x = Bx + 2, E1y = By + 2, E1z = D == 3 ? Bz + 2 : 1;
    static constexpr int E2x = Bx + 4, E2y = By + 4, E2z = D == 3 ? Bz + 4 : 1;
    static constexpr int n1 = E1x * E1y * E1z, n2 = E2x * E2y * E2z;
    static constexpr int NF0 = (Bx + 1) * By * Bz;
    static constexpr int NF1 = Bx * (By + 1) * Bz;
    static constexpr int NF2 = D == 3 ? Bx * By * (Bz + 1) : 0;
    // cells whose slopes some face of the tile needs: the tile's own, then the
    // ones across its low and high x, y (and z) faces
    static constexpr int NC = Bx * By * Bz, HX = By * Bz, HY = Bx * Bz, HZ = D == 3 ? Bx * By : 0;
    static constexpr int ns = NC + 2 * (HX + HY + HZ);
    __device__ static int slot(int x, int y, int z) {  // tile coordinates, at most one of them outside
        if (x < 0 || x >= Bx) return NC + (x < 0 ? 0 : HX) + y + By * z;
        if (y < 0 || y >= By) return NC + 2 * HX + (y < 0 ? 0 : HY) + x + Bx * z;
        if (z < 0 || z >= Bz) return NC + 2 * (HX + HY) + (z < 0 ? 0 : HZ) + x + Bx * y;
        return x + Bx * (y + By * z);
    }
    __device__ static void coords(int q, int l[3]) {
        if (q < NC) { l[0] = q % Bx; l[1] = (q / Bx) % By; l[2] = q / (Bx * By); return; }
        q -= NC;
        if (q < 2 * HX) { l[0] = q < HX ? -1 : Bx; q %= HX; l[1] = q % By; l[2] = q / By; return; }
        q -= 2 * HX;
        if (q < 2 * HY) { l[1] = q < HY ? -1 : By; q %= HY; l[0] = q % Bx; l[2] = q / Bx; return; }
        q -= 2 * HY;
        l[2] = q < HZ ? -1 : Bz;
        q %= HZ > 0 ? HZ : 1;
        l[0] = q % Bx;
        l[1] = q / Bx;
    }
    static constexpr size_t slopes = (size_t)ns * (D + 1) * V;  // [D slopes, dW/dt][V][cell]
    static constexpr size_t wold = (size_t)n2 * V;
    static_assert(ThetaTile<D, P, TX, TY, TZ>::scratch <= slopes * sizeof(R), "theta scratch fits the slopes' area");
    static constexpr size_t bytes = (slopes + wold) * sizeof(R) + ((size_t)n1 + 15) / 16 * 16;
};

template <typename R, int D, int P, int TX, int TY, int TZ>
__device__ __forceinline__ void fv_blend_kernel_body(const DevGrid& G, const DevMatsT<R>& M, const BlendArgsT<R>& A,
                                                     long long bidx) {
    using SM = BlendSmem<R, D, P, TX, TY, TZ>;
    constexpr int n = P + 1, nf = P + 2, V = D + 2, NPT = Shape<D, P>::NPT, NFP = Shape<D, P>::NFP;
    constexpr int Bx = SM::Bx, By = SM::By, Bz = SM::Bz;
    constexpr int E1x = SM::E1x, E1y = SM::E1y, E2x = SM::E2x, E2y = SM::E2y, ns = SM::ns;
    const int dz = D == 3 ? 1 : 0;
    int o[3], oe[3];
    {
        int b = (int)bidx;
        const int tx = (G.N[0] + TX - 1) / TX, ty = (G.N[1] + TY - 1) / TY;
        oe[0] = (b % tx) * TX;
        b /= tx;
        oe[1] = (b % ty) * TY;
        b /= ty;
        oe[2] = D == 3 ? b * TZ : 0;
        o[0] = oe[0] * n;
        o[1] = oe[1] * n;
        o[2] = oe[2] * n;
    }
    extern __shared__ __align__(128) unsigned char smem_raw[];
    R* SL = reinterpret_cast<R*>(smem_raw);  // slopes and dW/dt on the tile + 1 halo
    R* Wo = SL + SM::slopes;                 // W_old on the tile + 2 halo
    uint8_t* th = (uint8_t*)(Wo + SM::wold);
    __shared__ CellMap<D, P, TX, TY, TZ, 3> map;
    map.fill(G, o, 3);
    __syncthreads();
    // W_old = prim(U_cv), reflective images flipped
    for (int q = threadIdx.x; q < SM::n2; q += blockDim.x) {
        const int x = q % E2x + 1, y = (q / E2x) % E2y + 1, z = q / (E2x * E2y) + dz;
        const int cid = map.cell(x, y, z);
        if (cid < 0) continue;
        const bool fl[3] = {map.flip[x] != 0, map.flip[map.Lx + y] != 0, D == 3 && map.flip[map.Lx + map.Ly + z] != 0};
        const long long ge = cid / NPT;
        const int pt = cid % NPT;
        R u[V], w[V];
#pragma unroll
        for (int v = 0; v < V; v++) u[v] = A.ucv[(ge * V + v) * NPT + pt];
        primitives<D>(u, w, (R)G.gm);
#pragma unroll
        for (int d = 0; d < D; d++)
            if (fl[d]) w[1 + d] = -w[1 + d];
#pragma unroll
        for (int v = 0; v < V; v++) Wo[(size_t)q * V + v] = w[v];
    }
    theta_on_tile<D, P, TX, TY, TZ>(G, map, A.trouble, o, reinterpret_cast<uint8_t*>(SL), th, A.theta);
    __syncthreads();
    // slopes of the tile's cells and of the cells across its faces, where
    // one of the cell's faces blends
    for (int q = threadIdx.x; q < ns; q += blockDim.x) {
        int l[3];
        SM::coords(q, l);
        int a[3] = {o[0] + l[0], o[1] + l[1], o[2] + l[2]};
        if (!has_image<D, P>(G, a, 1)) continue;
        const bool ox = l[0] < 0 || l[0] == Bx, oy = l[1] < 0 || l[1] == By, oz = D == 3 && (l[2] < 0 || l[2] == Bz);
        const int t0 = (l[0] + 1) + E1x * ((l[1] + 1) + E1y * (l[2] + dz));
        int near = th[t0];
        if (!oy && !oz) near |= (l[0] >= 0 ? th[t0 - 1] : 0) | (l[0] < Bx ? th[t0 + 1] : 0);
        if (!ox && !oz) near |= (l[1] >= 0 ? th[t0 - E1x] : 0) | (l[1] < By ? th[t0 + E1x] : 0);
        if (D == 3 && !ox && !oy)
            near |= (l[2] >= 0 ? th[t0 - E1x * E1y] : 0) | (l[2] < Bz ? th[t0 + E1x * E1y] : 0);
        if (!near) continue;
        int fa[3] = {a[0] + 2, a[1] + 2, a[2] + 2};
        auto Wc = [&](int oi, int oj, int ok) -> const R* {
            return Wo + (size_t)((l[0] + 2 + oi) + E2x * ((l[1] + 2 + oj) + E2y * (l[2] + 2 * dz + ok))) * V;
        };
        R dW[D][V], dwt[V];
        muscl_slopes<D, R>(G, fa, Wc, dW, dwt);
#pragma unroll
        for (int d = 0; d < D; d++)
#pragma unroll
            for (int v = 0; v < V; v++) SL[(d * V + v) * ns + q] = dW[d][v];
#pragma unroll
        for (int v = 0; v < V; v++) SL[(D * V + v) * ns + q] = dwt[v];
    }
    __syncthreads();
    const R wdt = M.wt[A.t] * (R)(*A.dt);
    const long long E = G.E;
    const int nfaces[3] = {SM::NF0, SM::NF1, SM::NF2};
#pragma unroll
    for (int d = 0; d < D; d++) {
        const int ex = Bx + (d == 0), ey = By + (d == 1);
        const int Bd = d == 0 ? Bx : (d == 1 ? By : Bz);
        for (int q = threadIdx.x; q < nfaces[d]; q += blockDim.x) {
            const int a[3] = {q % ex, (q / ex) % ey, q / (ex * ey)};  // the low face of cell a
            const int sR = (a[0] + 1) + E1x * ((a[1] + 1) + E1y * (a[2] + dz));
            const int sL = sR - (d == 0 ? 1 : (d == 1 ? E1x : E1x * E1y));
            const R tR = (R)(th[sR] * 0.125), tL = (R)(th[sL] * 0.125);
            const R tf = smax(tR, tL);
            if (!(tf > 0)) continue;
            bool in = true;
#pragma unroll
            for (int e = 0; e < D; e++) in &= o[e] + a[e] < G.N[e] * n + (e == d);
            if (!in) continue;
            const int wR = (a[0] + 2) + E2x * ((a[1] + 2) + E2y * (a[2] + 2 * dz));
            const int wL = wR - (d == 0 ? 1 : (d == 1 ? E2x : E2x * E2y));
            const int cR = SM::slot(a[0], a[1], a[2]);
            const int cL = SM::slot(a[0] - (d == 0), a[1] - (d == 1), a[2] - (d == 2));
            const Width hR = G.fw[d][o[d] + a[d] + 2], hL = G.fw[d][o[d] + a[d] + 1];
            R whi[V], wlo[V];
#pragma unroll
            for (int v = 0; v < V; v++) {
                whi[v] = Wo[(size_t)wL * V + v] + SL[(d * V + v) * ns + cL] +
                         div_width(G, SL[(D * V + v) * ns + cL] * wdt, hL);
                wlo[v] = Wo[(size_t)wR * V + v] - SL[(d * V + v) * ns + cR] +
                         div_width(G, SL[(D * V + v) * ns + cR] * wdt, hR);
            }
            R uL[V], uR[V], fL[V];
            conservatives<D>(whi, uL, (R)G.gm);
            conservatives<D>(wlo, uR, (R)G.gm);
            riemann_hllc<D>(fL, uL, uR, d, (R)G.gm);
            // the copies of the face in the tile's elements: of the element
            // on its high side (flux point 0 at an interface) and, at an
            // interface, of the one on its low side
            const bool iface = a[d] % n == 0;
#pragma unroll
            for (int side = 0; side < 2; side++) {
                if (side == 0 ? a[d] == Bd || o[d] + a[d] >= G.N[d] * n : !iface || a[d] == 0) continue;
                int c[3] = {a[0], a[1], a[2]};
                c[d] -= side;
                const long long ge = ((long long)(oe[2] + c[2] / n) * G.N[1] + (oe[1] + c[1] / n)) * G.N[0] + oe[0] + c[0] / n;
                int p[3] = {c[0] % n, c[1] % n, c[2] % n};
                p[d] += side;
                R* F = A.ff[d] + ((long long)A.t * E + ge) * V * NFP + fp_index<n, nf>(d, p);
#pragma unroll
                for (int v = 0; v < V; v++) {
                    const R f = F[v * NFP];
                    F[v * NFP] = f + tf * (fL[v] - f);
                }
            }
        }
    }
}

// resident blocks the blend kernel's registers are sized for: what its shared
// memory admits (2D FP64 at p = 3: 31 KB; 3D FP64 at p = 5: 110 KB, two blocks)
template <typename R, int D>
constexpr int kBlendBlocksPerSM = sizeof(R) == 4 ? (D == 2 ? 4 : 3) : (D == 2 ? 3 : 2);

template <typename R, int D, int P, int TX, int TY, int TZ>
__global__ void __launch_bounds__(kThreads, kBlendBlocksPerSM<R, D>) fv_blend_kernel(DevGrid G, DevMatsT<R> M, BlendArgsT<R> A) {
    pdl_wait();
    if (gate_closed(G)) return;
    const int count = *A.list.count;
    for (int i = blockIdx.x; i < count; i += gridDim.x) {
        const int tile = A.list.tiles[i];
        fv_blend_kernel_body<R, D, P, TX, TY, TZ>(G, M, A, tile);
        __syncthreads();  // the next tile reuses the shared memory
        if (threadIdx.x == 0) A.list.mark[tile] = 0;
    }
}

// resident blocks the update kernel's registers are sized for (48 registers a
// thread in FP32, 64 in FP64: 16 bytes of spills at most where the inputs arrive
// as bulk copies). The 3D orders that gather them, p = 2 and 4, spill 212 to 260
// bytes there: in FP32 the spills cost more than the fifth block gains (24^3 p=4
// steps 5576 us at 5 blocks, 5384 us at 4), in FP64 less than the fourth (11454 us
// at 4, 11690 us at 3)
template <typename R, int D, int P>
constexpr int kUpdateBlocksPerSM = sizeof(R) == 8 || (D == 3 && P % 2 == 0) ? 4 : 5;

// elements of an update block: consecutive ones (no neighbour is read), as
// many as give every thread a sub-cell
template <int D, int P>
struct UpdateBlock {
    static constexpr int NPT = Shape<D, P>::NPT;
    static constexpr int NE = kThreads / NPT > 0 ? kThreads / NPT : 1;
};

template <typename R, int D, int P>
struct UpdateSmem {
    static constexpr int n = P + 1, V = D + 2;
    static constexpr int NPT = Shape<D, P>::NPT;
    static constexpr int NE = UpdateBlock<D, P>::NE;
    static constexpr int NFP = Shape<D, P>::NFP;
    // the block's inputs arrive as bulk copies (its elements are consecutive
    // in every array) where an element's blocks are whole 16-byte units
    static constexpr bool bulk = (V * NFP * sizeof(R)) % 16 == 0 && (V * NPT * sizeof(R)) % 16 == 0;
    static constexpr size_t faces = (size_t)D * NE * V * NFP;                  // face fluxes of one slice
    static constexpr size_t ucv = (size_t)NE * V * NPT;
    static constexpr size_t epi = 2 * ucv;                                     // U_cv and sweep scratch
    static constexpr size_t ind = (size_t)NE * NPT * 16 + NE * 8;               // indicator scratch (bytes)
    static constexpr size_t in0 = bulk ? (ucv + faces) * sizeof(R) : 0;         // slice t
    static constexpr size_t in1 = bulk ? faces * sizeof(R) : 0;                 // slice t + 1, else the epilogue's
    static constexpr size_t epi_bytes = (epi * sizeof(R) + 15) / 16 * 16;       // the indicator's pairs follow
    static constexpr size_t out = epi_bytes + ind;
    static constexpr size_t bytes = in0 + (in1 > out ? in1 : out);
};

// ---------------------------------------------------------------------------
// The corrected sub-cell update of slice t (src/transforms.cpp:483-543 with
// update=1) from the blended face fluxes, then either the next slice's
// candidate or, after the last slice, U_sp = cv_to_sp(U_cv), the RK
// combination, W_cv and the next dt. Blocks of consecutive elements: a
// sub-cell reads only its own element's state and face fluxes. Bounded by
// HBM: the inputs of a block (its U_cv, and the face fluxes of slices t and
// t + 1) are contiguous, so one thread fetches them as a handful of bulk
// copies instead of every thread waiting for its own 36 gathers: 256^2 p=3 FP64
// 105 -> 64 us a launch (58 us cold, 52 % of HBM), FP32 41 -> 37 us, KH 16^3 p=5
// FP64 156 -> 96 us.
// ---------------------------------------------------------------------------
template <typename R, int D, int P>
__device__ __forceinline__ void fv_update_kernel_body(const DevGrid& G, const DevMatsT<R>& M, const FallbackArgsT<R>& A, long long bidx) {
    using SM = UpdateSmem<R, D, P>;
    constexpr int n = P + 1, nf = P + 2, V = D + 2, NPT = SM::NPT, NFP = Shape<D, P>::NFP, NE = SM::NE;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    R* Uin = reinterpret_cast<R*>(smem_raw);                   // [NE][V][NPT] U_cv of slice t
    R* F0 = Uin + SM::ucv;                                      // [D][NE][V][NFP] face fluxes of slice t
    R* F1 = reinterpret_cast<R*>(smem_raw + SM::in0);           // ... of slice t + 1
    R* Ub = F1;                                                 // last slice: [NE][V][NPT] new U_cv
    R* Tmp = Ub + SM::ucv;
    __shared__ R Mcs[n * n], Mcv[n * n];  // cv_to_sp, sp_to_cv (lane-dependent rows)
    __shared__ uint64_t bar;
    if (bidx == 0 && threadIdx.x == 0) *A.blend_count = 0;
    const long long E = G.E, e0 = bidx * NE;
    const int ne = (int)(E - e0 < NE ? E - e0 : NE);  // elements of this block
    if constexpr (SM::bulk) {
        if (threadIdx.x == 0) {
            mbar_init(&bar, 1);
            mbar_fence_init();
            const uint32_t ub = (uint32_t)(ne * V * NPT * sizeof(R)), fb = (uint32_t)(ne * V * NFP * sizeof(R));
            mbar_expect_tx(&bar, ub + D * fb * (A.last ? 1 : 2));
            bulk_g2s(Uin, A.ucv_in + e0 * V * NPT, ub, &bar);
#pragma unroll
            for (int d = 0; d < D; d++) {
                const R* src = A.ff[d] + ((long long)A.t * E + e0) * V * NFP;
                bulk_g2s(F0 + d * NE * V * NFP, src, fb, &bar);
                if (!A.last) bulk_g2s(F1 + d * NE * V * NFP, src + E * V * NFP, fb, &bar);
            }
        }
    }
    if (A.last)
        for (int i = threadIdx.x; i < n * n; i += blockDim.x) {
            Mcs[i] = M.cv_to_sp[i];
            Mcv[i] = M.sp_to_cv[i];
        }
    const R dt = (R)(*A.dt);
    const R wdt = M.wt[A.t] * dt;
    if constexpr (SM::bulk) {
        __syncthreads();  // the barrier is initialised
        mbar_wait_bounded(&bar, 0, G.status);
    }
    for (int q = threadIdx.x; q < ne * NPT; q += blockDim.x) {
        const int el = q / NPT, pt = q % NPT;
        const long long ge = e0 + el;
        int c[3], eg[3];
        pt_coords<n>(pt, c);
        elem_pos(G, (int)ge, eg);
        Width hd[D];
        int fl_[D], fr_[D];
        const R* f0[D];
        const R* f1[D];
        const R* u0;
        if constexpr (SM::bulk) {
            u0 = Uin + el * V * NPT + pt;
#pragma unroll
            for (int d = 0; d < D; d++) {
                f0[d] = F0 + (d * NE + el) * V * NFP;
                f1[d] = F1 + (d * NE + el) * V * NFP;
            }
        } else {
            u0 = A.ucv_in + ge * V * NPT + pt;
            face_blocks<D, P, R>(G, A.ff, A.t, (int)ge, f0);
            face_blocks<D, P, R>(G, A.ff, A.last ? A.t : A.t + 1, (int)ge, f1);
        }
#pragma unroll
        for (int d = 0; d < D; d++) {
            hd[d] = G.fw[d][eg[d] * n + c[d] + 2];
            int cc[3] = {c[0], c[1], c[2]};
            fl_[d] = fp_index<n, nf>(d, cc);
            cc[d] = c[d] + 1;
            fr_[d] = fp_index<n, nf>(d, cc);
        }
        R un[V];
#pragma unroll
        for (int v = 0; v < V; v++) {
            R F = 0;
#pragma unroll
            for (int d = 0; d < D; d++) F += div_width(G, f0[d][v * NFP + fr_[d]] - f0[d][v * NFP + fl_[d]], hd[d]);
            if (G.grav && v != 0) {
                R s;
                if (v <= D) s = un[0] * (R)G.g[v - 1];
                else {
                    s = un[1] * (R)G.g[0] + un[2] * (R)G.g[1];
                    if (D == 3) s = s + un[3] * (R)G.g[2];
                }
                F -= s;
            }
            un[v] = u0[v * NPT] - wdt * F;
        }
        if (A.last) {
#pragma unroll
            for (int v = 0; v < V; v++) Ub[(el * V + v) * NPT + pt] = un[v];
        } else {
#pragma unroll
            for (int v = 0; v < V; v++) A.ucv_out[(ge * V + v) * NPT + pt] = un[v];
            // candidate of slice t+1 from the new U_cv
            R uc[V];
            fv_candidate<D, P, R>(G, f1, eg, pt, un, M.wt[A.t + 1] * dt, uc);
            A.rp_old_next[ge * NPT + pt] = rho_p_fp64<D>(un, G.gm);
            A.rp_new_next[ge * NPT + pt] = rho_p_fp64<D>(uc, G.gm);
        }
    }
    if (!A.last) return;
    __syncthreads();
    // U_sp = cv_to_sp(U_cv) (src/hydro_ader.hpp:570)
    double2* RPs = reinterpret_cast<double2*>(reinterpret_cast<unsigned char*>(Ub) + SM::epi_bytes);
    {
        R* bufs[2] = {Tmp, Ub};
        const R* src = Ub;
        for (int d = 0; d < D; d++) {
            R* dst = bufs[d % 2];
            sweep_smem<D, P, R>(src, dst, Mcs, d, ne * V * NPT);
            __syncthreads();
            src = dst;
        }
        R* Wsp = (R*)(src == Ub ? Tmp : Ub);
        for (int q = threadIdx.x; q < ne * NPT; q += blockDim.x) {
            const int el = q / NPT, pt = q % NPT;
            const long long ge = e0 + el;
            R u[V];
#pragma unroll
            for (int v = 0; v < V; v++) {
                const long long gi = (ge * V + v) * NPT + pt;
                R val = src[(el * V + v) * NPT + pt];
                if (A.rk_a > 0) {
                    const R ra = (R)A.rk_a;
                    val = ra * A.u0[gi] + ((R)1.0 - ra) * val;
                }
                u[v] = val;
                A.u[gi] = val;
            }
            if (A.final_stage && A.feat) {
                // (rho, p) of the new state for the indicator's features
                double r, pr;
                feature_rho_p(u, 1, V, G.gm, &r, &pr);
                RPs[q] = make_double2(r, pr);
            }
            if (A.final_stage) {
                R w[V];
                primitives<D>(u, w, (R)G.gm);
#pragma unroll
                for (int v = 0; v < V; v++) Wsp[(el * V + v) * NPT + pt] = w[v];
            }
        }
        if (!A.final_stage) return;
        __syncthreads();
        if (A.feat) {
            // element means summed in point order, then the nodal features
            // rho / mean - 1 and p / mean - 1 as BF16 (the values of the
            // indicator's feature kernels)
            float2* Mn = reinterpret_cast<float2*>(RPs + NE * NPT);
            for (int el = threadIdx.x; el < ne; el += blockDim.x) {
                double sr = 0, sp = 0;
                for (int pt = 0; pt < NPT; pt++) {
                    sr = __dadd_rn(sr, RPs[el * NPT + pt].x);
                    sp = __dadd_rn(sp, RPs[el * NPT + pt].y);
                }
                const float2 mn = make_float2((float)__ddiv_rn(sr, (double)NPT), (float)__ddiv_rn(sp, (double)NPT));
                Mn[el] = mn;
                A.means[e0 + el] = mn;
            }
            __syncthreads();
            for (int q = threadIdx.x; q < ne * NPT; q += blockDim.x) {
                const int el = q / NPT, pt = q % NPT;
                const double2 v = RPs[q];
                const float2 mn = Mn[el];
                uint16_t* row = A.feat + (e0 + el) * A.n_in;
                row[pt] = bf16_bits(feature_ratio(v.x, mn.x));
                row[NPT + pt] = bf16_bits(feature_ratio(v.y, mn.y));
            }
        }
        R* bufs2[2] = {(R*)src, Wsp};
        const R* s2 = Wsp;
        for (int d = 0; d < D; d++) {
            R* dst = bufs2[d % 2];
            sweep_smem<D, P, R>(s2, dst, Mcv, d, ne * V * NPT);
            __syncthreads();
            s2 = dst;
        }
        double dtl = 1.7976931348623157e308;
        for (int q = threadIdx.x; q < ne * NPT; q += blockDim.x) {
            const int el = q / NPT, pt = q % NPT;
            const long long ge = e0 + el;
            R w[V];
#pragma unroll
            for (int v = 0; v < V; v++) w[v] = s2[(el * V + v) * NPT + pt];
            if (A.wcv)
#pragma unroll
                for (int v = 0; v < V; v++) A.wcv[(ge * V + v) * NPT + pt] = w[v];
            dtl = smin(dtl, point_dt<D>(G, w, n));
        }
        block_min_dt(dtl, A.dtmin);
    }
}

template <typename R, int D, int P>
__global__ void __launch_bounds__(kThreads, kUpdateBlocksPerSM<R, D, P>) fv_update_kernel(DevGrid G, DevMatsT<R> M, FallbackArgsT<R> A) {
    pdl_wait();
    if (gate_closed(G)) return;
    fv_update_kernel_body<R, D, P>(G, M, A, blockIdx.x);
}

}  // namespace spdk
