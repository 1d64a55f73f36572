// Fused Picard pass of 2D runs: one thread per solution-point line.
//
// Of the slices of U_ader (PicardArgsT): the fluxes at the flux points, LLF at
// the interfaces, then the predictor's next slices, the corrected state or the
// FV face fluxes, organised by lines:
//
// * Phase A (fluxes at the flux points of one slice). A thread takes one x or
//   y line of an element, all variables: the line's low interface (its own
//   trace, and the neighbour's from the neighbour's line) and its interior
//   flux points. The interpolation coefficients are compile-time offsets of
//   the kernel parameters, and a line is read twice instead of once per flux
//   point. The interfaces on the tile's high edges, which no line of the tile
//   owns, go to one more warp or two, so that no thread solves two.
// * Phase B (divergence at the solution points). A thread owns one row of
//   points of V / H variables of one element for the whole pass: the x
//   fluxes of the row and all y fluxes of the element are read as vectors,
//   the x coefficients are constant bank operands. Each point's sum keeps
//   the reference's order (flux points outer, directions inner:
//   src/transforms.cpp:296-303), so the FP64 plain form is unchanged bit for
//   bit; the precision form scales the sum once.
// * Rows are contiguous in memory, so the step-start state is read and the
//   slices are written straight from registers (16-byte vectors where a row
//   is whole vectors).
// * Tiles at the high edges may hang over the domain: their outside elements
//   are staged as periodic images (or not at all), take part in nothing
//   that is stored, and any element counts run on the same tiles.
//
// What bounds it: instruction issue (the point-per-thread pass before it read
// every line nf - 2 + 2 times through shared memory with its coefficients,
// and ran 2.2 of 4 issue slots).
#pragma once
#include <type_traits>

namespace spdk {

// 16-byte vector of R
template <typename R> struct Vec16;
template <> struct Vec16<float> { using T = float4; };
template <> struct Vec16<double> { using T = double2; };

// the widest vector (in values) that divides a row of n values: 16 or 8 bytes, or single values
template <typename R, int n>
constexpr int kRowVec = sizeof(R) == 4 ? (n % 4 == 0 ? 4 : (n % 2 == 0 ? 2 : 1)) : (n % 2 == 0 ? 2 : 1);

// n consecutive values between memory and registers, W at a time
template <typename R, int n, int W = kRowVec<R, n>>
__device__ __forceinline__ void row_load(const R* p, R* out) {
    if constexpr (W == 1) {
#pragma unroll
        for (int i = 0; i < n; i++) out[i] = p[i];
    } else {
        using VT = typename std::conditional<W * sizeof(R) == 16, typename Vec16<R>::T, float2>::type;
#pragma unroll
        for (int c = 0; c < n / W; c++) {
            __align__(16) R t[W];
            *reinterpret_cast<VT*>(t) = reinterpret_cast<const VT*>(p)[c];
#pragma unroll
            for (int w = 0; w < W; w++) out[c * W + w] = t[w];
        }
    }
}
template <typename R, int n, int W = kRowVec<R, n>>
__device__ __forceinline__ void row_store(R* p, const R* in) {
    if constexpr (W == 1) {
#pragma unroll
        for (int i = 0; i < n; i++) p[i] = in[i];
    } else {
        using VT = typename std::conditional<W * sizeof(R) == 16, typename Vec16<R>::T, float2>::type;
#pragma unroll
        for (int c = 0; c < n / W; c++) {
            __align__(16) R t[W];
#pragma unroll
            for (int w = 0; w < W; w++) t[w] = in[c * W + w];
            reinterpret_cast<VT*>(p)[c] = *reinterpret_cast<const VT*>(t);
        }
    }
}

// element stride of a flux-point array: V * NFP plus the pad (whole 16-byte
// units) that leaves the fewest bank conflicts when a warp's lanes run over
// the n lines of an element, then over elements
template <typename R, int n>
constexpr int flux_stride() {
    constexpr int nf = n + 1, V = 4, W = (int)sizeof(R) / 4, lanes = 32 / W;
    constexpr int base = V * n * nf;
    int best = 0, best_c = 1 << 30;
    for (int pad = 0; pad < 32 / W; pad += 4 / W) {
        int cnt[32] = {};
        for (int l = 0; l < lanes; l++) cnt[(((l % n) * nf + (l / n) * (base + pad)) * W) % 32]++;
        int c = 0;
        for (int b = 0; b < 32; b++) c = cnt[b] > c ? cnt[b] : c;
        c = c * 64 + pad;
        if (c < best_c) { best_c = c; best = pad; }
    }
    return base + best;
}

// Thread organisation and shared memory of the 2D pass on TX x TY elements.
// Phase A: the x lines, then the y lines (each padded to whole warps, so that
// a warp runs one direction), then the interfaces on the tile's high edges.
// Phase B: rows of points x H groups of variables.
// A thread has registers for either the predictor's divergences of every slice
// or the flux evaluation at the occupancy that hides its latency, so the
// predictor keeps the divergences in shared memory (one private column per
// thread) and forms the sums over slices once, at the end: 4 nt accesses a
// point. (Summing as the slices pass rewrites every sum in every slice, 2 nt^2
// accesses, which outweigh the FP64 arithmetic from p = 4 on: 128^2 steps without
// the fallback, p=5 FP64 1744 -> 1498 us, p=5 FP32 678 -> 550 us, p=7 FP32 2052 ->
// 1615 us, 64^2 p=4 FP64 298 -> 248 us.) A pass has one staging and one flux-point
// buffer: the next slice's copy starts when phase A is over and runs under
// phase B, and the shared memory saved is more resident blocks.
template <typename R, int P, int TX, int TY, int MODE>
struct Line2 {
    static constexpr int n = P + 1, nf = P + 2, V = 4, NPT = n * n, NFP = n * nf, NE = TX * TY;
    static constexpr int NS = Tile<2, TX, TY, 1>::NS;
    static constexpr int warps(int items) { return (items + 31) / 32 * 32; }
    static constexpr int H = P <= 3 ? 2 : 4;
    static constexpr int VB = V / H;                           // variables of a phase-B thread
    static constexpr int LINES = NE * n;                       // lines of one direction
    static constexpr int LW = warps(LINES);
    static constexpr int EDGE0 = TY * n, EDGE1 = TX * n;       // interfaces on the high x / y edge
    static constexpr int ROWS = NE * n * H;                    // phase-B threads
    static constexpr int A = 2 * LW + warps(EDGE0 + EDGE1);
    static constexpr int threads = A > warps(ROWS) ? A : warps(ROWS);
    static constexpr bool shared_sums = MODE == kPredict;
    static constexpr int SS = PicardPad<2, P, R>::SS;          // staged element
    static constexpr int FE = flux_stride<R, n>();             // flux points of an element, one direction
    static constexpr size_t stage = (size_t)NS * SS;
    static constexpr size_t fx = (size_t)2 * NE * FE;
    static constexpr size_t sums = shared_sums ? (size_t)VB * n * n * ROWS : 0;
    static constexpr size_t grav = MODE == kPredict ? (size_t)n * 3 * NE * NPT : 0;  // predictor slices of rho, m (gravity)
    static constexpr size_t epi = 2 * (size_t)NE * V * NPT;         // W_sp / U_sp and sweep scratch
    static constexpr size_t m0 = stage + fx > grav ? stage + fx : grav;
    static constexpr size_t m1 = m0 > epi ? m0 : epi;
    static constexpr size_t bytes = (m1 + sums) * sizeof(R);
};

// tile of the 2D pass: 4 x 4 elements up to p = 3 and 4 x 2 above (160
// threads at p = 2, 3 and 4, 192 at p = 5)
template <int P> constexpr int kLineTX = 4;
template <int P> constexpr int kLineTY = P <= 3 ? 4 : 2;

// resident blocks per SM the 2D pass's registers are sized for
// (threads x blocks leave 64 registers a thread at p = 3 in FP32 and 96 to 128
// in FP64, where the inviscid predictor spills 24 bytes at most and the corrector
// 52 to 204; FP64 flux pass at p = 3: 347 us at 3 blocks, 304 us at 4; FP32 with
// double buffers at 5 blocks 138 us, single at 5 and 6 134 and 125 us; the FP64
// predictor's shared memory admits one block above p = 5: 128^2 p=7 steps 7100
// us at the registers of two, 5830 us at those of one)
template <typename R, int P, int MODE>
constexpr int kLineBlocksPerSM =
    sizeof(R) == 4 ? (P == 1 ? 8 : P <= 3 ? 6 : P == 4 ? 5 : P == 5 ? 4 : 2)
                   : (P == 1 ? 5 : P <= 4 ? (MODE == kPredict ? 3 : 4) : P == 5 ? (MODE == kPredict ? 2 : 3)
                                                                               : (MODE == kPredict ? 1 : 2));
// (viscous passes carry the interface's viscous fluxes too)
template <typename R, int P, int MODE>
constexpr int kLineBlocksPerSMVisc =
    sizeof(R) == 4 ? (P == 1 ? 6 : P <= 3 ? 4 : P == 4 ? 4 : P == 5 ? 3 : 2)
                   : (P == 1 ? 4 : P <= 4 ? (MODE == kPredict ? 2 : 3) : P == 5 ? 2 : 1);

// The values of one line of one variable's point block: x lines are
// contiguous, y lines strided by n.
//
// The direction of the code below is a value: a compile-time one in the passes
// of several slices (x lines as vectors, no selects), or one that differs
// between warps (RT), which halves the code a pass fetches: a single-slice
// SSP-RK stage runs it once, from a cold instruction cache (64^2 p=2 FP64 RK3
// steps 41 -> 39 us, 128^2 p=6 304 -> 276 us; the predictor is up to 1.3 times
// slower so, its slices find the code cached).
template <bool RT, typename R, int n>
__device__ __forceinline__ void load_line(int d, const R* src, int tp, R (&u)[n]) {
    if (!RT && d == 0) row_load<R, n>(src + n * tp, u);
    else {
        const R* p = src + (d == 0 ? n * tp : tp);
        const int st = d == 0 ? 1 : n;
#pragma unroll
        for (int l = 0; l < n; l++) u[l] = p[l * st];
    }
}
template <typename R>
__device__ __forceinline__ R along2(const R* w, int d) { return d == 0 ? w[0] : w[1]; }

// euler_flux and riemann_llf of that direction, and the mirrored state
template <typename R>
__device__ __forceinline__ void euler_flux2(const R* u, const R* w, R* f, int d) {
    const R vn = along2(w + 1, d);
    f[0] = u[0] * vn;
#pragma unroll
    for (int v = 1; v <= 2; v++) f[v] = (v == 1 + d) ? (u[v] * vn + w[3]) : (u[v] * vn);
    f[3] = (u[3] + w[3]) * vn;
}
template <typename R>
__device__ __forceinline__ void riemann_llf2(R* F, const R* uL, const R* uR, int d, R gm) {
    R wL[4], wR[4], fL[4], fR[4];
    primitives<2>(uL, wL, gm);
    primitives<2>(uR, wR, gm);
    euler_flux2(uL, wL, fL, d);
    euler_flux2(uR, wR, fR, d);
    R cL = sound_speed(wL[0], wL[3], gm) + fabs(along2(wL + 1, d));
    R cR = sound_speed(wR[0], wR[3], gm) + fabs(along2(wR + 1, d));
    R cmax = smax(cL, cR);
#pragma unroll
    for (int v = 0; v < 4; v++) F[v] = R(0.5) * (fR[v] + fL[v]) - R(0.5) * cmax * (uR[v] - uL[v]);
}
template <typename R>
__device__ __forceinline__ void ghost2(const DevGrid& G, const R* in, R* out, int d) {
    const bool flip = G.bc[d] == kReflective;
#pragma unroll
    for (int v = 0; v < 4; v++) out[v] = (flip && v == 1 + d) ? -in[v] : in[v];
}

// the state at a line's end: E = 0 low, 1 high
template <bool RT, int P, int END, typename R>
__device__ __forceinline__ void trace2(const DevMatsT<R>& M, int d, const R* src, int tp, R (&t)[4]) {
    constexpr int n = P + 1, NPT = n * n, o = END ? (P + 1) * n : 0;
#pragma unroll
    for (int v = 0; v < 4; v++) {
        R ul[n];
        load_line<RT>(d, src + v * NPT, tp, ul);
        R a = 0;
#pragma unroll
        for (int l = 0; l < n; l++) a += ul[l] * M.sp_to_fp[o + l];
        t[v] = a;
    }
}

// interface flux between the states of the two sides: the ghost image at a
// non-periodic domain edge (src/boundary.cpp:48-113), LLF, and in viscous
// runs the interface sum of the sides' viscous fluxes (src/hydro.cpp:420-455)
template <int P, bool VISC, typename R>
__device__ __forceinline__ void interface2(const DevGrid& G, int d, R (&uL)[4], R (&uR)[4], bool ghostL, bool ghostR,
                                           R (&F)[4], const R* vg, int eL, int eR, int vt, int tp) {
    constexpr int V = 4, NTP = P + 1;
    if (ghostL) ghost2(G, uR, uL, d);
    if (ghostR) ghost2(G, uL, uR, d);
    riemann_llf2(F, uL, uR, d, (R)G.gm);
    if constexpr (VISC) {
        R gL[V], gR[V];
        if (!ghostL) {
            const R* g = vg + ((((long long)vt * G.E + eL) * 2 + 1) * V) * NTP + tp;
#pragma unroll
            for (int v = 0; v < V; v++) gL[v] = g[v * NTP];
        }
        if (!ghostR) {
            const R* g = vg + ((((long long)vt * G.E + eR) * 2 + 0) * V) * NTP + tp;
#pragma unroll
            for (int v = 0; v < V; v++) gR[v] = g[v * NTP];
        }
        if (ghostL) ghost2(G, gR, gL, d);
        if (ghostR) ghost2(G, gL, gR, d);
#pragma unroll
        for (int v = 0; v < V; v++) F[v] += wind_mix(gR[v], gL[v], R(-0.5));
    }
}

template <typename R, int P, int TX, int TY, int MODE, bool VISC, bool RT = false>
__device__ __forceinline__ void picard2d_body(const DevGrid& G, const DevMatsT<R>& M, const PicardArgsT<R>& A,
                                              long long bidx) {
    constexpr int D = 2;
    using S = Shape<2, P>;
    using TL = Tile<2, TX, TY, 1>;
    using LN = Line2<R, P, TX, TY, MODE>;
    constexpr int n = S::n, nf = S::nf, V = S::V, NPT = S::NPT, NFP = S::NFP;
    constexpr int NE = TL::NE, NS = TL::NS, NTH = LN::threads;
    constexpr int NT = MODE == kFlux ? 1 : (P + 1);
    constexpr int ND = MODE == kPredict ? NT : 1;  // divergence values kept per point
    constexpr int SS = LN::SS, FE = LN::FE, VB = LN::VB;
    constexpr int Q = 16 / (int)sizeof(R);
    using VT = typename Vec16<R>::T;
    static_assert((V * NPT * sizeof(R)) % 16 == 0, "2D element chunks are whole 16-byte units");
    static_assert((V * NFP * sizeof(R)) % 16 == 0 && FE % Q == 0, "flux blocks are whole 16-byte units");

    extern __shared__ __align__(128) unsigned char smem_raw[];
    R* smem = reinterpret_cast<R*>(smem_raw);
    R* Sbuf = smem;                       // [NS][SS]
    R* FX = Sbuf + LN::stage;             // [2][NE][FE]
    __shared__ int sl_elem[NS];           // staged element (a periodic image outside the domain), -1: none
    __shared__ int el_own[NE];            // element of the tile, -1 outside the domain
    __shared__ uint64_t bar;

    const int tid = threadIdx.x;
    int o[2];
    {
        const int tx = (G.N[0] + TX - 1) / TX;
        o[0] = ((int)bidx % tx) * TX;
        o[1] = ((int)bidx / tx) * TY;
    }
    for (int s = tid; s < NS; s += NTH) {
        int l[3];
        TL::coords(s, l);
        int g[2];
        bool none = false;
#pragma unroll
        for (int d = 0; d < 2; d++) {
            g[d] = o[d] + l[d];
            if (g[d] < 0 || g[d] >= G.N[d]) {
                none |= G.bc[d] != kPeriodic;
                g[d] = (g[d] + G.N[d]) % G.N[d];
            }
        }
        sl_elem[s] = none ? -1 : g[1] * G.N[0] + g[0];
        if (s < NE) {
            const int gx = o[0] + l[0], gy = o[1] + l[1];
            el_own[s] = gx < G.N[0] && gy < G.N[1] ? gy * G.N[0] + gx : -1;
        }
    }
    if (tid == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
    }
    const R dt = (R)(*A.dt);
    const int nt = MODE == kPredict ? P + 1 : G.nt;
    const long long E = G.E;

    // phase B: row br of variables bv .. bv + VB - 1 of element bel
    const int bh = tid / (NE * n), bel = (tid / n) % NE, br = tid % n, bv = bh * VB;
    const bool brow = tid < LN::ROWS;
    // kPredict: dudt of every slice (of one where all are equal), replaced by
    // the du of every slice at the end; kCorrect: du
    R dreg[VB][n][LN::shared_sums ? 1 : ND];
    R* sums = smem + LN::m1 + tid;
    auto acc = [&](int k, int i, int tt) -> R& {
        if constexpr (LN::shared_sums) return sums[((k * n + i) * ND + tt) * LN::ROWS];
        else return dreg[k][i][tt];
    };
    // du of slice tt += dudt of slice ll, invader(tt,l) w_l dt times (the
    // precision form takes invader(tt,l) w_l from one product and dt at the end)
    auto add_term = [&](R& du, R dudt, int tt, int ll) {
        if constexpr (sizeof(R) == 4) du += dudt * M.pred[tt * (P + 1) + ll];
        else du += dudt * M.invader[tt * (P + 1) + ll] * M.wt[ll] * dt;
    };
    R cy[nf];           // derivative coefficients of the row
    if (MODE != kFlux) {
        if (MODE == kCorrect) {
#pragma unroll
            for (int k = 0; k < VB; k++)
#pragma unroll
                for (int i = 0; i < n; i++) acc(k, i, 0) = 0;
        }
#pragma unroll
        for (int ll = 0; ll < nf; ll++) cy[ll] = M.dfp_to_sp[br * nf + ll];
        if constexpr (sizeof(R) == 4) {
            // the precision form scales the sum by 1/h_x alone
            const R ratio = (R)(G.h[0] / G.h[1]);
#pragma unroll
            for (int ll = 0; ll < nf; ll++) cy[ll] *= ratio;
        }
    }
    __syncthreads();
    // the last warp issues the bulk copies of slice t, one
    // staged element per lane
    auto issue = [&](int t) {
        if (tid < NTH - 32) return;
        const int lane = tid & 31;
        const R* src = A.in_slices > 1 ? A.ua_in + (long long)t * E * V * NPT : A.ua_in;
        int cnt = 0;
        for (int s = lane; s < NS; s += 32) cnt += sl_elem[s] >= 0;
        cnt = __reduce_add_sync(0xffffffffu, cnt);
        if (lane == 0) {
            fence_proxy_async_smem();
            mbar_expect_tx(&bar, (uint32_t)(cnt * V * NPT * sizeof(R)));
        }
        __syncwarp();
        for (int s = lane; s < NS; s += 32)
            if (sl_elem[s] >= 0)
                bulk_g2s(Sbuf + s * SS, src + (long long)sl_elem[s] * V * NPT, V * NPT * sizeof(R), &bar);
    };
    const bool multi = A.in_slices > 1;
    const int nt_eval = (MODE == kPredict && !multi) ? 1 : nt;
    issue(0);
    for (int t = 0; t < nt_eval; t++) {
        const R* Ss = Sbuf;
        if (t == 0 || multi) mbar_wait_bounded(&bar, t & 1, G.status);
        // ---- phase A: fluxes at every flux point of the slice ----
        bool bad = false;  // a flux value outside div_range
        const bool check = MODE != kFlux && sizeof(R) == 8 && !G.uniform_pow2;
        const int vt = multi ? t : 0;
        auto line = [&](auto dir, int q) {
            const int d = dir;
            // x lines: 8 elements, then their rows (16-byte loads of 8 lanes
            // fall into distinct banks); y lines: an element's columns first
            int el, r;
            if (NE % 8 == 0 && d == 0) { el = (q & 7) + 8 * (q / (8 * n)); r = (q >> 3) % n; }
            else { el = q / n; r = q % n; }
            const int lx = el % TX, ly = el / TX;
            const int sN = d == 0 ? TL::slot(lx - 1, ly, 0) : TL::slot(lx, ly - 1, 0);
            const int gface = o[d] + (d == 0 ? lx : ly);
            // beyond the domain's edge, or in a row outside it: nothing reads it
            if (gface > G.N[d] || o[1 - d] + (d == 0 ? ly : lx) >= G.N[1 - d]) return;
            const bool edge = G.bc[d] != kPeriodic;
            const bool ghostL = edge && gface == 0, ghostR = edge && gface == G.N[d];
            const R* src = Ss + el * SS;
            R* dst = FX + d * NE * FE + el * FE + (d == 0 ? r * nf : r);
            const int st = d == 0 ? 1 : n;  // stride between the line's flux points
            // the plain form reads the line again after the interface instead
            // of holding it across, for its registers
            constexpr bool hold = sizeof(R) == 4;
            R ul[V][n];
            auto load = [&]() {
#pragma unroll
                for (int v = 0; v < V; v++) load_line<RT>(d, src + v * NPT, r, ul[v]);
            };
            if (hold) load();
            {
                R uL[V], uR[V], F[V];
                if constexpr (hold) {
#pragma unroll
                    for (int v = 0; v < V; v++) {
                        R a = 0;
#pragma unroll
                        for (int l = 0; l < n; l++) a += ul[v][l] * M.sp_to_fp[l];
                        uR[v] = a;
                    }
                } else if (!ghostR) {
                    trace2<RT, P, 0>(M, d, src, r, uR);
                }
                if (!ghostL) trace2<RT, P, 1>(M, d, Ss + sN * SS, r, uL);
                interface2<P, VISC>(G, d, uL, uR, ghostL, ghostR, F, VISC ? along2(A.vg, d) : nullptr, VISC ? sl_elem[sN] : 0,
                                          VISC ? sl_elem[el] : 0, vt, r);
                R* dl = FX + d * NE * FE + sN * FE + (d == 0 ? r * nf : r) + (nf - 1) * st;
                const bool inside = d == 0 ? lx > 0 : ly > 0;
#pragma unroll
                for (int v = 0; v < V; v++) {
                    dst[v * NFP] = F[v];
                    if (inside) dl[v * NFP] = F[v];
                    if (check) bad |= !div_range(F[v]);
                }
            }
            if (gface == G.N[d]) return;  // the domain's high edge: only the interface is inside
            if (!hold) load();
#pragma unroll
            for (int ll = 1; ll < nf - 1; ll++) {
                R u[V], w[V], f[V];
#pragma unroll
                for (int v = 0; v < V; v++) {
                    R a = 0;
#pragma unroll
                    for (int l = 0; l < n; l++) a += ul[v][l] * M.sp_to_fp[ll * n + l];
                    u[v] = a;
                }
                primitives<2>(u, w, (R)G.gm);
                euler_flux2(u, w, f, d);
#pragma unroll
                for (int v = 0; v < V; v++) {
                    dst[v * NFP + ll * st] = f[v];
                    if (check) bad |= !div_range(f[v]);
                }
            }
        };
        auto edge = [&](auto dir, int q) {
            const int d = dir;
            const int r = q % n, k = q / n;
            const int el = d == 0 ? (TX - 1) + TX * k : k + TX * (TY - 1);
            const int sN = d == 0 ? TL::slot(TX, k, 0) : TL::slot(k, TY, 0);
            const int gface = o[d] + (d == 0 ? TX : TY);
            if (gface > G.N[d] || o[1 - d] + k >= G.N[1 - d]) return;
            const bool ghostR = G.bc[d] != kPeriodic && gface == G.N[d];
            R uL[V], uR[V], F[V];
            trace2<RT, P, 1>(M, d, Ss + el * SS, r, uL);
            if (!ghostR) trace2<RT, P, 0>(M, d, Ss + sN * SS, r, uR);
            interface2<P, VISC>(G, d, uL, uR, false, ghostR, F, VISC ? along2(A.vg, d) : nullptr, VISC ? sl_elem[el] : 0,
                                      VISC ? sl_elem[sN] : 0, vt, r);
            R* dst = FX + d * NE * FE + el * FE + (d == 0 ? r * nf + nf - 1 : r + n * (nf - 1));
#pragma unroll
            for (int v = 0; v < V; v++) {
                dst[v * NFP] = F[v];
                if (check) bad |= !div_range(F[v]);
            }
        };
        using D0 = std::integral_constant<int, 0>;
        using D1 = std::integral_constant<int, 1>;
        if constexpr (RT) {
            if (tid < 2 * LN::LW) {
                const int d = tid >= LN::LW, q = tid - d * LN::LW;
                if (LN::LW == LN::LINES || q < LN::LINES) line(d, q);
            } else if (tid < 2 * LN::LW + LN::EDGE0 + LN::EDGE1) {
                const int q = tid - 2 * LN::LW, d = q >= LN::EDGE0;
                edge(d, q - d * LN::EDGE0);
            }
        } else if (tid < LN::LW) {
            if (LN::LW == LN::LINES || tid < LN::LINES) line(D0{}, tid);
        } else if (tid < 2 * LN::LW) {
            if (LN::LW == LN::LINES || tid < LN::LW + LN::LINES) line(D1{}, tid - LN::LW);
        } else if (tid < 2 * LN::LW + LN::EDGE0) {
            edge(D0{}, tid - 2 * LN::LW);
        } else if (tid < 2 * LN::LW + LN::EDGE0 + LN::EDGE1) {
            edge(D1{}, tid - 2 * LN::LW - LN::EDGE0);
        }
        // spacings that are no power of two: the FP64 form divides every term
        // by h, from h's reciprocal unless some flux value of the tile is so
        // small or large that the quotient could under- or overflow
        bool slow = false;
        if (check) slow = __syncthreads_or(bad || !G.safe_div);
        else __syncthreads();
        // one staging buffer: the next slice's copy may start, unless phase B
        // still reads this slice's state
        const bool reads = MODE == kCorrect && G.grav;
        if (multi && t + 1 < nt && !reads) issue(t + 1);
        if constexpr (MODE != kFlux) {
            // ---- phase B: divergence of the thread's rows ----
            if (brow) {
#pragma unroll
                for (int k = 0; k < VB; k++) {
                    const int v = bv + k;
                    const R* Fx = FX + bel * FE + v * NFP + br * nf;
                    const R* Fy = FX + NE * FE + bel * FE + v * NFP;
                    R dd[n];
                    if constexpr (sizeof(R) == 4) {
#pragma unroll
                        for (int i = 0; i < n; i++) dd[i] = 0;
#pragma unroll
                        for (int ll = 0; ll < nf; ll++) {
                            R fy[n];
                            row_load<R, n>(Fy + n * ll, fy);
                            const R fx = Fx[ll];
#pragma unroll
                            for (int i = 0; i < n; i++) {
                                dd[i] += fx * M.dfp_to_sp[i * nf + ll];
                                dd[i] += fy[i] * cy[ll];
                            }
                        }
                        // (the predictor without gravity scales at the end)
                        if (MODE != kPredict || G.grav) {
                            const R ihx = (R)G.ih[0];
#pragma unroll
                            for (int i = 0; i < n; i++) dd[i] *= ihx;
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < n; i++) dd[i] = 0;
                        auto sum = [&](auto term) {
#pragma unroll
                            for (int ll = 0; ll < nf; ll++) {
                                R fy[n];
                                row_load<R, n>(Fy + n * ll, fy);
                                const R fx = Fx[ll];
#pragma unroll
                                for (int i = 0; i < n; i++) {
                                    dd[i] += term(fx * M.dfp_to_sp[i * nf + ll], 0);
                                    dd[i] += term(fy[i] * cy[ll], 1);
                                }
                            }
                        };
                        if (G.uniform_pow2) {
                            // every active h is the same power of two: the
                            // scaling of each term by 1/h is exact and
                            // commutes with the rounding of the sum
                            sum([](R x, int) { return x; });
#pragma unroll
                            for (int i = 0; i < n; i++) dd[i] *= G.ih[0];
                        } else if (!slow) {
                            sum([&](R x, int d) { return div_const(x, G.h[d], G.ih[d], G.ihl[d]); });
                        } else {
                            sum([&](R x, int d) { return x / G.h[d]; });
                        }
                    }
#pragma unroll
                    for (int i = 0; i < n; i++) {
                        if constexpr (MODE == kPredict) {
                            acc(k, i, t) = dd[i];
                        } else {
                            R dudt = dd[i];
                            if (G.grav && v != 0) {
                                const R* uv = Ss + bel * SS + br * n + i;
                                R s;
                                if (v <= D) s = uv[0] * (R)G.g[v - 1];
                                else s = uv[NPT] * (R)G.g[0] + uv[2 * NPT] * (R)G.g[1];
                                dudt -= s;
                            }
                            acc(k, i, 0) += dudt * M.wt[t] * dt;
                        }
                    }
                }
            }
        } else {
            // ---- FV face fluxes of slice t (src/transforms.cpp:378-481):
            // the averages across each set of transverse points replace the
            // points in place, then the element blocks are copied out ----
            constexpr int ITEMS = NE * V * nf;
            for (int q = tid; q < 2 * ITEMS; q += NTH) {
                const int d = q >= ITEMS, w = d ? q - ITEMS : q;
                const int ll = w % nf, k = w / nf;  // k = element x variable
                R* src = FX + d * NE * FE + (k / V) * FE + (k % V) * NFP + (d ? n * ll : ll);
                const int st = d ? 1 : nf;
                R in[n];
#pragma unroll
                for (int m = 0; m < n; m++) in[m] = src[st * m];
#pragma unroll
                for (int c = 0; c < n; c++) {
                    R f = 0;
#pragma unroll
                    for (int m = 0; m < n; m++) f += in[m] * M.sp_to_cv[c * n + m];
                    src[st * c] = f;
                }
            }
            __syncthreads();
            constexpr int CF = V * NFP / Q;  // vectors per element block
            for (int q = tid; q < 2 * NE * CF; q += NTH) {
                const int d = q >= NE * CF, w = d ? q - NE * CF : q;
                const int el = w / CF, c = w - el * CF;
                const int ge = el_own[el];
                if (ge >= 0)
                    reinterpret_cast<VT*>(A.ff[d] + ((long long)t * E + ge) * V * NFP)[c] =
                        reinterpret_cast<const VT*>(FX + d * NE * FE + el * FE)[c];
            }
        }
        __syncthreads();  // the next slice's phase A overwrites this slice's fluxes
        if (multi && t + 1 < nt && reads) issue(t + 1);
    }
    const int bge = brow ? el_own[bel] : -1;

    if constexpr (MODE == kPredict) {
        // ---- ADER predictor (src/transforms.cpp:309-323) ----
        // with gravity the source of a momentum (energy) slot uses the
        // updated density (momenta) of the same point and slice
        // (src/transforms.cpp:16-27 on U_ader being written): variables are
        // finished in three rounds that pass those on through shared memory
        R* O = smem;  // [slice][rho, m_x, m_y][element][point]
        const int rounds = G.grav ? 3 : 1;
        for (int round = 0; round < rounds; round++) {
            if (brow) {
#pragma unroll
                for (int k = 0; k < VB; k++) {
                    const int v = bv + k;
                    if (G.grav && (v == 0 ? 0 : (v <= D ? 1 : 2)) != round) continue;
                    R uo[n];
                    if (bge >= 0) row_load<R, n>(A.u + ((long long)bge * V + v) * NPT + br * n, uo);
                    else {
#pragma unroll
                        for (int i = 0; i < n; i++) uo[i] = 0;
                    }
                    if (G.grav && v != 0) {
                        // (from the last slice down: where all are equal, slice 0 holds dudt)
#pragma unroll
                        for (int tt = NT - 1; tt >= 0; tt--)
#pragma unroll
                            for (int i = 0; i < n; i++) {
                                const R* nw = O + ((tt * 3) * NE + bel) * NPT + br * n + i;
                                R s;
                                if (v <= D) s = nw[0] * (R)G.g[v - 1];
                                else s = nw[NE * NPT] * (R)G.g[0] + nw[2 * NE * NPT] * (R)G.g[1];
                                acc(k, i, tt) = acc(k, i, multi ? tt : 0) - s;
                            }
                    }
                    // the sums over slices, in place
#pragma unroll (n > 4 ? 1 : n)
                    for (int i = 0; i < n; i++) {
                        R q[NT];
#pragma unroll
                        for (int ll = 0; ll < NT; ll++) q[ll] = acc(k, i, multi || (G.grav && v != 0) ? ll : 0);
#pragma unroll
                        for (int tt = 0; tt < NT; tt++) {
                            R du = 0;
#pragma unroll
                            for (int ll = 0; ll < NT; ll++) add_term(du, q[ll], tt, ll);
                            acc(k, i, tt) = du;
                        }
                    }
#pragma unroll
                    for (int tt = 0; tt < NT; tt++) {
                        R val[n];
#pragma unroll
                        for (int i = 0; i < n; i++) {
                            R du = acc(k, i, tt);
                            if constexpr (sizeof(R) == 4) du *= G.grav ? dt : dt * (R)G.ih[0];
                            val[i] = uo[i] - du;
                        }
                        if (bge >= 0) row_store<R, n>(A.ua_out + (((long long)tt * E + bge) * V + v) * NPT + br * n, val);
                        if (G.grav && v <= D) {
#pragma unroll
                            for (int i = 0; i < n; i++) O[((tt * 3 + v) * NE + bel) * NPT + br * n + i] = val[i];
                        }
                    }
                }
            }
            if (G.grav) __syncthreads();
        }
    } else if constexpr (MODE == kCorrect) {
        // ---- corrector / RK stage (src/transforms.cpp:327-374, 252-261) ----
        R* Wsp = smem;                     // [NE][V][NPT]
        R* Tmp = smem + NE * V * NPT;
        if (brow) {
#pragma unroll
            for (int k = 0; k < VB; k++) {
                const int v = bv + k;
                const long long g = ((long long)bge * V + v) * NPT + br * n;
                R val[n];
                if (bge >= 0) {
                    row_load<R, n>(A.u + g, val);
#pragma unroll
                    for (int i = 0; i < n; i++) val[i] -= acc(k, i, 0);
                    if (A.rk_a > 0) {
                        const R ra = (R)A.rk_a;
                        R u0[n];
                        row_load<R, n>(A.u0 + g, u0);
#pragma unroll
                        for (int i = 0; i < n; i++) val[i] = ra * u0[i] + ((R)1.0 - ra) * val[i];
                    }
                    row_store<R, n>(A.u_out + g, val);
                } else {
#pragma unroll
                    for (int i = 0; i < n; i++) val[i] = 1;
                }
#pragma unroll
                for (int i = 0; i < n; i++) Wsp[(bel * V + v) * NPT + br * n + i] = val[i];
            }
        }
        if (A.final_stage) {
            __shared__ R Mcv[S::n * S::n];
            for (int i = tid; i < S::n * S::n; i += NTH) Mcv[i] = M.sp_to_cv[i];
            __syncthreads();
            for (int q = tid; q < NE * NPT; q += NTH) {
                const int el = q / NPT, pt = q % NPT;
                R un[V], w[V];
#pragma unroll
                for (int v = 0; v < V; v++) un[v] = Wsp[(el * V + v) * NPT + pt];
                primitives<D>(un, w, (R)G.gm);
#pragma unroll
                for (int v = 0; v < V; v++) Wsp[(el * V + v) * NPT + pt] = w[v];
            }
            __syncthreads();
            // W_cv = sp_to_cv(W_sp): x, y sweeps (src/transforms.cpp:99-117)
            sweep_smem<D, P, R>(Wsp, Tmp, Mcv, 0, NE * V * NPT);
            __syncthreads();
            sweep_smem<D, P, R>(Tmp, Wsp, Mcv, 1, NE * V * NPT);
            __syncthreads();
            double dtl = 1.7976931348623157e308;
            for (int q = tid; q < NE * NPT; q += NTH) {
                const int el = q / NPT, pt = q % NPT;
                const long long ge = el_own[el];
                if (ge < 0) continue;
                R w[V];
#pragma unroll
                for (int v = 0; v < V; v++) w[v] = Wsp[(el * V + v) * NPT + pt];
                if (A.wcv)
#pragma unroll
                    for (int v = 0; v < V; v++) A.wcv[(ge * V + v) * NPT + pt] = w[v];
                dtl = smin(dtl, point_dt<D>(G, w, n));
            }
            block_min_dt(dtl, A.dtmin);
        }
    } else {
        if (A.labels)
            for (int el = tid; el < NE; el += NTH)
                if (el_own[el] >= 0) A.labels[el_own[el]] = 0;
        // ---- U_cv = sp_to_cv(U) and the slice-0 FV candidate: a thread
        // averages its rows in x, then, from the rows' x averages, in y ----
        R* Tx = smem;                      // [NE][V][NPT]
        R* src = smem + NE * V * NPT;
        if (brow && bge >= 0) {
#pragma unroll
            for (int k = 0; k < VB; k++) {
                R u[n], a[n];
                row_load<R, n>(A.u + ((long long)bge * V + bv + k) * NPT + br * n, u);
#pragma unroll
                for (int c = 0; c < n; c++) {
                    a[c] = 0;
#pragma unroll
                    for (int l = 0; l < n; l++) a[c] += u[l] * M.sp_to_cv[c * n + l];
                }
                row_store<R, n>(Tx + (bel * V + bv + k) * NPT + br * n, a);
            }
        }
        __syncthreads();
        if (brow && bge >= 0) {
            R m[n];
#pragma unroll
            for (int l = 0; l < n; l++) m[l] = M.sp_to_cv[br * n + l];
#pragma unroll
            for (int k = 0; k < VB; k++) {
                R a[n];
#pragma unroll
                for (int c = 0; c < n; c++) a[c] = 0;
#pragma unroll
                for (int l = 0; l < n; l++) {
                    R u[n];
                    row_load<R, n>(Tx + (bel * V + bv + k) * NPT + l * n, u);
#pragma unroll
                    for (int c = 0; c < n; c++) a[c] += u[c] * m[l];
                }
                row_store<R, n>(src + (bel * V + bv + k) * NPT + br * n, a);
                row_store<R, n>(A.ucv + ((long long)bge * V + bv + k) * NPT + br * n, a);
            }
        }
        __syncthreads();
        for (int q = tid; q < NE * NPT; q += NTH) {
            const int el = q / NPT, pt = q % NPT;
            const long long ge = el_own[el];
            if (ge < 0) continue;
            R uo[V], un[V];
#pragma unroll
            for (int v = 0; v < V; v++) uo[v] = src[(el * V + v) * NPT + pt];
            int eg[3];
            const R* fb[D];
            elem_pos(G, (int)ge, eg);
            face_blocks<D, P, R>(G, A.ff, 0, (int)ge, fb);
            fv_candidate<D, P, R>(G, fb, eg, pt, uo, M.wt[0] * dt, un);
            A.rp_old[ge * NPT + pt] = rho_p_fp64<D>(uo, G.gm);
            A.rp_new[ge * NPT + pt] = rho_p_fp64<D>(un, G.gm);
        }
    }
}

}  // namespace spdk
