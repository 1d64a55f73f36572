// Fused Picard pass of 3D runs: one thread per solution-point line, blocks of
// consecutive elements.
//
// Same inputs, outputs and FP64 arithmetic as the 2D pass
// (spdk_picard2d.cuh), with these differences:
//
// * A block takes EB consecutive elements and stages only their own slices;
//   both faces of every element are solved by its block (a tile of several
//   elements with staged neighbours held 7 elements' slices for one, which
//   left one block of 8 warps on an SM at p = 5 in FP64). The neighbours'
//   lines are read from global memory (L2) by the threads that need them.
// * Phase A has two kinds of threads, about equally long: the interior flux
//   points of a line, and both interfaces at its ends. The direction is a
//   runtime value (strides and selects), so one copy of the code serves
//   all three and a warp may mix them.
// * Element counts do not matter to the blocks.
//
// The predictor keeps its sums in shared memory, as in 2D. Measured per launch
// (predictor, average of a step's passes / flux pass): KH 16^3 p=5 FP64 925 /
// 1578 -> 737 / 1242 us, 32^3 p=3 FP32 591 / 1205 -> 410 / 854 us.
#pragma once

namespace spdk {

template <typename R, int P, int MODE>
struct Line3 {
    static constexpr int n = P + 1, nf = P + 2, V = 5, L = n * n, NPT = n * n * n, NFP = L * nf;
    static constexpr int EB = P == 1 ? 8 : P == 2 ? 4 : P == 3 ? 2 : 1;  // elements of a block
    static constexpr int LINES = 3 * EB * L;                   // lines of all directions
    static constexpr int warps(int items) { return (items + 31) / 32 * 32; }
    static constexpr int LW = warps(LINES);
    static constexpr int ROWS = EB * L * V;                     // phase-B threads
    static constexpr int threads = 2 * LW > warps(ROWS) ? 2 * LW : warps(ROWS);
    // the EB slices as one bulk copy where an element is whole 16-byte units
    static constexpr bool bulk = (V * NPT * sizeof(R)) % 16 == 0;
    static constexpr size_t stage = ((size_t)EB * V * NPT + 3) / 4 * 4;
    static constexpr int FE = V * NFP;                          // flux points of an element, one direction
    static constexpr size_t fx = (size_t)3 * EB * FE;
    static constexpr size_t sums = MODE == kPredict ? (size_t)n * n * ROWS : 0;
    static constexpr size_t grav = MODE == kPredict ? (size_t)n * 4 * EB * NPT : 0;  // predictor slices of rho, m
    static constexpr size_t epi = 2 * (size_t)EB * V * NPT;
    static constexpr size_t m0 = stage + fx > grav ? stage + fx : grav;
    static constexpr size_t m1 = m0 > epi ? m0 : epi;
    static constexpr size_t bytes = (m1 + sums) * sizeof(R);
};

// resident blocks per SM the 3D pass's registers are sized for
template <typename R, int P, int MODE>
constexpr int kLine3BlocksPerSM = sizeof(R) == 8 ? (P <= 3 ? 3 : 2) : (P <= 3 ? 4 : 3);

// the component along d of (x, y, z) values
template <typename R>
__device__ __forceinline__ R along(const R* w, int d) { return d == 0 ? w[0] : (d == 1 ? w[1] : w[2]); }

// euler_flux, riemann_llf and the reflected state with a runtime direction
template <typename R>
__device__ __forceinline__ void euler_flux3(const R* u, const R* w, R* f, int n) {
    const R vn = along(w + 1, n);
    f[0] = u[0] * vn;
#pragma unroll
    for (int d = 1; d <= 3; d++) f[d] = (d == 1 + n) ? (u[d] * vn + w[4]) : (u[d] * vn);
    f[4] = (u[4] + w[4]) * vn;
}
template <typename R>
__device__ __forceinline__ void riemann_llf3(R* F, const R* uL, const R* uR, int n, R gm) {
    R wL[5], wR[5], fL[5], fR[5];
    primitives<3>(uL, wL, gm);
    primitives<3>(uR, wR, gm);
    euler_flux3(uL, wL, fL, n);
    euler_flux3(uR, wR, fR, n);
    R cL = sound_speed(wL[0], wL[4], gm) + fabs(along(wL + 1, n));
    R cR = sound_speed(wR[0], wR[4], gm) + fabs(along(wR + 1, n));
    R cmax = smax(cL, cR);
#pragma unroll
    for (int v = 0; v < 5; v++) F[v] = R(0.5) * (fR[v] + fL[v]) - R(0.5) * cmax * (uR[v] - uL[v]);
}
template <typename R>
__device__ __forceinline__ void ghost3(const DevGrid& G, const R* in, R* out, int d) {
    const bool flip = G.bc[d] == kReflective;
#pragma unroll
    for (int v = 0; v < 5; v++) out[v] = (flip && v == 1 + d) ? -in[v] : in[v];
}

// ANY: the corrector's u, u0 and u_out are a caller's buffers that start on no
// 16-byte boundary; their rows move value by value
template <typename R, int P, int MODE, bool VISC, bool ANY = false>
__device__ __forceinline__ void picard3d_body(const DevGrid& G, const DevMatsT<R>& M, const PicardArgsT<R>& A,
                                              long long bidx) {
    constexpr int D = 3;
    using LN = Line3<R, P, MODE>;
    constexpr int n = LN::n, nf = LN::nf, V = LN::V, L = LN::L, NPT = LN::NPT, NFP = LN::NFP, FE = LN::FE;
    constexpr int EB = LN::EB, NTH = LN::threads, NT = P + 1;
    constexpr int ND = MODE == kPredict ? NT : 1;
    constexpr int Q = 16 / (int)sizeof(R);
    using VT = typename Vec16<R>::T;

    extern __shared__ __align__(128) unsigned char smem_raw[];
    R* smem = reinterpret_cast<R*>(smem_raw);
    R* Ss = smem;                    // [EB][V][NPT]
    R* FX = smem + LN::stage;        // [3][EB][V][NFP]
    __shared__ uint64_t bar;

    const int tid = threadIdx.x;
    const long long E = G.E;
    const int e0 = (int)bidx * EB;
    const int ne = E - e0 < EB ? (int)(E - e0) : EB;
    if (tid == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
    }
    const R dt = (R)(*A.dt);
    const int nt = MODE == kPredict ? P + 1 : G.nt;

    // phase A: the line of this thread (interior points, or both interfaces)
    const int ia = tid < LN::LW ? tid : tid - LN::LW;
    const bool interior = tid < LN::LW;
    const int ld = ia / (EB * L), lel = (ia / L) % EB, lt = ia % L;  // direction, element, transverse point
    const bool has_line = ia < LN::LINES && tid < 2 * LN::LW && lel < ne;
    const int ta = lt % n, tb = lt / n;
    // the line's first point and step among solution points and flux points
    const int ps = ld == 0 ? 1 : (ld == 1 ? n : n * n);
    const int p0 = ld == 0 ? n * ta + n * n * tb : (ld == 1 ? ta + n * n * tb : ta + n * tb);
    const int f0 = ld == 0 ? nf * (ta + n * tb) : (ld == 1 ? ta + n * nf * tb : ta + n * tb);
    const int lg = e0 + (lel < ne ? lel : 0);
    // neighbours of the line's element across its low and high face, -1: none
    int nb[2];
    {
        int g[3];
        elem_pos(G, lg, g);
        const int gd = ld == 0 ? g[0] : (ld == 1 ? g[1] : g[2]);
        const int Nd = ld == 0 ? G.N[0] : (ld == 1 ? G.N[1] : G.N[2]);
        const int st = ld == 0 ? 1 : (ld == 1 ? G.N[0] : G.N[0] * G.N[1]);
        const bool per = G.bc[ld < 3 ? ld : 0] == kPeriodic;
        nb[0] = gd > 0 ? lg - st : (per ? lg + (Nd - 1) * st : -1);
        nb[1] = gd < Nd - 1 ? lg + st : (per ? lg - (Nd - 1) * st : -1);
    }

    // phase B: row br of variable bv of element bel
    const int bel = tid / (L * V), bv = (tid / L) % V, br = tid % L;
    const bool brow = tid < LN::ROWS && bel < ne;
    const int bj = br % n, bk = br / n;
    const long long bge = e0 + bel;
    R dreg[n];
    R* sums = smem + LN::m1 + tid;
    auto acc = [&](int i, int tt) -> R& {
        if constexpr (MODE == kPredict) return sums[(i * ND + tt) * LN::ROWS];
        else return dreg[i];
    };
    auto add_term = [&](R& du, R dudt, int tt, int ll) {
        if constexpr (sizeof(R) == 4) du += dudt * M.pred[tt * (P + 1) + ll];
        else du += dudt * M.invader[tt * (P + 1) + ll] * M.wt[ll] * dt;
    };
    R cy[nf], cz[nf];
    if (MODE != kFlux) {
        if (MODE == kCorrect) {
#pragma unroll
            for (int i = 0; i < n; i++) acc(i, 0) = 0;
        }
        R ry = 1, rz = 1;  // the precision form scales the sum by 1/h_x alone
        if constexpr (sizeof(R) == 4) {
            ry = (R)(G.h[0] / G.h[1]);
            rz = (R)(G.h[0] / G.h[2]);
        }
#pragma unroll
        for (int ll = 0; ll < nf; ll++) {
            cy[ll] = M.dfp_to_sp[bj * nf + ll];
            cz[ll] = M.dfp_to_sp[(bk < n ? bk : 0) * nf + ll];
            if constexpr (sizeof(R) == 4) {
                cy[ll] *= ry;
                cz[ll] *= rz;
            }
        }
    }
    __syncthreads();
    const bool multi = A.in_slices > 1;
    auto slice = [&](int t) { return multi ? A.ua_in + (long long)t * E * V * NPT : A.ua_in; };
    // the block's own slices: one bulk copy, or plain loads
    auto issue = [&](int t) {
        const R* src = slice(t) + (long long)e0 * V * NPT;
        if constexpr (LN::bulk) {
            if (tid == 0) {
                const uint32_t bytes = (uint32_t)(ne * V * NPT * sizeof(R));
                fence_proxy_async_smem();
                mbar_expect_tx(&bar, bytes);
                bulk_g2s(Ss, src, bytes, &bar);
            }
        } else {
            for (int q = tid; q < ne * V * NPT; q += NTH) Ss[q] = src[q];
        }
    };
    const int nt_eval = (MODE == kPredict && !multi) ? 1 : nt;
    const bool reads = MODE == kCorrect && G.grav;  // phase B reads the staged state
    issue(0);
    for (int t = 0; t < nt_eval; t++) {
        if (t == 0 || multi) {
            if constexpr (LN::bulk) mbar_wait_bounded(&bar, t & 1, G.status);
            else __syncthreads();
        }
        // ---- phase A ----
        bool bad = false;
        const bool check = MODE != kFlux && sizeof(R) == 8 && !G.uniform_pow2;
        if (has_line) {
            const R* src = Ss + lel * V * NPT + p0;
            R* dst = FX + ((ld * EB + lel) * V) * NFP + f0;
            if (interior) {
                R ul[V][n];
#pragma unroll
                for (int v = 0; v < V; v++)
#pragma unroll
                    for (int l = 0; l < n; l++) ul[v][l] = src[v * NPT + l * ps];
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
                    primitives<3>(u, w, (R)G.gm);
                    euler_flux3(u, w, f, ld);
#pragma unroll
                    for (int v = 0; v < V; v++) {
                        dst[v * NFP + ll * ps] = f[v];
                        if (check) bad |= !div_range(f[v]);
                    }
                }
            } else {
                const R* gs = slice(t);
#pragma unroll 1
                for (int side = 0; side < 2; side++) {
                    // own trace at the face, and the neighbour's from its line
                    const R* Mo = M.sp_to_fp + (side ? (nf - 1) * n : 0);
                    const R* Mn = M.sp_to_fp + (side ? 0 : (nf - 1) * n);
                    const int e = side ? nb[1] : nb[0];
                    R own[V], oth[V];
                    if (e >= 0) {
                        const R* o = gs + (long long)e * V * NPT + p0;
#pragma unroll
                        for (int v = 0; v < V; v++) {
                            R a = 0;
#pragma unroll
                            for (int l = 0; l < n; l++) a += o[v * NPT + l * ps] * Mn[l];
                            oth[v] = a;
                        }
                    }
#pragma unroll
                    for (int v = 0; v < V; v++) {
                        R a = 0;
#pragma unroll
                        for (int l = 0; l < n; l++) a += src[v * NPT + l * ps] * Mo[l];
                        own[v] = a;
                    }
                    if (e < 0) ghost3(G, own, oth, ld);
                    R uL[V], uR[V], F[V];
#pragma unroll
                    for (int v = 0; v < V; v++) {
                        uL[v] = side ? own[v] : oth[v];
                        uR[v] = side ? oth[v] : own[v];
                    }
                    riemann_llf3(F, uL, uR, ld, (R)G.gm);
                    if constexpr (VISC) {
                        // viscous interface flux (src/hydro.cpp:420-455), as in 2D
                        const R* vg = ld == 0 ? A.vg[0] : (ld == 1 ? A.vg[1] : A.vg[2]);
                        const int vt = multi ? t : 0;
                        auto side_flux = [&](int el, int s, R* g) {
                            const R* p = vg + ((((long long)vt * E + el) * 2 + s) * V) * L + lt;
#pragma unroll
                            for (int v = 0; v < V; v++) g[v] = p[v * L];
                        };
                        R go[V], gn[V];
                        side_flux(lg, side, go);
                        if (e >= 0) side_flux(e, 1 - side, gn);
                        else ghost3(G, go, gn, ld);
#pragma unroll
                        for (int v = 0; v < V; v++)
                            F[v] += side ? wind_mix(gn[v], go[v], R(-0.5)) : wind_mix(go[v], gn[v], R(-0.5));
                    }
#pragma unroll
                    for (int v = 0; v < V; v++) {
                        dst[v * NFP + (side ? (nf - 1) * ps : 0)] = F[v];
                        if (check) bad |= !div_range(F[v]);
                    }
                }
            }
        }
        bool slow = false;
        if (check) slow = __syncthreads_or(bad || !G.safe_div);
        else __syncthreads();
        if (multi && t + 1 < nt && !reads) issue(t + 1);
        if constexpr (MODE != kFlux) {
            // ---- phase B: divergence of the thread's row ----
            if (brow) {
                const R* Fx = FX + ((0 * EB + bel) * V + bv) * NFP + br * nf;
                const R* Fy = FX + ((1 * EB + bel) * V + bv) * NFP + n * nf * bk;
                const R* Fz = FX + ((2 * EB + bel) * V + bv) * NFP + n * bj;
                R dd[n];
#pragma unroll
                for (int i = 0; i < n; i++) dd[i] = 0;
                auto sum = [&](auto term) {
#pragma unroll
                    for (int ll = 0; ll < nf; ll++) {
                        R fy[n], fz[n];
                        row_load<R, n>(Fy + n * ll, fy);
                        row_load<R, n>(Fz + n * n * ll, fz);
                        const R fx = Fx[ll];
#pragma unroll
                        for (int i = 0; i < n; i++) {
                            dd[i] += term(fx * M.dfp_to_sp[i * nf + ll], 0);
                            dd[i] += term(fy[i] * cy[ll], 1);
                            dd[i] += term(fz[i] * cz[ll], 2);
                        }
                    }
                };
                if (sizeof(R) == 4) {
                    sum([](R x, int) { return x; });
                    if (MODE != kPredict || G.grav) {
#pragma unroll
                        for (int i = 0; i < n; i++) dd[i] *= (R)G.ih[0];
                    }
                } else if (G.uniform_pow2) {
                    // the scaling of each term by 1/h is exact and commutes
                    // with the rounding of the sum
                    sum([](R x, int) { return x; });
#pragma unroll
                    for (int i = 0; i < n; i++) dd[i] *= (R)G.ih[0];
                } else if (!slow) {
                    sum([&](R x, int d) { return (R)div_const(x, G.h[d], G.ih[d], G.ihl[d]); });
                } else {
                    sum([&](R x, int d) { return x / (R)G.h[d]; });
                }
#pragma unroll
                for (int i = 0; i < n; i++) {
                    if constexpr (MODE == kPredict) {
                        acc(i, t) = dd[i];
                    } else {
                        R dudt = dd[i];
                        if (G.grav && bv != 0) {
                            const R* uv = Ss + bel * V * NPT + br * n + i;
                            R s;
                            if (bv <= D) s = uv[0] * (R)G.g[bv - 1];
                            else s = uv[NPT] * (R)G.g[0] + uv[2 * NPT] * (R)G.g[1] + uv[3 * NPT] * (R)G.g[2];
                            dudt -= s;
                        }
                        acc(i, 0) += dudt * M.wt[t] * dt;
                    }
                }
            }
        } else {
            // ---- FV face fluxes of slice t (src/transforms.cpp:378-481): the
            // averages along the first, then the second transverse direction
            // (next(d), next(next(d))) replace the points in place ----
            constexpr int PER = V * nf * n, ITEMS = EB * PER;  // lines of one direction's points
#pragma unroll 1
            for (int pass = 1; pass <= 2; pass++) {
                for (int q = tid; q < 3 * ITEMS; q += NTH) {
                    const int d = q / ITEMS, el = (q / PER) % EB, k = q % PER;
                    const int v = k / (nf * n), id = (k / n) % nf, ir = k % n;
                    const int sd = pass == 1 ? (d == 2 ? 0 : d + 1) : (d == 0 ? 2 : d - 1);  // averaged along
                    const int rd = 3 - d - sd;                                             // the remaining one
                    auto stride = [&](int a) {
                        return a == 0 ? 1 : (a == 1 ? (d == 0 ? nf : n) : (d == 2 ? n * n : nf * n));
                    };
                    R* p = FX + ((d * EB + el) * V + v) * NFP + id * stride(d) + ir * stride(rd);
                    const int st = stride(sd);
                    R in[n];
#pragma unroll
                    for (int m = 0; m < n; m++) in[m] = p[st * m];
#pragma unroll
                    for (int c = 0; c < n; c++) {
                        R f = 0;
#pragma unroll
                        for (int m = 0; m < n; m++) f += in[m] * M.sp_to_cv[c * n + m];
                        p[st * c] = f;
                    }
                }
                __syncthreads();
            }
#pragma unroll
            for (int d = 0; d < D; d++) {
                R* out = A.ff[d] + ((long long)t * E + e0) * FE;
                const R* in = FX + d * EB * FE;
                if constexpr ((FE * sizeof(R)) % 16 == 0 && (LN::stage * sizeof(R)) % 16 == 0) {
                    for (int q = tid; q < ne * FE / Q; q += NTH)
                        reinterpret_cast<VT*>(out)[q] = reinterpret_cast<const VT*>(in)[q];
                } else {
                    for (int q = tid; q < ne * FE; q += NTH) out[q] = in[q];
                }
            }
        }
        __syncthreads();  // the next slice's phase A overwrites the flux points
        if (multi && t + 1 < nt && reads) issue(t + 1);
    }

    if constexpr (MODE == kPredict) {
        // ---- ADER predictor (src/transforms.cpp:309-323), gravity in rounds as in 2D ----
        R* O = smem;  // [slice][rho, m_x, m_y, m_z][element][point]
        const int rounds = G.grav ? 3 : 1;
        for (int round = 0; round < rounds; round++) {
            if (brow && !(G.grav && (bv == 0 ? 0 : (bv <= D ? 1 : 2)) != round)) {
                R uo[n];
                row_load<R, n>(A.u + (bge * V + bv) * NPT + br * n, uo);
                if (G.grav && bv != 0) {
                    // (from the last slice down: where all are equal, slice 0 holds dudt)
#pragma unroll
                    for (int tt = NT - 1; tt >= 0; tt--)
#pragma unroll
                        for (int i = 0; i < n; i++) {
                            const R* nw = O + ((tt * 4) * EB + bel) * NPT + br * n + i;
                            R s;
                            if (bv <= D) s = nw[0] * (R)G.g[bv - 1];
                            else s = nw[EB * NPT] * (R)G.g[0] + nw[2 * EB * NPT] * (R)G.g[1] + nw[3 * EB * NPT] * (R)G.g[2];
                            acc(i, tt) = acc(i, multi ? tt : 0) - s;
                        }
                }
                // the sums over slices, in place
#pragma unroll (n > 4 ? 1 : n)
                for (int i = 0; i < n; i++) {
                    R q[NT];
#pragma unroll
                    for (int ll = 0; ll < NT; ll++) q[ll] = acc(i, multi || (G.grav && bv != 0) ? ll : 0);
#pragma unroll
                    for (int tt = 0; tt < NT; tt++) {
                        R du = 0;
#pragma unroll
                        for (int ll = 0; ll < NT; ll++) add_term(du, q[ll], tt, ll);
                        acc(i, tt) = du;
                    }
                }
#pragma unroll
                for (int tt = 0; tt < NT; tt++) {
                    R val[n];
#pragma unroll
                    for (int i = 0; i < n; i++) {
                        R du = acc(i, tt);
                        if constexpr (sizeof(R) == 4) du *= G.grav ? dt : dt * (R)G.ih[0];
                        val[i] = uo[i] - du;
                    }
                    row_store<R, n>(A.ua_out + (((long long)tt * E + bge) * V + bv) * NPT + br * n, val);
                    if (G.grav && bv <= D) {
#pragma unroll
                        for (int i = 0; i < n; i++) O[((tt * 4 + bv) * EB + bel) * NPT + br * n + i] = val[i];
                    }
                }
            }
            if (G.grav) __syncthreads();
        }
    } else {
        __shared__ R Mcv[n * n];
        R* B0 = smem;                     // [EB][V][NPT]
        R* B1 = smem + EB * V * NPT;
        for (int i = tid; i < n * n; i += NTH) Mcv[i] = M.sp_to_cv[i];
        // the x, y, z sweeps of sp_to_cv: B0 -> B1 -> B0 -> B1
        auto to_averages = [&]() {
            sweep_smem<D, P, R>(B0, B1, Mcv, 0, ne * V * NPT);
            __syncthreads();
            sweep_smem<D, P, R>(B1, B0, Mcv, 1, ne * V * NPT);
            __syncthreads();
            sweep_smem<D, P, R>(B0, B1, Mcv, 2, ne * V * NPT);
            __syncthreads();
        };
        if constexpr (MODE == kCorrect) {
            // ---- corrector / RK stage (src/transforms.cpp:327-374, 252-261) ----
            constexpr int W = ANY ? 1 : kRowVec<R, n>;
            if (brow) {
                const long long g = (bge * V + bv) * NPT + br * n;
                R val[n];
                row_load<R, n, W>(A.u + g, val);
#pragma unroll
                for (int i = 0; i < n; i++) val[i] -= acc(i, 0);
                if (A.rk_a > 0) {
                    const R ra = (R)A.rk_a;
                    R u0[n];
                    row_load<R, n, W>(A.u0 + g, u0);
#pragma unroll
                    for (int i = 0; i < n; i++) val[i] = ra * u0[i] + ((R)1.0 - ra) * val[i];
                }
                row_store<R, n, W>(A.u_out + g, val);
#pragma unroll
                for (int i = 0; i < n; i++) B0[(bel * V + bv) * NPT + br * n + i] = val[i];
            }
            if (A.final_stage) {
                __syncthreads();
                for (int q = tid; q < ne * NPT; q += NTH) {
                    R* p = B0 + (q / NPT) * V * NPT + q % NPT;
                    R un[V], w[V];
#pragma unroll
                    for (int v = 0; v < V; v++) un[v] = p[v * NPT];
                    primitives<D>(un, w, (R)G.gm);
#pragma unroll
                    for (int v = 0; v < V; v++) p[v * NPT] = w[v];
                }
                __syncthreads();
                to_averages();
                double dtl = 1.7976931348623157e308;
                for (int q = tid; q < ne * NPT; q += NTH) {
                    const int el = q / NPT, pt = q % NPT;
                    R w[V];
#pragma unroll
                    for (int v = 0; v < V; v++) w[v] = B1[(el * V + v) * NPT + pt];
                    if (A.wcv)
#pragma unroll
                        for (int v = 0; v < V; v++) A.wcv[((long long)(e0 + el) * V + v) * NPT + pt] = w[v];
                    dtl = smin(dtl, point_dt<D>(G, w, n));
                }
                block_min_dt(dtl, A.dtmin);
            }
        } else {
            if (A.labels && tid < ne) A.labels[e0 + tid] = 0;
            // ---- U_cv = sp_to_cv(U) and the slice-0 FV candidate ----
            for (int q = tid; q < ne * V * NPT; q += NTH) B0[q] = A.u[(long long)e0 * V * NPT + q];
            __syncthreads();
            to_averages();
            for (int q = tid; q < ne * V * NPT; q += NTH) A.ucv[(long long)e0 * V * NPT + q] = B1[q];
            for (int q = tid; q < ne * NPT; q += NTH) {
                const int el = q / NPT, pt = q % NPT;
                const long long ge = e0 + el;
                R uo[V], un[V];
#pragma unroll
                for (int v = 0; v < V; v++) uo[v] = B1[(el * V + v) * NPT + pt];
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
}

}  // namespace spdk
