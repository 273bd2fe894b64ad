// aeo_positive.cuh -- positivity-preserving scalar advection
// (advect_positive!, src/AdvectionSchemes.jl:1100-1160, the limiter
// apply_positivity_limiter! :998-1098).
//
// -div(u phi) with the face fluxes limited so that a forward-Euler update
// with the same dt keeps a non-negative phi non-negative (under the
// first-order CFL condition):
//   F  = vel * face value, WENO-JS5 or WENO-Z5 reconstruction upwinded on the
//        face velocity (_reconstructed_fluxes! :868-892),
//   L  = vel * the upwind cell value (_upwind_fluxes! :899-909),
//   R  = min(1, Q / P) per cell, P = dt * the antidiffusive outflow
//        sum(max(+-(F - L), 0) / h), Q = max(phi - dt div L, 0), 1 where
//        nothing flows out (_b_limit_ratio! :1015-1043),
//   F' = L + c (F - L) with c the donor's R, R wrapped periodically one layer
//        beyond the interior (_wrap_one_layer! :951-958, the default without
//        boundary conditions; at walls the face velocity and flux are zero),
//   tend (+)= -div F' (_b_flux_div! :911-926).
// Two kernels, because each limited flux needs the R of its donor: the face
// fluxes F (WENO) and the ratios; the limited fluxes and their divergence (each face's limited
// flux evaluated by both of its cells, from the same values, so the two see
// the same flux and the update conserves phi).
//
// Arrays: u, v, w, phi, tend in the reference storage layout (halos hx, hy,
// hz >= 3, filled), x fastest; F on the interior faces ((nx+1) ny nz,
// nx (ny+1) nz, nx ny (nz+1)); R on the interior cells.
#pragma once

#include "aeo_sweep_wpair.cuh"   // the paired reconstruction

struct PosGeo {
    int nx, ny, nz, hx, hy, hz;
    long long sx, sy, sz;   // storage strides: 1, NX, NX*NY
    double idx, idy, idz;
};

__device__ __forceinline__ long long pos_sidx(const PosGeo& g, int i, int j, int k) {
    return (long long)(i + g.hx) + g.sy * (j + g.hy) + g.sz * (k + g.hz);
}

// The face fluxes F and the ratios R in one pass: a CTA marches a tile of TX x TY
// columns through ZC levels.  A row of the tile is a warp, a thread N cells of it
// 32 apart (FP32: a pair, on the paired instructions), its column's six values
// around a z face a register ring, the levels' phi planes a ring in shared memory
// that cp.async fills a level ahead.  Each face is computed once but for the tile's
// east and north faces, which one more warp computes for the ratios of the last
// cells; F and the upwind flux L of x and y faces pass through shared memory, so
// that the ratios read no flux from memory and form no L twice.
// Bound by the reconstruction's instructions (three faces a cell).
template <typename R> struct PosTile {
    using VT = typename std::conditional<sizeof(R) == 4, F2, double>::type;   // a thread's values
    static constexpr int N = sizeof(R) == 4 ? 2 : 1, TX = 32 * N, TY = 8, ROWT = 32 * TY, THREADS = ROWT + 32;
    static constexpr int PW = TX + 6, PH = TY + 6, PSZ = PW * PH, RING = 5;
};
template <typename R, int S>
__global__ void __launch_bounds__(PosTile<R>::THREADS, 2) pos_flux_ratio_kernel(
    PosGeo g, const R* __restrict__ u, const R* __restrict__ v, const R* __restrict__ w, const R* __restrict__ f,
    const double* __restrict__ dtp, int zc, R* __restrict__ Fx, R* __restrict__ Fy, R* __restrict__ Fz,
    R* __restrict__ Rr) {
    using T = PosTile<R>;
    using VT = typename T::VT;
    constexpr int N = T::N;
    __shared__ R ring[T::RING][T::PSZ];
    __shared__ R xFs[2][T::TY][T::TX + 1], xLs[2][T::TY][T::TX + 1], yFs[2][T::TY + 1][T::TX], yLs[2][T::TY + 1][T::TX];
    const int t = threadIdx.x, lane = t & 31, row = t >> 5;
    const int i0 = blockIdx.x * T::TX, j0 = blockIdx.y * T::TY, k0 = blockIdx.z * zc, k1 = min(k0 + zc, g.nz);
    const bool edge = row == T::TY;   // the warp of the tile's east and north faces
    const int i = i0 + lane, j = j0 + row;

    // a plane of phi, columns i0 - 3 .. i0 + TX + 2 and rows j0 - 3 .. j0 + TY + 2 as far as the faces
    // reach: the thread's elements lie the same way in every plane
    constexpr int NF = (T::PSZ + T::THREADS - 1) / T::THREADS;
    long long fo[NF];
#pragma unroll
    for (int s = 0; s < NF; ++s) {
        const int q = t + s * T::THREADS, r = q / T::PW, c = q - r * T::PW;
        fo[s] = q < T::PSZ && i0 + c - 3 <= g.nx + 2 && j0 + r - 3 <= g.ny + 2 ? pos_sidx(g, i0 + c - 3, j0 + r - 3, 0) : -1;
    }
    auto fetch = [&](int k) {
        const unsigned d = (unsigned)__cvta_generic_to_shared(ring[k % T::RING] + t);
        const R* a = f + g.sz * k;
#pragma unroll
        for (int s = 0; s < NF; ++s)
            if (fo[s] >= 0)
                asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d + unsigned(s * T::THREADS * sizeof(R))),
                             "l"(a + fo[s]), "n"(sizeof(R)) : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto arrive = [&] {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
    };
    // the N values a[q], a[q + 32] where the mask has them
    auto at = [&](const R* a, long long q, const bool (&on)[2]) {
        if constexpr (N == 2) return F2(on[0] ? a[q] : R(0), on[1] ? a[q + 32] : R(0));
        else return on[0] ? a[q] : R(0);
    };
    auto tile = [&](const R* a) {
        if constexpr (N == 2) return F2(a[0], a[32]);
        else return a[0];
    };
    auto comp = [&](auto x, int c) {
        if constexpr (N == 2) return c ? x.v.y : x.v.x;
        else return x;
    };
    // F and L of a face from its velocity and the six values around it
    auto face = [&](VT vel, VT f0, VT f1, VT f2, VT f3, VT f4, VT f5, VT* F, VT* L) {
        if constexpr (N == 2) {
            *F = vel * weno_upwind_f2<S>(vel, f0, f1, f2, f3, f4, f5);
            *L = F2(vel.v.x * (vel.v.x >= R(0) ? f2.v.x : f3.v.x), vel.v.y * (vel.v.y >= R(0) ? f2.v.y : f3.v.y));
        } else {
            *F = vel * weno_upwind<R, S>(vel >= R(0), f0, f1, f2, f3, f4, f5);
            *L = vel * (vel >= R(0) ? f2 : f3);
        }
    };
    const bool inx[2] = {i < g.nx, N == 2 && i + 32 < g.nx};
    const bool fx[2] = {!edge && i <= g.nx && j < g.ny, !edge && N == 2 && i + 32 <= g.nx && j < g.ny};
    const bool fy[2] = {inx[0] && j <= g.ny, inx[1] && j <= g.ny};   // the edge warp's row is TY: the north faces
    const bool cell[2] = {!edge && inx[0] && j < g.ny, !edge && inx[1] && j < g.ny};

    for (int k = k0; k < k0 + 4; ++k)
        if (k <= g.nz + 2) fetch(k);
    const long long col = pos_sidx(g, i, j, 0);
    const R dt = R(*dtp), z = R(0), idx = R(g.idx), idy = R(g.idy), idz = R(g.idz);
    const int centre = (row + 3) * T::PW + lane + 3;
    VT h[6];   // the column's values at k - 3 .. k + 2
    for (int q = 0; q < 3; ++q) h[q] = at(f, col + g.sz * (k0 + q - 3), cell);
    VT Fb, Lb, Ft, Lt;
    const long long zplane = (long long)g.nx * g.ny, zface = (long long)g.nx * j + i;
    auto put = [&](R* dst, VT x, const bool (&on)[2]) {
#pragma unroll
        for (int c = 0; c < N; ++c)
            if (on[c]) dst[32 * c] = comp(x, c);
    };
    arrive();
    if (!edge) {
        for (int q = 0; q < 3; ++q) h[3 + q] = tile(&ring[(k0 + q) % T::RING][centre]);
        face(at(w, col + g.sz * k0, cell), h[0], h[1], h[2], h[3], h[4], h[5], &Fb, &Lb);
        put(Fz + zplane * k0 + zface, Fb, cell);
    }
    const R *pu = u + col + g.sz * k0, *pv = v + col + g.sz * k0, *pw = w + col + g.sz * (k0 + 1);
    const R* pe = u + pos_sidx(g, i0 + T::TX, j0 + lane, k0);   // the edge warp's east faces
    R* ox = Fx + (long long)(g.nx + 1) * (j + (long long)g.ny * k0) + i;
    R* oy = Fy + (long long)g.nx * (j + (long long)(g.ny + 1) * k0) + i;
    R* oz = Fz + zplane * (k0 + 1) + zface;
    R* orr = Rr + zplane * k0 + zface;
    const long long nxp = (long long)(g.nx + 1) * g.ny, nyp = (long long)g.nx * (g.ny + 1);
    // lanes 0 .. TY - 1 of the edge warp: one a row of the tile
    const bool fe = edge && lane < T::TY && i0 + T::TX <= g.nx && j0 + lane < g.ny;
    const bool fown[2] = {fy[0] && (!edge || j == g.ny), fy[1] && (!edge || j == g.ny)};
    for (int k = k0;; ++k, pu += g.sz, pv += g.sz, pw += g.sz, pe += g.sz, ox += nxp, oy += nyp, oz += zplane, orr += zplane) {
        // the faces' velocities of level k, on their way across the barrier
        const bool last = k == k1;
        VT vx = VT(z), vy = VT(z), vz = VT(z);
        if (!last) {
            if (edge) {
                const R ue = fe ? *pe : z;
                if constexpr (N == 2) vx = F2(ue, ue);
                else vx = ue;
            } else {
                vx = at(pu, 0, fx);
                vz = at(pw, 0, cell);
            }
            vy = at(pv, 0, fy);
        }
        if (k > k0) {
            arrive();
            if (!edge) {
                // the ratios of level k - 1, whose faces the barrier has completed
                const auto &xF = xFs[(k - 1) & 1], &xL = xLs[(k - 1) & 1];
                const auto &yF = yFs[(k - 1) & 1], &yL = yLs[(k - 1) & 1];
#pragma unroll
                for (int c = 0; c < N; ++c) {
                    const int x = lane + 32 * c;
                    const R le = xL[row][x + 1], lw = xL[row][x], ln = yL[row + 1][x], ls = yL[row][x], lt = comp(Lt, c), lb = comp(Lb, c);
                    const R axe = xF[row][x + 1] - le, axw = xF[row][x] - lw, ayn = yF[row + 1][x] - ln, ays = yF[row][x] - ls,
                            azt = comp(Ft, c) - lt, azb = comp(Fb, c) - lb;
                    const R Pm = dt * ((fmax(axe, z) + fmax(-axw, z)) * idx + (fmax(ayn, z) + fmax(-ays, z)) * idy +
                                       (fmax(azt, z) + fmax(-azb, z)) * idz);
                    const R div_lo = (le - lw) * idx + (ln - ls) * idy + (lt - lb) * idz;
                    const R Q = fmax(comp(h[2], c) - dt * div_lo, z);
                    if (cell[c]) orr[32 * c - zplane] = Pm > z ? fmin(R(1), Q / Pm) : R(1);
                }
                Fb = Ft;
                Lb = Lt;
            }
        }
        if (last) break;
        if (k + 1 < k1) fetch(k + 4);   // plane k + 4 (at most nz + 2) over plane k - 1
        auto &xF = xFs[k & 1], &xL = xLs[k & 1];
        auto &yF = yFs[k & 1], &yL = yLs[k & 1];
        const R* P = ring[k % T::RING];
        const R* Y = P + centre;
        auto yface = [&](VT* F, VT* L) {
            face(vy, tile(Y - 3 * T::PW), tile(Y - 2 * T::PW), tile(Y - T::PW), tile(Y), tile(Y + T::PW), tile(Y + 2 * T::PW), F, L);
        };
        auto keep = [&](R* dF, R* dL, VT F, VT L) {
#pragma unroll
            for (int c = 0; c < N; ++c) {
                dF[32 * c] = comp(F, c);
                dL[32 * c] = comp(L, c);
            }
        };
        if (edge) {
            VT F, L, Fe, Le;
            yface(&F, &L);
            const R* X = P + ((lane & (T::TY - 1)) + 3) * T::PW + T::TX + 3;
            auto dup = [&](R a) { if constexpr (N == 2) return F2(a, a); else return a; };
            face(vx, dup(X[-3]), dup(X[-2]), dup(X[-1]), dup(X[0]), dup(X[1]), dup(X[2]), &Fe, &Le);
            keep(&yF[row][lane], &yL[row][lane], F, L);
            put(oy, F, fown);
            if (fe) {
                xF[lane][T::TX] = comp(Fe, 0);
                xL[lane][T::TX] = comp(Le, 0);
                if (i0 + T::TX == g.nx) Fx[(long long)(g.nx + 1) * (j0 + lane + (long long)g.ny * k) + g.nx] = comp(Fe, 0);
            }
        } else {
            // the three faces' chains side by side
            VT Fy_, Ly_, Fx_, Lx_;
#pragma unroll
            for (int q = 0; q < 5; ++q) h[q] = h[q + 1];
            h[5] = tile(&ring[(k + 3) % T::RING][centre]);
            yface(&Fy_, &Ly_);
            face(vx, tile(Y - 3), tile(Y - 2), tile(Y - 1), tile(Y), tile(Y + 1), tile(Y + 2), &Fx_, &Lx_);
            face(vz, h[0], h[1], h[2], h[3], h[4], h[5], &Ft, &Lt);
            keep(&yF[row][lane], &yL[row][lane], Fy_, Ly_);
            keep(&xF[row][lane], &xL[row][lane], Fx_, Lx_);
            put(oy, Fy_, fown);
            put(ox, Fx_, fx);
            if (k + 1 < k1 || k1 == g.nz) put(oz, Ft, cell);
        }
    }
}

// The limited fluxes and their divergence, on the tiles of pos_flux_ratio_kernel: each
// thread limits the west, south and top faces of its cells (the bottom one is the
// level before's top), the edge warp the tile's east and north faces, and x and y fluxes
// pass through shared memory (two buffers, one barrier a level).  Bound by memory: eight
// arrays in, one out.  With both cells of a face limiting it, a cell loaded 30 values
// (256^3 FP32: 207 us against 189 now, both from a cold cache).
template <typename R>
__global__ void __launch_bounds__(PosTile<R>::THREADS) pos_apply_kernel(
    PosGeo g, const R* __restrict__ u, const R* __restrict__ v, const R* __restrict__ w, const R* __restrict__ f,
    const R* __restrict__ Fx, const R* __restrict__ Fy, const R* __restrict__ Fz, const R* __restrict__ Rr, int zc,
    R* __restrict__ tend, int accumulate) {
    using T = PosTile<R>;
    constexpr int N = T::N;
    __shared__ R xG[2][T::TY][T::TX + 1], yG[2][T::TY + 1][T::TX];
    const int t = threadIdx.x, lane = t & 31, row = t >> 5;
    const int i0 = blockIdx.x * T::TX, j0 = blockIdx.y * T::TY, k0 = blockIdx.z * zc, k1 = min(k0 + zc, g.nz);
    const bool edge = row == T::TY;
    const int j = j0 + row;
    // the limited flux lo + c (F - lo), c the ratio of the donor (the low cell where the
    // antidiffusive flux is >= 0)
    auto limited = [&](R F, R vel, R fl, R fh, R rl, R rh) {
        const R lo = vel * (vel >= R(0) ? fl : fh);
        const R a = F - lo;
        return lo + (a >= R(0) ? rl : rh) * a;
    };
    const R idx = R(g.idx), idy = R(g.idy), idz = R(g.idz);
    // Cells and faces beyond the domain are clamped to its last ones (their results are not
    // used), so that a level's loads have no branch between them and leave together.
    R fc[N], rc[N], gb[N];   // phi, R and the bottom face's limited flux of the thread's cells
    const int jc = min(j, g.ny), jw = jc < g.ny ? jc : 0, js = jc > 0 ? jc - 1 : g.ny - 1;
    const long long nxy = (long long)g.nx * g.ny;
    int rw[N], rm[N], rs[N];          // in-plane indices of R at the cell, its west and its south neighbour
    long long pc[N], qx[N], qy[N];    // storage, x face and y face indices at level k
#pragma unroll
    for (int c = 0; c < N; ++c) {
        const int i = min(i0 + lane + 32 * c, g.nx), iw = i < g.nx ? i : 0, im = i > 0 ? i - 1 : g.nx - 1;
        rw[c] = g.nx * jw + iw;
        rm[c] = g.nx * jw + im;
        rs[c] = g.nx * js + iw;
        pc[c] = pos_sidx(g, i, jc, k0);
        qx[c] = (long long)(g.nx + 1) * (min(jc, g.ny - 1) + (long long)g.ny * k0) + i;
        qy[c] = (long long)g.nx * (jc + (long long)(g.ny + 1) * k0) + min(i, g.nx - 1);
        fc[c] = f[pc[c]];
        rc[c] = Rr[nxy * k0 + rw[c]];
        gb[c] = limited(Fz[nxy * k0 + rw[c]], w[pc[c]], f[pc[c] - g.sz], fc[c], Rr[nxy * (k0 > 0 ? k0 - 1 : g.nz - 1) + rw[c]], rc[c]);
    }
    // the edge warp's east faces: lanes 0 .. TY - 1, one a row of the tile
    const int ie = min(i0 + T::TX, g.nx), je = min(j0 + (lane & (T::TY - 1)), g.ny - 1);
    for (int k = k0; k < k1; ++k) {
        const int buf = (k - k0) & 1;
        const long long rk = nxy * k, rt = nxy * (k + 1 < g.nz ? k + 1 : 0);
        R gt[N], fn[N], rn[N], td[N];
        R yv[N], yF[N], yf[N], yr[N], xv[N], xF[N], xf[N], xr[N], zv[N], zF[N];
#pragma unroll
        for (int c = 0; c < N; ++c) {
            yv[c] = v[pc[c]];
            yF[c] = Fy[qy[c]];
            yf[c] = f[pc[c] - g.sy];
            yr[c] = Rr[rk + rs[c]];
            if (!edge) {
                xv[c] = u[pc[c]];
                xF[c] = Fx[qx[c]];
                xf[c] = f[pc[c] - 1];
                xr[c] = Rr[rk + rm[c]];
                zv[c] = w[pc[c] + g.sz];
                zF[c] = Fz[rk + nxy + rw[c]];
                fn[c] = f[pc[c] + g.sz];
                rn[c] = Rr[rt + rw[c]];
                td[c] = accumulate ? tend[pc[c]] : R(0);
            } else {
                fn[c] = f[pc[c] + g.sz];
                rn[c] = Rr[rt + rw[c]];
            }
        }
        if (edge) {
            const long long p = pos_sidx(g, ie, je, k);
            const R ue = u[p], Fe = Fx[(long long)(g.nx + 1) * (je + (long long)g.ny * k) + ie], fw = f[p - 1], fe = f[p];
            const R rl = Rr[rk + (long long)g.nx * je + ie - 1], rh = Rr[rk + (long long)g.nx * je + (ie < g.nx ? ie : 0)];
            if (lane < T::TY) xG[buf][lane][T::TX] = limited(Fe, ue, fw, fe, rl, rh);
        }
#pragma unroll
        for (int c = 0; c < N; ++c) {
            const int x = lane + 32 * c;
            yG[buf][row][x] = limited(yF[c], yv[c], yf[c], fc[c], yr[c], rc[c]);
            if (edge) continue;
            xG[buf][row][x] = limited(xF[c], xv[c], xf[c], fc[c], xr[c], rc[c]);
            gt[c] = limited(zF[c], zv[c], fc[c], fn[c], rc[c], rn[c]);
        }
        __syncthreads();
#pragma unroll
        for (int c = 0; c < N; ++c) {
            const int x = lane + 32 * c;
            if (!edge) {
                const R d = (xG[buf][row][x + 1] - xG[buf][row][x]) * idx + (yG[buf][row + 1][x] - yG[buf][row][x]) * idy +
                            (gt[c] - gb[c]) * idz;
                if (i0 + x < g.nx && j < g.ny) tend[pc[c]] = accumulate ? td[c] - d : -d;
                gb[c] = gt[c];
            }
            fc[c] = fn[c];
            rc[c] = rn[c];
            pc[c] += g.sz;
            qx[c] += (long long)(g.nx + 1) * g.ny;
            qy[c] += (long long)g.nx * (g.ny + 1);
        }
    }
}
