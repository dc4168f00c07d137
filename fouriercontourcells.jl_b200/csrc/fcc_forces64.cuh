// fcc_forces64.cuh — FP64 force evaluation of the step (forces_warp64).
//
// Same work per body as the FP32 forces_warp (fcc_kernels.cuh), arranged for
// the FP64 units.  8 lanes per body, 4 bodies per warp; lane l of a body owns
// the contour nodes l + 8 s, s < S (5, or 8 in variant 7), of a chunk and the
// modes m = l (and lane 0 m = 8 too).  The contractions over modes and nodes run
// on the FP64 tensor cores (mma.sync m8n8k4, IEEE double products and sums):
//   synthesis  [R_b ; R'_b] (8 rows) = [c_b ; c'_b] (8 x 20) . M^T (20 x 8 S)
//   pullback   [g_b ; h_b]  (8 rows) = [GR_b ; GD_b] (8 x 8 S) . M (8 S x 20)
// with rows 2b + h (b the body, h = bit 2 of the lane: value or derivative),
// M[k] = (cos 2 phi_k, sin 2 phi_k, ..., cos 10 phi_k, sin 10 phi_k, 1, 0),
// c the R0-scaled lab coefficients of the record and c' the derivative's
// (n beta, -n alpha, 0), so that R' = M c' (src/geometry.jl:113-122, 248-257)
// and glab = g + D h (alpha: -n h[beta], beta: +n h[alpha];
// src/gradients.jl:374-386).  A row's A fragment lives in the four lanes that
// share its body and h, and a tile's column c is the node (c >> 1) + 4 (c &
// 1), so a lane finds its own node or mode, or its partner's across one
// shuffle with lane ^ 4: no transposition through shared memory.

#pragma once

namespace fcc {

__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// R_j(psi) of a staged FP64 record by two complex Horner chains (even and odd
// modes), as the FP32 radius_at.
__device__ __forceinline__ double radius_at64(const double* p, double cp, double sp) {
    const double wr = cp * cp - sp * sp, wi = 2.0 * cp * sp;  // z^2
    const double2* q = reinterpret_cast<const double2*>(p + R_A0);
    auto step = [&](double& r, double& im, double al, double be) {
        const double t = fma(r, wr, fma(-im, wi, al));
        im = fma(r, wi, fma(im, wr, -be));
        r = t;
    };
    // pairs: (a0 al2) (be2 al3) (be3 al4) (be4 al5) (be5 al6) (be6 al7) (be7 al8) (be8 al9) (be9 al10) (be10 theta)
    const double2 v9 = q[9], v8 = q[8], v7 = q[7], v6 = q[6];
    double er = v8.y, ei = -v9.x;   // c10
    double orr = v7.y, oi = -v8.x;  // c9
    step(er, ei, v6.y, v7.x);       // c8
    const double2 v5 = q[5], v4 = q[4];
    step(orr, oi, v5.y, v6.x);  // c7
    step(er, ei, v4.y, v5.x);   // c6
    const double2 v3 = q[3], v2 = q[2];
    step(orr, oi, v3.y, v4.x);  // c5
    step(er, ei, v2.y, v3.x);   // c4
    const double2 v1 = q[1], v0 = q[0];
    step(orr, oi, v1.y, v2.x);  // c3
    step(er, ei, v0.y, v1.x);   // c2
    const double qr = fma(orr, cp, fma(-oi, sp, er));
    const double qi = fma(orr, sp, fma(oi, cp, ei));
    return fma(wr, qr, fma(-wi, qi, v0.x));
}

// Euler-Maruyama update of body g (update_body) in FP64, lane l with modes l
// and (lane 0) 8.  scf: the body-frame coefficients, then sin and cos of the
// old theta and 1/(2 a0).
// What does not depend on the shape's sums (the displacement, the wrap, the
// distance from the skin reference) is computed by every lane before them:
// a straight line of independent chains, where lane 0 alone after the sums
// added 700 cycles to a warp group.
__device__ __forceinline__ void update_body64(const DevPtrs<double>& d, const SimDesc<double>& P, bool act, int g, int s,
                                              int l, int par, double xo, double yo, double wo, double tho, double r0,
                                              int ti, double fx, double fy, double tt, double gl0, const double (&gA)[2],
                                              const double (&gB)[2], const double* scf, double x0, double y0,
                                              double rmax0, int fl, const double (&nz)[2], int* rbp, double* own,
                                              double* scf_w, bool keep) {
    typedef double T;
    constexpr int L = 8;
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int MPL = 2;
    const T dt = P.dt;
    // standard normals of this body and step (src/random.jl:88-100): lane 0
    // holds block 1 (orientation), lane 1 block 0 (translation)
    const T z3 = __shfl_sync(FULL, nz[0], 0, L);
    const T xi1 = __shfl_sync(FULL, nz[0], 1, L);
    const T xi2 = __shfl_sync(FULL, nz[1], 1, L);
    const T sig_r = P.sigr[ti];
    const T thn = fma(sig_r, z3, fma(-(dt * P.muth[ti]), tt, tho));
    const T so1 = scf[NCM], co1 = scf[NCM + 1];
    T sn1, cn1;
    t_sincos(thn, &sn1, &cn1);

    // displacement and wrap
    const T sig = P.sigt[ti];
    const T dxp = fma(dt, fma(P.v0[ti], co1, -(P.mur[ti] * fx)), sig * xi1);
    const T dyp = fma(dt, fma(P.v0[ti], so1, -(P.mur[ti] * fy)), sig * xi2);
    int sx, sy;
    const T xw = wrap_exact(add_rn(xo, dxp), P.Lx, sx);
    const T yw = wrap_exact(add_rn(yo, dyp), P.Ly, sy);
    // distance from the skin reference (src/neighbors.jl:198-205)
    const T dx = minimum_image_exact(sub_rn(xw, x0), P.Lx);
    const T dy = minimum_image_exact(sub_rn(yw, y0), P.Ly);
    const T moved = t_sqrt(add_rn(mul_rn(dx, dx), mul_rn(dy, dy)));

    T* cf = d.coef + (size_t)(act ? g : 0) * NCM;
    const T ga0 = r0 * gl0;
    // dE/da0 * da0/da_n = -h0 a_n (area constraint)
    const T h0 = ga0 * scf[NCM + 2];
    const T dtmu = dt * P.muab[ti];
    const int K = P.K;
    const int Kt = min(K, P.kmax[ti]);  // modes of this type; the rest stay zero
    // Every lane computes its MPL modes without branches (those of a lane
    // beyond Kt give zero), so their chains overlap; a simulation whose modes
    // fit one per lane skips the second
    T an[MPL], bn[MPL], nrm[MPL];
    double sp = 0.0, qp = 0.0;
    T bp = T(0);
#pragma unroll
    for (int u = 0; u < MPL; ++u) {
        an[u] = bn[u] = nrm[u] = T(0);
        if (u > 0 && K <= u * L) continue;  // uniform
        const int m = l + u * L;
        const bool on = m < Kt;
        const T ga = gA[u] * r0, gb = gB[u] * r0;
        T so, co;
        cis_pow(co1, so1, m + 2, co, so);
        const T a = m < KM ? scf[1 + m] : T(0), b = m < KM ? scf[1 + KM + m] : T(0);
        const T gca = fma(-h0, a, fma(ga, co, gb * so));
        const T gcb = fma(-h0, b, fma(-ga, so, gb * co));
        const T a1 = fma(-dtmu, gca, a), b1 = fma(-dtmu, gcb, b);
        an[u] = on ? a1 : T(0);
        bn[u] = on ? b1 : T(0);
        nrm[u] = mode_norm(an[u], bn[u]);
    }
    // enforce_shape! (src/dynamics.jl:44-64) with FP64 sums: the three sums of
    // the shape as it is at once; a body beyond the bound (rare) is scaled and
    // summed again
    auto sums = [&] {
        sp = qp = 0.0;
        bp = T(0);
#pragma unroll
        for (int u = 0; u < MPL; ++u) {
            if (u > 0 && K <= u * L) continue;
            sp += (double)nrm[u];
            qp += mode_sq(an[u], bn[u]);
            bp += nrm[u];
        }
        sp = group_sum<L>(sp);
        qp = group_sum<L>(qp);
        bp = group_sum<L>(bp);
    };
    sums();
    if (__any_sync(FULL, sp > SHAPE_BOUND)) {
        if (sp > SHAPE_BOUND) {
            const double f = SHAPE_BOUND / sp;
#pragma unroll
            for (int u = 0; u < MPL; ++u) {
                an[u] = T((double)an[u] * f);
                bn[u] = T((double)bn[u] * f);
                nrm[u] = mode_norm(an[u], bn[u]);
            }
        }
        sums();
    }
    const T a0n = T(sqrt(1.0 - qp * 0.5));

    // lab frame of the new state (src/geometry.jl:208-227)
    T* rn = rec_next(d, par) + (size_t)(act ? g : 0) * RECW;
#pragma unroll
    for (int u = 0; u < MPL; ++u) {
        const int m = l + u * L;
        if (m < K) {
            T so, co, al, be;
            cis_pow(cn1, sn1, m + 2, co, so);
            to_lab(an[u], bn[u], co, so, al, be);
            if (act) {
                rn[r_al(m)] = r0 * al;
                rn[r_be(m)] = r0 * be;
                cf[1 + m] = an[u];
                cf[1 + KM + m] = bn[u];
                if (keep) {
                    own[r_al(m)] = r0 * al;
                    own[r_be(m)] = r0 * be;
                    scf_w[1 + m] = an[u];
                    scf_w[1 + KM + m] = bn[u];
                }
            }
        }
    }
    const T rmax = r0 * (a0n + bp);

    if (act && l == 0) {
        if (sx) d.imgx[g] += sx;  // image counters change only on a wrap
        if (sy) d.imgy[g] += sy;
        rn[R_X] = xw;
        rn[R_Y] = yw;
        rn[R_RMAX] = rmax;
        rn[R_W] = wo;
        rn[R_A0] = r0 * a0n;
        rn[R_TH] = thn;
        cf[0] = a0n;
        if (keep) {  // where the next step reads them (Resident)
            own[R_X] = xw;
            own[R_Y] = yw;
            own[R_RMAX] = rmax;
            own[R_A0] = r0 * a0n;
            own[R_TH] = thn;
            scf_w[0] = a0n;
            scf_w[NCM] = sn1;
            scf_w[NCM + 1] = cn1;
            scf_w[NCM + 2] = T(0.5) / a0n;
        }
        // skin check of the new state (src/neighbors.jl:198-205); the flags of
        // this step (read at its start) already carry F_VALID of a rebuild
        if ((fl & F_CONTACT) && (fl & F_VALID) && P.skin > T(0)) {
            const T grow = sub_rn(rmax, rmax0);
            const T delta = add_rn(moved, grow > T(0) ? grow : T(0));
            if (mul_rn(T(2), delta) > P.skin) {
                atomicOr(&d.flags[s], F_REBUILD);
                if (rbp) *rbp = 1;  // the block's arrival at the step barrier reports it
            }
        }
        if (!(isfinite(xw) && isfinite(yw) && isfinite(thn) && isfinite(rmax))) atomicOr(&d.flags[s], F_NONFINITE);
    }
}

// Forces on the 4 bodies of warp group `wg`, and in MODE_FUSED their update
// (references: forces_warp).  `stage` is this warp's shared memory; `tab` the
// block's copy of M and of the nodes' (cos, sin) (one chunk), else null.
template <int S, bool ONE, int MODE, bool USER, bool LAT>
__device__ __forceinline__ void forces_warp64(const DevPtrs<double>& d, int wg, double* stage, int par,
                                              const SimDesc<double>* sim0, const double* tab, int* rbp,
                                              const BarrierLocal* lone, bool drawn, Resident<double, 8>* res) {
    typedef double T;
    constexpr int L = 8, BPW = 4;
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int IDS = (NBMAX64 + L - 1) / L;
    constexpr int MPL = 2;  // modes per lane
    // slot of a staged neighbour's coupling: its record word, which user terms need, or its theta
    constexpr int COUPLING = USER ? R_TH : R_W;
    const int lane = threadIdx.x & 31;
    const int l = lane & 7, tq = lane & 3, b = lane >> 3;
    const bool h = lane & 4;  // this lane's MMA row is a derivative row
    const int g = wg * BPW + b;
    int s = 0;
    if (!sim0) {
        const int gf = wg * BPW;
        s = gf < d.Ntot ? __ldg(d.sim_of + gf) : -1;
        if (s < 0) return;
    }
    // a pool's descriptors are read where they are (constant during a launch)
    const SimDesc<T>& P = sim0 ? *sim0 : d.sims[s];
    const bool valid = sim0 ? g < d.Ntot : g < P.body_off + P.n;
    const int gg = valid ? g : (sim0 ? 0 : wg * BPW);
    const T* rc = rec_cur(d, par);

    // warp's shared memory: own records, neighbour records, walk slots, own body-frame coefficients
    T* own = stage + (size_t)b * SREC64;
    T* snb = stage + (size_t)(BPW + b * NBMAX64) * SREC64;
    T* wx = stage + (size_t)BPW * (1 + NBMAX64) * SREC64 + lane;  // node offsets x, y and pressure: [3][S][32]
    T* wy = wx + S * 32;
    T* wp = wy + S * 32;
    T* scf = stage + (size_t)BPW * (1 + NBMAX64) * SREC64 + 3 * S * 32 + (size_t)b * SCF64;

    // the matrix and the nodes' (cos, sin): in shared memory but for a contour of many chunks
    const T* mat = ONE || tab ? tab : d.basis;
    const T* cst = ONE || tab ? tab + m64_rows(ONE, S) * M64_COLS : d.cs;

    // ---- independent loads first
    const T* grec = rc + (size_t)gg * RECW;
    T xi, yi, rmi, wf, r0;
    const bool kept = LAT && res->have;
    if (kept) {  // the own state is where the last update left it
        xi = own[R_X], yi = own[R_Y], wf = own[R_W];
        r0 = res->r0;
    } else {
        for (int c = l; c < RECW / 2; c += L) cp_async16(own + 2 * c, grec + 2 * c);
        if (MODE != MODE_FORCES) {
            const T* cf = d.coef + (size_t)gg * NCM;  // written by this block only (during a launch)
#pragma unroll
            for (int u = 0; u < 3; ++u)
                if (l + u * L < NCM) cp_async8(scf + l + u * L, cf + l + u * L);
        }
        load_head(grec, xi, yi, rmi, wf);
        r0 = __ldg(d.R0 + gg);
    }
    cp_async_commit();
    int cnt_raw, ids[IDS];
    static_assert(IDS == 1, "one neighbour id per lane");
    if (kept && res->lists) {
        cnt_raw = res->cnt;
        ids[0] = res->ids[0];
    } else {
        cnt_raw = ldcg(d.nb_count + gg);
        ids[0] = l < min(d.cap, NBMAX64) ? ldcg(d.nb_idx + (size_t)gg * d.cap + l) : gg;
    }
    const bool ref = kept && res->lists;  // the skin references of the last rebuild are at hand
    if constexpr (LAT) {
        res->r0 = r0;
        res->cnt = cnt_raw;
        res->ids[0] = ids[0];
        res->lists = true;
    }
    const int fl = lone ? lone->flags : ldcg(d.flags + s);
    const long long clk = lone ? lone->clock : ldcg(d.clock + s);
    bool act = valid;
    if (MODE != MODE_DIAG) act = act && (fl & F_ACTIVE) && !(fl & (F_FROZEN | F_HOLD));
    const int nth = P.nth;
    const T dphi = P.dphi;

    // ---- Philox normals early (lane 1: translation, the others: orientation)
    // unless they were drawn during the last step barrier (draw_ahead)
    T nz[2] = {T(0), T(0)};
    if (MODE == MODE_FUSED && drawn) nz[0] = wx[0], nz[1] = wx[32];
    else if (MODE == MODE_FUSED && P.has_noise)
        philox_pair<T>(P.k0, P.k1, (uint32_t)(gg - P.body_off + 1), (uint64_t)clk, l == 1 ? 0u : 1u, nz[0], nz[1]);

    // ---- neighbour records into shared memory, a record by the 8 lanes of its
    // body (whole lines; a record per lane took 32 lines an instruction); once
    // there, lane q replaces the head of record q by what the contact phases
    // use: the minimum-image centre offset r_i - r_j, the squared reach and
    // (without user terms) the pair's coupling
    const bool contact = act && (fl & F_CONTACT);
    const int cnt = contact ? min(cnt_raw, d.cap) : 0;
    const int maxc = __reduce_max_sync(FULL, cnt);
    const int wv = unpack_w(wf);
    const int ti = wv & 7;
    const int pi = wv >> 3;
    const T Lx = P.Lx, Ly = P.Ly;
    const T cB = P.cB[ti];
    auto stage_batch = [&](int base, bool have) {  // have: ids holds the batch's ids
        const int npre = min(cnt - base, NBMAX64);
        __syncwarp();
        if (!have) {
#pragma unroll
            for (int u = 0; u < IDS; ++u) {
                const int q = l + u * L;
                ids[u] = q < npre ? ldcg(d.nb_idx + (size_t)gg * d.cap + base + q) : gg;
            }
        }
        int j[NBMAX64];
#pragma unroll
        for (int q = 0; q < NBMAX64; ++q) j[q] = __shfl_sync(FULL, ids[q / L], q % L, L);
#pragma unroll
        for (int q = 0; q < NBMAX64; ++q)
            if (q < npre) {
                const T* src = rc + (size_t)j[q] * RECW;
                cp_async16(snb + q * SREC64 + 2 * l, src + 2 * l);
                if (l < RECW / 2 - L) cp_async16(snb + q * SREC64 + 2 * (l + L), src + 2 * (l + L));
            }
        cp_async_commit();
    };
    auto finish_batch = [&](int base) {
        const int npre = min(cnt - base, NBMAX64);
        cp_async_wait_all();
        __syncwarp();
#pragma unroll
        for (int u = 0; u < IDS; ++u) {
            const int q = l + u * L;
            if (q < npre) {
                T* r = snb + q * SREC64;
                const T lim = r[R_RMAX] + P.crange;
                r[R_X] = minimum_image_fast(xi - r[R_X], Lx, P.invLx);
                r[R_Y] = minimum_image_fast(yi - r[R_Y], Ly, P.invLy);
                r[R_RMAX] = lim * lim;
                const int wj = unpack_w(r[R_W]);
                r[COUPLING] = P.cA[(wj >> 3) == pi ? 1 : 0][ti][wj & 7];
            }
        }
        __syncwarp();
    };
    stage_batch(0, true);
    int staged_base = 0;

    // ---- contour chunks of 8 ns nodes (ns <= S), evenly filled
    const int nch = ONE ? 1 : (nth + L * S - 1) / (L * S);
    const int ns = ONE ? S : (nth + 8 * nch - 1) / (8 * nch);
    T R[S], R1[S], R2[S];
    unsigned vmask = 0;
    T fa[5];  // synthesis A fragment of this lane's row, one value per k-step
    auto load_row = [&]() {
        const T n0 = T((tq >> 1) + 2);
        const T f0 = h ? ((tq & 1) ? -n0 : n0) : T(1), df = h ? ((tq & 1) ? T(-2) : T(2)) : T(0);
#pragma unroll
        for (int kt = 0; kt < 5; ++kt) {
            const int j = 4 * kt + tq;  // column of M
            T v = T(0);
            if (j < 18) v = (f0 + T(kt) * df) * own[R_A0 + 1 + (h ? (j ^ 1) : j)];
            else if (j == 18 && !h) v = own[R_A0];
            fa[kt] = v;
        }
    };
    auto m_at = [&](int row, int col) -> T { return mat[row * M64_COLS + col]; };
    auto cs_at = [&](int k) -> double2 { return reinterpret_cast<const double2*>(cst)[k]; };
    auto synth = [&](int ch) {
        vmask = 0;
        if (!ONE) load_row();
        const int k0 = ch * 8 * ns, c = lane >> 2;
        const int row0 = k0 + (c >> 1) + 4 * (c & 1);
        double acc[S][2];
#pragma unroll
        for (int sl = 0; sl < S; ++sl) acc[sl][0] = acc[sl][1] = 0.0;
#pragma unroll
        for (int kt = 0; kt < 5; ++kt)  // the S chains of products side by side
#pragma unroll
            for (int sl = 0; sl < S; ++sl)
                if (ONE || sl < ns) mma_f64(acc[sl], fa[kt], m_at(row0 + 8 * sl, 4 * kt + tq));
#pragma unroll
        for (int sl = 0; sl < S; ++sl) {
            const T recv = __shfl_xor_sync(FULL, h ? acc[sl][0] : acc[sl][1], 4);
            const bool v = (ONE || sl < ns) && k0 + l + 8 * sl < nth;
            vmask |= v ? 1u << sl : 0u;
            R[sl] = v ? (h ? recv : acc[sl][0]) : T(0);
            R1[sl] = v ? (h ? acc[sl][1] : recv) : T(0);
            R2[sl] = T(0);
        }
        if constexpr (USER) {  // R'' = M c'' with c'' = -n^2 c: both rows of a body carry it
            T f2[5];
#pragma unroll
            for (int kt = 0; kt < 5; ++kt) {
                const int j = 4 * kt + tq;
                const T n = T(2 * kt + (tq >> 1) + 2);
                f2[kt] = j < 18 ? -(n * n) * own[R_A0 + 1 + j] : T(0);
            }
#pragma unroll
            for (int sl = 0; sl < S; ++sl) acc[sl][0] = acc[sl][1] = 0.0;
#pragma unroll
            for (int kt = 0; kt < 5; ++kt)
#pragma unroll
                for (int sl = 0; sl < S; ++sl) mma_f64(acc[sl], f2[kt], m_at(row0 + 8 * sl, 4 * kt + tq));
#pragma unroll
            for (int sl = 0; sl < S; ++sl)
                if (vmask & (1u << sl)) R2[sl] = h ? acc[sl][1] : acc[sl][0];
        }
    };

    cp_async_wait_group<1>();  // the own records (the neighbour copies may still fly)
    __syncwarp();
    if (ONE) load_row();
    // ---- pass 1: contour integral Q
    T Qp = T(0);
    for (int ch = 0; ch < nch; ++ch) {
        synth(ch);
#pragma unroll
        for (int sl = 0; sl < S; ++sl) {
            // the smallest normal number is lost in any sum but at R = R' = 0: a node
            // beyond the contour, or one where a shape at its bound touches the
            // centre.  There it makes the root of 0 0 to 1e-154, where x times its
            // reciprocal root is 0 times infinity, at no cost (1024 bodies 877 -> 875
            // us a pass; with a mask a node 882 -> 889, with a comparison 885 -> 904)
            const T x2 = fma(R[sl], R[sl], fma(R1[sl], R1[sl], T(2.2250738585072014e-308)));
            Qp = add_rn(Qp, mul_rn(x2, rsqrt_normal(x2)));  // not fused: every launch shape the same bits
        }
    }
    const T Q = group_sum<L>(Qp) * dphi;
    T W, E;
    body_terms(P, ti, Q, r0, dphi, W, E);
    UserBody<T> ub;
    if constexpr (USER) {
        ub.template integrals<L, S>(P, ti, vmask, R, R1, R2, dphi);
        ub.energies(P, ti, r0, dphi, E);
    }

    // what the update needs of the own state alone, while the neighbours' copies arrive
    if (MODE == MODE_FUSED && !kept && l == 0) {
        T so, co;
        t_sincos(own[R_TH], &so, &co);
        scf[NCM] = so;
        scf[NCM + 1] = co;
        scf[NCM + 2] = T(0.5) / scf[0];
    }

    // ---- pass 2: contact pressure, contour gradients, force/torque, pullback
    T fx = T(0), fy = T(0), tt = T(0);
    double pb[3][2], pb2[3][2];  // pullback accumulators (pb2: the R'' rows of user terms)
#pragma unroll
    for (int nt = 0; nt < 3; ++nt) pb[nt][0] = pb[nt][1] = pb2[nt][0] = pb2[nt][1] = 0.0;
    finish_batch(0);
    const bool rewrap = P.rewrap != 0;
    for (int ch = 0; ch < nch; ++ch) {
        if (!ONE) synth(ch);
        const int k0 = ch * 8 * ns;
        if (maxc > 0) {
            {
                T X[S], Y[S];
#pragma unroll
                for (int sl = 0; sl < S; ++sl) {
                    const double2 e = cs_at(vmask & (1u << sl) ? k0 + l + 8 * sl : 0);
                    X[sl] = R[sl] * e.x;
                    Y[sl] = R[sl] * e.y;
                    wx[sl * 32] = X[sl];
                    wy[sl * 32] = Y[sl];
                    wp[sl * 32] = T(0);
                }
                constexpr int QB = 64 / S;  // neighbours per 64-bit hit mask
                static_assert(QB >= NBMAX64, "one hit mask per batch");
                for (int base = 0; base < maxc; base += NBMAX64) {
                    if (base != staged_base) {  // lists longer than the stage: restage
                        stage_batch(base, false);
                        finish_batch(base);
                        staged_base = base;
                    }
                    const int qn = min(cnt - base, NBMAX64);
                    // (1) nodes inside each neighbour's bounding circle (`wrap`: a box of
                    // fewer than 3 cells a side re-images every node)
                    unsigned long long hm = 0;
                    auto test = [&](auto wrap) {
                        for (int q = 0; q < qn; ++q) {
                            const T* r = snb + q * SREC64;
                            const double2 o = *reinterpret_cast<const double2*>(r);
                            const T lim2 = r[R_RMAX];
                            unsigned m = 0;
#pragma unroll
                            for (int sl = 0; sl < S; ++sl) {
                                T dx = X[sl] + o.x, dy = Y[sl] + o.y;
                                if constexpr (decltype(wrap)::value) {
                                    dx = minimum_image_fast(dx, Lx, P.invLx);
                                    dy = minimum_image_fast(dy, Ly, P.invLy);
                                }
                                m |= (dx * dx + dy * dy <= lim2) ? (1u << sl) : 0u;
                            }
                            hm |= (unsigned long long)(m & vmask) << (q * S);
                        }
                    };
                    if (rewrap) test(Flag<true>{});
                    else test(Flag<false>{});
                    // (2) each lane walks its hits in (neighbour, node) order, two at a
                    // time: one is a chain of some 400 cycles, and two overlap
                    while (hm) {
                        int bit[2], sl[2];
                        const T* r[2];
                        T dx[2], dy[2], dd[2], gv[2];
                        bit[0] = __ffsll((long long)hm) - 1;
                        hm &= hm - 1;
                        const bool two = hm != 0;
                        bit[1] = two ? __ffsll((long long)hm) - 1 : bit[0];
                        hm &= hm - 1;
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const int q = bit[i] / S;
                            sl[i] = bit[i] - q * S;
                            r[i] = snb + q * SREC64;
                            const double2 o = *reinterpret_cast<const double2*>(r[i]);
                            dx[i] = wx[sl[i] * 32] + o.x;
                            dy[i] = wy[sl[i] * 32] + o.y;
                        }
                        if (rewrap) {
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                dx[i] = minimum_image_fast(dx[i], Lx, P.invLx);
                                dy[i] = minimum_image_fast(dy[i], Ly, P.invLy);
                            }
                        }
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const T d2 = dx[i] * dx[i] + dy[i] * dy[i];
                            // psi = 0 at u = r_j, like atan(0, 0) (at distances below 2e-154, where d2 is subnormal, too)
                            const bool off = d2 >= T(2.2250738585072014e-308);
                            const T inv = rsqrt_normal(off ? d2 : T(1));
                            const T dist = off ? d2 * inv : T(0);
                            dd[i] = radius_at64(r[i], off ? dx[i] * inv : T(1), off ? dy[i] * inv : T(0)) - dist;
                            // pair coupling of the terms (src/energies/contact.jl:267-293)
                            gv[i] = dd[i] >= T(0) ? r[i][COUPLING] : T(0);
                            gv[i] = dd[i] > T(0) ? fma(cB, dd[i], gv[i]) : gv[i];
                        }
                        if constexpr (USER) {
                            const int wj[2] = {unpack_w(r[0][R_W]), unpack_w(r[1][R_W])};
                            user_pressure(P, dd, ti, wj, pi, gv);
                        }
                        wp[sl[0] * 32] += gv[0];
                        if (two) wp[sl[1] * 32] += gv[1];
                    }
                }
            }
        }
        // contour gradients of node k: GR = W R/q + p dphi R, GD = W R'/q
        T GR[S], GD[S], GDD[S];
#pragma unroll
        for (int sl = 0; sl < S; ++sl) {
            // beyond the contour r = r1 = p = 0: every contribution is zero
            const bool v = vmask & (1u << sl);
            const int k = k0 + l + 8 * sl;
            const T r = R[sl], r1 = R1[sl];
            const T p = maxc > 0 ? wp[sl * 32] : T(0);
            const double2 e = cs_at(v ? k : 0);
            const T iq = rsqrt_normal(v ? r * r + r1 * r1 : T(1));
            const T pw = p * dphi;
            GR[sl] = W * r * iq + pw * r;
            GD[sl] = W * r1 * iq;
            GDD[sl] = T(0);
            fx += pw * (r * e.x + r1 * e.y);
            fy += pw * (r * e.y - r1 * e.x);
            tt += (-pw * r) * r1;
            if (MODE == MODE_DIAG && act && v) d.P[(size_t)g * nth + k] = p;
        }
        if constexpr (USER) ub.gradients(P, ti, vmask, R, R1, R2, GR, GD, GDD);
        if (MODE == MODE_DIAG && act) {
#pragma unroll
            for (int sl = 0; sl < S; ++sl)
                if (vmask & (1u << sl)) {
                    const size_t o = (size_t)g * nth + k0 + l + 8 * sl;
                    d.GR[o] = GR[sl];
                    d.GD[o] = GD[sl];
                    d.GDD[o] = GDD[sl];
                }
        }
        // pullback of the chunk
        const int c = lane >> 2;
#pragma unroll
        for (int sl = 0; sl < S; ++sl) {
            if (!ONE && sl >= ns) continue;
            const T recv = __shfl_xor_sync(FULL, h ? GR[sl] : GD[sl], 4);
            const T a0 = h ? recv : GR[sl], a1 = h ? GD[sl] : recv;
            const int row = k0 + 8 * sl + tq;
            T u0 = T(0), u1 = T(0);
            if constexpr (USER) {
                const T rd = __shfl_xor_sync(FULL, GDD[sl], 4);
                u0 = h ? rd : GDD[sl];
                u1 = h ? GDD[sl] : rd;
            }
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int nt = 0; nt < 3; ++nt) {
                    const int col = 8 * nt + c;
                    const T m = col < M64_COLS ? m_at(row + 4 * e, col) : T(0);
                    mma_f64(pb[nt], e ? a1 : a0, m);
                    if constexpr (USER) mma_f64(pb2[nt], e ? u1 : u0, m);
                }
        }
    }
    // skin reference of the update: under way during the sums
    T x0 = T(0), y0 = T(0), rmax0 = T(0);
    if (LAT && ref) {
        x0 = res->pre.x0, y0 = res->pre.y0, rmax0 = res->pre.rmax0;
    } else if (MODE == MODE_FUSED) {
        x0 = ldcg(d.x0 + gg);
        y0 = ldcg(d.y0 + gg);
        rmax0 = ldcg(d.rmax0 + gg);
        if constexpr (LAT) res->pre.x0 = x0, res->pre.y0 = y0, res->pre.rmax0 = rmax0;
    }
    // ---- mode gradients of the lab frame (/ R0): lane l has those of mode l,
    // lane 0 those of mode 8 too; dE/da0 to every lane of the body
    T gA[MPL], gB[MPL], gl0;
    {
        const T sa = h ? pb[0][0] : pb[1][0], sb = h ? pb[0][1] : pb[1][1];
        const T ra = __shfl_xor_sync(FULL, sa, 4), rb = __shfl_xor_sync(FULL, sb, 4);
        const T r8a = __shfl_xor_sync(FULL, pb[2][0], 4), r8b = __shfl_xor_sync(FULL, pb[2][1], 4);
        const T n = T(l + 2);
        const T va = h ? ra : pb[0][0], vb = h ? rb : pb[0][1];  // (g) of alpha_l, beta_l
        const T ha = h ? pb[1][0] : ra, hb = h ? pb[1][1] : rb;  // (h)
        gA[0] = va - n * hb;
        gB[0] = vb + n * ha;
        gA[1] = pb[2][0] - T(10) * r8b;
        gB[1] = pb[2][1] + T(10) * r8a;
        gl0 = __shfl_sync(FULL, pb[2][0], 1, L);
        if constexpr (USER) {
            const T n2 = n * n;
            gA[0] -= n2 * (h ? pb2[1][0] : pb2[0][0]);
            gB[0] -= n2 * (h ? pb2[1][1] : pb2[0][1]);
            gA[1] -= T(100) * pb2[2][0];
            gB[1] -= T(100) * pb2[2][1];
        }
    }
    fx = group_sum<L>(fx);
    fy = group_sum<L>(fy);
    tt = group_sum<L>(tt);
    if (act) bond_forces<T, USER>(d, P, rc, g, ti, xi, yi, fx, fy);

    if (MODE == MODE_FORCES || MODE == MODE_DIAG) {
        if (act) {
            T* gl = d.glab + (size_t)g * NCM;
            if (l == 0) {
                d.gx[g] = fx;
                d.gy[g] = fy;
                d.gth[g] = tt;
                d.E[g] = E;
                gl[0] = gl0;
                gl[KM] = gA[1];
                gl[2 * KM] = gB[1];
            }
            gl[1 + l] = gA[0];
            gl[1 + KM + l] = gB[0];
        }
        if (MODE == MODE_DIAG && act) {
            // body-frame gradient gcoef (src/gradients.jl:347-362), frame = true
            const T ga0 = r0 * gl0;
            const T h0 = ga0 / (T(2) * scf[0]);
            const T th = own[R_TH];
#pragma unroll
            for (int u = 0; u < MPL; ++u) {
                const int m = l + u * L;
                if (m >= P.K) continue;
                const T ga = gA[u] * r0, gb = gB[u] * r0;
                T so, co;
                t_sincos(T(m + 2) * th, &so, &co);
                d.gcoef[(size_t)g * NCM + 1 + m] = ga * co + gb * so - h0 * scf[1 + m];
                d.gcoef[(size_t)g * NCM + 1 + KM + m] = -ga * so + gb * co - h0 * scf[1 + KM + m];
            }
            if (l == 0) d.gcoef[(size_t)g * NCM] = ga0;
        }
        return;
    }

    // the last step's centre gradients and body energy stay readable
    if (act && l == 0) {
        d.gx[g] = fx;
        d.gy[g] = fy;
        d.gth[g] = tt;
        d.E[g] = E;
    }
    if (valid && !act) carry_record_staged<T, L>(d, g, l, par, own);
    update_body64(d, P, act, g, s, l, par, xi, yi, wf, own[R_TH], r0, ti, fx, fy, tt, gl0, gA, gB, scf, x0, y0, rmax0, fl,
                  nz, rbp, own, scf, LAT && res->on);
}

}  // namespace fcc
