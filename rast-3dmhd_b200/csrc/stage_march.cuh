// stage_march.cuh -- the stage kernel of the FMA build, included by
// stage_impl.cuh: the column march of march.cuh in FP64.
//
// Stage 1 writes no Z: Z = U1 + ZETA1*DT*F1 follows in stage 2 from U1 and the
// state U0 the step began with, which is still in the buffer stage 2 writes
// (a cell is read by the thread that then overwrites it, and by no other).
// That is 64 of the 640 bytes a cell and step, and one rounding less: errors
// against 80-bit arithmetic fall by 13-15 % in every field.  U1-U0 carries the
// rounding of U1, which ZETA1/GAM1 scales: a scheme with |ZETA1| > |GAM1| (the
// reference's ratio is -0.53) would lose by it, up to GAM1 = 0, where U1 holds
// no F1 at all, so it has Z stored by stage 1.
//
// GEN instances (StageArgs.general) are for what the others leave out to stay
// as fast as they are: Z stored by stage 1, and wall values that BCON does not
// rewrite (BZ with IBC not 0, TT on the top wall with ITC=3).  A step by them
// takes 10.08 ms at 512x512x256 against 9.43, 1256 us at 256x256x128 against 1207.
//
// Bound by DRAM traffic in flight (12 warps an SM, two planes in the ring
// beyond the two in use, three in stage 1) together with the latency of a
// plane's instructions (690, 808 and 870 in stages 1, 2, 3 with a magnetic
// field).  Measured at 512x512x256 (ms a step; stages): one plane in flight,
// planes k-1, k, k+1 read for every cell 10.61 (3.18 / 3.58 / 3.79); the march
// 9.76 (2.98 / 3.31 / 3.37); stage 1 without Z, rows on 128-byte lines and
// 32-plane chunks 9.39 (2.62 / 3.24 / 3.39).  At 256x256x128 1581, 1413 and
// 1241 us; 1207 with the chunks that z_chunks now chooses there.
// Tried against the march in one run: 4 CTAs an SM at 128 registers with a
// three-slot ring and one Z slot 1425 us and 10.4 ms; 32x8 tiles, 2 CTAs an
// SM, three slots 1410 us and 10.16 ms, four slots and one Z slot 1529 us and
// 10.8 ms; planes 1, 2, 4 beyond the ring prefetched into L2 10.09, 10.52,
// 11.64 ms against 9.91 (neighbours' halo rows leave L2 earlier).

// 1/x by two Newton-Raphson steps y <- y + y(1 - xy) from the approximate
// reciprocal rcp.approx.ftz.f64 (each step squares the relative error, so
// two reach the rounding level): within an ulp or so of the correctly rounded
// 1/x for the positive normal densities it is used on.  A full
// division of every arriving plane measured 0.1 ms more a step at 512x512x256.
__device__ __forceinline__ double recip(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double e = fma(-x, y, 1.0);
    y = fma(y, e, y);
    e = fma(-x, y, 1.0);
    return fma(y, e, y);
}

constexpr int NZS = 2;   // Z slots (stages 2, 3)
template <bool MAG, int STAGE>
struct Lay {
    static constexpr int NF = MAG ? 8 : 5;
    static constexpr int NR = STAGE >= 2 ? NRAW : NRAW + 1;   // ring slots: stages without Z hold a plane more
    static constexpr int REC = (NF * BSLOT * 8 + 127) / 128 * 128 / 8;   // plane constants behind the fields
    static constexpr int RAW_SLOT = REC + 16;
    static constexpr int ZT = NF * TY * TX;
    static constexpr int RI_OFF = NR * RAW_SLOT;
    static constexpr int Z_OFF = ((RI_OFF + 2 * BSLOT) * 8 + 127) / 128 * 128 / 8;
    static constexpr int BAR_OFF = Z_OFF + (STAGE >= 2 ? NZS : 0) * ZT;
    static constexpr int RED_OFF = BAR_OFF + (NR + NZS + 1) / 2 * 2;   // an mbarrier a slot
    static constexpr int FLAG_OFF = RED_OFF + (NT / 32) * 8;
    static constexpr int TOTAL = FLAG_OFF + 2;
    static constexpr size_t BYTES = (size_t)TOTAL * 8 + 128;
};

// STAGE 0: right-hand side only (written to f_out); STAGE 1..3: the RK3
// substeps of STEP (3dmhdsub.f:874-1169).
template <bool MAG, bool ROT, int STAGE, bool GEN = false>
__global__ void __launch_bounds__(NT, MHD3D_MINB) k_stage(const __grid_constant__ StageArgs a)
{
    using L = Lay<MAG, STAGE>;
    constexpr int NR = L::NR;
    using Mc = March<MAG, ROT, BW, BSLOT>;
    constexpr int NF = L::NF;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    // 128-byte aligned base, formed by pointer arithmetic on the shared array
    // so that every access below stays a shared-window (32-bit) access
    double* const sbase = reinterpret_cast<double*>(smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u));
    double* const sri = sbase + L::RI_OFF;
    double* const sz = sbase + L::Z_OFF;
    unsigned long long* const bars = reinterpret_cast<unsigned long long*>(sbase + L::BAR_OFF);
    unsigned long long* const red = reinterpret_cast<unsigned long long*>(sbase + L::RED_OFF);
    int* const sflag = reinterpret_cast<int*>(sbase + L::FLAG_OFF);

    const Control* ctl = a.ctl;
    const Scalars& s = a.s;
    const Metrics& m = a.m;
    const MarchRun& run = a.run;
    const int npx = s.npx, npy = s.npy, npz = s.npz;
    const int tid = threadIdx.x;
    const int tx = tid % TX, ty = tid / TX;
    const int tile = blockIdx.x;
    const int x0 = (tile % a.ntx) * TX, y0 = (tile / a.ntx) * TY;
    const int chunk = blockIdx.y;
    const int k0 = chunk_start(chunk, npz, a.nchunks), k1 = chunk_start(chunk + 1, npz, a.nchunks);
    const int gi = x0 + tx, gj = y0 + ty;
    const bool active = gi < npx && gj < npy;
    const int o = (ty + 1) * BW + tx + BXO;   // own cell in a plane slot

    grid_wait();   // what follows reads what the kernels before wrote
    const double DT = ctl->dt;
    const double cu = STAGE == 1 ? s.gam1 * DT : STAGE == 2 ? s.gam2 * DT : s.gam3 * DT;
    const double cz = (STAGE == 1 ? s.zeta1 : s.zeta2) * DT;
    const double C13 = s.c13, C23 = s.c23, C43 = s.c43;
    MarchCol col;
    {
        const int i = active ? gi + 1 : 1, j = active ? gj + 1 : 1;
        col.ax = m.fax[i];
        col.xp = m.fbx[i] + m.fcx[i];
        col.xm = m.fbx[i] - m.fcx[i];
        col.ay = m.fay[j];
        col.yp = m.fby[j] + m.fcy[j];
        col.ym = m.fby[j] - m.fcy[j];
    }
    const unsigned raw_bytes = (unsigned)(NF * BSLOT * 8 + sizeof(PlaneZ));
    const unsigned z_bytes = (unsigned)(NF * TY * TX * 8);
    const size_t ucol = (size_t)(gj + 1) * a.upitch + (gi + 1);
    const size_t zcol = (size_t)gj * a.zpitch + gi;
    const HaloCols hc = halo_cols(npx, npy, a.upitch, gi, gj);

    // the stop flag is read once, by one thread, so the CTA takes one path
    if (tid == 0) {
        const bool stopped = STAGE != 0 && ctl->stop;
        *sflag = stopped ? -1 : 0;
        if (!stopped) {
            for (int i = 0; i < NR + NZS; ++i) mbar_init(&bars[i], 1);
            fence_mbar_init();
        }
    }
    if (STAGE == 3 && (tid & 31) == 0) {
        unsigned long long* r = red + (tid >> 5) * 3;
        r[0] = ~0ull;
        r[1] = 0ull;
        r[2] = 0ull;
    }
    if (STAGE == 3) cfl_screen_init(red, a.acc, a.s, MAG);
    __syncthreads();
    if (*sflag < 0) return;

    // plane q (-1 .. npz) is fill n = q-(k0-1) of the CTA: raw slot n % NR,
    // 1/RO slot n & 1; the plane's constants arrive with it
    int hi_issued = k0 - 2;
    auto issue_plane = [&](int q) {
        const int sl = (q - (k0 - 1)) % NR;
        fence_proxy_async();
        mbar_expect_tx(&bars[sl], raw_bytes);
        tma_load4(sbase + (size_t)sl * L::RAW_SLOT, &a.map_u, &bars[sl], x0 + BX0, y0, q + 1, 0);
        bulk_load(sbase + (size_t)sl * L::RAW_SLOT + L::REC, a.pz + (q + 1), (unsigned)sizeof(PlaneZ), &bars[sl]);
        hi_issued = q;
    };
    auto wait_plane = [&](int q, long limit) -> bool {
        const int n = q - (k0 - 1);
        return mbar_wait(&bars[n % NR], (unsigned)(n / NR) & 1u, limit);
    };
    auto derive_ri = [&](int q) {
        const int n = q - (k0 - 1);
        const double* r = sbase + (size_t)(n % NR) * L::RAW_SLOT + F_RO * BSLOT;
        double* d = sri + (size_t)(n & 1) * BSLOT;
        for (int p = tid; p < BSLOT; p += NT) d[p] = recip(r[p]);
    };
    int z_hi = k0 - 1;
    auto issue_z = [&](int k) {
        const int zs = (k - k0) % NZS;
        fence_proxy_async();
        mbar_expect_tx(&bars[NR + zs], z_bytes);
        // stage 2: the state the step began with, still in the output buffer
        if (STAGE == 2 && !GEN) tma_load4(sz + (size_t)zs * L::ZT, &a.map_o, &bars[NR + zs], x0 + UOFS + 1, y0 + 1, k + 1, 0);
        else tma_load4(sz + (size_t)zs * L::ZT, &a.map_z, &bars[NR + zs], x0, y0, k, 0);
        z_hi = k;
    };
    auto wait_z = [&](int k) -> bool {
        return mbar_wait(&bars[NR + (k - k0) % NZS], (unsigned)(((k - k0) / NZS) & 1));
    };
    if (tid == 0) {
        for (int q = k0 - 1; q <= k0 - 2 + NR && q <= k1; ++q) issue_plane(q);
        if (STAGE >= 2) {
            for (int k = k0; k < k0 + NZS && k < k1; ++k) issue_z(k);
        }
    }
    if (wait_plane(k0 - 1, (long)a.wait_first)) derive_ri(k0 - 1);
    else atomicOr(sflag, 1);
    __syncthreads();

    CflAcc cfa;
    const CflCol ccol = cfl_col(m, gi, gj, active);
    Mc c;
    bool zok = true;
    if (!*sflag) {
        int slot = 0, pslot = NR - 1;   // of planes q and q-1
#pragma unroll 1
        for (int q = k0 - 1; q <= k1; ++q) {
            const double* const raw = sbase + (size_t)slot * L::RAW_SLOT;
            const double* const rip = sri + (size_t)((q - (k0 - 1)) & 1) * BSLOT;
            const double* const rawk = sbase + (size_t)pslot * L::RAW_SLOT;
            const int k = q - 1;   // the plane this arrival completes
            if (active) {
                const PlaneZ& zq = *reinterpret_cast<const PlaneZ*>(raw + L::REC);
                const PlaneZ& zk = *reinterpret_cast<const PlaneZ*>(rawk + L::REC);
                c.arrive(raw, rip, o, col);
                if (q > k0) {
                    c.cell(raw, rip, o);
                    c.recall(rawk, o);
                    const bool top = (k == 0), bot = (k == npz - 1), wall = top || bot;
                    const double ghost = c.nri;
                    double l1 = 0.0, l2 = 0.0;
                    if (bot) {
                        // own column one, two and three planes inside the wall
                        const double* u = a.u_in + ucol + (size_t)(npz - 1) * a.uz;
                        const double* u2 = u - a.uz;
                        const double rwm = u[F_RW * a.uf], rw2 = u2[F_RW * a.uf];
                        c.nrw = rw2 - 3.0 * rwm;
                        c.nw = rw2 * (1.0 / u2[F_RO * a.uf]) - 3.0 * (rwm * (1.0 / u[F_RO * a.uf]));
                        if (MAG) {
                            const double* u3 = u2 - a.uz;
                            l1 = Mc::wall_d2(zk, -1.0, c.bx, u[F_BX * a.uf], u2[F_BX * a.uf], u3[F_BX * a.uf]);
                            l2 = Mc::wall_d2(zk, -1.0, c.by, u[F_BY * a.uf], u2[F_BY * a.uf], u3[F_BY * a.uf]);
                        }
                    }
                    c.complete(zk, run, bot, l1, l2);
                    const size_t zc = (size_t)k * a.zz + zcol;
                    if (STAGE != 0 && bot)
                        store_cell<1>(a.u_out + (size_t)(npz + 1) * a.uz, a.uf, ucol, hc, {F_RO}, {ghost});
                    if (GEN && top) {
                        // FT's dw/dz is central on the wall, with the ghost plane
                        const double* g = a.u_in + ucol;
                        const double wz = (c.nw - g[F_RW * a.uf] * (1.0 / g[F_RO * a.uf])) * zk.az;
                        c.ft += c.ri * run.tmpa * run.c43 * (wz * (wz - c.s) - c.wz * (c.wz - c.s))
                              - run.ocv * c.tt * (wz - c.wz);
                    }
                    if (STAGE == 0) {
                        a.f_out[zc + 0 * a.zf] = wall ? 0.0 : c.fu;
                        a.f_out[zc + 1 * a.zf] = wall ? 0.0 : c.fv;
                        a.f_out[zc + 2 * a.zf] = wall ? 0.0 : c.fw;
                        a.f_out[zc + 3 * a.zf] = c.fr;
                        a.f_out[zc + 4 * a.zf] = wall ? 0.0 : c.ft;
                        if (MAG) {
                            a.f_out[zc + 5 * a.zf] = c.w1;
                            a.f_out[zc + 6 * a.zf] = c.w2;
                            a.f_out[zc + 7 * a.zf] = wall ? 0.0 : c.w3;
                        }
                    } else {
                        // RK3 update: U = Z + COEF*F (stage 1: Z = U)
                        double zu, zv, zw, zr, zt, zbx = 0, zby = 0, zbz = 0;
                        if (STAGE == 1) {
                            zu = c.ru; zv = c.rv; zw = c.rw; zr = c.ro; zt = c.tt;
                            if (MAG) { zbx = c.bx; zby = c.by; zbz = c.bz; }
                        } else {
                            zok = wait_z(k);
                            const double* zt_ = sz + (size_t)((k - k0) % NZS) * L::ZT + tid;
                            zu = zt_[F_RU * NT];
                            zv = zt_[F_RV * NT];
                            zw = zt_[F_RW * NT];
                            zt = zt_[F_TT * NT];
                            zr = zt_[F_RO * NT];
                            if (MAG) {
                                zbx = zt_[F_BX * NT];
                                zby = zt_[F_BY * NT];
                                zbz = zt_[F_BZ * NT];
                            }
                            if (STAGE == 2 && !GEN) {
                                // Z = U1 + ZETA1*DT*F1 with GAM1*DT*F1 = U1 - U0
                                zu = fma(s.zr10, c.ru - zu, c.ru);
                                zv = fma(s.zr10, c.rv - zv, c.rv);
                                zw = fma(s.zr10, c.rw - zw, c.rw);
                                zt = fma(s.zr10, c.tt - zt, c.tt);
                                zr = fma(s.zr10, c.ro - zr, c.ro);
                                if (MAG) {
                                    zbx = fma(s.zr10, c.bx - zbx, c.bx);
                                    zby = fma(s.zr10, c.by - zby, c.by);
                                    zbz = fma(s.zr10, c.bz - zbz, c.bz);
                                }
                            }
                        }
                        const double nu = zu + cu * c.fu, nv = zv + cu * c.fv, nw = zw + cu * c.fw;
                        const double nr = zr + cu * c.fr, nt = zt + cu * c.ft;
                        const double nbx = zbx + cu * c.w1, nby = zby + cu * c.w2, nbz = zbz + cu * c.w3;
                        const int kz = k + 1;
                        if (zok) {
                            // on the walls RU, RV, RW, TT, BZ are rewritten by BCON below
                            double* const pl = a.u_out + (size_t)kz * a.uz;
                            if (MAG)
                                store_cell<8>(pl, a.uf, ucol, hc, {F_RO, F_BX, F_BY, F_RU, F_RV, F_RW, F_TT, F_BZ},
                                              {nr, nbx, nby, nu, nv, nw, nt, nbz});
                            else
                                store_cell<5>(pl, a.uf, ucol, hc, {F_RO, F_RU, F_RV, F_RW, F_TT}, {nr, nu, nv, nw, nt});
                            // Z for the next stage: Z = U + ZETA*DT*F; on the walls only RO, BX,
                            // BY, and what else BCON does not rewrite (GEN)
                            if (STAGE == 2 || (STAGE == 1 && GEN)) {
                                double* zo = a.z + zc;
                                zo[F_RO * a.zf] = nr + cz * c.fr;
                                if (MAG) {
                                    zo[F_BX * a.zf] = nbx + cz * c.w1;
                                    zo[F_BY * a.zf] = nby + cz * c.w2;
                                }
                                if (!wall || GEN) {
                                    zo[F_RU * a.zf] = nu + cz * c.fu;
                                    zo[F_RV * a.zf] = nv + cz * c.fv;
                                    zo[F_RW * a.zf] = nw + cz * c.fw;
                                    zo[F_TT * a.zf] = nt + cz * c.ft;
                                    if (MAG) zo[F_BZ * a.zf] = nbz + cz * c.w3;
                                }
                            }
                        }
                        // BCON (3dmhdsub.f:2751-2955) and the CFL parts of the next step
                        if (!wall && STAGE == 3)
                            cfl_acc_cell<MAG>(cfa, s, m, cfl_screen_of(red), ccol, gi, gj, k, nu, nv, nw, nr, nt, nbx, nby, nbz);
                        if (k == 2 && k0 == 0) {
                            // top wall: new values of planes K=3 (read back) and K=4 (this plane);
                            // this thread wrote planes K=2 and K=3 of u_out itself
                            const double* ub = a.u_out + ucol;
                            const size_t c0 = 1 * a.uz, c1 = 2 * a.uz;
                            const double h1_ru = ub[F_RU * a.uf + c1], h1_rv = ub[F_RV * a.uf + c1];
                            const double h1_ro = ub[F_RO * a.uf + c1], h1_tt = ub[F_TT * a.uf + c1];
                            const double w0_ro = ub[F_RO * a.uf + c0], w0_tt = ub[F_TT * a.uf + c0];
                            const double w0_bx = MAG ? ub[F_BX * a.uf + c0] : 0.0, w0_by = MAG ? ub[F_BY * a.uf + c0] : 0.0;
                            const double w0_bz = MAG ? ub[F_BZ * a.uf + c0] : 0.0;
                            const double ru_w = w0_ro * (C43 * h1_ru / h1_ro - C13 * nu / nr);
                            const double rv_w = w0_ro * (C43 * h1_rv / h1_ro - C13 * nv / nr);
                            double tt_w = w0_tt;
                            if (s.plume) {
                                const double tpr = (s.tc != 0.0) ? s.tp + (1.0 - s.tp) * exp(-ctl->timt / s.tc) : s.tp;
                                const double gx = m.plume_gx[gi + 1], gy = m.plume_gy[gj + 1];
                                if (s.itcon == 0) tt_w = 1.0 - (1.0 - tpr) * gx / s.hh * gy / s.hh;
                                else tt_w = C43 * h1_tt - C13 * nt - C23 * s.top_dz * (s.theta - (s.theta - tpr) * gx / s.hh * gy / s.hh);
                            } else if (s.itcon == 0 || s.itcon == 2 || s.itcon == 4) {
                                tt_w = 1.0;
                                if (s.itcon == 4 && gi + 2 <= (npx + 2) / 2) tt_w = 1.0 - s.tp;
                            } else if (s.itcon == 1) {
                                tt_w = C43 * h1_tt - C13 * nt - s.top_flux;
                            }
                            const double bz_w = (MAG && s.ibcon == 0) ? 0.0 : w0_bz;
                            if (zok) {
                                double* const pl = a.u_out + a.uz;
                                if (MAG)
                                    store_cell<5>(pl, a.uf, ucol, hc, {F_RU, F_RV, F_RW, F_TT, F_BZ}, {ru_w, rv_w, 0.0, tt_w, bz_w});
                                else
                                    store_cell<4>(pl, a.uf, ucol, hc, {F_RU, F_RV, F_RW, F_TT}, {ru_w, rv_w, 0.0, tt_w});
                            }
                            if (STAGE == 3)
                                cfl_acc_direct<MAG>(cfa, s, m, cfl_screen_of(red), ccol, gi, gj, 0, ru_w, rv_w, 0.0, w0_ro, tt_w, w0_bx, w0_by, bz_w);
                        }
                        if (bot) {
                            // bottom wall: new values of planes K=NZ-2 and K=NZ-3, read back
                            const double* ub = a.u_out + ucol;
                            const size_t c1 = (size_t)(npz - 1) * a.uz, c2 = (size_t)(npz - 2) * a.uz;
                            const double h1_ru = ub[F_RU * a.uf + c1], h1_rv = ub[F_RV * a.uf + c1];
                            const double h1_ro = ub[F_RO * a.uf + c1], h1_tt = ub[F_TT * a.uf + c1];
                            const double h2_ru = ub[F_RU * a.uf + c2], h2_rv = ub[F_RV * a.uf + c2];
                            const double h2_ro = ub[F_RO * a.uf + c2], h2_tt = ub[F_TT * a.uf + c2];
                            const double ru_w = nr * (C43 * h1_ru / h1_ro - C13 * h2_ru / h2_ro);
                            const double rv_w = nr * (C43 * h1_rv / h1_ro - C13 * h2_rv / h2_ro);
                            const double tt_w = (s.izcon == 0) ? s.tb : C43 * h1_tt - C13 * h2_tt + s.bot_flux;
                            const double bz_w = (MAG && s.ibcon == 0) ? 0.0 : nbz;
                            if (zok) {
                                double* const pl = a.u_out + (size_t)kz * a.uz;
                                if (MAG)
                                    store_cell<5>(pl, a.uf, ucol, hc, {F_RU, F_RV, F_RW, F_TT, F_BZ}, {ru_w, rv_w, 0.0, tt_w, bz_w});
                                else
                                    store_cell<4>(pl, a.uf, ucol, hc, {F_RU, F_RV, F_RW, F_TT}, {ru_w, rv_w, 0.0, tt_w});
                            }
                            if (STAGE == 3) cfl_acc_cell<MAG>(cfa, s, m, cfl_screen_of(red), ccol, gi, gj, k, ru_w, rv_w, 0.0, nr, tt_w, nbx, nby, bz_w);
                        }
                    }
                }
                if (q >= k0 && q < k1) {
                    const bool top = (q == 0);
                    double l1 = 0.0, l2 = 0.0, rwt = 0.0, wt = 0.0;
                    asm volatile("" ::: "memory");
                    if (top) {
                        // ghost RO plane: FLUXES leaves 1/RO behind (3dmhdsub.f:1386-1391)
                        if (STAGE != 0) store_cell<1>(a.u_out, a.uf, ucol, hc, {F_RO}, {c.ri});
                        const double* u = a.u_in + ucol + 2 * a.uz;
                        const double* u2 = u + a.uz;
                        const double rwp = u[F_RW * a.uf], rw2 = u2[F_RW * a.uf];
                        rwt = rw2 - 3.0 * rwp;
                        wt = rw2 * (1.0 / u2[F_RO * a.uf]) - 3.0 * (rwp * (1.0 / u[F_RO * a.uf]));
                        if (MAG) {
                            const double* u3 = u2 + a.uz;
                            l1 = Mc::wall_d2(zq, 1.0, raw[F_BX * BSLOT + o], u[F_BX * a.uf], u2[F_BX * a.uf], u3[F_BX * a.uf]);
                            l2 = Mc::wall_d2(zq, 1.0, raw[F_BY * BSLOT + o], u[F_BY * a.uf], u2[F_BY * a.uf], u3[F_BY * a.uf]);
                        }
                    }
                    c.begin(raw, rip, o, zq, rawk, col, run, top, rwt, wt, l1, l2);
                }
                c.shift(rip[o]);
            } else if (STAGE >= 2 && q > k0) {
                // columns outside the domain still see the Z fill of this plane land
                zok = wait_z(k);
            }
            if (!zok) atomicOr(sflag, 1);
            if (STAGE == 3 && q > k0) cfl_fold_plane(red, cfa, 0.0, s);
            if (q < k1) {
                if (wait_plane(q + 1, WAIT_LIMIT)) derive_ri(q + 1);
                else atomicOr(sflag, 1);
            }
            __syncthreads();
            if (*sflag) break;
            // the slot of plane q-1 and, from q = k0+1 on, the Z slot of plane q-1 are free
            if (tid == 0) {
                if (q >= k0 && q - 1 + NR <= k1) issue_plane(q - 1 + NR);
                if (STAGE >= 2 && q > k0 && q - 1 + NZS < k1) issue_z(q - 1 + NZS);
            }
            pslot = slot;
            slot = slot + 1 == NR ? 0 : slot + 1;
        }
    }
    if (*sflag) {
        // a bounded wait gave up: let every fill still in flight land (again
        // bounded), report, and leave without touching the reduction
        if (tid == 0) {
            for (int q = hi_issued - (NR - 1); q <= hi_issued; ++q)
                if (q >= k0 - 1) wait_plane(q, WAIT_LIMIT);
            for (int k = z_hi - (NZS - 1); k <= z_hi; ++k)
                if (k >= k0) wait_z(k);
            atomicExch(&a.ctl->status, MHD3D_ERR_TIMEOUT);
            atomicExch(&a.ctl->stop, 1);
        }
        return;
    }
    if (STAGE == 3) {
        cfl_commit_acc(a.acc, red, cfa);
        if (tid == 0) step_end(a);
    }
}
