// march.cuh -- the right-hand side of FLUXES (3dmhdsub.f:1249-2634) for a
// column that marches down z.
//
// When plane q arrives in shared memory, the thread forms every x and y
// difference of its cell there and keeps in registers what the plane's
// right-hand side still lacks, the z differences.  Those are linear in the
// planes above and below, or squares of sums that start with the plane above:
//   arrive()    the gradients of plane q that plane q-1 needs
//   complete()  plane q-1 gets its terms from plane q and is complete
//   begin()     plane q's x, y terms and its terms from plane q-1
// Planes q-1 (own cell only) and q are in use, the other ring slots in flight.
// The cells of both planes are read again by begin(): holding them across the
// update and stores of plane q-1 spilled registers and cost 20 % in stage 1.
//
// Second differences are sums of first differences weighted b+c and b-c (b, c
// the metric factors of (f+ - f-) and (f+ + f- - 2f)): neighbours of a smooth
// field subtract almost exactly, so this rounds no worse than f+ + f- - 2f.
// The pressure gradient meets gravity in complete(), both at once: either one
// in the carried sum would have every small term rounded at its size.  The
// rounded P of plane q-1 cancels between its two differences.
#pragma once
#include "mhd3d_dev.cuh"

namespace mhd3d {

// per-column constants: HX*DXXDX, and HX*D2XXDX2 +- H2X*DXXDX**2, likewise y
struct MarchCol {
    double ax, xp, xm, ay, yp, ym;
};

// BWV, BS: row length and field size of a plane slot in shared memory.
template <bool MAG, bool ROT, int BWV, int BS>
struct March {
    // plane q-1: its cell, read again from its slot
    double ru, rv, rw, tt, ro, p, u, v, w;
    double bx, by, bz;
    // carried between arrivals for plane q-1
    double ri;
    double wx, wy, s;                                 // dw/dx, dw/dy, du/dx + dv/dy
    double fu, fv, fw, fr, ft, heat, w1, w2, w3;      // what its right-hand side holds so far
    double exz, eyz, wz, jx, jy;                      // du/dz + dw/dx, dv/dz + dw/dy, dw/dz, currents: without plane q
    double dp;                                        // pressure less that of the plane above
    // plane q
    double nru, nrv, nrw, ntt, nro, nri, nu, nv, nw, np, nbx, nby, nbz;
    double nwx, nwy, ns;

    static __device__ __forceinline__ double ld(const double* __restrict__ raw, int f, int off)
    {
        return raw[f * BS + off];
    }
    // the pressure, a product rounded by itself (never part of an FMA)
    static __device__ __forceinline__ double pres(double ro_, double tt_) { return __dmul_rn(ro_, tt_); }
    // difference of two pressures of a plane
    static __device__ __forceinline__ double dpres(double rop, double tp, double rom, double tm)
    {
        return fma(rop, tp, -pres(rom, tm));
    }

    // the cell of plane q
    __device__ __forceinline__ void cell(const double* __restrict__ raw, const double* __restrict__ rip, int o)
    {
        nru = ld(raw, F_RU, o);
        nrv = ld(raw, F_RV, o);
        nrw = ld(raw, F_RW, o);
        ntt = ld(raw, F_TT, o);
        nro = ld(raw, F_RO, o);
        nri = rip[o];
        if (MAG) {
            nbx = ld(raw, F_BX, o);
            nby = ld(raw, F_BY, o);
            nbz = ld(raw, F_BZ, o);
        }
        nu = nru * nri;
        nv = nrv * nri;
        nw = nrw * nri;
        np = pres(nro, ntt);
    }

    __device__ __forceinline__ void arrive(const double* __restrict__ raw, const double* __restrict__ rip, int o,
                                           const MarchCol& c)
    {
        const double rxp = rip[o + 1], rxm = rip[o - 1], ryp = rip[o + BWV], rym = rip[o - BWV];
        nwx = fma(ld(raw, F_RW, o + 1), rxp, -ld(raw, F_RW, o - 1) * rxm) * c.ax;
        nwy = fma(ld(raw, F_RW, o + BWV), ryp, -ld(raw, F_RW, o - BWV) * rym) * c.ay;
        ns = fma(fma(ld(raw, F_RU, o + 1), rxp, -ld(raw, F_RU, o - 1) * rxm), c.ax,
                     fma(ld(raw, F_RV, o + BWV), ryp, -ld(raw, F_RV, o - BWV) * rym) * c.ay);
    }

    // plane q-1's terms from plane q (z: the constants of plane q-1).  bot: it
    // is the bottom wall, whose d2BX/dz2, d2BY/dz2 are one-sided (l1, l2).
    __device__ __forceinline__ void complete(const PlaneZ& z, const MarchRun& r, bool bot, double l1, double l2)
    {
        const double du = nu - u, dv = nv - v, dw = nw - w, dt = ntt - tt;
        fr = fma(rw - nrw, z.az, fr);
        fu = fma(-nru * nw, z.az, fu);
        fv = fma(-nrv * nw, z.az, fv);
        fw = fma(fma(rw, w, -nrw * nw), z.az, fw);
        fu = fma(z.ozp, du, fma(z.t13az, nwx, fu));
        fv = fma(z.ozp, dv, fma(z.t13az, nwy, fv));
        fw = fma(z.ozp, r.c43 * dw, fma(z.t13az, ns, fw));
        fw = fma(r.grav, ro, fma(-(dp + fma(nro, ntt, -p)), z.az, fw));
        exz = fma(du, z.az, exz);
        eyz = fma(dv, z.az, eyz);
        wz = fma(dw, z.az, wz);
        ft = fma(dt, fma(ri * r.tmpc, z.kzp, -w * z.az), ft);
        ft = fma(-r.ocv * tt, wz, ft);
        heat = fma(r.tmpa, fma(exz, exz, fma(eyz, eyz, r.c43 * (wz * (wz - s)))), heat);
        if (MAG) {
            const double dbx = nbx - bx, dby = nby - by, dbz = nbz - bz;
            jy = fma(dbx, z.az, jy);
            jx = fma(dby, z.az, jx);
            w1 += bot ? l1 : z.mzp * dbx;
            w2 += bot ? l2 : z.mzp * dby;
            w1 = fma(bz, exz, fma(-bx, wz, fma(-w, jy, w1)));
            w2 = fma(bz, eyz, fma(-by, wz, fma(-w, jx, w2)));
            w3 = fma(dbz, fma(-w, z.az, z.mzp), w3);
            const double oy = r.obeta * jy, ox = r.obeta * jx;
            fu = fma(bz, oy, fu);
            fv = fma(bz, ox, fv);
            fw -= fma(bx, oy, by * ox);
            heat = fma(r.tmpm, fma(jx, jx, jy * jy), heat);
        }
        ft = fma(ri, heat, ft);
    }

    // plane q's x, y terms and its terms from plane q-1 (z: the constants of
    // plane q).  top: it is the top wall, as in complete().
    __device__ __forceinline__ void begin(const double* __restrict__ raw, const double* __restrict__ rip, int o,
                                          const PlaneZ& z, const double* __restrict__ rawk, const MarchCol& c,
                                          const MarchRun& r, bool top, double rwt, double wt, double l1, double l2)
    {
        cell(raw, rip, o);
        recall(rawk, o);
        if (top) {   // one-sided dRW/dz, dw/dz
            rw = rwt;
            w = wt;
        }
        const double du = nu - u, dv = nv - v, dw = nw - w, dt = ntt - tt;
        double gu, gv, gw, gr, gt, gh;
        // terms from the plane above, and dw/dz, strain and current sums that start with it
        gr = (rw - nrw) * z.az;
        gu = fma(ru * w, z.az, fma(z.ozm, du, -z.t13az * wx));
        gv = fma(rv * w, z.az, fma(z.ozm, dv, -z.t13az * wy));
        dp = np - p;
        gw = fma(fma(rw, w, -nrw * nw), z.az, fma(z.ozm, r.c43 * dw, -z.t13az * s));
        const double q = nri * r.tmpc;
        gt = dt * fma(q, z.kzm, -nw * z.az);
        exz = fma(du, z.az, nwx);
        eyz = fma(dv, z.az, nwy);
        wz = dw * z.az;
        gt = fma(-r.ocv * ntt, ns, gt);
        if (ROT) {
            gu = fma(r.omz, nrv, gu);
            gv = fma(r.omx, nrw, fma(-r.omz, nru, gv));
            gw = fma(-r.omx, nrv, gw);
        }
        double lt;   // x, y part of the Laplacian of T
        double vx, ux;
        {   // x
            const double rxp = rip[o + 1], rxm = rip[o - 1];
            const double rup = ld(raw, F_RU, o + 1), rum = ld(raw, F_RU, o - 1);
            const double rvp = ld(raw, F_RV, o + 1), rvm = ld(raw, F_RV, o - 1);
            const double rwp = ld(raw, F_RW, o + 1), rwm = ld(raw, F_RW, o - 1);
            const double tp = ld(raw, F_TT, o + 1), tm = ld(raw, F_TT, o - 1);
            const double dpx = dpres(ld(raw, F_RO, o + 1), tp, ld(raw, F_RO, o - 1), tm);
            const double vp = rvp * rxp, vm = rvm * rxm, uxp = rup * rxp, uxm = rum * rxm;
            const double wxp = rwp * rxp, wxm = rwm * rxm;
            gr = fma(-(rup - rum), c.ax, gr);
            gu = fma(-fma(rup, uxp, fma(-rum, uxm, dpx)), c.ax, gu);
            gv = fma(-fma(rvp, uxp, -rvm * uxm), c.ax, gv);
            gw = fma(-fma(rwp, uxp, -rwm * uxm), c.ax, gw);
            gu = fma(r.ore43, fma(uxp - nu, c.xp, (nu - uxm) * c.xm), gu);
            gv = fma(r.ore, fma(vp - nv, c.xp, (nv - vm) * c.xm), gv);
            gw = fma(r.ore, fma(wxp - nw, c.xp, (nw - wxm) * c.xm), gw);
            gt = fma(-nu, (tp - tm) * c.ax, gt);
            lt = fma(tp - ntt, c.xp, (ntt - tm) * c.xm);
            ux = (uxp - uxm) * c.ax;
            vx = (vp - vm) * c.ax;
        }
        double uy, vy;
        {   // y
            const double ryp = rip[o + BWV], rym = rip[o - BWV];
            const double rup = ld(raw, F_RU, o + BWV), rum = ld(raw, F_RU, o - BWV);
            const double rvp = ld(raw, F_RV, o + BWV), rvm = ld(raw, F_RV, o - BWV);
            const double rwp = ld(raw, F_RW, o + BWV), rwm = ld(raw, F_RW, o - BWV);
            const double tp = ld(raw, F_TT, o + BWV), tm = ld(raw, F_TT, o - BWV);
            const double dpy = dpres(ld(raw, F_RO, o + BWV), tp, ld(raw, F_RO, o - BWV), tm);
            const double up = rup * ryp, um = rum * rym, vyp = rvp * ryp, vym = rvm * rym;
            const double wyp = rwp * ryp, wym = rwm * rym;
            gr = fma(-(rvp - rvm), c.ay, gr);
            gu = fma(-fma(rup, vyp, -rum * vym), c.ay, gu);
            gv = fma(-fma(rvp, vyp, fma(-rvm, vym, dpy)), c.ay, gv);
            gw = fma(-fma(rwp, vyp, -rwm * vym), c.ay, gw);
            gu = fma(r.ore, fma(up - nu, c.yp, (nu - um) * c.ym), gu);
            gv = fma(r.ore43, fma(vyp - nv, c.yp, (nv - vym) * c.ym), gv);
            gw = fma(r.ore, fma(wyp - nw, c.yp, (nw - wym) * c.ym), gw);
            gt = fma(-nv, (tp - tm) * c.ay, gt);
            lt += fma(tp - ntt, c.yp, (ntt - tm) * c.ym);
            uy = (up - um) * c.ay;
            vy = (vyp - vym) * c.ay;
        }
        gt = fma(q * z.rka, lt, gt);
        {   // corners: d2v/dxdy, d2u/dxdy
            const double rpp = rip[o + BWV + 1], rmp = rip[o + BWV - 1], rpm = rip[o - BWV + 1], rmm = rip[o - BWV - 1];
            const double sxy = r.t13 * (c.ax * c.ay);
            const double vv = fma(ld(raw, F_RV, o + BWV + 1), rpp, -ld(raw, F_RV, o + BWV - 1) * rmp)
                       - fma(ld(raw, F_RV, o - BWV + 1), rpm, -ld(raw, F_RV, o - BWV - 1) * rmm);
            const double uu = fma(ld(raw, F_RU, o + BWV + 1), rpp, -ld(raw, F_RU, o + BWV - 1) * rmp)
                       - fma(ld(raw, F_RU, o - BWV + 1), rpm, -ld(raw, F_RU, o - BWV - 1) * rmm);
            gu = fma(sxy, vv, gu);
            gv = fma(sxy, uu, gv);
        }
        {
            const double e = uy + vx;
            gh = r.tmpa * fma(e, e, r.c43 * fma(ns, ns, -3.0 * ux * vy));
        }
        if (MAG) {
            const double dbx = nbx - bx, dby = nby - by, dbz = nbz - bz;
            double g1 = top ? l1 : z.mzm * dbx, g2 = top ? l2 : z.mzm * dby, g3 = dbz * fma(-nw, z.az, z.mzm);
            double cy = dbx * z.az, cx = dby * z.az;   // currents without d/dx BZ, d/dy BZ
            double lx, jz;
            {   // x
                const double b1p = ld(raw, F_BX, o + 1), b1m = ld(raw, F_BX, o - 1);
                const double b2p = ld(raw, F_BY, o + 1), b2m = ld(raw, F_BY, o - 1);
                const double b3p = ld(raw, F_BZ, o + 1), b3m = ld(raw, F_BZ, o - 1);
                const double d2 = (b2p - b2m) * c.ax, d3 = (b3p - b3m) * c.ax;
                lx = fma(b1p - nbx, c.xp, (nbx - b1m) * c.xm);
                g1 = fma(r.orm, lx, fma(-nu, (b1p - b1m) * c.ax, g1));
                lx = fma(b2p - nby, c.xp, (nby - b2m) * c.xm);
                g2 = fma(r.orm, lx, fma(-nu, d2, g2));
                lx = fma(b3p - nbz, c.xp, (nbz - b3m) * c.xm);
                g3 = fma(r.orm, lx, fma(-nu, d3, g3));
                g1 = fma(-nw, d3, g1);
                cy -= d3;
                jz = -d2;
            }
            {   // y
                const double b1p = ld(raw, F_BX, o + BWV), b1m = ld(raw, F_BX, o - BWV);
                const double b2p = ld(raw, F_BY, o + BWV), b2m = ld(raw, F_BY, o - BWV);
                const double b3p = ld(raw, F_BZ, o + BWV), b3m = ld(raw, F_BZ, o - BWV);
                const double d1 = (b1p - b1m) * c.ay, d3 = (b3p - b3m) * c.ay;
                lx = fma(b1p - nbx, c.yp, (nbx - b1m) * c.ym);
                g1 = fma(r.orm, lx, fma(-nv, d1, g1));
                lx = fma(b2p - nby, c.yp, (nby - b2m) * c.ym);
                g2 = fma(r.orm, lx, fma(-nv, (b2p - b2m) * c.ay, g2));
                lx = fma(b3p - nbz, c.yp, (nbz - b3m) * c.ym);
                g3 = fma(r.orm, lx, fma(-nv, d3, g3));
                g2 = fma(-nw, d3, g2);
                cx -= d3;
                jz += d1;
            }
            g1 = fma(nby, uy, fma(-nbx, vy, fma(-nbz, nwx, g1)));
            g2 = fma(nbx, vx, fma(-nby, ux, fma(-nbz, nwy, g2)));
            g3 = fma(nbx, nwx, fma(nby, nwy, fma(-nbz, ns, g3)));
            const double oz = r.obeta * jz;
            gu = fma(nby, oz, gu);
            gv = fma(-nbx, oz, gv);
            gh = fma(r.tmpm * jz, jz, gh);
            w1 = g1;
            w2 = g2;
            w3 = g3;
            jx = cx;
            jy = cy;
        }
        fu = gu;
        fv = gv;
        fw = gw;
        fr = gr;
        ft = gt;
        heat = gh;
    }

    // one-sided d2B/dz2 on a wall (3dmhdsub.f:1510-1513 and the like) without the
    // part the march adds for the neighbour inside: b0 the wall, b1..b3 the
    // planes inside it, sg +1 on the top wall, -1 on the bottom wall
    static __device__ __forceinline__ double wall_d2(const PlaneZ& z, double sg, double b0, double b1, double b2,
                                                     double b3)
    {
        const double B = sg * (0.5 * (z.mzp + z.mzm)), C = 0.5 * (z.mzp - z.mzm);
        const double d1 = b1 - b0, d2 = b2 - b1, d3 = b3 - b2;
        return fma(2.0 * d1 - d2, B, (3.0 * (d2 - d1) - d3) * C);
    }

    // the cell of plane q-1, from its slot
    __device__ __forceinline__ void recall(const double* __restrict__ raw, int o)
    {
        ru = ld(raw, F_RU, o);
        rv = ld(raw, F_RV, o);
        rw = ld(raw, F_RW, o);
        tt = ld(raw, F_TT, o);
        ro = ld(raw, F_RO, o);
        if (MAG) {
            bx = ld(raw, F_BX, o);
            by = ld(raw, F_BY, o);
            bz = ld(raw, F_BZ, o);
        }
        u = ru * ri;
        v = rv * ri;
        w = rw * ri;
        p = pres(ro, tt);
    }

    // plane q becomes the carried plane (rq: its 1/RO)
    __device__ __forceinline__ void shift(double rq)
    {
        ri = rq;
        wx = nwx;
        wy = nwy;
        s = ns;
    }
};

}  // namespace mhd3d
