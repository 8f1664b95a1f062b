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
template <typename T>
struct MarchCol {
    T ax, xp, xm, ay, yp, ym;
};

template <typename T>
__device__ __forceinline__ T mfma(T a, T b, T c);
template <>
__device__ __forceinline__ double mfma<double>(double a, double b, double c) { return fma(a, b, c); }
template <>
__device__ __forceinline__ float mfma<float>(float a, float b, float c) { return fmaf(a, b, c); }

// a product that is rounded by itself (never part of an FMA)
template <typename T>
__device__ __forceinline__ T mmul(T a, T b);
template <>
__device__ __forceinline__ double mmul<double>(double a, double b) { return __dmul_rn(a, b); }
template <>
__device__ __forceinline__ float mmul<float>(float a, float b) { return __fmul_rn(a, b); }

// T: arithmetic type; BG: fields are perturbations from per-plane backgrounds,
// whose z differences join as constants of the plane; BWV, BS: row length and
// field size of a plane slot in shared memory; PZ: a plane's constants.
template <typename T, bool MAG, bool ROT, bool BG, int BWV, int BS, typename PZ>
struct March {
    // plane q-1: its cell, read again from its slot (b: without its background)
    T ru, rv, rw, tt, ro, p, u, v, w;
    T bx, by, bz;
    // carried between arrivals for plane q-1
    T ri;
    T wx, wy, s;                                 // dw/dx, dw/dy, du/dx + dv/dy
    T fu, fv, fw, fr, ft, heat, w1, w2, w3;      // what its right-hand side holds so far
    T exz, eyz, wz, jx, jy;                      // du/dz + dw/dx, dv/dz + dw/dy, dw/dz, currents: without plane q
    T dp;                                        // pressure less that of the plane above
    // plane q
    T nru, nrv, nrw, ntt, nro, nri, nu, nv, nw, np, nbx, nby, nbz;
    T nwx, nwy, ns;

    static __device__ __forceinline__ T ld(const T* __restrict__ raw, int f, int off) { return raw[f * BS + off]; }
    // pressure, or its perturbation RHOb*T' + RO'*(Tb + T')
    static __device__ __forceinline__ T pres(T ro_, T tt_, const PZ& z)
    {
        if constexpr (BG) return mfma<T>(ro_, z.ttb + tt_, z.rob * tt_);
        else return mmul<T>(ro_, tt_);
    }
    // difference of two pressures of a plane
    static __device__ __forceinline__ T dpres(T rop, T tp, T rom, T tm, const PZ& z)
    {
        if constexpr (BG) return pres(rop, tp, z) - pres(rom, tm, z);
        else return mfma<T>(rop, tp, -mmul<T>(rom, tm));
    }
    __device__ __forceinline__ T bfull(T b, T b0) const
    {
        if constexpr (BG) return b0 + b;
        else return b;
    }

    // the cell of plane q
    __device__ __forceinline__ void cell(const T* __restrict__ raw, const T* __restrict__ rip, int o, const PZ& z)
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
        np = pres(nro, ntt, z);
    }

    __device__ __forceinline__ void arrive(const T* __restrict__ raw, const T* __restrict__ rip, int o,
                                           const MarchCol<T>& c)
    {
        const T rxp = rip[o + 1], rxm = rip[o - 1], ryp = rip[o + BWV], rym = rip[o - BWV];
        nwx = mfma<T>(ld(raw, F_RW, o + 1), rxp, -ld(raw, F_RW, o - 1) * rxm) * c.ax;
        nwy = mfma<T>(ld(raw, F_RW, o + BWV), ryp, -ld(raw, F_RW, o - BWV) * rym) * c.ay;
        ns = mfma<T>(mfma<T>(ld(raw, F_RU, o + 1), rxp, -ld(raw, F_RU, o - 1) * rxm), c.ax,
                     mfma<T>(ld(raw, F_RV, o + BWV), ryp, -ld(raw, F_RV, o - BWV) * rym) * c.ay);
    }

    // plane q-1's terms from plane q (z: the constants of plane q-1).  bot: it
    // is the bottom wall, whose d2BX/dz2, d2BY/dz2 are one-sided (l1, l2).
    __device__ __forceinline__ void complete(const PZ& z, const MarchRun<T>& r, bool bot, T l1, T l2)
    {
        const T du = nu - u, dv = nv - v, dw = nw - w, dt = ntt - tt;
        fr = mfma<T>(rw - nrw, z.az, fr);
        fu = mfma<T>(-nru * nw, z.az, fu);
        fv = mfma<T>(-nrv * nw, z.az, fv);
        fw = mfma<T>(mfma<T>(rw, w, -nrw * nw), z.az, fw);
        fu = mfma<T>(z.ozp, du, mfma<T>(z.t13az, nwx, fu));
        fv = mfma<T>(z.ozp, dv, mfma<T>(z.t13az, nwy, fv));
        fw = mfma<T>(z.ozp, r.c43 * dw, mfma<T>(z.t13az, ns, fw));
        if constexpr (BG) fw += mfma<T>(-(dp + (np - p)), z.az, mfma<T>(r.grav, ro, z.fw));
        else fw = mfma<T>(r.grav, ro, mfma<T>(-(dp + mfma<T>(nro, ntt, -p)), z.az, fw));
        exz = mfma<T>(du, z.az, exz);
        eyz = mfma<T>(dv, z.az, eyz);
        wz = mfma<T>(dw, z.az, wz);
        ft = mfma<T>(dt, mfma<T>(ri * r.tmpc, z.kzp, -w * z.az), ft);
        if constexpr (BG) ft = mfma<T>(-r.ocv * (z.ttb + tt), wz, ft);
        else ft = mfma<T>(-r.ocv * tt, wz, ft);
        heat = mfma<T>(r.tmpa, mfma<T>(exz, exz, mfma<T>(eyz, eyz, r.c43 * (wz * (wz - s)))), heat);
        if (MAG) {
            const T dbx = nbx - bx, dby = nby - by, dbz = nbz - bz;
            const T fbx = bfull(bx, bgx(z)), fby = bfull(by, bgy(z)), fbz = bfull(bz, bgz(z));
            jy = mfma<T>(dbx, z.az, jy);
            jx = mfma<T>(dby, z.az, jx);
            w1 += bot ? l1 : z.mzp * dbx;
            w2 += bot ? l2 : z.mzp * dby;
            w1 = mfma<T>(fbz, exz, mfma<T>(-fbx, wz, mfma<T>(-w, jy, w1)));
            w2 = mfma<T>(fbz, eyz, mfma<T>(-fby, wz, mfma<T>(-w, jx, w2)));
            w3 = mfma<T>(dbz, mfma<T>(-w, z.az, z.mzp), w3);
            const T oy = r.obeta * jy, ox = r.obeta * jx;
            fu = mfma<T>(fbz, oy, fu);
            fv = mfma<T>(fbz, ox, fv);
            fw -= mfma<T>(fbx, oy, fby * ox);
            heat = mfma<T>(r.tmpm, mfma<T>(jx, jx, jy * jy), heat);
        }
        ft = mfma<T>(ri, heat, ft);
    }

    static __device__ __forceinline__ T bgx(const PZ& z) { if constexpr (BG) return z.bx; else return T(0); }
    static __device__ __forceinline__ T bgy(const PZ& z) { if constexpr (BG) return z.by; else return T(0); }
    static __device__ __forceinline__ T bgz(const PZ& z) { if constexpr (BG) return z.bz; else return T(0); }

    // plane q's x, y terms and its terms from plane q-1 (z: the constants of
    // plane q).  top: it is the top wall, as in complete().
    __device__ __forceinline__ void begin(const T* __restrict__ raw, const T* __restrict__ rip, int o, const PZ& z,
                                          const T* __restrict__ rawk, const PZ& zk,
                                          const MarchCol<T>& c, const MarchRun<T>& r, bool top, T rwt, T wt, T l1, T l2)
    {
        cell(raw, rip, o, z);
        recall(rawk, o, zk);
        if (top) {   // one-sided dRW/dz, dw/dz
            rw = rwt;
            w = wt;
        }
        const T du = nu - u, dv = nv - v, dw = nw - w, dt = ntt - tt;
        T gu, gv, gw, gr, gt, gh;
        // terms from the plane above, and dw/dz, strain and current sums that start with it
        gr = (rw - nrw) * z.az;
        gu = mfma<T>(ru * w, z.az, mfma<T>(z.ozm, du, -z.t13az * wx));
        gv = mfma<T>(rv * w, z.az, mfma<T>(z.ozm, dv, -z.t13az * wy));
        dp = np - p;
        gw = mfma<T>(mfma<T>(rw, w, -nrw * nw), z.az, mfma<T>(z.ozm, r.c43 * dw, -z.t13az * s));
        const T q = nri * r.tmpc;
        gt = dt * mfma<T>(q, z.kzm, -nw * z.az);
        exz = mfma<T>(du, z.az, nwx);
        eyz = mfma<T>(dv, z.az, nwy);
        wz = dw * z.az;
        T tf = ntt;   // full temperature
        if constexpr (BG) {
            gt = mfma<T>(q, z.kbg, mfma<T>(-nw, z.tzaz, gt));
            tf += z.ttb;
        }
        gt = mfma<T>(-r.ocv * tf, ns, gt);
        if (ROT) {
            gu = mfma<T>(r.omz, nrv, gu);
            gv = mfma<T>(r.omx, nrw, mfma<T>(-r.omz, nru, gv));
            gw = mfma<T>(-r.omx, nrv, gw);
        }
        T lt;   // x, y part of the Laplacian of T
        T vx, ux;
        {   // x
            const T rxp = rip[o + 1], rxm = rip[o - 1];
            const T rup = ld(raw, F_RU, o + 1), rum = ld(raw, F_RU, o - 1);
            const T rvp = ld(raw, F_RV, o + 1), rvm = ld(raw, F_RV, o - 1);
            const T rwp = ld(raw, F_RW, o + 1), rwm = ld(raw, F_RW, o - 1);
            const T tp = ld(raw, F_TT, o + 1), tm = ld(raw, F_TT, o - 1);
            const T dpx = dpres(ld(raw, F_RO, o + 1), tp, ld(raw, F_RO, o - 1), tm, z);
            const T vp = rvp * rxp, vm = rvm * rxm, uxp = rup * rxp, uxm = rum * rxm, wxp = rwp * rxp, wxm = rwm * rxm;
            gr = mfma<T>(-(rup - rum), c.ax, gr);
            gu = mfma<T>(-mfma<T>(rup, uxp, mfma<T>(-rum, uxm, dpx)), c.ax, gu);
            gv = mfma<T>(-mfma<T>(rvp, uxp, -rvm * uxm), c.ax, gv);
            gw = mfma<T>(-mfma<T>(rwp, uxp, -rwm * uxm), c.ax, gw);
            gu = mfma<T>(r.ore43, mfma<T>(uxp - nu, c.xp, (nu - uxm) * c.xm), gu);
            gv = mfma<T>(r.ore, mfma<T>(vp - nv, c.xp, (nv - vm) * c.xm), gv);
            gw = mfma<T>(r.ore, mfma<T>(wxp - nw, c.xp, (nw - wxm) * c.xm), gw);
            gt = mfma<T>(-nu, (tp - tm) * c.ax, gt);
            lt = mfma<T>(tp - ntt, c.xp, (ntt - tm) * c.xm);
            ux = (uxp - uxm) * c.ax;
            vx = (vp - vm) * c.ax;
        }
        T uy, vy;
        {   // y
            const T ryp = rip[o + BWV], rym = rip[o - BWV];
            const T rup = ld(raw, F_RU, o + BWV), rum = ld(raw, F_RU, o - BWV);
            const T rvp = ld(raw, F_RV, o + BWV), rvm = ld(raw, F_RV, o - BWV);
            const T rwp = ld(raw, F_RW, o + BWV), rwm = ld(raw, F_RW, o - BWV);
            const T tp = ld(raw, F_TT, o + BWV), tm = ld(raw, F_TT, o - BWV);
            const T dpy = dpres(ld(raw, F_RO, o + BWV), tp, ld(raw, F_RO, o - BWV), tm, z);
            const T up = rup * ryp, um = rum * rym, vyp = rvp * ryp, vym = rvm * rym, wyp = rwp * ryp, wym = rwm * rym;
            gr = mfma<T>(-(rvp - rvm), c.ay, gr);
            gu = mfma<T>(-mfma<T>(rup, vyp, -rum * vym), c.ay, gu);
            gv = mfma<T>(-mfma<T>(rvp, vyp, mfma<T>(-rvm, vym, dpy)), c.ay, gv);
            gw = mfma<T>(-mfma<T>(rwp, vyp, -rwm * vym), c.ay, gw);
            gu = mfma<T>(r.ore, mfma<T>(up - nu, c.yp, (nu - um) * c.ym), gu);
            gv = mfma<T>(r.ore43, mfma<T>(vyp - nv, c.yp, (nv - vym) * c.ym), gv);
            gw = mfma<T>(r.ore, mfma<T>(wyp - nw, c.yp, (nw - wym) * c.ym), gw);
            gt = mfma<T>(-nv, (tp - tm) * c.ay, gt);
            lt += mfma<T>(tp - ntt, c.yp, (ntt - tm) * c.ym);
            uy = (up - um) * c.ay;
            vy = (vyp - vym) * c.ay;
        }
        gt = mfma<T>(q * z.rka, lt, gt);
        {   // corners: d2v/dxdy, d2u/dxdy
            const T rpp = rip[o + BWV + 1], rmp = rip[o + BWV - 1], rpm = rip[o - BWV + 1], rmm = rip[o - BWV - 1];
            const T sxy = r.t13 * (c.ax * c.ay);
            const T vv = mfma<T>(ld(raw, F_RV, o + BWV + 1), rpp, -ld(raw, F_RV, o + BWV - 1) * rmp)
                       - mfma<T>(ld(raw, F_RV, o - BWV + 1), rpm, -ld(raw, F_RV, o - BWV - 1) * rmm);
            const T uu = mfma<T>(ld(raw, F_RU, o + BWV + 1), rpp, -ld(raw, F_RU, o + BWV - 1) * rmp)
                       - mfma<T>(ld(raw, F_RU, o - BWV + 1), rpm, -ld(raw, F_RU, o - BWV - 1) * rmm);
            gu = mfma<T>(sxy, vv, gu);
            gv = mfma<T>(sxy, uu, gv);
        }
        {
            const T e = uy + vx;
            gh = r.tmpa * mfma<T>(e, e, r.c43 * mfma<T>(ns, ns, T(-3) * ux * vy));
        }
        if (MAG) {
            const T fbx = bfull(nbx, bgx(z)), fby = bfull(nby, bgy(z)), fbz = bfull(nbz, bgz(z));
            const T dbx = nbx - bx, dby = nby - by, dbz = nbz - bz;
            T g1 = top ? l1 : z.mzm * dbx, g2 = top ? l2 : z.mzm * dby, g3 = dbz * mfma<T>(-nw, z.az, z.mzm);
            T cy = dbx * z.az, cx = dby * z.az;   // currents without d/dx BZ, d/dy BZ
            if constexpr (BG) {
                g1 += z.ml1;
                g2 += z.ml2;
                g3 += mfma<T>(-nw, z.bzz, z.ml3);
                cy += z.bxz;
                cx += z.byz;
            }
            T lx, jz;
            {   // x
                const T b1p = ld(raw, F_BX, o + 1), b1m = ld(raw, F_BX, o - 1);
                const T b2p = ld(raw, F_BY, o + 1), b2m = ld(raw, F_BY, o - 1);
                const T b3p = ld(raw, F_BZ, o + 1), b3m = ld(raw, F_BZ, o - 1);
                const T d2 = (b2p - b2m) * c.ax, d3 = (b3p - b3m) * c.ax;
                lx = mfma<T>(b1p - nbx, c.xp, (nbx - b1m) * c.xm);
                g1 = mfma<T>(r.orm, lx, mfma<T>(-nu, (b1p - b1m) * c.ax, g1));
                lx = mfma<T>(b2p - nby, c.xp, (nby - b2m) * c.xm);
                g2 = mfma<T>(r.orm, lx, mfma<T>(-nu, d2, g2));
                lx = mfma<T>(b3p - nbz, c.xp, (nbz - b3m) * c.xm);
                g3 = mfma<T>(r.orm, lx, mfma<T>(-nu, d3, g3));
                g1 = mfma<T>(-nw, d3, g1);
                cy -= d3;
                jz = -d2;
            }
            {   // y
                const T b1p = ld(raw, F_BX, o + BWV), b1m = ld(raw, F_BX, o - BWV);
                const T b2p = ld(raw, F_BY, o + BWV), b2m = ld(raw, F_BY, o - BWV);
                const T b3p = ld(raw, F_BZ, o + BWV), b3m = ld(raw, F_BZ, o - BWV);
                const T d1 = (b1p - b1m) * c.ay, d3 = (b3p - b3m) * c.ay;
                lx = mfma<T>(b1p - nbx, c.yp, (nbx - b1m) * c.ym);
                g1 = mfma<T>(r.orm, lx, mfma<T>(-nv, d1, g1));
                lx = mfma<T>(b2p - nby, c.yp, (nby - b2m) * c.ym);
                g2 = mfma<T>(r.orm, lx, mfma<T>(-nv, (b2p - b2m) * c.ay, g2));
                lx = mfma<T>(b3p - nbz, c.yp, (nbz - b3m) * c.ym);
                g3 = mfma<T>(r.orm, lx, mfma<T>(-nv, d3, g3));
                g2 = mfma<T>(-nw, d3, g2);
                cx -= d3;
                jz += d1;
            }
            g1 = mfma<T>(fby, uy, mfma<T>(-fbx, vy, mfma<T>(-fbz, nwx, g1)));
            g2 = mfma<T>(fbx, vx, mfma<T>(-fby, ux, mfma<T>(-fbz, nwy, g2)));
            g3 = mfma<T>(fbx, nwx, mfma<T>(fby, nwy, mfma<T>(-fbz, ns, g3)));
            const T oz = r.obeta * jz;
            gu = mfma<T>(fby, oz, gu);
            gv = mfma<T>(-fbx, oz, gv);
            gh = mfma<T>(r.tmpm * jz, jz, gh);
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
    static __device__ __forceinline__ T wall_d2(const PZ& z, T sg, T b0, T b1, T b2, T b3)
    {
        const T B = sg * (T(0.5) * (z.mzp + z.mzm)), C = T(0.5) * (z.mzp - z.mzm);
        const T d1 = b1 - b0, d2 = b2 - b1, d3 = b3 - b2;
        return mfma<T>(T(2) * d1 - d2, B, (T(3) * (d2 - d1) - d3) * C);
    }

    // the cell of plane q-1, from its slot (z: its constants)
    __device__ __forceinline__ void recall(const T* __restrict__ raw, int o, const PZ& z)
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
        p = pres(ro, tt, z);
    }

    // plane q becomes the carried plane (rq: its 1/RO)
    __device__ __forceinline__ void shift(T rq)
    {
        ri = rq;
        wx = nwx;
        wy = nwy;
        s = ns;
    }
};

}  // namespace mhd3d
