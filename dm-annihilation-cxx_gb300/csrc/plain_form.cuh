// plain_form.cuh -- the plain FP64 precision form of the disc engine: the
// reference CPU path's per-pixel arithmetic (pix2vec of each disc pixel,
// w = exp(-0.5 (acos(v_pix . v)/ar)^2 / 0.333), src/genmap.cpp:133-145,
// FP64 normalisation and FP64 atomic deposits, genmap.cpp:148-153).
// Shared by the plain render kernels (disc_plain.cu) and the adjoint
// kernels (adjoint.cu); both translation units are compiled with
// -fmad=false so the weights round exactly as the CPU path's do.
#pragma once
#include "disc_engine.cuh"

namespace dmann {

// a / b, correctly rounded, from r = RN(1 / b): the quotient a r is within
// two ulp, one correction makes it faithful, and by Markstein's theorem (IBM
// J. Res. Dev. 34, 1990) a second one rounds it correctly.  Five FP64
// operations where the general division takes about twice as many; the
// divisors here serve a whole disc.
__device__ __forceinline__ double div_by(double a, double b, double r) {
    double q = __dmul_rn(a, r);
    q = __fma_rn(__fma_rn(-q, b, a), r, q);
    return __fma_rn(__fma_rn(-q, b, a), r, q);
}

// The azimuth of pixel k (from 0) of a cap ring (ipole rings from its pole)
// and of an equatorial ring (pf: 1/2 or 1), as pix2vec forms them.
__device__ __forceinline__ double cap_phi(int k, int ipole) {
    return ((double)(k + 1) - 0.5) * kHalfPi / (double)ipole;
}
__device__ __forceinline__ double belt_phi(int k, double pf, double fact1) {
    return ((double)(k + 1) - pf) * kPi * 0.75 * fact1;
}

struct PlainForm {
    static constexpr bool kFastChord = false;  // the exact FP64 chord test
    static constexpr int kMinBlocks = 1;
    struct alignas(16) Seg {
        int start, nr, lo, off;
        double z, st, pf;
        int cap, ipole;
        const double2 *trig;   // (sin, cos) of the ring's pixels, or null
    };
    struct SegReg {
        int start, nr, lo;
        double z, st, pf;
        int cap, ipole;
        const double2 *trig;
    };
    struct Ext {
        double vx, vy, vz, ar, fact1, inv_ar;
    };
    struct Dep {
        double S, inv_S, flux;
    };

    // anglefuncs.cpp:55-71 ang2vec, from the un-normalised phi of calc_angles
    __device__ static void particle_setup(const DiscArgs &a, const DiscHdr &d, double phi_raw,
                                          Ext &e) {
        const double sz = sin(d.theta0);
        e.vx = sz * cos(phi_raw);
        e.vy = sz * sin(phi_raw);
        e.vz = cos(d.theta0);
        e.ar = d.ar;
        e.inv_ar = __ddiv_rn(1.0, d.ar);
        e.fact1 = a.g.fact1;
    }

    __device__ static void fill_seg(const DiscArgs &a, const DiscHdr &d, const Ext &e, int ring,
                                    int lo, int cnt, Seg &s) {
        (void)d;
        (void)e;
        (void)cnt;
        const int ns = a.g.nside;
        s.start = (int)ring_start(a.g, ring);
        s.nr = ring_npix(a.g, ring);
        s.lo = lo;
        s.z = a.rt.z[ring];
        s.st = a.rt.st[ring];
        s.cap = (ring < ns) || (ring > 3 * ns);
        s.ipole = (ring < ns) ? ring : 4 * ns - ring;
        s.pf = ((ring + ns) & 1) ? 1.0 : 0.5;
        if (s.cap) s.trig = a.trig_cap ? a.trig_cap + 2LL * s.ipole * (s.ipole - 1) : nullptr;
        else s.trig = a.trig_belt ? a.trig_belt + (s.pf == 1.0 ? 4 * ns : 0) : nullptr;
    }

    __device__ static void load_seg(const Seg &s, SegReg &r) {
        r.start = s.start;
        r.nr = s.nr;
        r.lo = s.lo;
        r.z = s.z;
        r.st = s.st;
        r.pf = s.pf;
        r.cap = s.cap;
        r.ipole = s.ipole;
        r.trig = s.trig;
    }

    // pix2vec of a pixel of the segment's ring, as the oracle restates it
    __device__ static void pixel_vec(const Ext &e, const SegReg &sr, int pix, double &px,
                                     double &py, double &pz) {
        const int k = pix - sr.start;
        double sp, cp;
        if (sr.trig) {
            const double2 t = __ldg(sr.trig + k);
            sp = t.x;
            cp = t.y;
        } else {
            sincos(sr.cap ? cap_phi(k, sr.ipole) : belt_phi(k, sr.pf, e.fact1), &sp, &cp);
        }
        px = sr.st * cp;
        py = sr.st * sp;
        pz = sr.z;
    }

    // src/genmap.cpp:135-143: the weight of angular distance alpha
    __device__ static double weight_at(const Ext &e, double alpha) {
        constexpr double kR = 1.0 / 0.333;
        double d2 = div_by(alpha, e.ar, e.inv_ar);
        d2 = d2 * d2;
        return exp(div_by(-0.5 * d2, 0.333, kR));
    }
    __device__ static double weight(const Ext &e, const SegReg &sr, int pix) {
        double px, py, pz;
        pixel_vec(e, sr, pix, px, py, pz);
        const double dot = px * e.vx + py * e.vy + pz * e.vz;
        return weight_at(e, acos(fmin(1.0, fmax(-1.0, dot))));
    }

    __device__ static void deposit_setup(const DiscHdr &d, double S, Dep &dep) {
        dep.S = S;
        dep.inv_S = __ddiv_rn(1.0, S);
        dep.flux = d.flux;
    }
    __device__ static void deposit(const DiscArgs &a, const Dep &dep, double w, int pix) {
        red_add_f64(a.acc.acc64 + pix, div_by(w, dep.S, dep.inv_S) * dep.flux);
    }
    __device__ static void single(const DiscArgs &a, const DiscHdr &d) {
        red_add_f64(a.acc.acc64 + d.cpix, d.flux);
    }
};

}  // namespace dmann
