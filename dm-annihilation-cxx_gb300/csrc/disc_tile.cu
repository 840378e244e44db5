// disc_tile.cu -- the compensated-FP32 render of the block-class discs by map
// tiles.
//
// A deposit per disc pixel is one reduction in L2, and at full overlap
// density those reductions bound a scatter (disc_seg.cu: 1.07e12 deposits/s
// on the 16M-particle workload, 0.75 of a bare sweep of FP32 reductions).
// Times below are of 1M of the 16M set's particles at Nside 2048 (4.6e10
// deposits): 34 ms in all.  The whole set takes 0.54 s, and 1.16 s by the
// segmented render.
// Here a warp owns a tile of the map -- 32 rings (one per lane) by kTileW
// in-ring pixel indices -- in registers, and walks the list of the discs
// that touch it: the sums never leave the SM until the tile is flushed, with
// one FP64 reduction per pixel for up to kUnitMax discs.
//
// Sequence (one stream, nothing waits for the host):
//   k_tile_hdr      a short header per disc; the giants and the long discs
//   k_tile_pairs<0> (disc, tile) pairs of the chunk, for its mode (where they
//                   could exceed the list)
//   k_tile_norm     weight sums S of the discs; k_tile_norm_giant of the
//                   giants, the largest and those that carry the map's flux
//   k_tile_fin      F = flux / S per disc, discs of fewer than two pixels
//   k_tile_pairs<1> pairs per (tile, octave of F)
//   k_tile_plan     each tile's range of the pair list, its octaves in
//                   ascending order, cut into work units
//   k_tile_pairs<2> the pair list
//   k_tile_dep<0>, <1> units of polynomial discs; <2>, k_tile_dep_px of the others
//
// Weight sums without visiting the pixels.  Along a ring the weight is a
// smooth even function f(x) of the half azimuth offset x (a Gaussian, cut at
// 3.5 sigma), sampled at a uniform step s over cnt pixels.  By the
// Euler-Maclaurin formula at midpoints
//     sum f = (1/s) int f - [f']/24 + 7 [f''']/5760 - 31 [f5]/967680 + ...
// (derivatives per pixel step, taken between the outer edges of the first
// and the last pixel), and since f is even the integral from 0 to an edge
// at distance X is half that from -X to X, which Gauss-Legendre's rule of
// 2 kNodes points gives from kNodes values of f.  Rings of up to
// kDirect pixels are summed pixel by pixel.  Above that the disc's
// radius is at least kDirect / 2 pixels, so sigma is at least 3.5 pixels and
// the truncation is below 6e-11 of the ring's sum; the rule's own error on
// the exponents that occur (at most 6.01) is 1.3e-11.  The rule's nodes
// (squared) are the FP32 numbers used and its weights are FP32 pairs, so the
// error of the constants does not add up over rings.  A chord of the 16M
// workload holds 130 pixels on average: 8 packed evaluations in its place.
//
// FP32 sums of a tile.  A unit's discs are visited in ascending octave of F
// (tile_class in tile_plan.h) and at most kUnitMax of them go into one FP32 sum:
// no small deposit is lost on a large total, and the rounding errors of the
// short sums are random.
#include "comp_engine.cuh"

namespace dmann {

namespace {

constexpr int kClsBits = 6;
constexpr int kCls = 1 << kClsBits;   // classes of F (tile_class)
static_assert(kCls == kTileClasses, "histogram size");

// How a disc's weights are evaluated.
enum Kind {
    K_POLY3 = 0,   // the ring's exponent polynomial without its y^4 term
    K_POLY = 1,    // the ring's exponent polynomial
    K_GEN = 2,     // run-time series per value
    K_GIANT = 3    // the same, summed pixel by pixel and deposited in two floats: radius beyond
                   // kGiantR (which may reach the kink at the antipode), or a share of the map's flux
};
constexpr int kKindMask = 3, kFlagH1 = 4, kFlagAll = 8, kFlagFast = 16, kFlagA2 = 32, kFlagLong = 64;
constexpr double kGiantR = 2.2;

// Discs with 1 / kShare and more of the flux kept so far are giants too.  The
// quadrature's sum of one disc scatters by 5e-9 (up to 2e-8: a few thousand nodes
// instead of the pixels, each exponent rounded to FP32), so the rest of a map is
// off by 5e-9 / sqrt(kShare) = 3e-10 of its flux at most, few discs or many.  A
// giant's own flux is off by 1e-12.  (kShareMax: with fluxes of both signs the
// sum of flux bounds nothing.)
constexpr int kShare = 256, kShareMax = 1024;

// Half azimuth offsets x below 0.1 rad (sin R / sin theta0 = sin 2x) of the
// three-term asin^2 tier (h < 4e-3) do without the y^4 term (y = x^2): up to 6e-8
// in the exponent of 2, most of it the share of h^3, which that of h^4, beyond the
// three terms, would cancel.  With it a map of 1M particles at Nside 512 is
// 1.17e-7 from the FP64 form instead of 8.9e-8, one of 200k at Nside 400 6.4e-8
// instead of 3.9e-8 (units of 512 discs), and the 16M workload took 632 ms
// instead of 604.
constexpr float kPoly3Sin = 0.1987f;

constexpr int kLongRings = 256;   // general discs of more are summed by several warps

// Rings from which a general disc's exponent is interpolated over 32 pixels
// (half azimuth offsets of 16 pixels below 0.06 rad: see add_gen).
constexpr int kFineNr = 838;

// ------------------------------------------------------------ one ring
struct RingT {
    float thh, thl;     // theta as a two-float
    float st, step;     // sin theta, 2 pi / nr
    float fnr;          // nr / 2 pi
    float nrf, shift;
    int nr;
};

__device__ __forceinline__ RingT ring_t(const DiscArgs &a, int ring) {
    RingT r;
    const float2 th = a.rt.th2[ring];
    r.thh = th.x;
    r.thl = th.y;
    r.st = a.rt.st32[ring];
    r.step = a.rt.step32[ring];
    r.nr = ring_npix(a.g, ring);
    r.nrf = (float)r.nr;
    r.fnr = r.nrf * 0.159154943091895336f;
    r.shift = ring_shifted(a.g, ring) ? 0.5f : 0.0f;
    return r;
}

// 1/x and 1/sqrt(x) to 2^-23 and 2^-22.9 relative (positive normal x: the
// subnormal handling of __fdividef and rsqrtf costs several instructions each)
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

constexpr float kPiHi = 3.14159274101257324f, kPiLo = -8.74227765734758577e-8f;

// The exact FP64 chord test.
__device__ __noinline__ int exact_run(const DiscArgs &a, int q, int ring, int &lo, float &d0h) {
    const DiscHdr &d = a.chdr[q].hdr;
    int cnt;
    ring_segment_t<true>(a.g, d, ring, lo, cnt);
    if (cnt <= 0) return 0;
    const double shift = ring_shifted(a.g, ring) ? 0.5 : 0.0;
    // azimuth of the first pixel relative to the particle, in [-pi, pi)
    double d0 = ((double)lo + shift) * a.rt.step[ring] - d.phi0;
    if (d0 < -kPi) d0 += kTwoPi;
    if (d0 >= kPi) d0 -= kTwoPi;
    d0h = (float)(0.5 * d0);
    return cnt;
}

// One ring's pixels inside the disc, as make_runs in comp_engine.cuh but in
// FP32 throughout: theta and the azimuth phi0 / 2 pi are two-floats (the FP64
// pipe, at 1/64 of the FP32 rate, was 65 % busy in the weight sums with FP64
// differences and conversions here), the polynomial discs (GEN false: |theta
// - theta0| < 0.29, dphi < 0.67) take sin and asin from short series, and the
// divisions are approximate.  The end points are c -+ w in pixels, c = nr phi0
// / 2 pi - shift, w = nr dphi / 2 pi; their error bound tau sums, in units of
// eps = 2^-24 = 6e-8:
//   A = sin^2(d/2): 8 eps (GEN: sinf, 10 eps); hR, num: 1 eps each;
//   q = num / B: 6 eps (sin theta, sin theta0, their product, the reciprocal
//   2, the product) besides num's error, eq in all;
//   dphi: eq sq / sqrt(1 - q), and 5.2 eps (root 2.2 + 1, asin 2; GEN: 7);
//   w: 3 eps; c: 2 eps absolute; c -+ w: 1 eps of (1 + w);
//   and the FP64 form's own rounding, which this must reproduce (1e-15 over
//   B sq and sin^2 theta sq; for the polynomial discs sin theta is within a
//   factor of 2.7 of sin theta0);
// each enlarged a little, 5 % on the sum and 4e-7 on tau.  Rings with an end
// point within tau of an integer take the exact test, so the pixels are the
// same (a bound four times as wide sent 8 % of the warps there and cost 20 %
// of the FP64 pipe).
// Returns the count; the first pixel is lo (modulo nr), pixel j lies at half
// azimuth offset d0h + j step / 2; A and B are the haversine terms (see Run).
template <bool GEN>
__device__ __forceinline__ int tile_run(const DiscArgs &a, const TileHdr &h, const RingT &rc, int ring, int &lo,
                                        float &d0h, float &A, float &B) {
    // nr phi0 / 2 pi - shift = fl + cf, fl an integer
    auto split_phi = [&](float &fl, float &cf) {
        const float hi = rc.nrf * h.ph;
        const float lw = fmaf(rc.nrf, h.ph, -hi) + fmaf(rc.nrf, h.pl, -rc.shift);
        fl = floorf(hi);
        cf = (hi - fl) + lw;
    };
    const float d = (rc.thh - h.t0h) + (rc.thl - h.t0l);
    float s;
    if (GEN) {
        s = sinf(0.5f * d);
    } else {
        const float x = 0.5f * d, x2 = x * x;
        float p = fmaf(x2, -1.0f / 5040.0f, 1.0f / 120.0f);
        p = fmaf(x2, p, -1.0f / 6.0f);
        s = fmaf(x * x2, p, x);
    }
    A = s * s;
    B = rc.st * h.sth0;
    if (GEN && ((h.flags & kFlagAll) || ring < h.irmin || ring > h.irmax)) {
        // a full ring, from the pixel behind the antipodal azimuth on (FP32 may
        // start it one pixel to the side of the FP64 form: the same pixels, the
        // first at an offset of -pi / 2 to an ulp)
        float fl, cf;
        split_phi(fl, cf);
        const float up = ceilf(cf);
        lo = (int)fl + (int)up - rc.nr / 2;
        d0h = fmaf(0.5f * rc.step, up - cf, -0.5f * kPiLo) - 0.5f * kPiHi;
        return rc.nr;
    }
    if ((h.flags & kFlagFast) && rc.st > 0.01f) {
        const float num = h.hR - A;
        const float dnum = 7e-8f * h.hR + (GEN ? 7e-7f : 5.5e-7f) * A + 7e-8f * fabsf(num);
        if (num < -4.0f * dnum && -num > 1e-9f * B) return 0;   // clearly outside
        const float rB = rcp_approx(B);
        const float q = num * rB;
        const float eq = fmaf(dnum, rcp_approx(num), 4e-7f);
        if (num > 4.0f * dnum && q < (GEN ? 0.9999f : 0.11f) && eq <= 1e-3f) {
            const float rsq = rsqrt_approx(q), sq = q * rsq;
            float dphi;
            if (GEN) {
                dphi = 2.0f * asinf(sq);
            } else {   // q < 0.11: 2.6e-9 of the next term
                float p = fmaf(q, 10395.0f / 599040.0f, 945.0f / 42240.0f);
                p = fmaf(q, p, 105.0f / 3456.0f);
                p = fmaf(q, p, 15.0f / 336.0f);
                p = fmaf(q, p, 3.0f / 40.0f);
                p = fmaf(q, p, 1.0f / 6.0f);
                dphi = 2.0f * fmaf(sq * q, p, sq);
            }
            const float amp = GEN ? rsqrt_approx(1.0f - q) : 1.07f;
            const float ddphi = 1.05f * (eq * sq * amp + (GEN ? 4.5e-7f : 3.3e-7f) * dphi) +
                                (GEN ? 1e-15f * (rB + rcp_approx(rc.st * rc.st)) : 4e-15f * rB) * rsq;
            float fl, cf;
            split_phi(fl, cf);
            const float w = rc.fnr * dphi;
            const float tau = rc.fnr * ddphi + 3e-7f * w + 6e-7f;
            const float xlo = cf - w, xhi = cf + w;
            const float flo = floorf(xlo), fhi = floorf(xhi);
            const float f0 = xlo - flo, f1 = xhi - fhi;
            if (fminf(f0, f1) >= tau && fmaxf(f0, f1) <= 1.0f - tau) {
                int ip = (int)fl + (int)flo + 1;
                const int cnt = (int)(fhi - flo);
                if (cnt <= 0) return 0;
                d0h = 0.5f * fmaf(rc.step, flo + 1.0f, -rc.step * cf);
                if (ip + cnt > rc.nr) ip -= rc.nr;
                if (GEN && (cnt > rc.nr || ip < -rc.nr || ip >= rc.nr)) return 0;  // cannot happen for finite input
                lo = ip;
                return cnt;
            }
        }
    }
    return exact_run(a, h.q, ring, lo, d0h);
}

// ------------------------------------------------------------ weight sums
// Gauss-Legendre of 2 n points on [-1, 1], the positive half: for the
// polynomial discs the squared nodes (n = 8), for the general ones the nodes
// (n = 12), as FP32 numbers; the weights for exactly these nodes (they
// integrate the even powers up to 2 n - 2) as FP32 pairs.
constexpr int kNodes = 8, kNodesGen = 12;
__device__ constexpr float kTau[kNodes] = {9.027376771e-03f, 7.930056006e-02f, 2.097793669e-01f, 3.817710578e-01f,
                                           5.706357956e-01f, 7.493174076e-01f, 8.922219872e-01f, 9.789142013e-01f};
__device__ constexpr float kGw[kNodes] = {1.894506067e-01f, 1.826034039e-01f, 1.691565365e-01f, 1.495959759e-01f,
                                          1.246289760e-01f, 9.515853971e-02f, 6.225349382e-02f, 2.715246566e-02f};
__device__ constexpr float kGwLo[kNodes] = {4.9362e-09f,  5.3504e-09f,  -5.5062e-09f, -5.3167e-09f,
                                            3.0101e-09f, -1.7361e-09f, 1.1800e-09f,  -5.5195e-11f};
__device__ constexpr float kNodeG[kNodesGen] = {6.405689567e-02f, 1.911188662e-01f, 3.150426745e-01f, 4.337935150e-01f,
                                                5.454214811e-01f, 6.480936408e-01f, 7.401241660e-01f, 8.200019598e-01f,
                                                8.864155412e-01f, 9.382745624e-01f, 9.747285843e-01f, 9.951872230e-01f};
__device__ constexpr float kGwG[kNodesGen] = {1.279381961e-01f, 1.258374453e-01f, 1.216704696e-01f, 1.155056953e-01f,
                                              1.074442416e-01f, 9.761864692e-02f, 8.619012684e-02f, 7.334652543e-02f,
                                              5.929858610e-02f, 4.427745566e-02f, 2.853137814e-02f, 1.234121434e-02f};
__device__ constexpr float kGwGLo[kNodesGen] = {1.0278e-09f, 6.3130e-09f, 1.3962e-09f, -3.0681e-09f,
                                                2.2970e-09f, 1.2565e-09f, 3.0315e-09f, 2.8634e-09f,
                                                1.7837e-09f, 1.6689e-09f, -6.9250e-11f, 1.2575e-10f};
constexpr int kDirect = 24, kDirectGen = 64;   // pixels up to which a ring is summed pixel by pixel
constexpr int kFullPts = 32;                   // points of a full ring's trapezoid rule

template <bool P3 = false>
__device__ __forceinline__ float2 poly_exp2(const float c[5], float2 y) {
    float2 t;
    if constexpr (P3) {
        t = fma2(y, f2(c[3]), f2(c[2]));
    } else {
        t = fma2(y, f2(c[4]), f2(c[3]));
        t = fma2(y, t, f2(c[2]));
    }
    t = fma2(y, t, f2(c[1]));
    return fma2(y, t, f2(c[0]));
}
__device__ __forceinline__ float2 ex2_2(float2 t) { return make_float2(ex2_approx(t.x), ex2_approx(t.y)); }

// ex2.approx is off by a fixed function of its argument: by -3.6e-8 on
// average over a disc's pixels, whatever the disc, less near 0 than below -1,
// with a scatter of 3e-8 from argument to argument.  The few nodes of a rule
// would sample that function at the same exponents in every disc of a size.
// So a ring's exponents are moved up (upwards they stay exact) by a fraction
// of 1/16, one of 32 dealt to the lanes anew for each disc, and its sum is
// scaled back: the nodes then see the function's local average, as the
// pixels do, but for 1.4e-9 (the mean over 300 discs of each of several radii
// and Nside).  Sets of thousands of discs of one kind and size are left with
// -5e-10 to 6e-10 of their flux (Nside 64 to 1024).
constexpr float kEx2Bias = -1.4e-9f;

struct Dither {
    float shift, hi, lo;   // 2^-shift = hi + lo
};

__device__ __forceinline__ Dither lane_dither() {
    Dither d;
    const float g = (float)(threadIdx.x & 31) * 0.61803399f;
    d.shift = floorf((g - floorf(g)) * 1024.0f) * (1.0f / 16384.0f);
    const double e = exp2(-(double)d.shift);
    d.hi = (float)e;
    d.lo = (float)(e - (double)d.hi);
    return d;
}

__device__ __forceinline__ Dither deal_dither(const Dither &d, long long q) {
    const int from = ((int)(q * 11) + (int)threadIdx.x) & 31;
    return Dither{__shfl_sync(0xffffffffu, d.shift, from), __shfl_sync(0xffffffffu, d.hi, from),
                  __shfl_sync(0xffffffffu, d.lo, from)};
}

// The end corrections of the midpoint Euler-Maclaurin formula for f at its
// two ends (f there, and the logarithmic derivatives per pixel step, each
// counted outwards).
__device__ __forceinline__ float2 end_terms(float2 f, float2 g1, float2 g2) {
    const float2 g1s = mul2(g1, g1);
    const float2 r3 = fma2(g2, f2(3.0f), g1s);   // third over first derivative
    const float2 r5 = fma2(g1s, fma2(g2, f2(10.0f), g1s), mul2(mul2(g2, g2), f2(15.0f)));   // fifth over first
    float2 k = fma2(r5, f2(-31.0f / 967680.0f), f2(-1.0f / 24.0f));
    k = fma2(r3, f2(7.0f / 5760.0f), k);
    return mul2(k, mul2(f, g1));
}

// Node sums of a rule, largest term first: s in FP32 (each rounding error
// exactly, Fast2Sum), the errors and the low halves of the weights in sl.
struct NodeSum {
    float2 s, sl;
    __device__ __forceinline__ void add(float2 w, float g, float gl) {
        const float2 t = fma2(w, f2(g), s);
        sl = add2(sl, fma2(w, f2(g), sub2(s, t)));
        sl = fma2(w, f2(gl), sl);
        s = t;
    }
};

// The ring's total as a two-float: X (s + sl) / steph of both sides plus the
// end terms k, scaled back by the dither.  (In plain FP32 the end terms and
// the low halves, below half an ulp, were lost in every ring, a bias of 3e-8,
// and the roundings left 8e-9 per disc of 100 rings.)
__device__ __forceinline__ float2 ring_total(const NodeSum &n, float2 X, float2 k, float steph, const Dither &di) {
    const float2 hi = mul2(n.s, X);
    const float2 lo = add2(fma2(n.s, X, make_float2(-hi.x, -hi.y)), fma2(n.sl, X, mul2(k, f2(steph))));
    float e;
    const float H = two_sum(hi.x, hi.y, e);
    const float rs = rcp_approx(steph);
    const float q = H * rs;
    const float ql = (fmaf(-q, steph, H) + (e + (lo.x + lo.y))) * rs;
    const float v = q * di.hi;
    return make_float2(v, fmaf(q, di.hi, -v) + fmaf(q, di.lo + kEx2Bias * di.hi, ql * di.hi));
}

// A short ring's weights pixel by pixel (w(j): those of pixels j, j + 1), each
// rounding of the sum kept: the sums start at 1, above every weight.
template <class W>
__device__ __forceinline__ float2 direct_sum(int cnt, W w) {
    float2 s = f2(1.0f), c = f2(0.0f);
    for (int j = 0; j < cnt; j += 2) {
        float2 v = w((float)j);
        if (j + 1 >= cnt) v.y = 0.0f;
        const float2 t = add2(s, v);
        c = add2(c, sub2(v, sub2(t, s)));
        s = t;
    }
    float e;
    const float H = two_sum(s.x - 1.0f, s.y - 1.0f, e);
    return make_float2(H, e + (c.x + c.y));
}

// The weight sum of one ring of a polynomial disc as a two-float.
__device__ __forceinline__ float2 ring_sum(const float c[5], float d0h, float steph, int cnt, const Dither &di) {
    if (cnt <= kDirect)
        return direct_sum(cnt, [&](float jf) {
            const float2 x = fma2(make_float2(jf, jf + 1.0f), f2(steph), f2(d0h));
            return ex2_2(poly_exp2(c, mul2(x, x)));
        });
    // outer edges of the run at -X.x and X.y
    const float2 X = make_float2(fmaf(0.5f, steph, -d0h), fmaf((float)cnt - 0.5f, steph, d0h));
    const float2 Y = mul2(X, X);
    const float cs[5] = {c[0] + di.shift, c[1], c[2], c[3], c[4]};
    NodeSum n{f2(0.0f), f2(0.0f)};
#pragma unroll
    for (int k = 0; k < kNodes; k++) n.add(ex2_2(poly_exp2(cs, mul2(Y, f2(kTau[k])))), kGw[k], kGwLo[k]);
    // with E the exponent of 2 and x = steph u: d ln f / du = g1 = ln2 2 x
    // steph E'(y), d2 ln f / du2 = g1 / u up to E''
    const float2 fe = ex2_2(poly_exp2(cs, Y));
    float2 dE = fma2(Y, f2(4.0f * c[4]), f2(3.0f * c[3]));
    dE = fma2(Y, dE, f2(2.0f * c[2]));
    dE = fma2(Y, dE, f2(c[1]));
    const float2 g2 = mul2(dE, f2(1.38629436112f * steph * steph));
    const float2 g1 = mul2(g2, mul2(X, f2(rcp_approx(steph))));
    return ring_total(n, X, end_terms(fe, g1, g2), steph, di);
}

// The weight sum of one ring of a general disc (run g, full: the whole ring
// of the map is inside).
__device__ inline float2 ring_sum_gen(const Ext &e, Run g, bool full, const Dither &di) {
    float2 sn, h, gg;
    if (g.cnt <= kDirectGen)
        return direct_sum(g.cnt, [&](float jf) {
            return ex2_2(exponent2x<-1, -1>(e, g, make_float2(jf, jf + 1.0f), sn, h, gg));
        });
    const float steph = g.steph, d0h = g.d0h;
    const int cnt = g.cnt;
    g.steph = 1.0f;   // exponents at half azimuth offsets instead of pixel indices
    g.d0h = 0.0f;
    if (full) {
        // f is periodic in the azimuth and analytic: equally spaced points
        // give its mean, from a phase of the lane's own (so that the rounding
        // of their positions is not the same in every disc; the spacing is a
        // two-float: a relative error of it is one of the sum)
        constexpr float hh = (float)(kPi / kFullPts), hl = (float)(kPi / kFullPts - (double)hh);
        NodeSum n{f2(0.0f), f2(0.0f)};
#pragma unroll 1
        for (int k = 0; k < kFullPts / 2; k++) {
            const float u = (float)(2 * k - kFullPts / 2) + 16.0f * di.shift;
            const float2 m = make_float2(u, u + 1.0f);
            const float2 t = exponent2x<-1, -1>(e, g, fma2(m, f2(hh), mul2(m, f2(hl))), sn, h, gg);
            n.add(ex2_2(add2(t, f2(di.shift))), 1.0f, 0.0f);
        }
        float err;
        const float H = two_sum(n.s.x, n.s.y, err), L = err + (n.sl.x + n.sl.y);
        // The pixels lie at multiples of the FP32 steph from the first, so they
        // cover not the period pi but cnt steph = pi (1 + eps): their sum is
        // cnt (mean - eps (mean - f)), f the weight where the two ends meet.
        // (eps is 2.8e-8 on every equatorial ring of a power-of-two Nside; left
        // out, maps of discs that hold a pole were 2e-9 to 4e-9 too faint.)
        const float eps = (fmaf(steph, (float)cnt, -kPiHi) - kPiLo) * (float)(1.0 / kPi);
        const float fe = ex2_approx(exponent2x<-1, -1>(e, g, f2((float)(0.5 * kPi)), sn, h, gg).x + di.shift);
        const float m = (float)cnt * (1.0f / kFullPts);   // exact
        const float q = H * m, ql = fmaf(H, m, -q) + fmaf(L, m, -eps * fmaf(-(float)cnt, fe, q));
        const float v = q * di.hi;
        return make_float2(v, fmaf(q, di.hi, -v) + fmaf(q, di.lo, ql * di.hi));
    }
    const float2 X = make_float2(fmaf(0.5f, steph, -d0h), fmaf((float)cnt - 0.5f, steph, d0h));
    NodeSum n{f2(0.0f), f2(0.0f)};
#pragma unroll 1
    for (int k = 0; k < kNodesGen; k++)
        n.add(ex2_2(add2(exponent2x<-1, -1>(e, g, mul2(X, f2(kNodeG[k])), sn, h, gg), f2(di.shift))), kGwG[k], kGwGLo[k]);
    const float2 fe = ex2_2(add2(exponent2x<-1, -1>(e, g, X, sn, h, gg), f2(di.shift)));
    // d ln f / du = -K' G'(h) B sin 2x steph, G' = alpha / sin alpha
    const float k1 = 0.693147180560f * e.nK * g.B * steph;
    float g1[2], g2[2];
#pragma unroll
    for (int p = 0; p < 2; p++) {
        const float hp = p ? h.y : h.x, gp = p ? gg.y : gg.x, sp = p ? sn.y : sn.x;
        const float G1 = hp > 1e-20f ? sqrtf(gp / (hp * fmaxf(1.0f - hp, 1e-7f))) : 1.0f;
        const float cp = sqrtf(fmaxf(1.0f - sp * sp, 0.0f));
        g1[p] = k1 * G1 * 2.0f * sp * cp;
        g2[p] = k1 * steph * G1 * 2.0f * (1.0f - 2.0f * sp * sp);
    }
    return ring_total(n, X, end_terms(fe, make_float2(g1[0], g1[1]), make_float2(g2[0], g2[1])), steph, di);
}

// Tile header of every block-class disc.
__global__ void __launch_bounds__(256) k_tile_hdr(DiscArgs a, TileArgs tg) {
    const long long nblk = a.ctr[C_ADD_BLOCK];
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < nblk; q += stride) {
        const CompHdr &c = a.chdr[q];
        TileHdr t;
        t.t0h = (float)c.hdr.theta0;
        t.t0l = (float)(c.hdr.theta0 - (double)t.t0h);
        t.hR = c.ch.hR;
        t.sth0 = c.ch.sth0;
        t.nK = c.ext.nK;
        t.F = t.Flo = t.sh = 0.0f;
        const double turns = c.hdr.phi0 * kInvTwoPi;
        t.ph = (float)turns;
        t.pl = (float)(turns - (double)t.ph);
        t.r_first = c.hdr.r_first;
        t.r_last = c.hdr.r_last;
        t.irmin = c.hdr.irmin;
        t.irmax = c.hdr.irmax;
        t.q = (int)q;
        int kind;
        if (c.ext.tier_x < 2 && c.ext.tier_h < 2)
            kind = c.ext.tier_h == 0 && sinf((float)c.hdr.R) < kPoly3Sin * c.ch.sth0 ? K_POLY3 : K_POLY;
        else
            kind = c.hdr.R < kGiantR ? K_GEN : K_GIANT;
        if (kind != K_GIANT && c.hdr.flux != 0.0 && fabs(c.hdr.flux) * kShare >= fabs(*tg.flux_sum) &&
            atomicAdd(tg.ctl + 2, 1) < kShareMax)
            kind = K_GIANT;
        t.flags = kind | (c.ext.tier_h >= 1 ? kFlagH1 : 0) | (c.hdr.allsky ? kFlagAll : 0) |
                  (c.ch.fast ? kFlagFast : 0) | (c.ext.tier_h == 2 ? kFlagA2 : 0);
        if (kind == K_GEN && t.r_last - t.r_first >= kLongRings) {
            t.flags |= kFlagLong;
            tg.gen[nblk - 1 - atomicAdd(tg.ctl + 3, 1)] = (int)q;
        }
        tg.hdr[q] = t;
        if (kind == K_GIANT) {
            const unsigned long long k = atomicAdd((unsigned long long *)(a.ctr + C_GEN), 1ull);
            tg.gen[k] = (int)q;
        }
    }
}

// A warp's copy of a tile header (callers __syncwarp).
__device__ __forceinline__ void load_thdr(const TileArgs &tg, long long q, TileHdr &dst) {
    const int lane = threadIdx.x & 31;
    if (lane < (int)(sizeof(TileHdr) / 16))
        reinterpret_cast<float4 *>(&dst)[lane] = __ldg(reinterpret_cast<const float4 *>(tg.hdr + q) + lane);
}

// hav(theta + theta0 - pi): the distance to the antipode (see Run).
__device__ __forceinline__ float antipode_term(const TileHdr &h, const RingT &rc) {
    const float d = ((rc.thh - kPiHi) + h.t0h) + ((rc.thl + h.t0l) - kPiLo);
    const float s = sinf(0.5f * d);
    return s * s;
}

// The series' tiers and -K of a general disc.
__device__ __forceinline__ Ext gen_ext(const DiscArgs &a, const TileHdr &h) { return a.chdr[h.q].ext; }

constexpr int kNormWarps = 4;
constexpr int kNormClaim = 4;   // discs per claim
constexpr int kLongParts = 32;  // claims per general disc of more than kLongRings rings

// S and the pixel count of every disc but the giants: a warp per disc, a ring
// per lane.  5.0 ms, bound by FP32 issue (the ring's chord test and 8 or 12
// node values; the segmented render's first pass visits every pixel: 0.41 s
// on the whole set).  A general disc of R = 2 at Nside 1522 has 3900 rings, 26 us
// for each 32 of them: on one warp it took 2.9 ms, half of a map of 3000
// particles.  The long ones come first, in parts.
__global__ void __launch_bounds__(kNormWarps * 32, 7)
    k_tile_norm(const __grid_constant__ DiscArgs a, const __grid_constant__ TileArgs tg) {
    if (tg.ctl[0] != 2) return;
    __shared__ TileHdr sh[kNormWarps];
    const int lane = threadIdx.x & 31;
    TileHdr &h = sh[threadIdx.x >> 5];
    const Dither mine = lane_dither();
    const long long nblk = a.ctr[C_ADD_BLOCK], nparts = (long long)tg.ctl[3] * kLongParts;
    auto claim = [&](unsigned long long *next, int k) {
        long long t = 0;
        if (lane == 0) t = (long long)atomicAdd(next, (unsigned long long)k);
        return __shfl_sync(0xffffffffu, t, 0);
    };
    long long deposits = 0, next = 0, end = 0;
    bool parts = nparts > 0;
    for (;;) {
        long long q;
        int part = -1;
        if (parts) {
            const long long t = claim((unsigned long long *)(tg.ctl + 4), 1);
            if (t >= nparts) {
                parts = false;
                continue;
            }
            q = tg.gen[nblk - 1 - t / kLongParts];
            part = (int)(t % kLongParts);
        } else {
            if (next == end) {
                next = claim((unsigned long long *)(a.ctr + C_TILE_NEXT), kNormClaim);
                if (next >= nblk) break;
                end = min(nblk, next + kNormClaim);
            }
            q = next++;
        }
        __syncwarp();
        load_thdr(tg, q, h);
        __syncwarp();
        const int kind = h.flags & kKindMask;
        if (kind == K_GIANT || (part < 0 && (h.flags & kFlagLong))) continue;
        int r_first = h.r_first, r_last = h.r_last;
        if (part >= 0) {   // whole warps of rings per part
            const int step = ((r_last - r_first) / (32 * kLongParts) + 1) * 32;
            r_first += part * step;
            r_last = min(r_last, r_first + step - 1);
            if (r_first > r_last) continue;
        }
        const Dither di = deal_dither(mine, q);
        float s = 0.0f, c = 0.0f;
        int total = 0;
        if (kind <= K_POLY) {
            const int th = (h.flags & kFlagH1) ? 1 : 0;
            const float nK = h.nK;
            for (int r0 = r_first; r0 <= r_last; r0 += 32) {
                const int ring = r0 + lane;
                if (ring > r_last) continue;
                const RingT rc = ring_t(a, ring);
                int lo;
                float d0h, A, B;
                const int cnt = tile_run<false>(a, h, rc, ring, lo, d0h, A, B);
                if (cnt <= 0) continue;
                float co[5];
                poly_coeffs(A, B, nK, th, co);
                if (kind == K_POLY3) co[4] = 0.0f;   // (the deposits' polynomial)
                const float2 v = ring_sum(co, d0h, 0.5f * rc.step, cnt, di);
                total += cnt;
                float err;
                s = two_sum(s, v.x, err);
                c += err + v.y;
            }
        } else {
            const Ext e = gen_ext(a, h);
            for (int r0 = r_first; r0 <= r_last; r0 += 32) {
                const int ring = r0 + lane;
                if (ring > r_last) continue;
                const RingT rc = ring_t(a, ring);
                Run g{};
                int lo;
                g.cnt = tile_run<true>(a, h, rc, ring, lo, g.d0h, g.A, g.B);
                if (g.cnt <= 0) continue;
                g.steph = 0.5f * rc.step;
                if (h.flags & kFlagA2) g.A2 = antipode_term(h, rc);
                const float2 v = ring_sum_gen(e, g, ring < h.irmin || ring > h.irmax, di);
                total += g.cnt;
                float err;
                s = two_sum(s, v.x, err);
                c += err + v.y;
            }
        }
        __syncwarp();
        warp_sum_ff(s, c);
        total = __reduce_add_sync(0xffffffffu, total);
        if (lane == 0) {
            if (part < 0) {
                tg.disc_S[q] = (double)s + (double)c;
                tg.disc_px[q] = total;
            } else {
                atomicAdd(tg.disc_S + q, (double)s + (double)c);
                atomicAdd((unsigned long long *)(tg.disc_px + q), (unsigned long long)total);
            }
            deposits += total;
        }
    }
    if (lane == 0 && deposits) atomicAdd((unsigned long long *)(a.ctr + C_DEPOSITS), (unsigned long long)deposits);
}

constexpr int kGiantRings = 8;   // rings per claim of a giant disc

// The giants, pixel by pixel: a warp takes kGiantRings rings of a disc, one per
// lane to build, and walks each with all lanes (a ring has up to 4 nside
// pixels, and few discs are giants: short claims spread them over the GPU; 0.34
// ms, and 1.0 ms with claims of 32 rings).
__global__ void __launch_bounds__(kNormWarps * 32)
    k_tile_norm_giant(const __grid_constant__ DiscArgs a, const __grid_constant__ TileArgs tg) {
    if (tg.ctl[0] != 2) return;
    __shared__ TileHdr sh[kNormWarps];
    const int lane = threadIdx.x & 31;
    TileHdr &h = sh[threadIdx.x >> 5];
    const long long parts = (a.g.nrings + kGiantRings - 1) / kGiantRings;
    const long long n = a.ctr[C_GEN] * parts;
    long long deposits = 0;
    for (;;) {
        long long t = 0;
        if (lane == 0) t = (long long)atomicAdd((unsigned long long *)(a.ctr + C_GEN_NEXT), 1ull);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= n) break;
        const long long q = tg.gen[t / parts];
        __syncwarp();
        load_thdr(tg, q, h);
        __syncwarp();
        const int ring = h.r_first + (int)(t % parts) * kGiantRings + lane;
        const Ext e = gen_ext(a, h);
        // each rounding of the sums kept: they start at 1, above every weight
        float2 ks = f2(1.0f), kc = f2(0.0f);
        Run g{};
        if (lane < kGiantRings && ring <= h.r_last) {
            const RingT rc = ring_t(a, ring);
            int lo;
            g.cnt = max(0, tile_run<true>(a, h, rc, ring, lo, g.d0h, g.A, g.B));
            g.steph = 0.5f * rc.step;
            g.A2 = antipode_term(h, rc);
        }
        __syncwarp();
        for (int k = 0; k < kGiantRings; k++) {
            Run r{};
            r.cnt = __shfl_sync(0xffffffffu, g.cnt, k);
            if (r.cnt == 0) continue;
            r.A = __shfl_sync(0xffffffffu, g.A, k);
            r.B = __shfl_sync(0xffffffffu, g.B, k);
            r.A2 = __shfl_sync(0xffffffffu, g.A2, k);
            r.d0h = __shfl_sync(0xffffffffu, g.d0h, k);
            r.steph = __shfl_sync(0xffffffffu, g.steph, k);
            for (int j = lane; j < r.cnt; j += 64) {
                const float jf = (float)j;
                float2 w = weight2<-1, -1>(e, r, make_float2(jf, jf + 32.0f));
                if (j + 32 >= r.cnt) w.y = 0.0f;
                const float2 t = add2(ks, w);
                kc = add2(kc, sub2(w, sub2(t, ks)));
                ks = t;
            }
        }
        float err;
        float s = two_sum(ks.x - 1.0f, ks.y - 1.0f, err), c = (kc.x + kc.y) + err;
        warp_sum_ff(s, c);
        const int total = __reduce_add_sync(0xffffffffu, g.cnt);
        if (lane == 0 && total > 0) {
            atomicAdd(tg.disc_S + q, (double)s + (double)c);
            atomicAdd((unsigned long long *)(tg.disc_px + q), (unsigned long long)total);
            deposits += total;
        }
    }
    if (lane == 0 && deposits) atomicAdd((unsigned long long *)(a.ctr + C_DEPOSITS), (unsigned long long)deposits);
}

// F = flux / S into the disc's tile header; a disc of fewer than two pixels
// puts its whole flux into the centre pixel (genmap.cpp:125-128) and has
// F = 0.  Also the chunk's largest and smallest octave of F.
//
// A deposit is one FMA with a float, and F rounded to one would be an error of
// up to 2^-24 in each of a disc's pixels (a two-float F took two more packed
// operations per pixel pair and 9 % more time).  w F = 2^(t + s) (2^-s F), so
// of kShifts small shifts s of the disc's exponents, which cost nothing, the one
// is taken whose 2^-s F is nearest to a float: within 2^-24 / kShifts on
// average.  The shifts are of either sign, so that ex2's errors on either side
// of an octave stay as the weight sums have them.
constexpr int kShifts = 16;
__device__ __forceinline__ float shift_of(int k) { return (float)(k - kShifts / 2) * (1.0f / 256.0f); }

__global__ void __launch_bounds__(256) k_tile_fin(DiscArgs a, TileArgs tg) {
    if (tg.ctl[0] != 2) return;
    const long long nblk = a.ctr[C_ADD_BLOCK];
    const long long stride = (long long)gridDim.x * blockDim.x;
    __shared__ float2 pow2[kShifts];   // 2^-shift as a two-float
    if (threadIdx.x < kShifts) {
        const double v = exp2(-(double)shift_of(threadIdx.x));
        pow2[threadIdx.x].x = (float)v;
        pow2[threadIdx.x].y = (float)(v - (double)(float)v);
    }
    __syncthreads();
    int hi = 0, lo = 0;   // largest octave, 255 - the smallest
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < nblk; q += stride) {
        const DiscHdr &d = a.chdr[q].hdr;
        const double fs = d.flux * a.f.inv_scale;
        const long long px = tg.disc_px[q];
        float F = 0.0f, Flo = 0.0f, sh = 0.0f;
        TileHdr &t = tg.hdr[q];
        if (px < 2) {
            red_add_f64(a.acc.acc64 + d.cpix, fs);
            atomicAdd((unsigned long long *)(a.ctr + C_DEPOSITS), (unsigned long long)(1 - px));
        } else {
            const double Fd = fs / tg.disc_S[q];
            F = (float)Fd;
            Flo = (float)(Fd - (double)F);
            if ((t.flags & kKindMask) != K_GIANT && Flo != 0.0f) {
                const float Fh = F, Fl = Flo;
                float best = fabsf(Flo);
                for (int k = 0; k < kShifts; k++) {
                    const float2 g = pow2[k];
                    const float v = Fh * g.x, e = fmaf(Fh, g.x, -v) + fmaf(Fh, g.y, Fl * g.x);
                    if (fabsf(e) < best) {
                        best = fabsf(e);
                        F = v;
                        Flo = e;
                        sh = shift_of(k);
                    }
                }
            }
        }
        t.F = F;
        t.Flo = Flo;
        t.sh = sh;
        if (F != 0.0f) {
            const int oct = (int)((__float_as_uint(F) >> 23) & 255);
            hi = max(hi, oct);
            lo = max(lo, 255 - oct);
        }
    }
    hi = __reduce_max_sync(0xffffffffu, hi);
    lo = __reduce_max_sync(0xffffffffu, lo);
    if ((threadIdx.x & 31) == 0) {
        int *const c = reinterpret_cast<int *>(a.ctr + C_OCT);
        if (hi > 0) atomicMax(c, hi);
        if (lo > 0) atomicMax(c + 1, lo);
    }
}

// ------------------------------------------------------------ pairs
// The tile columns that disc h can touch in strip s, conservatively (the
// deposit kernels test every pixel's run exactly): [c0, c1] and, where the
// disc wraps past azimuth 0, [c2, c3] behind it (c2 > c3: none).  The chord's
// half-width over the strip's rings is at most that of q = (hav R - A) /
// (sin theta sin theta0) with the strip's smallest A and sin theta (a concave
// function: at one of its ends), FP32 with the numerator enlarged by more
// than its rounding error.  A pixel's centre lies 0 or 1/2 pixel behind its
// index and FP32 places indices below 2^15 to 4e-3 pixels: 0.75 pixels of
// margin on either side.
__device__ inline void strip_cols(const DiscArgs &a, const TileHdr &h, int s, int &nlo, int &c0, int &c1,
                                  int &c2, int &c3) {
    const int ra = max(h.r_first, s * kTileR + 1), rb = min(h.r_last, s * kTileR + kTileR);
    const int na = ring_npix(a.g, ra), nb = ring_npix(a.g, rb);
    nlo = min(na, nb);
    const int nhi = (ra <= 3 * a.g.nside && rb >= a.g.nside) ? 4 * a.g.nside : max(na, nb);
    c2 = 1;
    c3 = 0;
    c0 = 0;
    c1 = (nhi - 1) / kTileW;
    if ((h.flags & kFlagAll) || ra < h.irmin || rb > h.irmax) return;
    const float d = fmaxf(0.0f, fmaxf(a.rt.th2[ra].x - h.t0h, h.t0h - a.rt.th2[rb].x) - 1e-6f);
    const float sd = __sinf(0.5f * d) * 0.9999f;
    const float smin = fminf(a.rt.st32[ra], a.rt.st32[rb]);
    const float num = fmaxf(h.hR * 1.00001f - sd * sd, 0.0f) + 1e-12f;
    const float q = num / (smin * h.sth0);
    if (!(q < 0.98f)) return;
    const float D = 2.0f * asinf(sqrtf(q)) * (1.0001f / 6.28318531f);   // in turns
    const float margin = 0.75f / (float)nlo;
    const float lo = h.ph - D - margin, hi = h.ph + D + margin;
    if (hi - lo >= 0.999f) return;
    const float fl = (float)nlo, fh = (float)nhi;
    auto col_lo = [&](float v) { return max(0, (int)floorf(fl * v)) / kTileW; };
    auto col_hi = [&](float v) { return min(nhi - 1, (int)floorf(fh * v)) / kTileW; };
    const int cmax = c1;
    if (lo < 0.0f || hi >= 1.0f) {
        c1 = col_hi(lo < 0.0f ? hi : hi - 1.0f);
        c2 = min(cmax, col_lo(lo < 0.0f ? lo + 1.0f : lo));
        c3 = cmax;
        if (c2 <= c1) {   // the two ranges meet: the whole strip
            c1 = cmax;
            c2 = 1;
            c3 = 0;
        }
        return;
    }
    c0 = min(col_lo(lo), cmax);
    c1 = max(c0, col_hi(hi));
}

constexpr int kPairLanes = 8;    // lanes (strips at a time) per disc
constexpr int kWideParts = 64, kWideStrips = 96;   // warps of a giant or long disc of more strips than that

// MODE 0: the chunk's pairs, before S is known (for its mode; at least those
// of mode 1, which leaves out discs with nothing to deposit); 1: pairs per
// (tile, octave); 2: the pair list.  Bound by the latency of the slot atomics:
// mode 2 takes 1.3 ms with four on their way, 2.7 ms one at a time.  The tallest
// of the giants and long discs have their strips dealt to kWideParts warps, a
// column per lane: one disc over the whole map at Nside 8192, half a million
// pairs, kept its 8 lanes busy for 11 ms.  (With every long disc dealt out the
// three modes take 1.16 ms of 1M particles at Nside 512 instead of 0.48.)
template <int MODE>
__global__ void __launch_bounds__(256) k_tile_pairs(DiscArgs a, TileArgs tg) {
    if (MODE != 0 && tg.ctl[0] != 2) return;
    const long long nblk = a.ctr[C_ADD_BLOCK];
    const int sl = threadIdx.x % kPairLanes, lane = threadIdx.x & 31;
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long threads = (long long)gridDim.x * blockDim.x;
    const int *const oc = reinterpret_cast<const int *>(a.ctr + C_OCT);
    const int omax = MODE ? oc[0] : 0, omin = MODE ? 255 - oc[1] : 0;
    const int NT = tg.nstrips * tg.ncol;
    long long total = 0, list[kTileLists] = {};
    // a disc's class, negative with nothing to deposit (weights are >= exp(-6))
    auto class_of = [&](const TileHdr &h) {
        if (MODE == 0) return 0;
        return h.F == 0.0f ? -1 : tile_class((int)((__float_as_uint(h.F) >> 23) & 255), omax, omin);
    };
    auto list_of = [](const TileHdr &h, int nlo) {
        const int kind = h.flags & kKindMask;
        return kind <= K_POLY ? kind : kind == K_GEN && nlo >= kFineNr ? 2 : 3;
    };
    auto tally = [&](int which, int np) {
        if (MODE == 0) total += np;
#pragma unroll
        for (int k = 0; k < kTileLists; k++) list[k] += which == k ? np : 0;
    };
    auto wide = [](const TileHdr &h) {
        return ((h.flags & kKindMask) == K_GIANT || (h.flags & kFlagLong)) && h.r_last - h.r_first >= kWideStrips * kTileR;
    };
    const long long ngiant = a.ctr[C_GEN];
    const long long nwide = tg.nstrips > kWideStrips ? (ngiant + tg.ctl[3]) * kWideParts : 0;
    for (long long t = tid / 32; t < nwide; t += threads / 32) {
        const long long k = t / kWideParts;
        const int q = tg.gen[k < ngiant ? k : nblk - 1 - (k - ngiant)];
        const TileHdr h = tg.hdr[q];
        const int cls = class_of(h);
        if (cls < 0 || !wide(h)) continue;
        const int s1 = (h.r_last - 1) / kTileR;
        for (int s = (h.r_first - 1) / kTileR + (int)(t % kWideParts); s <= s1; s += kWideParts) {
            int nlo, c0, c1, c2, c3;
            strip_cols(a, h, s, nlo, c0, c1, c2, c3);
            const int n0 = c1 - c0 + 1, np = n0 + max(0, c3 - c2 + 1), which = list_of(h, nlo);
            if (lane == 0) tally(which, np);
            if (MODE == 0) continue;
            for (int i = lane; i < np; i += 32) {
                const int tile = which * NT + s * tg.ncol + (i < n0 ? c0 + i : c2 + (i - n0));
                const unsigned slot = atomicAdd(tg.hist + ((size_t)tile << kClsBits) + cls, 1u);
                if (MODE == 2) tg.list[tg.base[tile] + slot] = (unsigned)q;
            }
        }
    }
    for (long long q = tid / kPairLanes; q < nblk; q += threads / kPairLanes) {
        TileHdr h = tg.hdr[q];
        const int cls = class_of(h);
        if (cls < 0 || wide(h)) continue;
        const int s1 = h.r_last >= h.r_first ? (h.r_last - 1) / kTileR : -1;
        for (int s = (h.r_first - 1) / kTileR + sl; s <= s1; s += kPairLanes) {
            int nlo, c0, c1, c2, c3;
            strip_cols(a, h, s, nlo, c0, c1, c2, c3);
            const int n0 = c1 - c0 + 1, np = n0 + max(0, c3 - c2 + 1), which = list_of(h, nlo), t0 = which * NT;
            tally(which, np);
            if (MODE == 0) continue;
            // the columns of both ranges, four atomics on their way at a time
            for (int i = 0; i < np; i += 4) {
                unsigned k[4];
                int t[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int c = i + u < n0 ? c0 + i + u : c2 + (i + u - n0);
                    t[u] = t0 + s * tg.ncol + c;
                    if (i + u < np) k[u] = atomicAdd(tg.hist + ((size_t)t[u] << kClsBits) + cls, 1u);
                }
                if (MODE == 2) {
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        if (i + u < np) tg.list[tg.base[t[u]] + k[u]] = (unsigned)q;
                }
            }
        }
    }
    auto count = [&](int at, long long v) {
        v = warp_sum_ll(v);
        if ((threadIdx.x & 31) == 0 && v) atomicAdd((unsigned long long *)(a.ctr + at), (unsigned long long)v);
    };
    if (MODE == 0) count(C_TILE_BOUND, total);
    if (MODE == 1)
        for (int k = 0; k < kTileLists; k++) count(C_TILE_PAIRS + k, list[k]);
}

// The first unit of list k.
__device__ __forceinline__ long long first_unit(const DiscArgs &a, const TileArgs &tg, int k) {
    long long f = 0;
    for (int j = 0; j < k; j++) f += tile_units_of(a.ctr[C_TILE_PAIRS + j], (long long)tg.nstrips * tg.ncol);
    return f;
}

// Each tile's range of the pair list and its units: a warp per tile.
__global__ void __launch_bounds__(256) k_tile_plan(DiscArgs a, TileArgs tg) {
    if (tg.ctl[0] != 2) return;
    const int lane = threadIdx.x & 31;
    const int NT = tg.nstrips * tg.ncol;
    const int nt = kTileLists * NT;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < nt; t += nw) {
        static_assert(kCls == 64, "two octaves per lane");
        uint2 *hp = reinterpret_cast<uint2 *>(tg.hist + ((size_t)t << kClsBits)) + lane;
        const uint2 v = *hp;
        int total;
        const int ex = warp_excl_scan((int)(v.x + v.y), total);
        if (total == 0) continue;
        *hp = make_uint2((unsigned)ex, (unsigned)ex + v.x);
        const int which = t / NT;
        const int ulen = tile_unit_len(a.ctr[C_TILE_PAIRS + which]), nu = (total + ulen - 1) / ulen;
        long long b = 0, u = 0;
        if (lane == 0) {
            b = (long long)atomicAdd((unsigned long long *)(a.ctr + C_TILE_CURSOR), (unsigned long long)total);
            u = (long long)atomicAdd((unsigned long long *)(a.ctr + C_UNITS + which), (unsigned long long)nu);
            tg.base[t] = b;
        }
        b = __shfl_sync(0xffffffffu, b, 0);
        u = __shfl_sync(0xffffffffu, u, 0);
        const int per = (total + nu - 1) / nu;
        TileUnit *out = tg.units + first_unit(a, tg, which) + u;
        for (int k = lane; k < nu; k += 32) {
            TileUnit w;
            w.start = b + (long long)k * per;
            w.len = min(per, total - k * per);
            w.tile = t - which * NT;
            out[k] = w;
        }
    }
}

// ------------------------------------------------------------ deposits
// One disc of a unit: the lane's run in tile coordinates as up to two pieces
// (the second behind the wrap of the ring index).  Tile pixel t of a piece is
// pixel t - a of the run.
struct Piece {
    int a;       // tile coordinate of the run's pixel 0 (as this piece sees it)
    int s, e;    // tile pixels [s, e)
};

template <int W = kTileW>
__device__ __forceinline__ Piece piece_of(int p, int lo, int cnt, int nr, int base) {
    // in-ring index of the run's first pixel and the pixels before the wrap
    const int i0 = lo < 0 ? lo + nr : lo;
    const int n0 = min(cnt, nr - i0);
    Piece r;
    r.a = p ? -base - n0 : i0 - base;
    const int first = p ? -base : r.a, end = p ? cnt - n0 - base : r.a + n0;
    r.s = max(first, 0);
    r.e = min(end, W);
    return r;
}

constexpr int kDepWarps = 4;
constexpr int kDepBlocks = 4;
constexpr int kGroupPx = 8;                      // pixels per skip test
constexpr int kGroups = kTileW / kGroupPx;

__device__ __forceinline__ unsigned mask_below(int n) {   // bits 0 .. n-1, n clamped to [0, 32]
    unsigned m;
    asm("bmsk.clamp.b32 %0, 0, %1;" : "=r"(m) : "r"(max(n, 0)));
    return m;
}

// A piece's pixels as a bit mask, and the pixel groups any lane of the warp
// touches.
struct Masks {
    unsigned m[kTileW / 32], groups;
};

__device__ __forceinline__ Masks masks_of(const Piece &pc) {
    Masks k;
#pragma unroll
    for (int i = 0; i < kTileW / 32; i++) k.m[i] = mask_below(pc.e - 32 * i) & ~mask_below(pc.s - 32 * i);
    unsigned gm = 0;
    if (pc.e > pc.s) gm = ((2u << ((pc.e - 1) / kGroupPx)) - 1u) & ~((1u << (pc.s / kGroupPx)) - 1u);
    k.groups = __reduce_or_sync(0xffffffffu, gm);
    return k;
}

// The deposits w F of group g (weights w, pair by pair) into the lane's row.
// (Packed products with F = 0 in the lanes outside, where no lane covers the
// group in part, took as long; and a weight outside the run may be infinite.)
__device__ __forceinline__ void add_group(float2 (&acc)[kTileW / 2], int g, const Masks &mk,
                                          const float2 (&w)[kGroupPx / 2], float2 F) {
    const unsigned mw = mk.m[g * kGroupPx / 32] >> (g * kGroupPx % 32);
#pragma unroll
    for (int k = 0; k < kGroupPx / 2; k++) {
        float2 &r = acc[g * (kGroupPx / 2) + k];
        if (mw & (1u << (2 * k))) r.x = fmaf(w[k].x, F.x, r.x);
        if (mw & (2u << (2 * k))) r.y = fmaf(w[k].y, F.y, r.y);
    }
}

// A piece of a polynomial disc.
template <bool P3>
__device__ __forceinline__ void add_poly(float2 (&acc)[kTileW / 2], const Piece &pc, const float c[5], float d0h,
                                         float steph, float2 F) {
    const Masks mk = masks_of(pc);
    const float2 jb = make_float2((float)(-pc.a), (float)(1 - pc.a));
    const float2 st2 = f2(steph), d02 = f2(d0h), two = f2(2.0f);
#pragma unroll
    for (int g = 0; g < kGroups; g++) {
        if (!(mk.groups & (1u << g))) continue;
        float2 j = add2(jb, f2((float)(g * kGroupPx)));   // exact: x is rounded as in the weight sums
        float2 w[kGroupPx / 2];
#pragma unroll
        for (int k = 0; k < kGroupPx / 2; k++) {
            const float2 x = fma2(j, st2, d02);
            w[k] = ex2_2(poly_exp2<P3>(c, mul2(x, x)));
            j = add2(j, two);
        }
        add_group(acc, g, mk, w, F);
    }
}

// A piece of a general disc: over 32 pixels at a time the exponent is the
// polynomial of degree 5 through its values (run-time series) at six
// Chebyshev points, on rings whose pixels are narrow enough.  With a = 16
// steps of the half azimuth offset the remainder is about 0.05 a^6 / R^2: 3e-8
// in the exponent of 2 for a < 0.06 (kFineNr) and R > 0.28, a tenth of the
// exponent's FP32 rounding.
constexpr int kSubPx = 32;

// (a call: inlined at its six places it pushes the kernel out of the
// instruction cache)
__device__ __noinline__ float2 gen_exponent(float nK, int tier_x, int tier_h, float A, float B, float A2, float2 x) {
    Ext e{};
    e.nK = nK;
    e.tier_x = tier_x;
    e.tier_h = tier_h;
    Run r{};
    r.A = A;
    r.B = B;
    r.A2 = A2;
    r.steph = 1.0f;   // x: half azimuth offsets
    float2 sn, h, g;
    return exponent2x<-1, -1>(e, r, x, sn, h, g);
}

__device__ __forceinline__ void add_gen(float2 (&acc)[kTileW / 2], const Piece &pc, const Ext &e, const Run &r,
                                        float2 F, float shift) {
    // near Chebyshev points (0.966, 0.707, 0.259 of 16 pixels) exact in FP32,
    // squares too; the reciprocals as FP32 pairs: an error of these constants
    // would be the same in every disc
    constexpr float n1 = 31.0f / 32.0f, n2 = 23.0f / 32.0f, n3 = 8.0f / 32.0f;
    constexpr float m2 = n2 * n2, m3 = n3 * n3;
    constexpr double r12 = 1024.0 / 432.0, r23 = 1024.0 / 465.0;
    constexpr float i12 = (float)r12, i12l = (float)(r12 - (double)i12), i23 = (float)r23, i23l = (float)(r23 - (double)i23);
    constexpr float i13 = (float)(1024.0 / 897.0);
    const Masks mk = masks_of(pc);
#pragma unroll
    for (int b = 0; b < kTileW / kSubPx; b++) {
        constexpr unsigned kSubGroups = (1u << (kSubPx / kGroupPx)) - 1u;
        if (!(mk.groups & (kSubGroups << (b * (kSubPx / kGroupPx))))) continue;
        const float2 jc = f2((float)(b * kSubPx - pc.a) + 0.5f * (kSubPx - 1));   // centre, in pixels of the run
        constexpr float hw = kSubPx / 2;
        auto value = [&](float n) {
            const float2 x = fma2(add2(jc, make_float2(-n * hw, n * hw)), f2(r.steph), f2(r.d0h));
            return gen_exponent(e.nK, e.tier_x, e.tier_h, r.A, r.B, r.A2, x);
        };
        const float2 v1 = value(n1), v2 = value(n2), v3 = value(n3);
        // even part and odd part over n, each a quadratic in n^2 through
        // three points (Newton's divided differences)
        constexpr double c1 = 16.0 / 31.0, c2 = 16.0 / 23.0;
        constexpr float c1h = (float)c1, c1l = (float)(c1 - (double)c1h), c2h = (float)c2, c2l = (float)(c2 - (double)c2h);
        const float o1 = v1.y - v1.x, o2 = v2.y - v2.x, o3 = v3.y - v3.x;
        const float2 p1 = make_float2(0.5f * (v1.y + v1.x), fmaf(o1, c1h, o1 * c1l));
        const float2 p2 = make_float2(0.5f * (v2.y + v2.x), fmaf(o2, c2h, o2 * c2l));
        const float2 p3 = make_float2(0.5f * (v3.y + v3.x), 2.0f * o3);
        const float2 s12 = sub2(p1, p2), s23 = sub2(p2, p3);
        const float2 d23 = fma2(s23, f2(i23), mul2(s23, f2(i23l)));
        const float2 q2 = mul2(sub2(fma2(s12, f2(i12), mul2(s12, f2(i12l))), d23), f2(i13));
        const float2 q1 = fma2(q2, f2(-(m2 + m3)), d23);
        float2 q0 = fma2(f2(-m3), fma2(q2, f2(-m2), d23), p3);
        q0.x += shift;
#pragma unroll
        for (int gg = 0; gg < kSubPx / kGroupPx; gg++) {
            const int gi = b * (kSubPx / kGroupPx) + gg;
            if (!(mk.groups & (1u << gi))) continue;
            float2 w[kGroupPx / 2];
#pragma unroll
            for (int k = 0; k < kGroupPx / 2; k++) {
                const float t = (float)(gg * kGroupPx + 2 * k) - 0.5f * (kSubPx - 1);
                const float2 v = make_float2(t * (2.0f / kSubPx), (t + 1.0f) * (2.0f / kSubPx));
                float2 x = fma2(v, f2(q2.y), f2(q2.x));
                x = fma2(v, x, f2(q1.y));
                x = fma2(v, x, f2(q1.x));
                x = fma2(v, x, f2(q0.y));
                w[k] = ex2_2(fma2(v, x, f2(q0.x)));
            }
            add_group(acc, gi, mk, w, F);
        }
    }
}

__device__ __forceinline__ void prefetch_hdr(const TileArgs &tg, unsigned q, TileHdr *dst) {
    const int lane = threadIdx.x & 31;
    if (lane < (int)(sizeof(TileHdr) / 16)) {
        const unsigned d = (unsigned)__cvta_generic_to_shared(reinterpret_cast<char *>(dst) + 16 * lane);
        const char *s = reinterpret_cast<const char *>(tg.hdr + q) + 16 * lane;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(s) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// Calls body(h) with the header of each disc of the unit, the next one on
// its way meanwhile (buf: two headers of the warp).
template <class Body>
__device__ __forceinline__ void for_items(const TileArgs &tg, const TileUnit &un, TileHdr *buf, Body body) {
    const int lane = threadIdx.x & 31;
    unsigned ids = 0, nids = lane < un.len ? tg.list[un.start + lane] : 0;
    __syncwarp();
    prefetch_hdr(tg, __shfl_sync(0xffffffffu, nids, 0), buf);
    for (int i = 0; i < un.len; i++) {
        if ((i & 31) == 0) {   // 32 list entries at a time, the next 32 ahead
            ids = nids;
            nids = i + 32 + lane < un.len ? tg.list[un.start + i + 32 + lane] : 0;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();   // this header is complete, the other buffer is free
        const unsigned q1 = __shfl_sync(0xffffffffu, ((i + 1) & 31) ? ids : nids, (i + 1) & 31);
        if (i + 1 < un.len) prefetch_hdr(tg, q1, buf + ((i + 1) & 1));
        body(buf[i & 1]);
    }
}

// Units of one list: 0 and 1 polynomial discs (K_POLY3, K_POLY), 2 general
// discs on fine rings, 3 the other general discs and the giants.  (Each list
// has a kernel of its own: together they do not fit the instruction cache.)
// Lists 0 to 2 take 20.3, 3.4 and 2.2 ms, the pixel kernel 0.7 ms.  Bound by
// issue (72 % of the slots): per (disc, tile) about 580 instructions -- a ring's
// chord test per lane, then 3.5 instructions a pixel (exponent, ex2, the
// predicated product) over the groups that any lane covers.
__device__ __forceinline__ bool claim_unit(const DiscArgs &a, const TileArgs &tg, int which, TileUnit &un) {
    long long u = 0;
    if ((threadIdx.x & 31) == 0) u = (long long)atomicAdd((unsigned long long *)(a.ctr + C_UNEXT + which), 1ull);
    u = __shfl_sync(0xffffffffu, u, 0);
    if (u >= a.ctr[C_UNITS + which]) return false;
    un = tg.units[first_unit(a, tg, which) + u];
    return true;
}

template <int LIST>
__global__ void __launch_bounds__(kDepWarps * 32, kDepBlocks)
    k_tile_dep(const __grid_constant__ DiscArgs a, const __grid_constant__ TileArgs tg) {
    if (tg.ctl[0] != 2) return;
    constexpr bool GEN = LIST == 2;
    __shared__ TileHdr sh[kDepWarps][2];
    __shared__ float tr[kDepWarps][32 * 33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    TileUnit un;
    while (claim_unit(a, tg, LIST, un)) {
        const int strip = un.tile / tg.ncol, base = (un.tile - strip * tg.ncol) * kTileW;
        const int ring = min(strip * kTileR + 1 + lane, a.g.nrings);
        const bool own = strip * kTileR + 1 + lane <= a.g.nrings;
        const RingT rc = ring_t(a, ring);
        float2 acc[kTileW / 2];
#pragma unroll
        for (int k = 0; k < kTileW / 2; k++) acc[k] = f2(0.0f);
        for_items(tg, un, sh[w], [&](const TileHdr &h) {
            int lo = 0, cnt = 0;
            Run r{};
            r.steph = 0.5f * rc.step;
            if (own && ring >= h.r_first && ring <= h.r_last)
                cnt = max(0, tile_run<GEN>(a, h, rc, ring, lo, r.d0h, r.A, r.B));
            __syncwarp();
            const float2 F = f2(h.F);
            Piece pc{0, 0, 0};
            if (cnt > 0) pc = piece_of(0, lo, cnt, rc.nr, base);
            const bool second = __any_sync(0xffffffffu, cnt > 0 && (lo < 0 || lo + cnt > rc.nr));
            bool some = __any_sync(0xffffffffu, pc.e > pc.s);
            if (!some && !second) return;
            float co[5];
            Ext e{};
            if constexpr (GEN) {
                if (h.flags & kFlagA2) r.A2 = antipode_term(h, rc);
                e = gen_ext(a, h);
            } else {
                poly_coeffs(r.A, r.B, h.nK, LIST == 1 && (h.flags & kFlagH1) ? 1 : 0, co);
                co[0] += h.sh;
            }
#pragma unroll 1
            for (int p = 0;; p++) {
                if (some) {
                    if constexpr (GEN) add_gen(acc, pc, e, r, F, h.sh);
                    else add_poly<LIST == 0>(acc, pc, co, r.d0h, r.steph, F);
                }
                if (p == 1 || !second) break;
                pc = Piece{0, 0, 0};
                if (cnt > 0) pc = piece_of(1, lo, cnt, rc.nr, base);
                some = __any_sync(0xffffffffu, pc.e > pc.s);
            }
        });
        // the tile into the FP64 plane: one reduction per non-zero pixel, 32
        // consecutive pixels of a ring per instruction (through shared
        // memory; a lane holds a row)
        const long long row = ring_start(a.g, ring) + base;
#pragma unroll
        for (int k = 0; k < kTileW / 32; k++) {
            __syncwarp();
#pragma unroll
            for (int t = 0; t < 16; t++) {
                tr[w][lane * 33 + 2 * t] = acc[16 * k + t].x;
                tr[w][lane * 33 + 2 * t + 1] = acc[16 * k + t].y;
            }
            __syncwarp();
            for (int r = 0; r < kTileR; r++) {
                const float v = tr[w][r * 33 + lane];
                const long long p = __shfl_sync(0xffffffffu, row, r);
                if (v != 0.0f) red_add_f64(a.acc.acc64 + (p + 32 * k + lane), (double)v);
            }
        }
        __syncwarp();
    }
}

// Exponents of eight consecutive pixels.  The far hemisphere's library calls
// stand side by side: behind a branch per pixel each waited for the one before
// (300 discs of R = 2.5 at Nside 1024: 16.9 -> 15.7 ms).
__device__ __forceinline__ void exponents8(const Ext &e, const Run &r, float j, float2 (&t)[4]) {
    float2 sn, h[4], g[4];
    if (e.tier_h < 2) {
#pragma unroll
        for (int k = 0; k < 4; k++) t[k] = exponent2x<-1, -1>(e, r, make_float2(j + 2 * k, j + 2 * k + 1), sn, h[k], g[k]);
        return;
    }
    float top = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        t[k] = exponent2x<-1, 3>(e, r, make_float2(j + 2 * k, j + 2 * k + 1), sn, h[k], g[k]);
        top = fmaxf(top, fmaxf(h[k].x, h[k].y));
    }
    if (!(top > 0.5f)) return;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float2 x = fma2(make_float2(j + 2 * k, j + 2 * k + 1), f2(r.steph), f2(r.d0h));
        const float2 far = make_float2(g_far(x.x, r), g_far(x.y, r));
        t[k] = mul2(make_float2(h[k].x > 0.5f ? far.x : g[k].x, h[k].y > 0.5f ? far.y : g[k].y), f2(e.nK));
    }
}

constexpr int kGenWarps = 2;
constexpr int kPxW = kTileW / 2;

// The general discs on coarser rings, and the giants: each pixel's weight from
// the run-time series, eight pixels at a time, into a pixel in shared memory
// that is a two-float, added to with TwoSum: one giant can be most of a map's
// flux, and its FP32 deposits and sums left 1e-9 of it.  A warp takes half of a
// tile's columns at a time (one row per lane, rows an odd number of words
// apart): with 8 KB a warp instead of 17 as many are resident as the registers
// allow.
__global__ void __launch_bounds__(kGenWarps * 32)
    k_tile_dep_px(const __grid_constant__ DiscArgs a, const __grid_constant__ TileArgs tg) {
    if (tg.ctl[0] != 2) return;
    constexpr int kRow = kPxW + 1, kStep = 8;
    __shared__ TileHdr sh[kGenWarps][2];
    __shared__ float2 tile[kGenWarps][32 * kRow];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float2 *const my = tile[w] + lane * kRow;
    const long long halves = 2 * a.ctr[C_UNITS + 3], first = first_unit(a, tg, 3);
    for (;;) {
        long long u = 0;
        if (lane == 0) u = (long long)atomicAdd((unsigned long long *)(a.ctr + C_UNEXT + 3), 1ull);
        u = __shfl_sync(0xffffffffu, u, 0);
        if (u >= halves) break;
        const TileUnit un = tg.units[first + (u >> 1)];
        const int strip = un.tile / tg.ncol, base = (un.tile - strip * tg.ncol) * kTileW + (int)(u & 1) * kPxW;
        const int ring = min(strip * kTileR + 1 + lane, a.g.nrings);
        const bool own = strip * kTileR + 1 + lane <= a.g.nrings;
        const RingT rc = ring_t(a, ring);
        for (int t = 0; t < kPxW; t++) my[t] = f2(0.0f);
        for_items(tg, un, sh[w], [&](const TileHdr &h) {
            Run r{};
            int lo = 0, cnt = 0;
            if (own && ring >= h.r_first && ring <= h.r_last)
                cnt = max(0, tile_run<true>(a, h, rc, ring, lo, r.d0h, r.A, r.B));
            __syncwarp();
            r.steph = 0.5f * rc.step;
            if (h.flags & kFlagA2) r.A2 = antipode_term(h, rc);
            const Ext e = gen_ext(a, h);
            const float2 F2 = f2(h.F), Fl2 = f2(h.Flo), sh2 = f2(h.sh);
#pragma unroll 1
            for (int p = 0; p < 2; p++) {
                Piece pc{0, kPxW, 0};
                if (cnt > 0) pc = piece_of<kPxW>(p, lo, cnt, rc.nr, base);
                if (pc.e <= pc.s) pc.s = kPxW, pc.e = 0;
                const int s = __reduce_min_sync(0xffffffffu, pc.s), end = __reduce_max_sync(0xffffffffu, pc.e);
                for (int t = s; t < end; t += kStep) {
                    float2 wt[kStep / 2], wl[kStep / 2];   // w (F + Flo) as a two-float
                    exponents8(e, r, (float)(t - pc.a), wl);
#pragma unroll
                    for (int k = 0; k < kStep / 2; k++) {
                        const float2 wk = ex2_2(add2(wl[k], sh2));
                        wt[k] = mul2(wk, F2);
                        wl[k] = fma2(wk, Fl2, fma2(wk, F2, make_float2(-wt[k].x, -wt[k].y)));
                    }
                    auto add = [&](int at, float v, float lo) {
                        if (at < pc.s || at >= pc.e) return;
                        const float2 m = my[at];
                        float err;
                        const float sum = two_sum(m.x, v, err);
                        my[at] = make_float2(sum, m.y + (err + lo));
                    };
#pragma unroll
                    for (int k = 0; k < kStep / 2; k++) {
                        add(t + 2 * k, wt[k].x, wl[k].x);
                        add(t + 2 * k + 1, wt[k].y, wl[k].y);
                    }
                }
            }
        });
        const long long row = ring_start(a.g, ring) + base;
        __syncwarp();
        for (int r = 0; r < kTileR; r++) {
            const long long p = __shfl_sync(0xffffffffu, row, r);
            const float2 v = tile[w][r * kRow + lane];
            if (v.x != 0.0f) red_add_f64(a.acc.acc64 + (p + lane), (double)v.x + (double)v.y);
        }
        __syncwarp();
    }
}
static_assert(kPxW == 32, "a lane per column of the half");

template <class K>
int resident(K k, int threads) {
    int o = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k, threads, 0) != cudaSuccess) {
        cudaGetLastError();
        o = 1;
    }
    return o < 1 ? 1 : o;
}

}  // namespace

cudaError_t launch_tile_hdr(const DiscArgs &a, const TileArgs &tg, bool count, int num_sms, cudaStream_t s) {
    k_tile_hdr<<<num_sms * 8, 256, 0, s>>>(a, tg);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || !count) return e;
    k_tile_pairs<0><<<num_sms * 8, 256, 0, s>>>(a, tg);
    return cudaGetLastError();
}

cudaError_t launch_tile_norm(const DiscArgs &a, const TileArgs &tg, int num_sms, cudaStream_t s) {
    static const int occ = resident(k_tile_norm, kNormWarps * 32), occg = resident(k_tile_norm_giant, kNormWarps * 32);
    k_tile_norm<<<num_sms * occ, kNormWarps * 32, 0, s>>>(a, tg);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_tile_norm_giant<<<num_sms * occg, kNormWarps * 32, 0, s>>>(a, tg);
    return cudaGetLastError();
}

cudaError_t launch_tile_deposits(const DiscArgs &a, const TileArgs &tg, int num_sms, cudaStream_t s) {
    static const int occ0 = resident(k_tile_dep<0>, kDepWarps * 32), occ1 = resident(k_tile_dep<1>, kDepWarps * 32),
                     occ2 = resident(k_tile_dep<2>, kDepWarps * 32), occp = resident(k_tile_dep_px, kGenWarps * 32);
    k_tile_fin<<<num_sms * 8, 256, 0, s>>>(a, tg);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_tile_pairs<1><<<num_sms * 8, 256, 0, s>>>(a, tg);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    k_tile_plan<<<num_sms * 4, 256, 0, s>>>(a, tg);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    k_tile_pairs<2><<<num_sms * 8, 256, 0, s>>>(a, tg);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    k_tile_dep<0><<<num_sms * occ0, kDepWarps * 32, 0, s>>>(a, tg);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    k_tile_dep<1><<<num_sms * occ1, kDepWarps * 32, 0, s>>>(a, tg);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    k_tile_dep<2><<<num_sms * occ2, kDepWarps * 32, 0, s>>>(a, tg);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    k_tile_dep_px<<<num_sms * occp, kGenWarps * 32, 0, s>>>(a, tg);
    return cudaGetLastError();
}

}  // namespace dmann
