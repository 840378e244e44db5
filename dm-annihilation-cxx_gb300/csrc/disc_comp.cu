// disc_comp.cu -- the compensated-FP32 form's per-disc kernels: a block or
// a warp renders one disc in two passes (normalisation, then deposits as
// FP64 reductions), the compensated adjoint, and the disc headers.  The
// arithmetic (chord test, weights, two-float sums) is in comp_engine.cuh.
#include "comp_engine.cuh"

namespace dmann {

namespace {

// Both passes of one disc particle (tiers TX, TH; see weight2x), after
// render_particle has staged its header.
template <int G, int RCH, int TX, int TH>
__device__ void render_disc(const DiscArgs &a, CompSmem<RCH> &sm, const Ext &e) {
    using Gp = Grp<G>;
    const int rk = Gp::rank();
    const int r_first = sm.h.hdr.r_first, r_last = sm.h.hdr.r_last;
    const int nring = r_last - r_first + 1;
    const int nchunk = nring > 0 ? (nring + RCH - 1) / RCH : 0;

    // pass 1: the normalisation, a compensated sum per lane (both halves).
    // The sums start at 1 and every weight is <= 1, so the running sum always
    // dominates the addend and Fast2Sum gives each step's rounding error
    // exactly; the errors are summed apart (not fed back into the next addend,
    // where Kahan's subtraction would round them away again).  The result is
    // independent of the order in which lanes meet the weights to ~1e-12.
    // The offset is removed exactly after the pass.
    float2 ks = f2(1.0f), kc = f2(0.0f);
    long long total = 0;
    int px = 0;   // of the staged chunk
    for (int c = 0; c < nchunk; c++) {
        const int r0 = r_first + c * RCH;
        const int n = min(RCH, r_last - r0 + 1);
        px = build_runs<G, RCH>(a, sm, r0, n);
        total += px;
        if (G > 32) {
            if (rk == 0) sm.next_run = 0;
            Gp::sync();
        }
        auto add = [&](const Run &r, int, int j, int off, bool second) {
            const float jf = (float)j;
            float2 w = weight2<TX, TH>(e, r, make_float2(jf, jf + (float)off));
            if (!second) w.y = 0.0f;
            const float2 t = add2(ks, w);
            kc = add2(kc, sub2(w, sub2(t, ks)));
            ks = t;
        };
        sum_walk<G, RCH>(sm, n, px, add);
        Gp::sync();
    }
    if (total < 2) {  // genmap.cpp:125-128: the whole flux into the centre pixel
        if (rk == 0) {
            red_add_f64(a.acc.acc64 + sm.h.hdr.cpix, (double)e.fs_hi + (double)e.fs_lo);
            atomicAdd((unsigned long long *)(a.ctr + C_DEPOSITS), 1ull);
        }
        Gp::sync();
        return;
    }
    if (rk == 0) atomicAdd((unsigned long long *)(a.ctr + C_DEPOSITS), (unsigned long long)total);
    // S = sum of the lanes' (ks - 1) + kc, all in FP32 two-floats: ks - 1 is
    // exact (1 <= ks < 2^24: a multiple of ulp(ks) below ks), the lane and
    // warp sums are TwoSum trees, and F = flux inv_scale / S is Dekker's
    // two-float division (relative error ~2^-44).  Every lane of a warp ends
    // with the same sums (the xor tree adds the same pairs on each).
    float S_hi, S_lo;
    {
        float err;
        S_hi = two_sum(ks.x - 1.0f, ks.y - 1.0f, err);
        S_lo = (kc.x + kc.y) + err;
        warp_sum_ff(S_hi, S_lo);
    }
    float F, Flo;
    if (G > 32) {
        if ((rk & 31) == 0) sm.red2[rk >> 5] = make_float2(S_hi, S_lo);
        Gp::sync();
        if (rk == 0) {
            for (int k = 1; k < Gp::kWarps; k++) {
                float err;
                S_hi = two_sum(S_hi, sm.red2[k].x, err);
                S_lo = (S_lo + sm.red2[k].y) + err;
            }
            sm.fq = div_ff(e.fs_hi, e.fs_lo, S_hi, S_lo);
        }
        Gp::sync();
        F = sm.fq.x;
        Flo = sm.fq.y;
    } else {
        const float2 q = div_ff(e.fs_hi, e.fs_lo, S_hi, S_lo);
        F = q.x;
        Flo = q.y;
    }
    // |F| and the sign apart: the products are then >= 0 for the exact
    // conversion to FP64 (f32_to_f64), and the sign goes into its bit.  The
    // weights are >= exp(-6) (the disc edge), so a product is zero only when
    // the flux is: such a particle deposits nothing.
    if (F == 0.0f && Flo == 0.0f) return;
    const unsigned bias = f64_bias(F < 0.0f);
    const float Fa = fabsf(F), Floa = F < 0.0f ? -Flo : Flo;
    double *const acc = a.acc.acc64;

    // pass 2: deposits, one FP64 reduction per pixel (see the file header).
    for (int c = 0; c < nchunk; c++) {
        const int r0 = r_first + c * RCH;
        const int n = min(RCH, r_last - r0 + 1);
        if (nchunk > 1) px = build_runs<G, RCH>(a, sm, r0, n);
        if (G > 32) {
            if (rk == 0) sm.next_run = 0;
            Gp::sync();
        }
        auto deposit = [&](const Run &r, int, int j, int off, bool second) {
            const float jf = (float)j;
            const float2 w = weight2<TX, TH>(e, r, make_float2(jf, jf + (float)off));
            const float2 p = fma2(w, f2(Fa), mul2(w, f2(Floa)));   // w |F|, rounded once
            double *const m = acc + (r.pix0 + j);
            red_add_f64(m, f32_to_f64(p.x, bias));
            if (second) red_add_f64(m + off, f32_to_f64(p.y, bias));
        };
        deposit_walk<G, RCH>(sm, n, px, deposit);
        Gp::sync();
    }
}


// Renders the particle of queue slot q with a group of G threads (a warp or
// a block).
template <int G, int RCH>
__device__ void render_particle(const DiscArgs &a, CompSmem<RCH> &sm, long long q) {
    using Gp = Grp<G>;
    stage_hdr<G>(a, q, sm.h);
    Gp::sync();
    const Ext e = sm.h.ext;
    with_tiers(e, [&](auto tx, auto th) {
        render_disc<G, RCH, decltype(tx)::value, decltype(th)::value>(a, sm, e);
    });
}

constexpr int kWPB = 8, kRCHW = 64;    // warp kernel

// One block per large disc, persistent over the block-class queue (largest
// discs first, claimed dynamically).  Block shapes: BT threads, runs of RCH
// rings staged per chunk, MINB resident blocks per SM -- every shape fills
// the SM with 2048 threads (fewer, with more registers each, measured slower)
// and about 200 KB of staged runs.  The autotuner picks the shape.  Returns
// at once when a large chunk's render took the block class (*a.block_skip).
template <int BT, int RCH, int MINB>
__global__ void __launch_bounds__(BT, MINB) k_comp_block(DiscArgs a) {
    if (a.block_skip && *a.block_skip) return;
    __shared__ CompSmem<RCH> sm;
    __shared__ int s_q;
    const long long nblk = a.ctr[C_ADD_BLOCK];
    for (;;) {
        if (threadIdx.x == 0) s_q = (int)atomicAdd((unsigned long long *)(a.ctr + C_QNEXT_BLOCK), 1ull);
        __syncthreads();
        const int q = s_q;
        __syncthreads();
        if (q >= nblk) break;
        render_particle<BT, RCH>(a, sm, q);
    }
}

// One warp per small disc over the warp-class queue (after the block class).
__global__ void __launch_bounds__(kWPB * 32) k_comp_warp(DiscArgs a) {
    __shared__ CompSmem<kRCHW> sm[kWPB];
    const long long nblk = a.ctr[C_ADD_BLOCK];
    const long long ndisc = a.ctr[C_ADD_DISC];
    const int w = threadIdx.x >> 5;
    const long long gw = (long long)blockIdx.x * kWPB + w;
    const long long nw = (long long)gridDim.x * kWPB;
    for (long long q = nblk + gw; q < ndisc; q += nw) render_particle<32, kRCHW>(a, sm[w], q);
}

template <int BT, int RCH, int MINB>
cudaError_t launch_block(const DiscArgs &a, int num_sms, int blocks_per_sm, cudaStream_t s) {
    int occ = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_comp_block<BT, RCH, MINB>, BT, 0);
    if (e != cudaSuccess) return e;
    int bps = blocks_per_sm > 0 ? min(blocks_per_sm, occ) : occ;
    if (bps < 1) bps = 1;
    k_comp_block<BT, RCH, MINB><<<num_sms * bps, BT, 0, s>>>(a);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ adjoint
// The adjoint of the map (the formulas of adjoint.cu) with the compensated
// form's FP32 weights.  The tangent vector v_p - cos(alpha) n of each pixel is
// taken in the particle's local basis (e_theta, e_phi), where
//   v . e_theta = sin(theta_r - theta0) - 2 cos(theta0) sin(theta_r) sin^2(dphi/2),
//   v . e_phi   = sin(theta_r) sin(dphi) = 2 sin(theta_r) sin(x) cos(x),  x = dphi/2,
// both accurate to FP32 relative precision however small alpha is (the 3-D
// difference v - cos(alpha) n is not); alpha / sin(alpha) =
// sqrt(g / (h (1 - h))) with h = hav(alpha) and g = alpha^2 / 4 from the
// weight.  Sums: S with the offset Fast2Sum, the signed ones (sum G w, V_theta,
// V_phi, T) with Kahan's compensation per lane, all reduced as two-floats; a
// kernel with one thread per disc turns V into the map frame and writes the
// gradient in FP64.
template <int RCH>
struct AdjcSmem {
    CompSmem<RCH> c;
    AdjRing aring[RCH];
    float2 red[5][32];
};

// A disc's sums over its pixels: S, sum G w, V_theta, V_phi, T (S = 0: fewer
// than two pixels).
struct AdjSums {
    double S, A, vt, vp, t;
};
static_assert(sizeof(AdjSums) == kAdjSumBytes, "the caller's buffer");

// Two-float sum over the group; every thread ends with the total.  red: one
// slot per warp, used for nothing else within a disc.
template <int G>
__device__ __forceinline__ void group_sum_ff(float2 &v, float2 *red) {
    warp_sum_ff(v.x, v.y);
    if (G > 32) {
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
        __syncthreads();
        v = red[0];
        for (int w = 1; w < G / 32; w++) {
            float err;
            v.x = two_sum(v.x, red[w].x, err);
            v.y = (v.y + red[w].y) + err;
        }
    }
}

__device__ __forceinline__ void kahan(float &s, float &c, float v) {
    const float y = v - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
}

__device__ __forceinline__ void kahan2(float2 &s, float2 &c, float2 v) {
    const float2 y = sub2(v, c);
    const float2 t = add2(s, y);
    c = sub2(sub2(t, s), y);
    s = t;
}

// a / b and sqrt(a), correctly rounded, two at a time and without branches
// (Markstein's corrections with exact FMA remainders: P. Markstein, IBM J. Res.
// Dev. 34 (1990) 111).  a, b and the results normal, b above 2^-100; the results
// equal __fdiv_rn's on 8e9 pairs with quotients of 2^-2 to 2^26 and
// __fsqrt_rn's on every float of [2^-100, 2^31).  sqrt2_rn(0) is NaN.
__device__ __forceinline__ float2 div2_rn(float2 a, float2 b) {
    const float2 nb = mul2(b, f2(-1.0f));
    float2 y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y.x) : "f"(b.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y.y) : "f"(b.y));
    y = fma2(y, fma2(nb, y, f2(1.0f)), y);
    const float2 q = mul2(a, y);
    return fma2(fma2(nb, q, a), y, q);
}
__device__ __forceinline__ float2 sqrt2_rn(float2 a) {
    float2 y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y.x) : "f"(a.x));
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y.y) : "f"(a.y));
    float2 g = mul2(a, y), h = mul2(y, f2(-0.5f));
    const float2 r = fma2(g, h, f2(0.5f));
    g = fma2(g, r, g);
    h = fma2(h, r, h);
    return fma2(fma2(g, g, mul2(a, f2(-1.0f))), h, g);
}

// The sums of the disc particle whose header is staged.  Bound by issue (78 %
// of the slots), so by the instructions per pixel pair: with the series'
// lengths TX, TH (see weight2x) read at run time 1M particles at Nside 512 took
// 60.0 ms, with them fixed 56.4, and 49.1 with the second pass in packed
// arithmetic and its division and square roots free of branches.  Each step
// kept every value, bit by bit: the gradient of the observer's position is a
// sum of cancelling terms.
template <int G, int RCH, int TX, int TH>
__device__ void adjc_disc(const adj::AdjArgs &a, AdjcSmem<RCH> &sm, long long q, AdjSums *sums) {
    using Gp = Grp<G>;
    const DiscArgs &da = a.d;
    const int rk = Gp::rank();
    const Ext e = sm.c.h.ext;
    const int r_first = sm.c.h.hdr.r_first, r_last = sm.c.h.hdr.r_last;
    const int nring = r_last - r_first + 1;
    const int nchunk = nring > 0 ? (nring + RCH - 1) / RCH : 0;
    const float *g32 = a.gmap32;

    // pass 1: S (offset Fast2Sum) and sum G w (Kahan)
    float2 ks = f2(1.0f), kc = f2(0.0f);
    float as = 0.0f, ac = 0.0f;
    long long total = 0;
    for (int c = 0; c < nchunk; c++) {
        const int r0 = r_first + c * RCH;
        const int n = min(RCH, r_last - r0 + 1);
        total += build_runs<G, RCH>(da, sm.c, r0, n, sm.aring);
        if (G > 32) {
            if (rk == 0) sm.c.next_run = 0;
            Gp::sync();
        }
        ring_walk<G, RCH>(sm.c, n, [&](const Run &r, int, int j, int off, bool second) {
            const float jf = (float)j;
            float2 sn, h, g;
            float2 w = weight2x<TX, TH>(e, r, make_float2(jf, jf + (float)off), sn, h, g);
            if (!second) w.y = 0.0f;
            const int pix = r.pix0 + j;
            const float gw = g32[pix] * w.x + (second ? g32[pix + off] * w.y : 0.0f);
            kahan(as, ac, gw);
            const float2 t = add2(ks, w);
            kc = add2(kc, sub2(w, sub2(t, ks)));
            ks = t;
        });
        Gp::sync();
    }
    // (ks - 1 is exact, and so are the error terms of the two-float trees: no
    // FP64, whose pipe -- 1/64 of the FP32 rate -- was 73 % busy with these
    // sums in every warp and the epilogue on one lane per disc)
    float err;
    float2 S2, A2;
    S2.x = two_sum(ks.x - 1.0f, ks.y - 1.0f, err);
    S2.y = (kc.x + kc.y) + err;
    A2 = make_float2(as, -ac);
    group_sum_ff<G>(S2, sm.red[0]);
    group_sum_ff<G>(A2, sm.red[1]);
    AdjSums &out = sums[q];
    if (total < 2) {  // genmap.cpp:125-128: the whole flux in the centre pixel
        if (rk == 0) {
            out.S = 0.0;
            atomicAdd((unsigned long long *)(da.ctr + C_DEPOSITS), 1ull);
        }
        Gp::sync();
        return;
    }
    if (rk == 0) atomicAdd((unsigned long long *)(da.ctr + C_DEPOSITS), (unsigned long long)total);
    const float2 gq = div_ff(A2.x, A2.y, S2.x, S2.y);
    const float gm = gq.x;   // sum G w / S rounded

    // pass 2: V_theta, V_phi, T with q = (G - Gm) w
    float2 vs = f2(0.0f), vc = f2(0.0f);
    float ts = 0.0f, tc = 0.0f;
    for (int c = 0; c < nchunk; c++) {
        const int r0 = r_first + c * RCH;
        const int n = min(RCH, r_last - r0 + 1);
        if (nchunk > 1) build_runs<G, RCH>(da, sm.c, r0, n, sm.aring);
        if (G > 32) {
            if (rk == 0) sm.c.next_run = 0;
            Gp::sync();
        }
        ring_walk<G, RCH>(sm.c, n, [&](const Run &r, int ring, int j, int off, bool second) {
            const float jf = (float)j;
            float2 sn, h, g;
            const float2 w = weight2x<TX, TH>(e, r, make_float2(jf, jf + (float)off), sn, h, g);
            const AdjRing ar = sm.aring[ring];
            const int pix = r.pix0 + j;
            const float2 q = mul2(sub2(make_float2(g32[pix], second ? g32[pix + off] : 0.0f), f2(gm)), w);
            // alpha / sin(alpha); 0 at the antipode, where the tangent is undefined
            const float2 om = sub2(f2(1.0f), h);
            float2 af = sqrt2_rn(div2_rn(g, mul2(h, om)));
            if (TH < 0) {
                if (!(om.x > 1e-7f)) af.x = 0.0f;
                if (!(om.y > 1e-7f)) af.y = 0.0f;
            }
            if (!(h.x > 1e-30f)) af.x = 1.0f;
            if (!(h.y > 1e-30f)) af.y = 1.0f;
            const float2 s2 = mul2(sn, sn);
            const float2 c2 = sub2(f2(1.0f), s2);
            float2 cs = sqrt2_rn(c2);
            if (TX < 0) {
                if (!(c2.x > 0.0f)) cs.x = 0.0f;
                if (!(c2.y > 0.0f)) cs.y = 0.0f;
            }
            const float2 eth = fma2(f2(-ar.cr), s2, f2(ar.sr));
            const float2 eph = mul2(mul2(f2(ar.st2), sn), cs);
            const float2 qa = mul2(q, af), g4 = mul2(f2(4.0f), g);
            float2 v = make_float2(__fmul_rn(qa.x, eth.x), __fmul_rn(qa.x, eph.x));
            float tt = __fmul_rn(q.x, g4.x);
            if (second) {   // (beyond the run its values may be infinite or NaN)
                v.x = fmaf(qa.y, eth.y, v.x);
                v.y = fmaf(qa.y, eph.y, v.y);
                tt = fmaf(q.y, g4.y, tt);
            }
            kahan2(vs, vc, v);
            kahan(ts, tc, tt);
        });
        Gp::sync();
    }
    float2 vt = make_float2(vs.x, -vc.x), vp = make_float2(vs.y, -vc.y), tt = make_float2(ts, -tc);
    group_sum_ff<G>(vt, sm.red[2]);
    group_sum_ff<G>(vp, sm.red[3]);
    group_sum_ff<G>(tt, sm.red[4]);
    if (rk == 0) {
        out.S = (double)S2.x + (double)S2.y;
        out.A = (double)A2.x + (double)A2.y;
        out.vt = (double)vt.x + (double)vt.y;
        out.vp = (double)vp.x + (double)vp.y;
        out.t = (double)tt.x + (double)tt.y;
    }
    Gp::sync();
}

template <int G, int RCH>
__device__ void adjc_particle(const adj::AdjArgs &a, AdjcSmem<RCH> &sm, long long q, AdjSums *sums) {
    stage_hdr<G>(a.d, q, sm.c.h);
    Grp<G>::sync();
    with_tiers(sm.c.h.ext, [&](auto tx, auto th) {
        adjc_disc<G, RCH, decltype(tx)::value, decltype(th)::value>(a, sm, q, sums);
    });
}

// The gradients of the disc particles from their sums (FP64), one thread per
// disc, and the observer terms.  Blocks of one warp for small sets, as k_comp_hdr.
template <int BT>
__global__ void __launch_bounds__(BT) k_adjc_grad(adj::AdjArgs a, const AdjSums *sums) {
    __shared__ double red[12][32];
    double acc[12] = {0.0};
    const long long ndisc = a.d.ctr[C_ADD_DISC];
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < ndisc; q += (long long)gridDim.x * blockDim.x) {
        const AdjSums s = sums[q];
        const int i = a.d.queue[q];
        if (s.S == 0.0) {
            const double KV[3] = {0.0, 0.0, 0.0};
            adj::write_grad(a, i, a.gmap[a.d.cpix[i]] * a.inv_dOmega, 0.0, KV, false, acc);
            continue;
        }
        double theta0, phi0, ar;
        if (a.d.chdr) {
            const DiscHdr &d = a.d.chdr[q].hdr;
            theta0 = d.theta0;
            phi0 = d.phi0;
            ar = d.ar;
        } else {
            DiscHdr d;
            disc_setup(a.d.g, a.d.theta[i], a.d.phi[i], a.d.ar[i], a.d.flux[i], a.d.cpix[i], i, d);
            theta0 = d.theta0;
            phi0 = d.phi0;
            ar = d.ar;
        }
        const double Gm = s.A / s.S;
        const double ct = cos(theta0), st = sin(theta0), cp = cos(phi0), sp = sin(phi0);
        const double V[3] = {s.vt * ct * cp - s.vp * sp, s.vt * ct * sp + s.vp * cp, -s.vt * st};
        const double K = adj::kInvC2 * a.d.flux[i] / (s.S * ar * ar) * a.inv_dOmega;
        const double KV[3] = {K * V[0], K * V[1], K * V[2]};
        adj::write_grad(a, i, Gm * a.inv_dOmega, K * s.t, KV, true, acc);
    }
    adj::group_sum<BT, 12>(acc, red);
    if (threadIdx.x == 0) adj::flush_acc(a.oacc, acc);
}

// One block per disc of the block class (1024 threads a SM, 64 registers each).
// 1M particles at Nside 512: 45.7 ms with blocks of 128 threads, 49.1 with 256,
// whose barriers wait for more warps, and 47.3 with 64.  Smaller sets wait for
// their largest discs, which wider blocks finish sooner: at Nside 486 4,189
// particles take 0.91 ms with 128 threads and 0.60 with 256, 200,001 take 12.9
// and 8.8 ms.
constexpr int kAdjWideMax = 1 << 18;   // particles up to which the blocks are of 256 threads

template <int BT, int RCH, int MINB>
__global__ void __launch_bounds__(BT, MINB) k_adjc_block(adj::AdjArgs a, AdjSums *sums) {
    __shared__ AdjcSmem<RCH> sm;
    __shared__ int s_q;
    const long long nblk = a.d.ctr[C_ADD_BLOCK];
    for (;;) {
        if (threadIdx.x == 0) s_q = (int)atomicAdd((unsigned long long *)(a.d.ctr + C_QNEXT_BLOCK), 1ull);
        __syncthreads();
        const int q = s_q;
        __syncthreads();
        if (q >= nblk) break;
        adjc_particle<BT, RCH>(a, sm, q, sums);
    }
}

constexpr int kWPBA = 4;   // warps per block of the adjoint's warp kernel (shared memory)

__global__ void __launch_bounds__(kWPBA * 32) k_adjc_warp(adj::AdjArgs a, AdjSums *sums) {
    __shared__ AdjcSmem<kRCHW> sm[kWPBA];
    const long long nblk = a.d.ctr[C_ADD_BLOCK];
    const long long ndisc = a.d.ctr[C_ADD_DISC];
    const int w = threadIdx.x >> 5;
    const long long gw = (long long)blockIdx.x * kWPBA + w;
    const long long nw = (long long)gridDim.x * kWPBA;
    for (long long q = nblk + gw; q < ndisc; q += nw) adjc_particle<32, kRCHW>(a, sm[w], q, sums);
}

// The headers of every disc in the queue, one thread per particle (the
// FP64 set-up at full warp width instead of on one lane of a waiting block).
// One warp per block: the FP64 set-up is bound by the FP64 pipe (a warp's
// instruction takes 16 cycles of its SM's), so a few thousand discs are
// spread over as many SMs as they fill warps (1000 discs: 23 us in blocks of
// 256 threads, on 4 SMs).
constexpr int kHdrWarps = 1;

__global__ void __launch_bounds__(kHdrWarps * 32) k_comp_hdr(DiscArgs a) {
    // each warp builds its 32 consecutive headers in shared memory and
    // stores them as one contiguous run of 16-byte words (a thread's own
    // 160-byte store would leave partial sectors for the L2 to merge)
    constexpr int kW16 = sizeof(CompHdr) / 16;
    static_assert(sizeof(CompHdr) % 16 == 0, "headers are stored in 16-byte words");
    __shared__ __align__(16) CompHdr stage[kHdrWarps][32];
    const long long ndisc = a.ctr[C_ADD_DISC];
    const long long stride = (long long)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (long long q0 = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); q0 < ndisc; q0 += stride) {
        const long long q = q0 + lane;
        if (q < ndisc) setup_hdr(a, a.queue[q], stage[w][lane]);
        __syncwarp();
        const int nh = (int)min(32LL, ndisc - q0);
        const float4 *src = reinterpret_cast<const float4 *>(&stage[w][0]);
        float4 *dst = reinterpret_cast<float4 *>(a.chdr + q0);
        for (int k = lane; k < nh * kW16; k += 32) dst[k] = src[k];
        __syncwarp();
    }
}

}  // namespace

cudaError_t launch_hdr(const DiscArgs &a, int num_sms, cudaStream_t s) {
    if (!a.chdr) return cudaSuccess;
    k_comp_hdr<<<num_sms * 32, kHdrWarps * 32, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_disc_comp_warp(const DiscArgs &a, int num_sms, cudaStream_t s) {
    int occw = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occw, k_comp_warp, kWPB * 32, 0);
    if (e != cudaSuccess) return e;
    if (occw < 1) occw = 1;
    k_comp_warp<<<num_sms * occw, kWPB * 32, 0, s>>>(a);
    return cudaGetLastError();
}

size_t comp_hdr_bytes() { return sizeof(CompHdr); }

cudaError_t launch_disc_comp_block(const DiscArgs &a, int num_sms, int blocks_per_sm, int block_threads,
                                   cudaStream_t s) {
    if (block_threads == 128) return launch_block<128, 192, 16>(a, num_sms, blocks_per_sm, s);
    if (block_threads == 512) return launch_block<512, 640, 4>(a, num_sms, blocks_per_sm, s);
    return launch_block<256, 384, 8>(a, num_sms, blocks_per_sm, s);
}

cudaError_t launch_disc_comp(const DiscArgs &a, int num_sms, int blocks_per_sm, int block_threads,
                             cudaStream_t s, cudaEvent_t mid, bool headers) {
    cudaError_t e = headers ? launch_hdr(a, num_sms, s) : cudaSuccess;
    if (e != cudaSuccess) return e;
    if (block_threads == 128) e = launch_block<128, 192, 16>(a, num_sms, blocks_per_sm, s);
    else if (block_threads == 512) e = launch_block<512, 640, 4>(a, num_sms, blocks_per_sm, s);
    else e = launch_block<256, 384, 8>(a, num_sms, blocks_per_sm, s);
    if (e != cudaSuccess) return e;
    if (mid && (e = cudaEventRecord(mid, s)) != cudaSuccess) return e;
    int occw = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occw, k_comp_warp, kWPB * 32, 0);
    if (e != cudaSuccess) return e;
    if (occw < 1) occw = 1;
    k_comp_warp<<<num_sms * occw, kWPB * 32, 0, s>>>(a);
    return cudaGetLastError();
}

// The compensated adjoint's disc kernels (block class, then warp class).
cudaError_t launch_adjoint_comp_discs(const adj::AdjArgs &a, void *sum_buf, int num_sms, cudaStream_t s) {
    AdjSums *const sums = (AdjSums *)sum_buf;
    cudaError_t e = launch_hdr(a.d, num_sms, s);
    if (e != cudaSuccess) return e;
    auto blocks = [&](auto kernel, int threads) {
        int occ = 0;
        const cudaError_t r = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, 0);
        if (r != cudaSuccess) return r;
        kernel<<<num_sms * (occ < 1 ? 1 : occ), threads, 0, s>>>(a, sums);
        return cudaGetLastError();
    };
    e = a.p.n <= kAdjWideMax ? blocks(k_adjc_block<256, 256, 4>, 256) : blocks(k_adjc_block<128, 128, 8>, 128);
    if (e != cudaSuccess) return e;
    int occw = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occw, k_adjc_warp, kWPBA * 32, 0);
    if (e != cudaSuccess) return e;
    if (occw < 1) occw = 1;
    k_adjc_warp<<<num_sms * occw, kWPBA * 32, 0, s>>>(a, sums);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (a.p.n <= num_sms * 256) k_adjc_grad<32><<<num_sms * 8, 32, 0, s>>>(a, sums);
    else k_adjc_grad<128><<<num_sms * 8, 128, 0, s>>>(a, sums);
    return cudaGetLastError();
}

}  // namespace dmann
