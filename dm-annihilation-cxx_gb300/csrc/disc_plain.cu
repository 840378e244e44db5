// disc_plain.cu -- the plain FP64 form of the disc kernels.
//
// The reference CPU path's arithmetic on the GPU: each disc pixel's centre
// vector as pix2vec computes it (z and sin(theta) of its ring, phi from the
// in-ring index), w = exp(-0.5 (acos(v_pix . v)/ar)^2 / 0.333)
// (src/genmap.cpp:133-145), the FP64 normalisation and w/norm*flux added to
// an FP64 map with FP64 atomics (src/genmap.cpp:148-153).  Compiled with
// -fmad=false so every expression rounds as the CPU path's does; results
// differ from it only by the order of the additions.
#include "plain_form.cuh"

namespace dmann {

namespace {

constexpr int kBT = 256, kRCH = 256;
constexpr int kWPB = 8, kRCHW = 64;

// (sin, cos) of the pixel azimuths, by the same expressions and functions as
// the kernels' own (the values are the same bits).
__global__ void __launch_bounds__(256) k_trig(int nside, double fact1, double2 *belt, double2 *cap) {
    const long long nb = 8LL * nside, nc = cap ? 2LL * nside * (nside - 1) : 0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nb + nc;
         i += (long long)gridDim.x * blockDim.x) {
        double phi, sp, cp;
        if (i < nb) {
            const int row = i >= 4 * nside;
            phi = belt_phi((int)i - row * 4 * nside, row ? 1.0 : 0.5, fact1);
        } else {
            const long long p = i - nb;   // pixel p of the cap: ring r from 2 r (r - 1)
            int r = (int)((1.0 + sqrt(1.0 + 2.0 * (double)p)) * 0.5);
            while (2LL * r * (r - 1) > p) r--;
            while (2LL * r * (r + 1) <= p) r++;
            phi = cap_phi((int)(p - 2LL * r * (r - 1)), r);
        }
        sincos(phi, &sp, &cp);
        (i < nb ? belt[i] : cap[i - nb]) = make_double2(sp, cp);
    }
}

}  // namespace

cudaError_t launch_trig(int nside, double fact1, double2 *belt, double2 *cap, cudaStream_t s) {
    k_trig<<<152 * 4, 256, 0, s>>>(nside, fact1, belt, cap);
    return cudaGetLastError();
}

cudaError_t launch_disc_plain(const DiscArgs &a, int num_sms, int blocks_per_sm, cudaStream_t s,
                              cudaEvent_t mid) {
    int occ = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &occ, k_disc_block<PlainForm, kBT, kRCH>, kBT, 0);
    if (e != cudaSuccess) return e;
    int bps = blocks_per_sm > 0 ? min(blocks_per_sm, occ) : occ;
    if (bps < 1) bps = 1;
    DiscArgs b = a;
    b.scratch_len = a.scratch_total / (num_sms * bps);
    k_disc_block<PlainForm, kBT, kRCH><<<num_sms * bps, kBT, 0, s>>>(b);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (mid && (e = cudaEventRecord(mid, s)) != cudaSuccess) return e;
    int occw = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occw, k_disc_warp<PlainForm, kWPB, kRCHW>,
                                                      kWPB * 32, 0);
    if (e != cudaSuccess) return e;
    if (occw < 1) occw = 1;
    b.scratch_len = a.scratch_total / (num_sms * occw * kWPB);
    k_disc_warp<PlainForm, kWPB, kRCHW><<<num_sms * occw, kWPB * 32, 0, s>>>(b);
    return cudaGetLastError();
}

}  // namespace dmann
