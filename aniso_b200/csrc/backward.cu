// The adjoint of the rasterizer (no counterpart in the reference, which has no backward pass; the
// forward it differentiates is render.cpp:39-104 / 195-220 on the GPU path's lists).
//
// blend_backward: one block per tile of a batch; a warp owns an 8x8 block, each quarter warp two of its
//   columns, with two pixels per lane. Each pixel walks its tile list back to front from its last
//   applied splat, replaying the forward's alpha tests bit for bit (same record, same exponent code) and
//   recovering the transmittance in front of each splat (T_j = T_{j+1} / (1 - a_j));
//   nothing per pixel is stored but the final T and the last contributor. As in the forward, each
//   quarter walks only the splats its own cell (2x8 pixels) can take, the four side by side. Per splat
//   and cell, the gradient with respect to the nine record parameters (u, v, A2, B2, C2, L, r, g, b)
//   is summed over the quarter's lanes (through shared memory: half the instructions of shuffling
//   nine values), and at the end of a round over the quarters and warps, all in a fixed order, and
//   written to the pair's slot in the pair list -- no atomics, so the result does not depend on
//   scheduling, and the sums are those of the whole warp's butterfly, bit for bit.
//   Bound by issue (2.65 of 4 instructions a cycle, every pipe below 40%) at the 24 warps per SM that
//   the sums' shared memory leaves. Measured at 2.2M / 1280x720: 647 us with one list per warp and
//   warp-wide shuffles, 587 us with lists per quarter, 569 us with the sums through shared memory and
//   room for 512 of them (6 CTAs per SM; 640 and 768: 585 us).
//   Sparse frames (sparse_frame) take rounds of 32 splats, whose masks and lists are one ballot each, and leave
//   empty tiles at once; 16x32 tiles are held to 85 registers for three CTAs instead of two. Forward and
//   backward of twelve 1600x900 views of three scenes of 10k to 20k: 1279 -> 1050 us in 16x32 tiles, 1102 -> 999
//   in 16x16 (with one list per warp 1115, 1010); of twelve 640x360 views of 200k to 400k, 16x32: 1724 -> 1664.
// gauss_backward: one launch per view over the Gaussians visible in it (compacted first, so no lane
//   idles on a culled one); each sums its pairs' slots (contiguous, in a fixed order), applies the
//   chain rule through the record
//   (conic, log2 opacity, SH colour), the EWA projection (2D covariance, clamped Jacobian, camera
//   transform), the 3D covariance M M^T with M = R(q) diag(s), and the activations (exp, sigmoid,
//   quaternion normalisation) to the 59 raw parameters, and adds them to the scene's gradients.
//   Views are launched one after another, so the sum over views also runs in a fixed order.
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace ab2 {
namespace {

constexpr int kBackwardBatch = 128, kBackwardSparseBatch = 32;  // splats of a round, and in a sparse frame
constexpr int kBackwardPlaces = 512;  // (splat, cell) sums a 16x16 tile's round has room for
constexpr int kG = 9;
constexpr float kLn2 = 0.69314718055994530942f;
constexpr float kHalfLog2e = -0.72134752044448170368f;  // A2 = kHalfLog2e * A, C2 likewise
constexpr float kNegLog2e = -1.44269504088896340736f;   // B2 = kNegLog2e * B

__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The backward state of a lane's two pixels, as pairs (x: the left pixel, y: the right one).
struct PixelState2 {
    float2 T;                 // transmittance behind the splat being visited (starts at the final T)
    float2 ar, ag, ab;        // colour accumulated from the splats behind it
    float2 gr, gg, gb;        // dL/dC of the pixel
    unsigned last0, last1;    // list position one past each pixel's last applied splat
};

// The exponentials and whether the splat at list position pos applied in the forward to each of the
// lane's pixels (not behind its last applied splat, and passing the alpha tests, replayed with the
// forward's exponent bits).
struct PixelTest2 {
    float e0, e1;
    bool v0, v1;
};
__device__ __forceinline__ PixelTest2 pixel_test2(const PixelState2& s, unsigned pos, float2 p, float L) {
    PixelTest2 t;
    t.e0 = ex2_approx(p.x);
    t.e1 = ex2_approx(p.y);
    t.v0 = pos < s.last0 && !(p.x > L) && fminf(0.99f, t.e0) >= 1.0f / 255.0f;
    t.v1 = pos < s.last1 && !(p.y > L) && fminf(0.99f, t.e1) >= 1.0f / 255.0f;
    return t;
}

// One adjoint step at both pixels of the lane, each pair of operations one packed FP32x2 instruction
// (sm_100; per component the rounding of the scalar form). A pixel the splat did not apply to takes
// alpha = 0, which leaves its state unchanged (1/(1 - 0) = 1, w = 0) and adds zeros, so every lane of
// a warp with any such pixel takes the step without a branch. g[k] receives the gradients of the nine
// record parameters (u, v, A2, B2, C2, L, r, g, b), the sum of the two pixels'. 1/(1 - alpha) is the
// approximate reciprocal (relative error below 2^-22): the recovered transmittance drifts by that
// much per splat, far inside the gradients' tolerance. Packing the two pixels took the fwd+bwd of
// the 2.2M-Gaussian view from 1.95 to 1.86 ms.
__device__ __forceinline__ void pixel_step2(PixelState2& s, const PixelTest2& t, float2 dx, float dy, const float4& r0,
                                            const float4& r1, float rb, float g[kG]) {
    const float2 alpha = make_float2(t.v0 ? fminf(0.99f, t.e0) : 0.f, t.v1 ? fminf(0.99f, t.e1) : 0.f);
    const float2 om = __fadd2_rn(make_float2(1.0f, 1.0f), make_float2(-alpha.x, -alpha.y));
    const float2 inv_om = make_float2(rcp_approx(om.x), rcp_approx(om.y));
    const float2 Tb = __fmul2_rn(s.T, inv_om);  // transmittance in front of the splat
    const float2 w = __fmul2_rn(alpha, Tb);
    const float2 G6 = __fmul2_rn(s.gr, w), G7 = __fmul2_rn(s.gg, w), G8 = __fmul2_rn(s.gb, w);
    const float2 tr = __ffma2_rn(make_float2(r1.z, r1.z), Tb, __fmul2_rn(make_float2(-s.ar.x, -s.ar.y), inv_om));
    const float2 tg = __ffma2_rn(make_float2(r1.w, r1.w), Tb, __fmul2_rn(make_float2(-s.ag.x, -s.ag.y), inv_om));
    const float2 tb = __ffma2_rn(make_float2(rb, rb), Tb, __fmul2_rn(make_float2(-s.ab.x, -s.ab.y), inv_om));
    const float2 dalpha = __ffma2_rn(s.gb, tb, __ffma2_rn(s.gg, tg, __fmul2_rn(s.gr, tr)));
    s.ar = __ffma2_rn(make_float2(r1.z, r1.z), w, s.ar);
    s.ag = __ffma2_rn(make_float2(r1.w, r1.w), w, s.ag);
    s.ab = __ffma2_rn(make_float2(rb, rb), w, s.ab);
    s.T = Tb;
    // d alpha / d p = alpha ln 2 unless clamped or not applied
    float2 dp = __fmul2_rn(__fmul2_rn(dalpha, alpha), make_float2(kLn2, kLn2));
    if (!t.v0 || t.e0 > 0.99f) dp.x = 0.f;
    if (!t.v1 || t.e1 > 0.99f) dp.y = 0.f;
    const float2 ndp = make_float2(-dp.x, -dp.y);
    const float bdy = r0.w * dy, cdy2 = 2.0f * r1.x * dy;
    const float2 G0 = __fmul2_rn(ndp, __ffma2_rn(make_float2(2.0f * r0.z, 2.0f * r0.z), dx, make_float2(bdy, bdy)));
    const float2 G1 = __fmul2_rn(ndp, __ffma2_rn(make_float2(r0.w, r0.w), dx, make_float2(cdy2, cdy2)));
    const float2 dpdx = __fmul2_rn(dp, dx);
    const float2 G2 = __fmul2_rn(dpdx, dx);
    const float2 G3 = __fmul2_rn(dpdx, make_float2(dy, dy));
    const float2 G4 = __fmul2_rn(dp, make_float2(dy * dy, dy * dy));
    g[0] = G0.x + G0.y;
    g[1] = G1.x + G1.y;
    g[2] = G2.x + G2.y;
    g[3] = G3.x + G3.y;
    g[4] = G4.x + G4.y;
    g[5] = dp.x + dp.y;
    g[6] = G6.x + G6.y;
    g[7] = G7.x + G7.y;
    g[8] = G8.x + G8.y;
}

constexpr int kRedPitch = 36;  // floats per value: a quarter's eight lanes as two 16-byte words, free of conflicts

// Shared memory of one CTA. A quarter warp's sums for the splats of its list go to consecutive places
// of grad; at[slot][list] is where a staged splat's sums of that list start (place kPlaces, which holds
// zeros, where the list leaves the splat out).
template <int TW, int TH, int kBatch>
struct BackwardShared {
    static constexpr int kLists = TW * TH / 16;           // quarter warps: cells of 2 x 8 pixels
    static constexpr int kRoom = TW * TH * kBackwardPlaces / 256;
    static constexpr int kPlaces = TW * TH == 64 || kBatch * kLists < kRoom ? kBatch * kLists : kRoom;
    float4 r0[kBatch + 1];                                // the last slot: a splat that no pixel takes
    float4 r1[kBatch + 1];
    unsigned short at[kBatch][kLists];
    float grad[(kPlaces + 1) * kG];
    float b[kBatch + 1];
    unsigned pos[kBatch];
    unsigned mask[kBatch];
    unsigned char list[kLists][kBatch + 4];
    __align__(16) float red[kLists / 4][8][kRedPitch];    // per warp: eight values of its 32 lanes
    unsigned places;                                      // of grad, taken in this round
    unsigned maxlast;
};

// A warp owns an 8x8 block as in the forward; its quarter q the block's columns 2q, 2q + 1 (lane & 7 is
// the row), so that the sum over a splat's pixels -- rows by shuffles within the quarter, then the
// quarters as (0 + 2) + (1 + 3), then the warps in order -- runs in a fixed order whichever quarters a
// splat reaches.
template <int TW, int TH, int kBatch>
__global__ void __launch_bounds__(TW * TH / 2, TW * TH == 512 ? 3 : 0) blend_backward_kernel(BackwardIn in, float* __restrict__ grad_pair) {
    chain_entry();
    constexpr int kThreads = TW * TH / 2;
    constexpr int kWarps = kThreads / 32;
    constexpr int kWarpsX = TW / 8;
    constexpr int kCells = TW / 2;  // cells per 8-row band of the tile
    using Shared = BackwardShared<TW, TH, kBatch>;
    constexpr unsigned kPlaces = Shared::kPlaces;
    extern __shared__ __align__(16) unsigned char s_raw[];
    Shared& sh = *reinterpret_cast<Shared*>(s_raw);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, quarter = lane >> 3;
    const unsigned gtile = blockIdx.x;
    const unsigned v = find_segment(in.tables.tile_base, in.tables.n_views, gtile);
    const ViewInfo& vi = in.views[v];
    const unsigned local = gtile - vi.tile_base;
    const int tx = static_cast<int>(local % vi.cam.tilesX), ty = static_cast<int>(local / vi.cam.tilesX);
    const int ox = tx * TW, oy = ty * TH;
    const int x0 = ox + (warp % kWarpsX) * 8 + 2 * quarter, y = oy + (warp / kWarpsX) * 8 + (lane & 7);
    const int width = vi.cam.width, height = vi.cam.height;
    const float px0 = x0 + 0.5f, py = y + 0.5f;
    const uint2 range = (in.ctrl->flags & kFlagOverflow) ? make_uint2(0, 0) : in.ranges[gtile];
    if (kBatch == kBackwardSparseBatch && range.x == range.y) return;
    const int cell0 = (warp / kWarpsX) * kCells + (warp % kWarpsX) * 4;  // the warp's first cell in a mask
    const int sumq = lane & 3, sumk = lane >> 2;  // the quarter and value whose eight lanes this lane sums

    PixelState2 st;
    st.T = make_float2(1.f, 1.f);
    st.ar = st.ag = st.ab = st.gr = st.gg = st.gb = make_float2(0.f, 0.f);
    st.last0 = st.last1 = range.x;
    if (x0 < width && y < height) {
        const size_t p = static_cast<size_t>(y) * width + x0;
        st.T.x = vi.t_final[p];
        st.last0 = vi.n_contrib[p];
        st.gr.x = vi.grad_img[3 * p];
        st.gg.x = vi.grad_img[3 * p + 1];
        st.gb.x = vi.grad_img[3 * p + 2];
    }
    if (x0 + 1 < width && y < height) {
        const size_t p = static_cast<size_t>(y) * width + x0 + 1;
        st.T.y = vi.t_final[p];
        st.last1 = vi.n_contrib[p];
        st.gr.y = vi.grad_img[3 * p];
        st.gg.y = vi.grad_img[3 * p + 1];
        st.gb.y = vi.grad_img[3 * p + 2];
    }
    if (tid == 0) {
        sh.maxlast = range.x;
        sh.r0[kBatch] = make_float4(0.f, 0.f, 0.f, 0.f);
        sh.r1[kBatch] = make_float4(0.f, -INFINITY, 0.f, 0.f);
        sh.b[kBatch] = 0.f;
    }
    if (tid < kG) sh.grad[kPlaces * kG + tid] = 0.f;
    __syncthreads();
    // Past each quarter's last applied splat, and the tile's.
    unsigned qlast = max(st.last0, st.last1);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) qlast = max(qlast, __shfl_xor_sync(0xFFFFFFFFu, qlast, o));
    unsigned lasts[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) lasts[q] = __shfl_sync(0xFFFFFFFFu, qlast, 8 * q);
    if ((lane & 7) == 0) atomicMax(&sh.maxlast, qlast);
    __syncthreads();
    const unsigned end = sh.maxlast;

    // Pairs behind every pixel's last applied splat get zero gradient.
    for (unsigned q = end + tid; q < range.y; q += kThreads) {
        const unsigned g = in.vals[q];
        const unsigned j = in.rank ? in.rank[g] : g;
        const unsigned long long rc = in.rect[j];
        const unsigned rx0 = rc & 0xFFFFu, ry0 = (rc >> 16) & 0xFFFFu, rx1 = (rc >> 32) & 0xFFFFu;
        float* out = grad_pair +
                     static_cast<size_t>(in.offs[j] + (static_cast<unsigned>(ty) - ry0) * (rx1 - rx0 + 1) +
                                         (static_cast<unsigned>(tx) - rx0)) * kG;
#pragma unroll
        for (int k = 0; k < kG; ++k) out[k] = 0.f;
    }

    for (unsigned top = end; top > range.x;) {
        const unsigned start = top > range.x + kBatch ? top - kBatch : range.x;
        const unsigned cnt = top - start;
        // Stage the batch [start, top): records, cell masks and each pair's gradient slot (the slot of
        // (entry g, tile t) is g's first one plus t's row-major index in g's rectangle).
        for (unsigned slot = tid; slot < kBatch; slot += kThreads) {
            unsigned m = 0;
            if (slot < cnt) {
                const unsigned g = in.vals[start + slot];
                const SplatRecord r = in.rec[g];
                constexpr float kMax = 3.40282347e38f;  // an infinite colour as the forward blends it
                sh.r0[slot] = r.r0;
                sh.r1[slot] = make_float4(r.r1.x, r.r1.y, fminf(r.r1.z, kMax), fminf(r.r1.w, kMax));
                sh.b[slot] = fminf(r.r2.x, kMax);
                m = staged_cell_mask<TW, TH, 2, 8>(r, ox, oy);
                const unsigned j = in.rank ? in.rank[g] : g;
                const unsigned long long rc = in.rect[j];
                const unsigned rx0 = rc & 0xFFFFu, ry0 = (rc >> 16) & 0xFFFFu, rx1 = (rc >> 32) & 0xFFFFu;
                sh.pos[slot] =
                    in.offs[j] + (static_cast<unsigned>(ty) - ry0) * (rx1 - rx0 + 1) + (static_cast<unsigned>(tx) - rx0);
            }
            sh.mask[slot] = m;
        }
        if (tid == 0) sh.places = 0;
        __syncthreads();
        // The round takes the staged splats from `first` on: as many, from the back, as surely find
        // places for their sums. Every warp finds the same number.
        unsigned first = 0;
        if (kPlaces < kBatch * Shared::kLists) {
            constexpr int kPer = kBatch / 32;
            unsigned need[kPer], total = 0;
#pragma unroll
            for (int k = kPer - 1; k >= 0; --k) {
                total += __popc(sh.mask[lane * kPer + k]);
                need[k] = total;
            }
            const unsigned behind = __reduce_add_sync(0xFFFFFFFFu, total) - warp_incl_scan(total);
            unsigned fit = 0;
#pragma unroll
            for (int k = 0; k < kPer; ++k) fit += need[k] + behind <= kPlaces;
            first = kBatch - __reduce_add_sync(0xFFFFFFFFu, fit);
        }
        // Each quarter's splats of the round, back to front, and the places of their sums.
        unsigned n[4] = {0, 0, 0, 0};
        unsigned base = 0;
        {
            unsigned bits[4][kBatch / 32];
#pragma unroll
            for (int c = kBatch / 32 - 1; c >= 0; --c) {
                const unsigned idx = c * 32 + lane;
                const unsigned m = idx >= first && idx < cnt ? sh.mask[idx] >> cell0 : 0u;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    bits[q][c] = __ballot_sync(0xFFFFFFFFu, ((m >> q) & 1u) && start + idx < lasts[q]);
                    n[q] += __popc(bits[q][c]);
                }
            }
            if (lane == 0) base = atomicAdd(&sh.places, n[0] + n[1] + n[2] + n[3]);
            base = __shfl_sync(0xFFFFFFFFu, base, 0);
            unsigned at0[4] = {base, base + n[0], base + n[0] + n[1], base + n[0] + n[1] + n[2]};
            unsigned seen[4] = {0, 0, 0, 0};
            const unsigned above = ~(lanemask_lt() | (1u << lane));
#pragma unroll
            for (int c = kBatch / 32 - 1; c >= 0; --c) {
                const unsigned idx = c * 32 + lane;
                unsigned short at[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const unsigned i = seen[q] + __popc(bits[q][c] & above);
                    const bool mine = (bits[q][c] >> lane) & 1u;
                    at[q] = static_cast<unsigned short>((mine ? at0[q] + i : kPlaces) * kG);
                    if (mine) sh.list[warp * 4 + q][i] = static_cast<unsigned char>(idx);
                    seen[q] += __popc(bits[q][c]);
                }
                *reinterpret_cast<ushort4*>(&sh.at[idx][warp * 4]) = make_ushort4(at[0], at[1], at[2], at[3]);
            }
        }
        const unsigned longest = max(max(n[0], n[1]), max(n[2], n[3]));
        const unsigned own = quarter == 0 ? n[0] : quarter == 1 ? n[1] : quarter == 2 ? n[2] : n[3];
        unsigned char* list = sh.list[warp * 4 + quarter];
        for (unsigned i = own + (lane & 7); i < longest; i += 8) list[i] = kBatch;
        __syncwarp();
        const auto place = [&](int q) {  // of the quarter's first sum
            return base + (q > 0 ? n[0] : 0u) + (q > 1 ? n[1] : 0u) + (q > 2 ? n[2] : 0u);
        };
        // This lane writes one of the first eight values of quarter sumq, and the ninth of its own.
        const unsigned sum_own = sumq == 0 ? n[0] : sumq == 1 ? n[1] : sumq == 2 ? n[2] : n[3];
        const unsigned last_own = (lane & 7) == 0 ? own : 0u;
        float* out = sh.grad + place(sumq) * kG + sumk;
        float* last = sh.grad + place(quarter) * kG + 8;
        float* red = sh.red[warp][0] + lane;
        const float4* redq = reinterpret_cast<const float4*>(sh.red[warp][sumk] + 8 * sumq);
        const auto walk = [&](auto guarded) {
            for (unsigned i = 0; i < longest; ++i, out += kG, last += kG) {
                const unsigned jj = list[i];
                const float4 r0 = sh.r0[jj];
                const float4 r1 = sh.r1[jj];
                const float rb = sh.b[jj];
                const float dy = __fsub_rn(py, r0.y);
                float2 dx;
                const float2 pp = splat_exponents2(r0, r1, make_float2(px0, px0 + 1.0f), dy, dx);
                const PixelTest2 test = pixel_test2(st, start + jj, pp, r1.y);
                float sum = 0.f, ninth = 0.f;
                if (__any_sync(0xFFFFFFFFu, test.v0 || test.v1)) {  // else the sums are zero
                    float g[kG];
                    pixel_step2(st, test, dx, dy, r0, r1, rb, g);
                    if (decltype(guarded)::value)  // the colour sums: the others are selected to zero already
#pragma unroll
                        for (int k = 6; k < kG; ++k) g[k] = test.v0 || test.v1 ? g[k] : 0.f;
#pragma unroll
                    for (int k = 0; k < 8; ++k) red[k * kRedPitch] = g[k];
                    ninth = g[8];
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1) ninth += __shfl_xor_sync(0xFFFFFFFFu, ninth, o);
                    __syncwarp();
                    // The eight rows in the order of the shuffles above: 4 apart, 2 apart, neighbours.
                    const float4 lo = redq[0], hi = redq[1];
                    const float2 even = __fadd2_rn(make_float2(lo.x, lo.y), make_float2(hi.x, hi.y));
                    const float2 odd = __fadd2_rn(make_float2(lo.z, lo.w), make_float2(hi.z, hi.w));
                    const float2 both = __fadd2_rn(even, odd);
                    sum = both.x + both.y;
                    __syncwarp();
                }
                if (i < sum_own) *out = sum;
                if (i < last_own) *last = ninth;
            }
        };
        // An infinite or NaN gradient times a weight of zero is NaN: where the warp holds one, a lane whose
        // pixels a splat does not apply to adds zeros to its sums all the same, in a walk of its own. (Asked for
        // only here, so that the gradients' loads stay in flight over the staging: asked for before it, 502
        // instead of 495 us of adjoint blend at 2.2M / 1280x720; selects in the one walk 506.)
        const float grads = st.gr.x + st.gg.x + st.gb.x + st.gr.y + st.gg.y + st.gb.y;
        if (__any_sync(0xFFFFFFFFu, !isfinite(grads))) walk(std::true_type{});
        else walk(std::false_type{});
        __syncthreads();
        // Fixed-order sum over the quarters and warps; every pair of the round is written. Neighbouring
        // threads take the values of one pair, so that a store covers whole pairs.
        for (unsigned e = first * kG + tid; e < cnt * kG; e += kThreads) {
            const unsigned slot = e / kG, k = e - slot * kG;
            float acc = 0.f;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
                const ushort4 at = *reinterpret_cast<const ushort4*>(&sh.at[slot][4 * w]);
                const float q0 = sh.grad[at.x + k], q1 = sh.grad[at.y + k];
                const float q2 = sh.grad[at.z + k], q3 = sh.grad[at.w + k];
                acc += (q0 + q2) + (q1 + q3);
            }
            grad_pair[static_cast<size_t>(sh.pos[slot]) * kG + k] = acc;
        }
        __syncthreads();
        top = start + first;
    }
}

// SH basis (sh.cpp:18-58 order) and its derivatives along x, y, z, for degree D.
// Adds one view's gradient to the caller's buffer. The add is rounded on its own (never fused with
// the product that formed v), so accumulating views here equals summing per-view gradients.
__device__ __forceinline__ void accumulate(float* p, float v) { *p = __fadd_rn(*p, v); }
// The same where the old value is known to be zero (the first view of a fresh gradient) and is not
// read: 0 + v rounds as the add would.
template <bool kFresh>
__device__ __forceinline__ void add_grad(float* p, float v) {
    *p = __fadd_rn(kFresh ? 0.f : *p, v);
}

template <int D>
__device__ __forceinline__ void sh_basis(float x, float y, float z, float b[16], float bx[16], float by[16],
                                         float bz[16]) {
    const float C0 = 0.28209479177387814f, C1 = 0.4886025119029199f;
    const float C20 = 1.0925484305920792f, C21 = -1.0925484305920792f, C22 = 0.31539156525252005f,
                C23 = -1.0925484305920792f, C24 = 0.5462742152960396f;
    const float C30 = -0.5900435899266435f, C31 = 2.890611442640554f, C32 = -0.4570457994644658f,
                C33 = 0.3731763325901154f, C34 = -0.4570457994644658f, C35 = 1.445305721320277f,
                C36 = -0.5900435899266435f;
#pragma unroll
    for (int k = 0; k < 16; ++k) b[k] = bx[k] = by[k] = bz[k] = 0.f;
    b[0] = C0;
    if (D >= 1) {
        b[1] = -C1 * y; by[1] = -C1;
        b[2] = C1 * z; bz[2] = C1;
        b[3] = -C1 * x; bx[3] = -C1;
    }
    if (D >= 2) {
        const float xx = x * x, yy = y * y, zz = z * z;
        b[4] = C20 * x * y; bx[4] = C20 * y; by[4] = C20 * x;
        b[5] = C21 * y * z; by[5] = C21 * z; bz[5] = C21 * y;
        b[6] = C22 * (2 * zz - xx - yy); bx[6] = -2 * C22 * x; by[6] = -2 * C22 * y; bz[6] = 4 * C22 * z;
        b[7] = C23 * x * z; bx[7] = C23 * z; bz[7] = C23 * x;
        b[8] = C24 * (xx - yy); bx[8] = 2 * C24 * x; by[8] = -2 * C24 * y;
        if (D >= 3) {
            b[9] = C30 * y * (3 * xx - yy); bx[9] = C30 * 6 * x * y; by[9] = C30 * (3 * xx - 3 * yy);
            b[10] = C31 * x * y * z; bx[10] = C31 * y * z; by[10] = C31 * x * z; bz[10] = C31 * x * y;
            b[11] = C32 * y * (4 * zz - xx - yy); bx[11] = -2 * C32 * x * y; by[11] = C32 * (4 * zz - xx - 3 * yy);
            bz[11] = 8 * C32 * y * z;
            b[12] = C33 * z * (2 * zz - 3 * xx - 3 * yy); bx[12] = -6 * C33 * x * z; by[12] = -6 * C33 * y * z;
            bz[12] = C33 * (6 * zz - 3 * xx - 3 * yy);
            b[13] = C34 * x * (4 * zz - xx - yy); bx[13] = C34 * (4 * zz - 3 * xx - yy); by[13] = -2 * C34 * x * y;
            bz[13] = 8 * C34 * x * z;
            b[14] = C35 * z * (xx - yy); bx[14] = 2 * C35 * x * z; by[14] = -2 * C35 * y * z; bz[14] = C35 * (xx - yy);
            b[15] = C36 * x * (xx - 3 * yy); bx[15] = C36 * (3 * xx - 3 * yy); by[15] = -6 * C36 * x * y;
        }
    }
}

constexpr int kListItems = 4;  // entries per thread of the visible-list compaction

// The Gaussians of one view that are visible in it, appended in any order: the adjoint of each is
// independent of where it sits in the list, so the order does not change any result.
__global__ void __launch_bounds__(256) visible_list_kernel(int64_t n, unsigned entry_base,
                                                           const unsigned* __restrict__ depth_key,
                                                           unsigned* __restrict__ list, unsigned* counter) {
    chain_entry();
    __shared__ unsigned s_tmp[8];
    __shared__ unsigned s_base;
    const int64_t i0 = static_cast<int64_t>(blockIdx.x) * (256 * kListItems) + threadIdx.x;
    bool vis[kListItems];
    unsigned mine = 0;
#pragma unroll
    for (int k = 0; k < kListItems; ++k) {
        const int64_t i = i0 + k * 256;
        vis[k] = i < n && depth_key[entry_base + static_cast<unsigned>(i)] != kCulledKey;
        mine += vis[k];
    }
    // One atomic per CTA on the shared counter (one per warp contended on it for ~50 us at 2.2M).
    unsigned total;
    unsigned at = block_excl_scan<256>(mine, s_tmp, total);
    if (threadIdx.x == 0) s_base = total ? atomicAdd(counter, total) : 0u;
    __syncthreads();
    at += s_base;
#pragma unroll
    for (int k = 0; k < kListItems; ++k)
        if (vis[k]) list[at++] = static_cast<unsigned>(i0 + k * 256);
}

// The view's camera, its scene's raw tensors and gradient buffers come from the frame's device
// tables (copied into shared memory by each CTA), not from kernel arguments, so a recorded CUDA graph
// of the backward stays valid when the parameters, gradients or cameras move between replays.
template <typename T>
__device__ __forceinline__ void copy_words(T& dst, const T& src) {
    static_assert(sizeof(T) % 4 == 0, "copied as 32-bit words");
    if (threadIdx.x < sizeof(T) / 4)
        reinterpret_cast<unsigned*>(&dst)[threadIdx.x] = reinterpret_cast<const unsigned*>(&src)[threadIdx.x];
}

// Tiles per row of a rectangle, and its tiles (none where it is empty: 1 .. 0).
__device__ __forceinline__ unsigned rect_width(unsigned long long r) {
    return static_cast<unsigned>((r >> 32) & 0xFFFFu) - static_cast<unsigned>(r & 0xFFFFu) + 1u;
}
__device__ __forceinline__ unsigned rect_tiles(unsigned long long r) {
    return rect_width(r) * (static_cast<unsigned>(r >> 48) - static_cast<unsigned>((r >> 16) & 0xFFFFu) + 1u);
}

// Held to 128 registers (four CTAs per SM): the kernel waits on memory, and the extra warps
// measured faster where it runs many times per step (the 8-scene training batch: 27.0 -> 25.2 ms a
// step; 102 registers spilled and was no faster; the adjoint blend held to 64 was slower).
template <int D, bool kFresh>
__global__ void __launch_bounds__(128, 4) gauss_backward_kernel(const BatchScene<RawParams>* __restrict__ scenes,
                                                             unsigned scene, const ViewInfo* __restrict__ views,
                                                             unsigned view, const RawGrads* __restrict__ grads_table,
                                                             const Ctrl* ctrl, const unsigned* __restrict__ list,
                                                             const unsigned* __restrict__ list_count,
                                                             const unsigned* __restrict__ rank,
                                                             const unsigned* __restrict__ offs,
                                                             const unsigned long long* __restrict__ rect,
                                                             const unsigned long long* __restrict__ whole,
                                                             const float* __restrict__ grad_pair) {
    chain_entry();
    __shared__ CamParams s_cam;
    __shared__ RawParams s_raw;
    __shared__ RawGrads s_out;
    __shared__ unsigned s_entry_base;
    copy_words(s_cam, views[view].cam);
    copy_words(s_raw, scenes[scene].src);
    copy_words(s_out, grads_table[scene]);
    if (threadIdx.x == 0) s_entry_base = views[view].entry_base;
    __syncthreads();
    const CamParams& cam = s_cam;
    const RawParams raw = s_raw;
    const RawGrads out = s_out;
    const unsigned entry_base = s_entry_base;
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (ctrl->flags & kFlagOverflow) return;
    // The view's visible entries in entry order (the compacted list), so that a warp's reads of the
    // raw parameters and its gradient writes fall on neighbouring rows. (Walking the depth-sorted
    // list instead makes the pair-slot reads contiguous but every parameter row a random gather:
    // measured 0.22 -> 0.30 ms at 2.2M Gaussians.)
    const unsigned count = *list_count;
    if (blockIdx.x * blockDim.x >= count) return;
    const int lane = threadIdx.x & 31;
    // Past the end of the list: no Gaussian, but the lane still helps its warp.
    const bool active = t < count;
    const unsigned e = active ? entry_base + list[t] : entry_base;
    const int64_t i = e - entry_base;
    // The slots are those of the (cut) rectangle; `whole` (NULL: the same) is the rectangle before the cut.
    unsigned cnt = 0, off = 0, cut = 0;
    unsigned long long rc = 0, wr = 0;
    if (active) {
        const unsigned j = rank ? rank[e] : e;
        rc = rect[j];
        wr = whole ? whole[j] : rc;
        cut = rect_tiles(rc);
        cnt = rect_tiles(wr);
        off = offs[j];
    }
    // The sum of the Gaussian's per-pair gradients, in a fixed order: a short list by its own lane,
    // slot after slot; a long one (the nearest splats own thousands of tiles) by the whole warp,
    // lane l taking tiles l, l + 32, ... of the whole rectangle, then a fixed shuffle tree -- so one
    // huge splat does not hold its warp for thousands of serial loads, and a cut rectangle's sum has the
    // bits of the whole one's (whose other tiles add zeros).
    constexpr unsigned kSolo = 16;
    float g9[kG] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (cnt <= kSolo) {
        const float* gp = grad_pair + static_cast<size_t>(off) * kG;
        for (unsigned k = 0; k < cut; ++k)
#pragma unroll
            for (int c = 0; c < kG; ++c) g9[c] += gp[k * kG + c];
    }
    for (unsigned big = __ballot_sync(0xFFFFFFFFu, cnt > kSolo); big; big &= big - 1) {
        const int src = __ffs(big) - 1;
        const unsigned bc = __shfl_sync(0xFFFFFFFFu, cnt, src), bo = __shfl_sync(0xFFFFFFFFu, off, src);
        const unsigned long long br = __shfl_sync(0xFFFFFFFFu, rc, src), bw = __shfl_sync(0xFFFFFFFFu, wr, src);
        const unsigned ww = rect_width(bw), cw = rect_width(br), ch = rect_tiles(br) / max(cw, 1u);
        // The cut rectangle's corner within the whole one (an empty one holds no tile).
        const unsigned dx = (br & 0xFFFFu) - (bw & 0xFFFFu), dy = (br >> 16 & 0xFFFFu) - (bw >> 16 & 0xFFFFu);
        const float* gp = grad_pair + static_cast<size_t>(bo) * kG;
        float part[kG] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (unsigned k = lane; k < bc; k += 32) {
            const unsigned row = k / ww, y = row - dy, x = k - row * ww - dx;
            if (x >= cw || y >= ch) continue;
            const float* slot = gp + static_cast<size_t>(y * cw + x) * kG;
#pragma unroll
            for (int c = 0; c < kG; ++c) part[c] += slot[c];
        }
#pragma unroll
        for (int c = 0; c < kG; ++c) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) part[c] += __shfl_down_sync(0xFFFFFFFFu, part[c], o);
            part[c] = __shfl_sync(0xFFFFFFFFu, part[c], 0);
            if (lane == src) g9[c] = part[c];
        }
    }
    if (!active) return;

    // ---- forward quantities (the preprocess kernel's, in the same order) ----
    float4 pg, sg, qn;
    raw.load(i, pg, sg, qn);
    const float4 qraw = raw.quats[i];
    const float qlen = sqrtf(qraw.x * qraw.x + qraw.y * qraw.y + qraw.z * qraw.z + qraw.w * qraw.w);
    const float gx = pg.x, gy = pg.y, gz = pg.z, o = pg.w;
    const float* W = cam.R;
    const float px = W[0] * gx + W[1] * gy + W[2] * gz + cam.t[0];
    const float py = W[3] * gx + W[4] * gy + W[5] * gz + cam.t[1];
    const float pz = W[6] * gx + W[7] * gy + W[8] * gz + cam.t[2];
    const float qw = qn.x, qx = qn.y, qy = qn.z, qz = qn.w;
    const float Rq[3][3] = {{1 - 2 * (qy * qy + qz * qz), 2 * (qx * qy - qw * qz), 2 * (qx * qz + qw * qy)},
                            {2 * (qx * qy + qw * qz), 1 - 2 * (qx * qx + qz * qz), 2 * (qy * qz - qw * qx)},
                            {2 * (qx * qz - qw * qy), 2 * (qy * qz + qw * qx), 1 - 2 * (qx * qx + qy * qy)}};
    const float s[3] = {sg.x * cam.splatScale, sg.y * cam.splatScale, sg.z * cam.splatScale};
    float M[3][3], S[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) M[r][c] = Rq[r][c] * s[c];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) S[r][c] = M[r][0] * M[c][0] + M[r][1] * M[c][1] + M[r][2] * M[c][2];
    const float limX = 1.3f * 0.5f * cam.width / cam.fx, limY = 1.3f * 0.5f * cam.height / cam.fy;
    const float rx = px / pz, ry = py / pz;
    const bool clx = rx < -limX || rx > limX, cly = ry < -limY || ry > limY;
    const float tx = fminf(limX, fmaxf(-limX, rx)) * pz;
    const float ty = fminf(limY, fmaxf(-limY, ry)) * pz;
    const float iz = 1.0f / pz, iz2 = iz * iz;
    const float J[2][3] = {{cam.fx * iz, 0.f, -cam.fx * tx * iz2}, {0.f, cam.fy * iz, -cam.fy * ty * iz2}};
    float T[2][3];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) T[r][c] = J[r][0] * W[c] + J[r][1] * W[3 + c] + J[r][2] * W[6 + c];
    float ST[2][3];  // S T_r^T for r = 0, 1 (S symmetric)
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) ST[r][c] = S[c][0] * T[r][0] + S[c][1] * T[r][1] + S[c][2] * T[r][2];
    const float a = T[0][0] * ST[0][0] + T[0][1] * ST[0][1] + T[0][2] * ST[0][2] + 0.3f;
    const float b = T[1][0] * ST[0][0] + T[1][1] * ST[0][1] + T[1][2] * ST[0][2];
    const float c = T[1][0] * ST[1][0] + T[1][1] * ST[1][1] + T[1][2] * ST[1][2] + 0.3f;
    const float det = a * c - b * b;

    // ---- record parameters -> conic, opacity, colour ----
    const float gu = g9[0], gv = g9[1];
    // What densification reads (gsplat's DefaultStrategy): the screen-space gradient in NDC units
    // (x width/2, x height/2), its norm added over views, and the number of views that saw it.
    if (out.grad2d) {
        const float nu = gu * (0.5f * cam.width), nv = gv * (0.5f * cam.height);
        accumulate(&out.grad2d[i], sqrtf(nu * nu + nv * nv));
        accumulate(&out.visible[i], 1.0f);
    }
    const float gA = g9[2] * kHalfLog2e, gB = g9[3] * kNegLog2e, gC = g9[4] * kHalfLog2e;
    const float go = g9[5] / (o * kLn2);  // L = log2(o)
    float* gsh = out.sh + static_cast<size_t>(i) * raw.sh_planes * 4;
    float gm[3] = {0.f, 0.f, 0.f};
    {
        float3 d = make_float3(gx - cam.eye[0], gy - cam.eye[1], gz - cam.eye[2]);
        const float len = sqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
        const float ux = d.x / len, uy = d.y / len, uz = d.z / len;
        float bs[16], bxs[16], bys[16], bzs[16];
        sh_basis<D>(ux, uy, uz, bs, bxs, bys, bzs);
        constexpr int count = (D + 1) * (D + 1);
        const float4* shp = raw.sh + static_cast<size_t>(i) * raw.sh_planes;
        float shv[48];
#pragma unroll
        for (int k = 0; k < (count * 3 + 3) / 4; ++k) {
            const float4 f = shp[k];
            shv[4 * k] = f.x;
            if (4 * k + 1 < 48) shv[4 * k + 1] = f.y;
            if (4 * k + 2 < 48) shv[4 * k + 2] = f.z;
            if (4 * k + 3 < 48) shv[4 * k + 3] = f.w;
        }
        float gdir[3] = {0.f, 0.f, 0.f};
        const float grgb[3] = {g9[6], g9[7], g9[8]};
        float gc3[3];
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) {
            float pre = 0.5f;
#pragma unroll
            for (int k = 0; k < count; ++k) pre += bs[k] * shv[k * 3 + ch];
            const float gc = pre > 0.f ? grgb[ch] : 0.f;  // rgb = max(0, pre)
            gc3[ch] = gc;
#pragma unroll
            for (int k = 0; k < count; ++k) {
                gdir[0] += shv[k * 3 + ch] * bxs[k] * gc;
                gdir[1] += shv[k * 3 + ch] * bys[k] * gc;
                gdir[2] += shv[k * 3 + ch] * bzs[k] * gc;
            }
        }
        // d rgb / d sh = basis (x) gc, added 16 bytes at a time: float f of the row is coefficient f/3,
        // channel f%3 (each element still gets its own rounded add).
        constexpr int kFloats = count * 3;
        float4* gsh4 = reinterpret_cast<float4*>(gsh);
#pragma unroll
        for (int pl = 0; pl < (kFloats + 3) / 4; ++pl) {
            const float4 o = kFresh ? make_float4(0.f, 0.f, 0.f, 0.f) : gsh4[pl];
            float w[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int f = 4 * pl + e;
                if (f < kFloats) w[e] = __fadd_rn(w[e], bs[f / 3] * gc3[f % 3]);
            }
            gsh4[pl] = make_float4(w[0], w[1], w[2], w[3]);
        }
        const float dd = ux * gdir[0] + uy * gdir[1] + uz * gdir[2];
        gm[0] += (gdir[0] - ux * dd) / len;
        gm[1] += (gdir[1] - uy * dd) / len;
        gm[2] += (gdir[2] - uz * dd) / len;
    }
    add_grad<kFresh>(&out.logits[i], go * o * (1.0f - o));

    // ---- conic (A, B, C) = (c, -b, a) / det -> 2D covariance (a, b, c) ----
    const float id2 = 1.0f / (det * det);
    const float ga = (-c * c * gA + b * c * gB - b * b * gC) * id2;
    const float gb = (2.0f * b * c * gA - (det + 2.0f * b * b) * gB + 2.0f * a * b * gC) * id2;
    const float gc2 = (-b * b * gA + a * b * gB - a * a * gC) * id2;

    // ---- covariance = T S T^T + 0.3 I -> S, T ----
    float gS[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int q = 0; q < 3; ++q)
            gS[r][q] = ga * T[0][r] * T[0][q] + gb * T[0][r] * T[1][q] + gc2 * T[1][r] * T[1][q];
    float gT[2][3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        gT[0][q] = 2.0f * ga * ST[0][q] + gb * ST[1][q];
        gT[1][q] = gb * ST[0][q] + 2.0f * gc2 * ST[1][q];
    }
    // ---- T = J W -> J -> camera-space position ----
    float gJ[2][3];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int k = 0; k < 3; ++k) gJ[r][k] = gT[r][0] * W[3 * k] + gT[r][1] * W[3 * k + 1] + gT[r][2] * W[3 * k + 2];
    float gpx = gu * cam.fx * iz, gpy = gv * cam.fy * iz;
    float gpz = -(gu * cam.fx * px + gv * cam.fy * py) * iz2;
    gpz += -(gJ[0][0] * cam.fx + gJ[1][1] * cam.fy) * iz2;
    const float iz3 = iz2 * iz;
    if (!clx) {
        gpx += gJ[0][2] * (-cam.fx * iz2);
        gpz += gJ[0][2] * (2.0f * cam.fx * tx * iz3);
    } else {
        gpz += gJ[0][2] * (cam.fx * (tx * iz) * iz2);  // tx = lim pz: J02 = -fx lim / pz
    }
    if (!cly) {
        gpy += gJ[1][2] * (-cam.fy * iz2);
        gpz += gJ[1][2] * (2.0f * cam.fy * ty * iz3);
    } else {
        gpz += gJ[1][2] * (cam.fy * (ty * iz) * iz2);
    }
    // camera transform p_cam = W p + t
    gm[0] += W[0] * gpx + W[3] * gpy + W[6] * gpz;
    gm[1] += W[1] * gpx + W[4] * gpy + W[7] * gpz;
    gm[2] += W[2] * gpx + W[5] * gpy + W[8] * gpz;
    add_grad<kFresh>(&out.means[3 * i], gm[0]);
    add_grad<kFresh>(&out.means[3 * i + 1], gm[1]);
    add_grad<kFresh>(&out.means[3 * i + 2], gm[2]);

    // ---- S = M M^T -> M = R(q) diag(s) -> s, R(q) ----
    float gM[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            gM[r][k] = (gS[r][0] + gS[0][r]) * M[0][k] + (gS[r][1] + gS[1][r]) * M[1][k] + (gS[r][2] + gS[2][r]) * M[2][k];
    float gR[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float gs = 0.f;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            gR[r][k] = gM[r][k] * s[k];
            gs += gM[r][k] * Rq[r][k];
        }
        add_grad<kFresh>(&out.log_scales[3 * i + k], gs * s[k]);  // s = exp(log s) * splat_scale
    }
    const float gqw = 2.0f * (-qz * gR[0][1] + qy * gR[0][2] + qz * gR[1][0] - qx * gR[1][2] - qy * gR[2][0] + qx * gR[2][1]);
    const float gqx = 2.0f * (qy * gR[0][1] + qz * gR[0][2] + qy * gR[1][0] - 2.0f * qx * gR[1][1] - qw * gR[1][2] +
                              qz * gR[2][0] + qw * gR[2][1] - 2.0f * qx * gR[2][2]);
    const float gqy = 2.0f * (-2.0f * qy * gR[0][0] + qx * gR[0][1] + qw * gR[0][2] + qx * gR[1][0] + qz * gR[1][2] -
                              qw * gR[2][0] + qz * gR[2][1] - 2.0f * qy * gR[2][2]);
    const float gqz = 2.0f * (-2.0f * qz * gR[0][0] - qw * gR[0][1] + qx * gR[0][2] + qw * gR[1][0] -
                              2.0f * qz * gR[1][1] + qy * gR[1][2] + qx * gR[2][0] + qy * gR[2][1]);
    // q_n = q / |q|
    const float dq = qw * gqw + qx * gqx + qy * gqy + qz * gqz;
    const float il = qlen > 0 ? 1.0f / qlen : 0.f;
    float4* gq4 = reinterpret_cast<float4*>(out.quats) + i;
    const float4 oq = kFresh ? make_float4(0.f, 0.f, 0.f, 0.f) : *gq4;
    *gq4 = make_float4(__fadd_rn(oq.x, (gqw - qw * dq) * il), __fadd_rn(oq.y, (gqx - qx * dq) * il),
                       __fadd_rn(oq.z, (gqy - qy * dq) * il), __fadd_rn(oq.w, (gqz - qz * dq) * il));
}

}  // namespace

namespace {
template <int TW, int TH, int kBatch>
void launch_blend_backward_t(const BackwardIn& in, unsigned tiles, float* grad_pair, cudaStream_t stream) {
    constexpr int kDevices = 64;
    constexpr size_t kShared = sizeof(BackwardShared<TW, TH, kBatch>);
    static std::atomic<bool> raised[kDevices];  // the dynamic shared memory limit, once per device
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kDevices && !raised[dev]) {
        if (cudaFuncSetAttribute(blend_backward_kernel<TW, TH, kBatch>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(kShared)) == cudaSuccess)
            raised[dev] = true;
    }
    cudaGetLastError();  // a failed raise shows up as the launch's error
    launch_chained_smem(blend_backward_kernel<TW, TH, kBatch>, dim3(tiles), dim3(TW * TH / 2), kShared, stream, in,
                        grad_pair);
}

template <int kBatch>
void launch_blend_backward_rounds(const BackwardIn& in, unsigned tiles, int tile_w, int tile_h, float* grad_pair,
                                  cudaStream_t stream) {
    if (tile_w == 8) launch_blend_backward_t<8, 8, kBatch>(in, tiles, grad_pair, stream);
    else if (tile_h == 32) launch_blend_backward_t<16, 32, kBatch>(in, tiles, grad_pair, stream);
    else launch_blend_backward_t<16, 16, kBatch>(in, tiles, grad_pair, stream);
}
}  // namespace

void launch_blend_backward(const BackwardIn& in, unsigned tiles, int tile_w, int tile_h, bool sparse, float* grad_pair,
                           cudaStream_t stream) {
    if (tiles == 0) return;
    if (sparse) launch_blend_backward_rounds<kBackwardSparseBatch>(in, tiles, tile_w, tile_h, grad_pair, stream);
    else launch_blend_backward_rounds<kBackwardBatch>(in, tiles, tile_w, tile_h, grad_pair, stream);
}

namespace {
// The fresh and the accumulating gradient passes are separate instantiations: a run-time flag
// inside the kernel made the accumulating one (a batch's later views) slower.
template <bool kFresh>
void launch_gauss_backward_t(const GaussBackwardArgs& a, const Ctrl* ctrl, const unsigned* list,
                             const unsigned* list_count, const unsigned* rank, const unsigned* offs,
                             const unsigned long long* rect, const unsigned long long* whole, const float* grad_pair,
                             dim3 grid, dim3 block,
                             cudaStream_t stream) {
    switch (a.sh_degree) {
        case 0: launch_chained(gauss_backward_kernel<0, kFresh>, grid, block, stream, a.scenes, a.scene, a.views,
                               a.view, a.grads, ctrl, list, list_count, rank, offs, rect, whole,
                               grad_pair); break;
        case 1: launch_chained(gauss_backward_kernel<1, kFresh>, grid, block, stream, a.scenes, a.scene, a.views,
                               a.view, a.grads, ctrl, list, list_count, rank, offs, rect, whole,
                               grad_pair); break;
        case 2: launch_chained(gauss_backward_kernel<2, kFresh>, grid, block, stream, a.scenes, a.scene, a.views,
                               a.view, a.grads, ctrl, list, list_count, rank, offs, rect, whole,
                               grad_pair); break;
        default: launch_chained(gauss_backward_kernel<3, kFresh>, grid, block, stream, a.scenes, a.scene, a.views,
                                a.view, a.grads, ctrl, list, list_count, rank, offs, rect, whole,
                               grad_pair); break;
    }
}
}  // namespace

void launch_gauss_backward(const GaussBackwardArgs& a, const Ctrl* ctrl, const unsigned* depth_key,
                           const unsigned* rank, const unsigned* offs, const unsigned long long* rect,
                           const unsigned long long* whole, const float* grad_pair, unsigned* list, unsigned* list_count, cudaStream_t stream) {
    const unsigned lblocks = static_cast<unsigned>((a.n + 256 * kListItems - 1) / (256 * kListItems));
    if (lblocks == 0) return;
    launch_chained(visible_list_kernel, dim3(lblocks), dim3(256), stream, a.n, a.entry_base, depth_key, list,
                   list_count);
    const dim3 grid(static_cast<unsigned>((a.n + 127) / 128)), block(128);
    if (a.fresh)
        launch_gauss_backward_t<true>(a, ctrl, list, list_count, rank, offs, rect, whole, grad_pair, grid, block,
                                      stream);
    else
        launch_gauss_backward_t<false>(a, ctrl, list, list_count, rank, offs, rect, whole, grad_pair, grid, block,
                                       stream);
}

}  // namespace ab2
