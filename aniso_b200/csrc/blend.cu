// Step 5 of the rasterizer: front-to-back blending, one block per tile of a batch (any view),
// for tile shapes TW x TH of 8x8, 16x16 (the reference's) and 16x32 pixels.
//
// Per pixel this is the blend of render.cpp:195-220 / gpu_render.cu:180-233:
//   power = -(A dx^2 + C dy^2)/2 - B dx dy; skip if power > 0
//   alpha = min(0.99, opacity * exp(power)); skip if alpha < 1/255
//   stop (without applying) once T (1 - alpha) < 1e-4; else C += rgb alpha T, T *= 1 - alpha
// evaluated in base 2 on the pre-scaled conic of the SplatRecord (one MUFU ex2 per evaluation).
//
// B200 mapping (the kernel is issue bound, its ALU pipe the busiest, so the layout minimises
// instructions per pixel):
//   * each warp owns one 8x8 pixel block, each quarter warp one of its 4x4 cells, with two
//     horizontally adjacent pixels per lane; the row terms of the exponent (with log2(opacity)
//     folded in) are shared, and the two pixels' offsets and FMAs are packed FP32x2 instructions
//     (three for both pixels' exponents);
//   * the block stages kBatch splat records per round in shared memory and, per splat, a mask of
//     the tile's cells it can touch (staged_cell_mask): its pixel bounds (the CPU 8x8-tile
//     rectangle cut by the bounding box of the ellipse where alpha can reach 1/255, with a margin)
//     and the ellipse itself -- splats that are left out could not pass the alpha test anywhere in
//     the cell, so every pixel takes the splat list of the CPU renderer whatever the tile shape;
//   * each quarter warp walks only its own cell's splats (listed once per round from the masks by
//     ballot and popcount), the four side by side: a splat costs a warp a step only as often as its
//     quarters need it, and 4x4 cells waste fewer pixels around a splat than 8x8 blocks. The
//     quarters meet at the end of a round, so longer rounds even out their lists. Measured per 740k
//     1280x720 frame: blend 139 -> 124 us (122.7M -> 96.3M warp instructions) with one list per
//     quarter instead of per warp, the frame 266 -> 259 us with 256-splat rounds instead of 128,
//     -> 253 us with the ellipse test (8x8 blocks against the ellipse, in each tile's staging, had
//     cost more than they saved);
//   * a finished pixel holds T = 0 (T >= 1e-4 while it is not finished), so no separate flag is
//     carried; the warp leaves once all 64 pixels are finished and the block stops loading once all
//     its warps have (__syncthreads_or).
//   * a sparse frame (sparse_frame: under 32 entries per tile) is bound by the latency of each tile's few
//     splats, not by issue: the ellipse test, the lists and their padding took longer than the steps they
//     saved, and 56 to 85 registers and 19 KB left room for fewer CTAs. It takes instantiations of their own:
//     rounds of 128 (16x32: 256) splats, cells by the bounds alone, no lists where a round holds at most
//     32 splats, empty tiles left at once, 48 registers (16x16, 16x32). Eight 1660x984 views of two scenes of
//     20k: 410 -> 258 us a batch in 8x8 tiles, 239 -> 192 in 16x16, 236 -> 186 in 16x32 (with one list per warp
//     333, 228, 234).
// Tried and slower: comparisons as 0 / 1 floats with packed products in place of the selects
// (+1.5% per frame), predicated scalar updates (+4%), operands staged in pairs (+5.5%), ten CTAs per
// SM by holding the kernel to 48 registers (+3%).
#include "common.cuh"
#include "kernels.h"

namespace ab2 {
namespace {

// Both of a lane's pixels' step for one splat. p is each pixel's base-2 exponent including
// log2(opacity) L, so alpha = min(0.99, 2^p) and the reference's "power > 0" skip is p > L. The
// new transmittance is T - alpha T (one instruction fewer than T (1 - alpha); it differs only in
// rounding); once it would fall below 1e-4 the pixel is finished: T = 0 and the splat is not
// applied (T = 0 keeps a finished pixel finished). The weights, new transmittances and colour sums
// are packed FP32x2 instructions (per component the rounding of the scalar ones; T + (-1) w in one
// rounding is T - w) and the conditions selects: a pixel that does not take the splat adds 0 x
// colour, which leaves its sum as it was for the finite colours the blend stages (measured 0.153
// -> 0.139 ms of blend per 740k frame against a scalar step with branches). In training mode tfin
// keeps the transmittance after the last applied splat and last the list position one past it.
template <bool kTrain>
__device__ __forceinline__ void blend_px2(float2 p, float L, float r, float g, float b, float2& T, float2& cr,
                                          float2& cg, float2& cb, float2& tfin, unsigned& last0, unsigned& last1,
                                          unsigned pos) {
    bool v0, v1;
    const float a0 = splat_alpha(p.x, L, v0), a1 = splat_alpha(p.y, L, v1);
    const float2 w = __fmul2_rn(make_float2(a0, a1), T);
    const float2 nt = __ffma2_rn(make_float2(-1.f, -1.f), w, T);
    const bool k0 = v0 && !(nt.x < 1e-4f), k1 = v1 && !(nt.y < 1e-4f);
    T.x = v0 ? (k0 ? nt.x : 0.f) : T.x;  // taken, finished, or skipped
    T.y = v1 ? (k1 ? nt.y : 0.f) : T.y;
    const float2 wk = make_float2(k0 ? w.x : 0.f, k1 ? w.y : 0.f);
    cr = __ffma2_rn(make_float2(r, r), wk, cr);
    cg = __ffma2_rn(make_float2(g, g), wk, cg);
    cb = __ffma2_rn(make_float2(b, b), wk, cb);
    if (kTrain) {
        tfin.x = k0 ? nt.x : tfin.x;
        tfin.y = k1 ? nt.y : tfin.y;
        last0 = k0 ? pos : last0;
        last1 = k1 ? pos : last1;
    }
}

// The training outputs of one pixel: float colour, final transmittance, one past the last splat.
__device__ __forceinline__ void store_train_px(const ViewInfo& vi, int x, int y, float tfin, float cr, float cg,
                                               float cb, unsigned last) {
    const int width = vi.cam.width;
    if (x >= width || y >= vi.cam.height) return;
    const size_t p = static_cast<size_t>(y) * width + x;
    vi.rgbf[p * 3 + 0] = cr;
    vi.rgbf[p * 3 + 1] = cg;
    vi.rgbf[p * 3 + 2] = cb;
    vi.t_final[p] = tfin;
    vi.n_contrib[p] = last;
}

// One 8-bit channel as render.cpp quantises it: clamp to [0, 1], scale by 255, round half up.
__device__ __forceinline__ unsigned quantise(float c) {
    return static_cast<unsigned>(static_cast<uint8_t>(fminf(fmaxf(c, 0.f), 1.f) * 255.f + 0.5f));
}

// Copies the tile's RGB8 pixels, staged in s_px (TH rows of TW * 3 bytes, 16-byte aligned), to
// the image as whole row segments: 16-byte stores where the image rows and the segment allow,
// else 4-byte ones, else single bytes. Wide contiguous stores matter most when `out` is pinned
// host memory written across PCIe during the blend (each store instruction becomes a few bus
// writes, where per-pixel bytes would become many partial ones); in device memory they cost no
// more than per-pixel stores. kBlack: zeros, nothing is read.
template <int TW, int TH, int kThreads, bool kBlack = false>
__device__ __forceinline__ void write_tile_rgb8(const unsigned char* s_px, uint8_t* out, int width, int height,
                                                int ox, int oy) {
    constexpr int kRow = TW * 3;
    const int rows = min(TH, height - oy), seg = min(TW, width - ox) * 3;  // both >= 1: the tile starts inside
    const size_t pitch = static_cast<size_t>(width) * 3;
    uint8_t* dst = out + static_cast<size_t>(oy) * pitch + static_cast<size_t>(ox) * 3;
    const uintptr_t a = reinterpret_cast<uintptr_t>(dst) | pitch | static_cast<unsigned>(seg) | kRow;
    if ((a & 15) == 0) {
        const int per = seg >> 4;
        for (int i = threadIdx.x; i < rows * per; i += kThreads) {
            const int r = i / per, c = i - r * per;
            *reinterpret_cast<uint4*>(dst + r * pitch + c * 16) =
                kBlack ? make_uint4(0, 0, 0, 0) : *reinterpret_cast<const uint4*>(s_px + r * kRow + c * 16);
        }
    } else if ((a & 3) == 0) {
        const int per = seg >> 2;
        for (int i = threadIdx.x; i < rows * per; i += kThreads) {
            const int r = i / per, c = i - r * per;
            *reinterpret_cast<unsigned*>(dst + r * pitch + c * 4) =
                kBlack ? 0u : *reinterpret_cast<const unsigned*>(s_px + r * kRow + c * 4);
        }
    } else {
        for (int i = threadIdx.x; i < rows * seg; i += kThreads) {
            const int r = i / seg, c = i - r * seg;
            dst[r * pitch + c] = kBlack ? static_cast<unsigned char>(0) : s_px[r * kRow + c];
        }
    }
}

template <int TW, int TH, int kBatch, bool kTrain, bool kSparse>
__global__ void __launch_bounds__(TW * TH / 2, kSparse ? 1280 / (TW * TH / 2) : 0) blend_kernel(const uint2* __restrict__ ranges,
                                                            const unsigned* __restrict__ vals,
                                                            const SplatRecord* __restrict__ rec, const Ctrl* ctrl,
                                                            const ViewInfo* __restrict__ views, BatchTables tables) {
    chain_entry();
    constexpr int kThreads = TW * TH / 2;  // two pixels per lane
    constexpr int kWarpsX = TW / 8;
    constexpr int kCells = TW / 4;         // 4x4-pixel cells per tile row
    __shared__ float4 s_r0[kBatch + 1];    // the last slot: a splat that no pixel takes
    __shared__ float4 s_r1[kBatch + 1];
    __shared__ float s_b[kBatch + 1];
    __shared__ unsigned s_mask[kBatch];
    __shared__ __align__(8) unsigned short s_list[kThreads / 8][kBatch + 4];  // each quarter warp's splats of the round
    __shared__ __align__(16) unsigned char s_px[TH * TW * 3];  // the tile's RGB8, staged for row stores

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, quarter = lane >> 3;
    const unsigned gtile = blockIdx.x;
    const unsigned v = find_segment(tables.tile_base, tables.n_views, gtile);
    const ViewInfo& vi = views[v];
    const int tiles_x = vi.cam.tilesX;
    const unsigned local = gtile - vi.tile_base;
    const int ox = static_cast<int>(local % tiles_x) * TW, oy = static_cast<int>(local / tiles_x) * TH;
    const int x0 = ox + (warp % kWarpsX) * 8 + 4 * (quarter & 1) + 2 * (lane & 1);
    const int y = oy + (warp / kWarpsX) * 8 + 4 * (quarter >> 1) + ((lane >> 1) & 3);
    const int width = vi.cam.width, height = vi.cam.height;
    const float px0 = x0 + 0.5f, py = y + 0.5f;
    const uint2 range = (ctrl->flags & kFlagOverflow) ? make_uint2(0, 0) : ranges[gtile];
    const unsigned lt = lanemask_lt();
    // The warp's cells in a staged splat's mask: quarters 0 and 1 at this bit, 2 and 3 one row below.
    const int cell0 = (warp / kWarpsX) * 2 * kCells + (warp % kWarpsX) * 2;

    if (kSparse && range.x == range.y) {  // an empty tile
        if (kTrain) {
            store_train_px(vi, x0, y, 1.0f, 0.f, 0.f, 0.f, range.x);
            store_train_px(vi, x0 + 1, y, 1.0f, 0.f, 0.f, 0.f, range.x);
        }
        if (vi.rgb8) write_tile_rgb8<TW, TH, kThreads, true>(nullptr, vi.rgb8, width, height, ox, oy);
        return;
    }
    if (tid == 0) {
        s_r0[kBatch] = make_float4(0.f, 0.f, 0.f, 0.f);
        s_r1[kBatch] = make_float4(0.f, -INFINITY, 0.f, 0.f);
        s_b[kBatch] = 0.f;
    }

    // Pixels outside the image start finished.
    float2 T = make_float2((x0 < width && y < height) ? 1.0f : 0.f, (x0 + 1 < width && y < height) ? 1.0f : 0.f);
    float2 cr = make_float2(0.f, 0.f), cg = cr, cb = cr;
    unsigned last0 = range.x, last1 = range.x;
    float2 tf = make_float2(1.0f, 1.0f);

    for (unsigned base = range.x; base < range.y; base += kBatch) {
        if (!__syncthreads_or(T.x + T.y > 0.f)) break;
#pragma unroll
        for (int h = 0; h < kBatch / kThreads; ++h) {
            const int slot = tid + h * kThreads;
            const unsigned j = base + slot;
            unsigned m = 0;
            if (j < range.y) {
                const SplatRecord r = rec[vals[j]];
                constexpr float kMax = 3.40282347e38f;  // an infinite colour quantises as the largest finite one
                s_r0[slot] = r.r0;
                s_r1[slot] = make_float4(r.r1.x, r.r1.y, fminf(r.r1.z, kMax), fminf(r.r1.w, kMax));
                s_b[slot] = fminf(r.r2.x, kMax);
                m = staged_cell_mask<TW, TH, 4, 4, !kSparse>(r, ox, oy);
            }
            s_mask[slot] = m;
        }
        __syncthreads();
        const unsigned cnt = min(static_cast<unsigned>(kBatch), range.y - base);
        const unsigned live = __ballot_sync(0xFFFFFFFFu, T.x + T.y > 0.f);
        if (!live) continue;  // the warp is finished
        const auto step = [&](unsigned id) {
            const float4 a = s_r0[id];
            const float4 k = s_r1[id];
            const float bb = s_b[id];
            float2 dx;
            const float2 pp = splat_exponents2(a, k, make_float2(px0, px0 + 1.0f), __fsub_rn(py, a.y), dx);
            blend_px2<kTrain>(pp, k.y, k.z, k.w, bb, T, cr, cg, cb, tf, last0, last1, base + id + 1);
        };
        if (kSparse && cnt <= 32) {
            // A short round: each quarter takes its splats from its ballot, without lists.
            const unsigned m = static_cast<unsigned>(lane) < cnt ? s_mask[lane] >> cell0 : 0u;
            unsigned todo = 0, steps = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const unsigned bits = __ballot_sync(0xFFFFFFFFu, (m >> ((q & 1) + (q >> 1) * kCells)) & 1u);
                if (quarter == q) todo = bits;
                steps = max(steps, static_cast<unsigned>(__popc(bits)));
            }
            for (; steps > 0; --steps) {
                step(todo ? __ffs(todo) - 1u : static_cast<unsigned>(kBatch));
                todo &= todo - 1;
            }
            continue;
        }
        // Each quarter's splats of the round in list order, compacted once (a ballot per quarter and 32
        // staged); a finished quarter takes none. Then every list is padded with the splat that no
        // pixel takes to the longest one's length, a multiple of four.
        unsigned n[4] = {0, 0, 0, 0};
        for (unsigned c = 0; c * 32 < cnt; ++c) {
            const unsigned idx = c * 32 + lane;
            const unsigned m = idx < cnt ? s_mask[idx] >> cell0 : 0u;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const bool mine = ((live >> (8 * q)) & 0xFFu) && ((m >> ((q & 1) + (q >> 1) * kCells)) & 1u);
                const unsigned bits = __ballot_sync(0xFFFFFFFFu, mine);
                if (mine) s_list[warp * 4 + q][n[q] + __popc(bits & lt)] = static_cast<unsigned short>(idx);
                n[q] += __popc(bits);
            }
        }
        const unsigned longest = (max(max(n[0], n[1]), max(n[2], n[3])) + 3u) & ~3u;
        const unsigned short* list = s_list[warp * 4 + quarter];
        const unsigned own = quarter == 0 ? n[0] : quarter == 1 ? n[1] : quarter == 2 ? n[2] : n[3];
        for (unsigned i = own + (lane & 7); i < longest; i += 8) s_list[warp * 4 + quarter][i] = kBatch;
        __syncwarp();
        for (unsigned i = 0; i < longest; i += 4) {
            const ushort4 four = *reinterpret_cast<const ushort4*>(list + i);
            const unsigned id[4] = {four.x, four.y, four.z, four.w};
            // Four splats per vote on whether the warp is finished.
#pragma unroll
            for (int u = 0; u < 4; ++u) step(id[u]);
            if (!__any_sync(0xFFFFFFFFu, T.x + T.y > 0.f)) break;
        }
    }
    if (kTrain) {
        store_train_px(vi, x0, y, tf.x, cr.x, cg.x, cb.x, last0);
        store_train_px(vi, x0 + 1, y, tf.y, cr.y, cg.y, cb.y, last1);
    }
    if (vi.rgb8) {  // the same for the whole block: one view per tile
        // The lane's two pixels are 6 bytes at an even pixel column: three 2-byte words.
        unsigned short* q = reinterpret_cast<unsigned short*>(s_px + ((y - oy) * TW + (x0 - ox)) * 3);
        q[0] = static_cast<unsigned short>(quantise(cr.x) | quantise(cg.x) << 8);
        q[1] = static_cast<unsigned short>(quantise(cb.x) | quantise(cr.y) << 8);
        q[2] = static_cast<unsigned short>(quantise(cg.y) | quantise(cb.y) << 8);
        __syncthreads();
        write_tile_rgb8<TW, TH, kThreads>(s_px, vi.rgb8, width, height, ox, oy);
    }
}

template <int TW, int TH, int kBatch, bool kSparse>
void launch_shape(unsigned tiles, const uint2* ranges, const unsigned* vals, const SplatRecord* rec, const Ctrl* ctrl,
                  const ViewInfo* views, const BatchTables& tables, bool train, cudaStream_t stream) {
    const auto kernel = train ? blend_kernel<TW, TH, kBatch, true, kSparse> : blend_kernel<TW, TH, kBatch, false, kSparse>;
    launch_chained(kernel, dim3(tiles), dim3(TW * TH / 2), stream, ranges, vals, rec, ctrl, views, tables);
}

}  // namespace

bool blend_shape_supported(int tile_w, int tile_h) {
    return (tile_w == 8 && tile_h == 8) || (tile_w == 16 && tile_h == 16) || (tile_w == 16 && tile_h == 32);
}

void launch_blend(unsigned tiles, const uint2* ranges, const unsigned* sorted_vals, const SplatRecord* rec,
                  const Ctrl* ctrl, const ViewInfo* views, const BatchTables& tables, int tile_w, int tile_h,
                  int batch, bool sparse, bool train, cudaStream_t stream) {
    if (tiles == 0) return;
    const bool big = batch >= 256;
    const auto launch = tile_w == 8    ? (sparse ? launch_shape<8, 8, 128, true>
                                          : big  ? launch_shape<8, 8, 256, false>
                                                 : launch_shape<8, 8, 128, false>)
                        : tile_h == 32 ? (sparse ? launch_shape<16, 32, 256, true> : launch_shape<16, 32, 256, false>)
                                       : (sparse ? launch_shape<16, 16, 128, true>
                                          : big  ? launch_shape<16, 16, 256, false>
                                                 : launch_shape<16, 16, 128, false>);
    launch(tiles, ranges, sorted_vals, rec, ctrl, views, tables, train, stream);
}

}  // namespace ab2
