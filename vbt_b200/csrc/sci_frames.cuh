// sci_frames.cuh -- (b') exact frames of scientific leaves, one warp per leaf and up to 16 frames.
// Included by kernels.cu.
//
// A frame of a leaf is 64 control values (a DCT sum each), their trilinear over 512 voxels, and the
// leaf's events or residual grid.  What the plain per-voxel form spends on it -- eight shared reads
// and seven lerps per voxel, every coefficient re-read and re-scaled per frame, events as
// read-modify-writes of stored voxels -- is taken apart here:
//  - controls: a lane keeps the coefficients of its two controls as doubles for all frames of the
//    item; a control value is `keep` fused multiply-adds in double (products of two floats are
//    exact there), the reference's own sum (render/src/scientific_decode.cpp:82-97);
//  - trilinear, separable as in rt_staged.cuh (the same lerps on the same operands): a lane makes one
//    x quad per frame, three y quads and four z quads.  The weights of a lane never change, so they
//    are registers; the upper half of an axis is taken in mirrored order (a (1 - t) + b t is b t +
//    a (1 - t)), which makes the control rows of every lane the same register names;
//  - events: the keys of a time bin are read once per bin, and the events of a frame go through a
//    shared-memory row of residuals that the z step adds; frames without events skip it.
// 64 frames of a 128^3 field (537 MB written, 83 us at the measured copy rate) on a B200: cache 162 us, dense
// frames 175 (voxel by voxel 1,203 and 1,388).  Bound by instruction issue (about 400 warp
// instructions per leaf and frame over all leaf kinds, 55 % of the slots) beside the stores.
#pragma once

namespace vbtb {

constexpr int kSciChunk = 16;   // frames of one item at most
constexpr int kSciWarps = 4;
constexpr int kSciWideFrames = 4;   // frames whose controls a WIDE item forms together
template <bool WIDE>
struct __align__(16) SciWarpShared {
    union {
        struct {
            float ctrl[WIDE ? kSciWideFrames * 64 : 64];   // control rows of 4 (WIDE: of four frames)
            float x[16 * 8];                // x-lerped control rows
            float residual[WIDE ? 1024 : 512];   // events of the frame (all 0 between frames), or residual grids of
                                                 // 64, in rows of 4 (WIDE: the temporal-basis grids of the leaf)
        };
        float general[64 + 16 * 64];   // sci_decode_controls' values, for leaves of no common shape
    };
    double basis[kSciChunk][4];
    int frames[kSciChunk];
    uint32_t code[kSciChunk];      // the frames' time bin << 7 | frame inside the bin (7 bits, as the keys hold it)
    uint32_t start[17];            // first event of each bin, and the event count
};

// The constant weights of a lane: x quad k = lane & 1 of row lane >> 1, y row (lane >> 1) & 7,
// z rows 0-3 (lanes 0-15) or 7-4 (lanes 16-31).  First / second: in mirrored order for the upper
// halves.
template <int R>
struct SciWeights {
    float xf[4], xs[4], yt, yo, zf[4], zs[4];
    int y0;
    __device__ __forceinline__ explicit SciWeights(int lane)
    {
        constexpr int g = R == 3 ? 1 : 0;
        const bool kx = (lane & 1) != 0, hz = lane >= 16;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float tx = g_sci_axis[g][kx ? 7 - i : i].t, tz = g_sci_axis[g][hz ? 7 - i : i].t;
            xf[i] = kx ? tx : __fsub_rn(1.0f, tx);
            xs[i] = kx ? __fsub_rn(1.0f, tx) : tx;
            zf[i] = hz ? tz : __fsub_rn(1.0f, tz);
            zs[i] = hz ? __fsub_rn(1.0f, tz) : tz;
        }
        const AxisWeight ay = g_sci_axis[g][(lane >> 1) & 7];
        yt = ay.t;
        yo = ay.omt;
        y0 = ay.i0;
    }
};

__device__ __forceinline__ float lerp_fs(float f, float s, float wf, float ws)
{
    return __fadd_rn(__fmul_rn(f, wf), __fmul_rn(s, ws));
}
__device__ __forceinline__ float4 add4(float4 a, float4 b)
{
    return make_float4(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z), __fadd_rn(a.w, b.w));
}
__device__ __forceinline__ float4 mul4(float4 a, float b)
{
    return make_float4(__fmul_rn(a.x, b), __fmul_rn(a.y, b), __fmul_rn(a.z, b), __fmul_rn(a.w, b));
}
__device__ __forceinline__ float4 lerp4(float4 a, float4 b, float wa, float wb)
{
    return make_float4(lerp_fs(a.x, b.x, wa, wb), lerp_fs(a.y, b.y, wa, wb), lerp_fs(a.z, b.z, wa, wb),
                       lerp_fs(a.w, b.w, wa, wb));
}

// The lane's four voxel quads of the trilinear of an R^3 grid (R = 3 or 4; rows of 4 floats in g):
// q[i] = voxels 4 (lane & 1) .. + 3 of row (lane >> 1) & 7 of layer i (lanes 0-15) or 7 - i.  Of a
// quad's positions (mirrored in the upper half) the first three lie between controls 0 and 1 and the
// fourth between 1 and 2 for R = 4, all between 0 and 1 for R = 3: the axis table of the positions
// p / 7 (R - 1).
template <int R>
__device__ __forceinline__ void sci_quads(const SciWeights<R>& W, const float* __restrict__ g, float* __restrict__ x,
                                          int lane, float4 q[4])
{
    const bool kx = (lane & 1) != 0, hz = lane >= 16;
    if (R == 4 || (lane >> 1) < R * R) {
        const float4 c = *reinterpret_cast<const float4*>(g + 4 * (lane >> 1));
        const float n0 = kx ? (R == 4 ? c.w : c.z) : c.x, n1 = kx ? (R == 4 ? c.z : c.y) : c.y, n2 = kx ? c.y : c.z;
        const float o0 = lerp_fs(n0, n1, W.xf[0], W.xs[0]), o1 = lerp_fs(n0, n1, W.xf[1], W.xs[1]);
        const float o2 = lerp_fs(n0, n1, W.xf[2], W.xs[2]);
        const float o3 = R == 4 ? lerp_fs(n1, n2, W.xf[3], W.xs[3]) : lerp_fs(n0, n1, W.xf[3], W.xs[3]);
        *reinterpret_cast<float4*>(x + 8 * (lane >> 1) + 4 * (lane & 1)) =
            kx ? make_float4(o3, o2, o1, o0) : make_float4(o0, o1, o2, o3);
    }
    __syncwarp();
    constexpr int N = R == 4 ? 3 : 2;
    float4 y[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
        const int z = hz ? R - 1 - n : n;
        const float* r = x + 8 * (z * R + W.y0) + 4 * (lane & 1);
        y[n] = lerp4(*reinterpret_cast<const float4*>(r), *reinterpret_cast<const float4*>(r + 8), W.yo, W.yt);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        q[i] = R == 4 && i == 3 ? lerp4(y[1], y[N - 1], W.zf[i], W.zs[i]) : lerp4(y[0], y[1], W.zf[i], W.zs[i]);
    __syncwarp();   // the x rows are read before the next grid or frame overwrites them
}

// The words of a leaf, read inside its part of the payload only.
struct SciWords {
    const uint32_t* __restrict__ w;
    uint32_t n;
    __device__ __forceinline__ uint32_t at(uint32_t i) const { return i < n ? __ldg(w + i) : 0u; }
    __device__ __forceinline__ uint32_t u32(uint32_t byte) const   // unaligned
    {
        return __funnelshift_r(at(byte >> 2), at((byte >> 2) + 1u), (byte & 3u) * 8u);
    }
    // The coefficients of the control record at byte cb: the DC half, then signed bytes times their AC
    // scales, rounded to float as the reference's coeff is (render/src/scientific_decode.cpp:86-93).
    __device__ __forceinline__ void coefficients(uint32_t cb, uint32_t keep, const float* __restrict__ scales,
                                                 double c[4]) const
    {
        const uint32_t i = cb >> 2, sh = (cb & 3u) * 8u, x1 = at(i + 1u);
        const uint32_t r0 = __funnelshift_r(at(i), x1, sh), r1 = __funnelshift_r(x1, at(i + 2u), sh);
        c[0] = (double)half_to_float_exact(r0 & 0xFFFFu);
        c[1] = keep > 1u ? (double)__fmul_rn(byte_to_float(r0, 2u), __ldg(scales)) : 0.0;
        c[2] = keep > 2u ? (double)__fmul_rn(byte_to_float(r0, 3u), __ldg(scales + 1)) : 0.0;
        c[3] = keep > 3u ? (double)__fmul_rn(byte_to_float(r1, 0u), __ldg(scales + 2)) : 0.0;
    }
    // Two controls (records at bytes ca and cb) at four frames f[0..3], any number of coefficients: the sum of
    // sci_control, term by term, with a word of four coefficients, their scales and four basis values of each
    // frame read at a time.
    __device__ __forceinline__ void sums(uint32_t ca, uint32_t cb, uint32_t keep, const float* __restrict__ scales,
                                         const float* __restrict__ basis, const int f[kSciWideFrames],
                                         double sa[kSciWideFrames], double sb[kSciWideFrames]) const
    {
        const double da = (double)half_to_float_exact(u32(ca) & 0xFFFFu), db = (double)half_to_float_exact(u32(cb) & 0xFFFFu);
#pragma unroll 1
        for (uint32_t k0 = 0; k0 < keep; k0 += 4u) {
            const uint32_t wa = u32(ca + 1u + k0), wb = u32(cb + 1u + k0);   // coefficient k is byte k + 1 of the record
            float4 b[kSciWideFrames];
#pragma unroll
            for (int j = 0; j < kSciWideFrames; ++j)
                b[j] = __ldg(reinterpret_cast<const float4*>(basis + (uint64_t)(uint32_t)f[j] * 64u + k0));
#pragma unroll
            for (uint32_t i = 0; i < 4u; ++i) {
                if (k0 + i >= keep) break;
                const bool dc = k0 + i == 0u;
                const float sc = dc ? 0.0f : __ldg(scales + k0 + i - 1u);
                const double qa = dc ? da : (double)__fmul_rn(byte_to_float(wa, i), sc);
                const double qb = dc ? db : (double)__fmul_rn(byte_to_float(wb, i), sc);
#pragma unroll
                for (int j = 0; j < kSciWideFrames; ++j) {
                    const double v = (double)(i == 0u ? b[j].x : i == 1u ? b[j].y : i == 2u ? b[j].z : b[j].w);
                    sa[j] = dc ? qa * v : __fma_rn(qa, v, sa[j]);
                    sb[j] = dc ? qb * v : __fma_rn(qb, v, sb[j]);
                }
            }
        }
    }
    // sample ci of the BFP grid whose codes start at byte `data` (bfp_sample: at most two bytes of a code)
    __device__ __forceinline__ uint32_t code(uint32_t data, uint32_t bit) const
    {
        return (u32(data + (bit >> 3)) & 0xFFFFu) >> (bit & 7u);
    }
    // event i of a SparseEvents leaf whose keys start at word kw: key, and residual q * es
    __device__ __forceinline__ uint32_t event_key(uint32_t kw, uint32_t i) const
    {
        return (at(kw + (i >> 1)) >> ((i & 1u) * 16u)) & 0xFFFFu;
    }
    __device__ __forceinline__ float event_value(uint32_t rw, uint32_t i, float es) const
    {
        int q = (int)((at(rw + (i >> 3)) >> ((i & 7u) * 4u)) & 0xFu);
        if (q & 8) q -= 16;
        return __fmul_rn((float)q, es);
    }
};

// Is the leaf of the common shape?  No events, or events that the visit of a bin finds as the search does
// (kFlagSorted); every section inside the payload; and, but for the WIDE kernel, at most four coefficients per
// control, no temporal-basis residual and codes of at most eight bits.
template <bool WIDE>
__device__ __forceinline__ bool sci_common_shape(const AssetGeom& g, const LeafEntry& e)
{
    const uint64_t room = 4ull * (g.payload_words - e.word_off);
    const uint32_t hdr = e.header, mode = hdr & 3u, keep = ((hdr >> 2) & 0x3Fu) + 1u;
    const uint64_t sb = 4u + 64u * (keep + 1u);
    if ((!WIDE && keep > 4u) || sb + 4u > room) return false;
    if (mode == 1u && ((hdr >> 16) & 0x0FFFu) != 0u) {
        const uint32_t tier = (hdr >> 8) & 3u;
        const uint32_t cap = tier == 0u ? 64u : tier == 1u ? 256u : tier == 2u ? 768u : 1024u;
        return (e.info & kFlagSorted) != 0u && sb + 100u + 2u * cap + cap / 2u <= room;
    }
    if (mode >= 2u) {
        const bool tb = ((hdr >> 12) & 7u) == 1u;
        const uint32_t per = mode == 2u ? 27u : 64u, bits = (hdr >> 8) & 0xFu;
        const uint64_t grids = tb ? ((hdr >> 15) & 0xFu) + 1u : g.frames;
        const uint64_t end = sb + grids * (2u + (per * bits + 7u) / 8u);
        return (WIDE || (!tb && bits <= 8u)) && end <= room && end < (1ull << 32);
    }
    return true;
}

// grid.x: one warp per leaf, so that the warps of a CTA write neighbouring leaves together (warps that
// stride over leaves drift apart, and partly written lines fall out of L2: 64 dense frames of
// 256 x 128 x 128 took 650 us instead of 380); grid.y: the chunks of the launch's frames in turn.
// Leaves of no common shape (sections that leave the payload, unsorted events) go through the per-frame
// functions.
// WIDE: for files with leaves of five or more coefficients, temporal-basis residuals or codes of over eight
// bits (AssetGeom::wide).  Controls are summed four frames at a time from the payload instead of from four
// registers; a temporal-basis residual keeps its decoded grids in shared memory and takes each one's
// trilinear, which no frame changes, once for two frames.  Bound by instruction issue as the other.  64 frames
// of 128^3 into the cache on a B200: 6 coefficients 206 us, 12 226, residuals of 8 basis grids 476 (leaf by leaf
// and frame by frame 1,221, 1,467 and 4,348).  An instantiation of its own, since its controls and sums cost
// the other kernel registers.
// Four CTAs of 128 registers: with 96 registers and five, the spills and the wider spread of the writes
// cost more than the warps hide (an earlier form of the loop: 265 us against 222).
// LOOSE: a cache that starts at any float, its frames any number of floats apart (an instantiation of its
// own: the test in the one kernel costs an aligned window of 64 frames of 128^3 1.5 %).
template <bool DENSE, bool LOOSE, bool WIDE>
__global__ void __launch_bounds__(kSciWarps * 32, 4) sci_frames_kernel(DeviceAsset a, FrameList fl, int chunk,
                                                                       float* __restrict__ out, uint64_t frame_stride)
{
    __shared__ SciWarpShared<WIDE> s_all[kSciWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    SciWarpShared<WIDE>& sh = s_all[warp];
    const uint32_t n_leaves = DENSE ? a.g.leaf_count : *(volatile const uint32_t*)a.counters;
    const int ly = (lane >> 1) & 7, lx0 = 4 * (lane & 1);
    const bool hz = lane >= 16;
    const SciWeights<4> W(lane);
    // 16-byte stores: every quad of every frame on a 16-byte boundary
    const bool aligned = DENSE ? (a.g.width & 3u) == 0u && (frame_stride & 3u) == 0u &&
                                     (reinterpret_cast<uintptr_t>(out) & 15u) == 0u
                               : !LOOSE;
    const int f0 = (int)blockIdx.y * chunk, n = min(chunk, fl.n - f0);
    for (uint64_t at = (uint64_t)blockIdx.x * kSciWarps + warp; at < n_leaves; at += (uint64_t)gridDim.x * kSciWarps) {
        const uint32_t rank = (uint32_t)at;
        const uint32_t leaf = DENSE ? rank : __ldg(a.active_list + rank);
        const LeafEntry e = a.entries[leaf];
        uint32_t bx, by, bz;
        int w, h, d;
        leaf_extent(a.g, leaf, bx, by, bz, w, h, d);
        const bool whole = w == 8 && h == 8 && d == 8;
        // the leaf's first voxel in a frame, and the steps of a row and a layer
        const uint64_t origin = DENSE ? ((uint64_t)(bz * 8u) * a.g.height + by * 8u) * a.g.width + bx * 8u : (uint64_t)rank * 512u;
        const uint64_t row = DENSE ? a.g.width : 8u, plane = DENSE ? (uint64_t)a.g.width * a.g.height : 64u;
        float* const fout = out + (uint64_t)f0 * frame_stride + origin;
        // whole quads at a lane's place: its first row, and the step from layer to layer
        const bool plain = whole && aligned;
        float* dst = fout + (hz ? 7u * plane : 0u) + (uint64_t)ly * row + (uint64_t)lx0;
        const int64_t zstep = hz ? -(int64_t)plane : (int64_t)plane;
        // voxels lx .. lx + 3 of a row: in the cache all four, 0 outside the extent; in dense frames
        // what lies inside
        auto put = [&](int j, int y, int z, int lx, float4 v) {
            float* o = fout + (uint64_t)j * frame_stride + (uint64_t)z * plane + (uint64_t)y * row + (uint64_t)lx;
            const bool in = y < h && z < d;
            if (!DENSE) {
                if (!whole) {
                    if (!in || lx >= w) v.x = 0.0f;
                    if (!in || lx + 1 >= w) v.y = 0.0f;
                    if (!in || lx + 2 >= w) v.z = 0.0f;
                    if (!in || lx + 3 >= w) v.w = 0.0f;
                }
                if (aligned) {
                    *reinterpret_cast<float4*>(o) = v;
                } else {
                    o[0] = v.x;
                    o[1] = v.y;
                    o[2] = v.z;
                    o[3] = v.w;
                }
            } else if (in) {
                if (aligned && w == 8) {
                    *reinterpret_cast<float4*>(o) = v;
                } else {
                    if (lx < w) o[0] = v.x;
                    if (lx + 1 < w) o[1] = v.y;
                    if (lx + 2 < w) o[2] = v.z;
                    if (lx + 3 < w) o[3] = v.w;
                }
            }
        };
        const uint32_t st = entry_status(e);
        if (st != kOk) {
            if (lane == 0) record_error(a.err, leaf, st);
            for (int j = 0; j < n; ++j)
                for (int i = 0; i < 4; ++i) put(j, ly, hz ? 7 - i : i, lx0, make_float4(0.f, 0.f, 0.f, 0.f));
            continue;
        }
        if (lane < n) sh.frames[lane] = clamp_frame(fl.f[f0 + lane], (int)a.g.frames);
        __syncwarp();
        if (!sci_common_shape<WIDE>(a.g, e)) {
            bool oob = false;
            for (int j = 0; j < n; ++j) {
                const uint32_t t = (uint32_t)sh.frames[j];
                sci_decode_controls(a, e, t, sh.general, lane, oob);
                __syncwarp();
                for (int r = lane; r < 64; r += 32) {
                    float v[8];
                    sci_row(a, e, sh.general, t, w, h, d, r & 7, r >> 3, v, oob);
                    put(j, r & 7, r >> 3, 0, make_float4(v[0], v[1], v[2], v[3]));
                    put(j, r & 7, r >> 3, 4, make_float4(v[4], v[5], v[6], v[7]));
                }
                __syncwarp();
            }
            if (__any_sync(0xFFFFFFFFu, oob) && lane == 0) record_error(a.err, leaf, kErrDecodeOob);
            continue;
        }
        const uint32_t hdr = e.header, mode = hdr & 3u;
        const uint32_t keep = ((hdr >> 2) & 0x3Fu) + 1u;
        const uint64_t room = a.g.payload_words - e.word_off;
        const SciWords lw{a.payload + e.word_off, room < 0x40000000ull ? (uint32_t)room : 0x40000000u};
        const uint32_t sb = 4u + 64u * (keep + 1u), sw = sb >> 2;
        // coefficients of controls lane and lane + 32, and the basis rows of the frames
        const uint32_t cb0 = 4u + (uint32_t)lane * (keep + 1u), cb1 = cb0 + 32u * (keep + 1u);
        double c0[4], c1[4];
        if constexpr (!WIDE) {
            lw.coefficients(cb0, keep, a.scales, c0);
            lw.coefficients(cb1, keep, a.scales, c1);
        }
        for (int i = lane; !WIDE && i < n * 4; i += 32)
            sh.basis[i >> 2][i & 3] = (double)__ldg(a.basis + (uint64_t)(uint32_t)sh.frames[i >> 2] * 64u + (uint32_t)(i & 3));
        // events of the item's time bins: each lane keeps two of them (64 in all; a 16-frame item of a
        // field with 0.5 % of its values stored as events has about 40), the others are read per frame
        const uint32_t count = mode == 1u ? (hdr >> 16) & 0x0FFFu : 0u;
        const uint32_t tier = (hdr >> 8) & 3u, cap = tier == 0u ? 64u : tier == 1u ? 256u : tier == 2u ? 768u : 1024u;
        const float es = count ? __uint_as_float(lw.at(sw)) : 0.0f;
        const bool events = es > 0.0f;
        const uint32_t kw = sw + 25u, rw = kw + cap / 2u;
        uint32_t ev_end = 0, ev_rest = 0, k0 = 0, k1 = 0, code0 = 0xFFFFFFFFu, code1 = 0xFFFFFFFFu;
        float v0e = 0.0f, v1e = 0.0f;
        if (events) {
            const uint32_t fpb = ((hdr >> 10) & 0xFu) + 1u;
            const uint32_t t = (uint32_t)sh.frames[lane < n ? lane : 0], b = min(t / fpb, 15u);
            if (lane < n) sh.code[lane] = (b << 7) | ((t - b * fpb) & 0x7Fu);
            if (lane < 16) sh.start[lane] = (lw.at(sw + 17u + ((uint32_t)lane >> 1)) >> ((lane & 1) * 16)) & 0xFFFFu;
            if (lane == 16) sh.start[16] = count;
            for (int i = lane; i < 128; i += 32) reinterpret_cast<float4*>(sh.residual)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            const uint32_t b0 = __reduce_min_sync(0xFFFFFFFFu, b), b1 = __reduce_max_sync(0xFFFFFFFFu, b);
            __syncwarp();
            const uint32_t first = sh.start[b0];
            ev_end = min(sh.start[b1 + 1u], cap);
            ev_rest = first + 64u;
            auto event = [&](uint32_t i, uint32_t& k, uint32_t& code, float& v) {
                if (i >= ev_end) return;
                const uint32_t key = lw.event_key(kw, i);
                uint32_t bin = b0;
                for (uint32_t c = b0 + 1u; c <= b1; ++c) bin += sh.start[c] <= i ? 1u : 0u;
                k = key & 511u;
                code = (bin << 7) | (key >> 9);
                v = lw.event_value(rw, i, es);
            };
            event(first + (uint32_t)lane, k0, code0, v0e);
            event(first + 32u + (uint32_t)lane, k1, code1, v1e);
        }
        const bool more = ev_end > ev_rest;
        // residual grid: code bits of samples lane and lane + 32, read one frame ahead
        const uint32_t per = mode == 2u ? 27u : 64u;
        const uint32_t bits = (hdr >> 8) & 0xFu, fbytes = (per * bits + 7u) / 8u;
        const uint32_t gb0 = (uint32_t)lane * bits, gb1 = (uint32_t)(lane + 32) * bits;
        uint32_t g0 = 0, g1 = 0, gs = 0;
        auto read_grid = [&](uint32_t t) {
            const uint32_t data = sb + 2u * a.g.frames + t * fbytes;
            g0 = WIDE ? lw.code(data, gb0) : lw.u32(data + (gb0 >> 3)) >> (gb0 & 7u);
            g1 = WIDE ? lw.code(data, gb1) : lw.u32(data + (gb1 >> 3)) >> (gb1 & 7u);
            gs = lw.u32(sb + 2u * t) & 0xFFFFu;
        };
        const bool tb = WIDE && mode >= 2u && ((hdr >> 12) & 7u) == 1u;   // the leaf's grids times basis values
        if (mode >= 2u && !tb) read_grid((uint32_t)sh.frames[0]);
        // a code's level, by lane: the division of decode_bfp once per item (up to 5 bits)
        const float level = mode >= 2u ? decode_bfp((uint32_t)lane, 1.0f, (int)bits) : 0.0f;
        // the controls of frames j .. j + 3, where j is the first of them
        auto controls = [&](int j) {
            int f[kSciWideFrames];
            double sa[kSciWideFrames], sb2[kSciWideFrames];
#pragma unroll
            for (int i = 0; i < kSciWideFrames; ++i) f[i] = sh.frames[min(j + i, n - 1)];
            lw.sums(cb0, cb1, keep, a.scales, a.basis, f, sa, sb2);
#pragma unroll
            for (int i = 0; i < kSciWideFrames; ++i) {
                sh.ctrl[64 * i + lane] = (float)sa[i];
                sh.ctrl[64 * i + 32 + lane] = (float)sb2[i];
            }
        };
        if constexpr (WIDE) {
            if (tb) {
                const uint32_t tkeep = ((hdr >> 15) & 0xFu) + 1u, grids = bits ? tkeep : 0u;   // no bits: no residual
                const uint32_t mask = (1u << bits) - 1u;
                for (uint32_t i = (uint32_t)lane; i < grids * per; i += 32u) {
                    const uint32_t k = i / per, ci = i - k * per;
                    const float sc = half_to_float_exact(lw.u32(sb + 2u * k) & 0xFFFFu);
                    sh.residual[64u * k + (mode == 2u ? ci / 3u * 4u + ci % 3u : ci)] =
                        decode_bfp(lw.code(sb + 2u * tkeep + k * fbytes, ci * bits) & mask, sc, (int)bits);
                }
                const SciWeights<3> W3(lane);
                __syncwarp();
                for (int j = 0; j < n; j += 2) {
                    if (j % kSciWideFrames == 0) controls(j);
                    const float* r0 = a.basis + (uint64_t)(uint32_t)sh.frames[j] * 64u;
                    const float* r1 = a.basis + (uint64_t)(uint32_t)sh.frames[min(j + 1, n - 1)] * 64u;
                    float4 sum[2][4], q[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) sum[0][i] = sum[1][i] = make_float4(0.f, 0.f, 0.f, 0.f);
                    __syncwarp();
#pragma unroll 1
                    for (uint32_t k = 0; k < grids; ++k) {
                        if (mode == 3u) sci_quads<4>(W, sh.residual + 64u * k, sh.x, lane, q);
                        else sci_quads<3>(W3, sh.residual + 64u * k, sh.x, lane, q);
                        const float b0 = __ldg(r0 + k), b1 = __ldg(r1 + k);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            sum[0][i] = add4(sum[0][i], mul4(q[i], b0));
                            sum[1][i] = add4(sum[1][i], mul4(q[i], b1));
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        if (j + u >= n) break;
                        sci_quads<4>(W, sh.ctrl + 64 * ((j + u) % kSciWideFrames), sh.x, lane, q);
#pragma unroll
                        for (int i = 0; i < 4; ++i) q[i] = add4(q[i], sum[u][i]);
                        if (plain) {
                            float* o = dst;
#pragma unroll
                            for (int i = 0; i < 4; ++i, o += zstep) __stcs(reinterpret_cast<float4*>(o), q[i]);
                            dst += frame_stride;
                        } else {
#pragma unroll
                            for (int i = 0; i < 4; ++i) put(j + u, ly, hz ? 7 - i : i, lx0, q[i]);
                        }
                    }
                }
                continue;
            }
        }
        __syncwarp();
        for (int j = 0; j < n; ++j) {
            const float* ctrl = sh.ctrl;
            if constexpr (WIDE) {
                if (j % kSciWideFrames == 0) controls(j);
                ctrl += 64 * (j % kSciWideFrames);
            } else {
                double s0 = c0[0] * sh.basis[j][0], s1 = c1[0] * sh.basis[j][0];
#pragma unroll
                for (int k = 1; k < 4; ++k)
                    if (k < (int)keep) {
                        const double b = sh.basis[j][k];
                        s0 = __fma_rn(c0[k], b, s0);
                        s1 = __fma_rn(c1[k], b, s1);
                    }
                sh.ctrl[lane] = (float)s0;
                sh.ctrl[lane + 32] = (float)s1;
            }
            bool hit0 = false, hit1 = false;
            uint32_t code = 0u, r0 = 0u, r1 = 0u;   // the frame's bin, and its events that no lane keeps
            if (events) {
                code = sh.code[j];
                hit0 = code0 == code;
                hit1 = code1 == code;
                if (hit0) sh.residual[k0] = v0e;
                if (hit1) sh.residual[k1] = v1e;
                if (more) {
                    r0 = max(sh.start[code >> 7], ev_rest) + (uint32_t)lane;
                    r1 = min(sh.start[(code >> 7) + 1u], ev_end);
                    for (uint32_t i = r0; i < r1; i += 32u) {
                        const uint32_t k = lw.event_key(kw, i);
                        if ((k >> 9) == (code & 0x7Fu)) sh.residual[k & 511u] = lw.event_value(rw, i, es);
                    }
                }
            }
            const bool add = events && (more || __any_sync(0xFFFFFFFFu, hit0 || hit1));
            float4 q[4];
            if (mode >= 2u) {
                const float sc = half_to_float_exact(gs);
                const uint32_t mask = (1u << bits) - 1u;
                float v0, v1;
                if (bits <= 5u) {
                    v0 = __fmul_rn(__shfl_sync(0xFFFFFFFFu, level, (int)(g0 & mask)), sc);
                    v1 = __fmul_rn(__shfl_sync(0xFFFFFFFFu, level, (int)(g1 & mask)), sc);
                } else {
                    v0 = decode_bfp(g0 & mask, sc, (int)bits);
                    v1 = decode_bfp(g1 & mask, sc, (int)bits);
                }
                if (j + 1 < n) read_grid((uint32_t)sh.frames[j + 1]);
                float4 qr[4];
                if (mode == 3u) {
                    sh.residual[lane] = v0;
                    sh.residual[lane + 32] = v1;
                    __syncwarp();
                    sci_quads<4>(W, sh.residual, sh.x, lane, qr);
                } else {
                    if (lane < 27) sh.residual[lane / 3 * 4 + lane % 3] = v0;
                    __syncwarp();
                    const SciWeights<3> W3(lane);
                    sci_quads<3>(W3, sh.residual, sh.x, lane, qr);
                }
                sci_quads<4>(W, ctrl, sh.x, lane, q);
#pragma unroll
                for (int i = 0; i < 4; ++i) q[i] = add4(q[i], qr[i]);
            } else {
                __syncwarp();
                sci_quads<4>(W, ctrl, sh.x, lane, q);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);   // a sum with +0 is not the value itself at -0
                    if (add) r = *reinterpret_cast<const float4*>(sh.residual + 64 * (hz ? 7 - i : i) + 8 * ly + lx0);
                    q[i] = add4(q[i], r);
                }
            }
            if (plain) {
                float* o = dst;
#pragma unroll
                for (int i = 0; i < 4; ++i, o += zstep) __stcs(reinterpret_cast<float4*>(o), q[i]);
                dst += frame_stride;
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) put(j, ly, hz ? 7 - i : i, lx0, q[i]);
            }
            if (add) {   // the residual row is all 0 again
                __syncwarp();
                if (hit0) sh.residual[k0] = 0.0f;
                if (hit1) sh.residual[k1] = 0.0f;
                for (uint32_t i = r0; i < r1; i += 32u) {
                    const uint32_t k = lw.event_key(kw, i);
                    if ((k >> 9) == (code & 0x7Fu)) sh.residual[k & 511u] = 0.0f;
                }
                __syncwarp();
            }
        }
        __syncwarp();
    }
}

// Frames per item: 16 where that leaves twelve or more items for every resident warp, else 8, and 4
// where those would not give each warp two (an item's set-up costs about three frames; an earlier form of the
// loop, 64 frames of 128^3: 8 frames per item 216 us, 16 235; of 256 x 128 x 128: 385 and 375).
template <bool DENSE, bool LOOSE, bool WIDE>
static void launch_sci_variant(const DeviceAsset& a, const FrameList& fl, float* out, uint64_t stride, int grid,
                               cudaStream_t s)
{
    static int full = 0;
    if (!full) {
        int dev = 0, sms = 0, per = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, sci_frames_kernel<DENSE, LOOSE, WIDE>, kSciWarps * 32, 0);
        full = sms * (per > 0 ? per : 1);
    }
    const uint64_t warps = (uint64_t)full * kSciWarps, L = a.g.leaf_count;
    auto items = [&](int c) { return L * (uint64_t)((fl.n + c - 1) / c); };
    const int chunk = items(16) >= 12u * warps ? 16 : items(8) >= 2u * warps ? 8 : 4;
    const uint64_t most = (L + kSciWarps - 1) / kSciWarps;
    sci_frames_kernel<DENSE, LOOSE, WIDE><<<dim3((unsigned)(grid > 0 && (uint64_t)grid < most ? (uint64_t)grid : most),
                                                 (unsigned)((fl.n + chunk - 1) / chunk)),
                                            kSciWarps * 32, 0, s>>>(a, fl, chunk, out, stride);
}

template <bool DENSE>
static void launch_sci_frames(const DeviceAsset& a, const FrameList& fl, float* out, uint64_t stride, int grid,
                              cudaStream_t s)
{
    const bool loose = !DENSE && ((stride & 3u) != 0u || (reinterpret_cast<uintptr_t>(out) & 15u) != 0u);
    if (a.g.wide) {
        if (loose) launch_sci_variant<DENSE, !DENSE, true>(a, fl, out, stride, grid, s);
        else launch_sci_variant<DENSE, false, true>(a, fl, out, stride, grid, s);
    } else {
        if (loose) launch_sci_variant<DENSE, !DENSE, false>(a, fl, out, stride, grid, s);
        else launch_sci_variant<DENSE, false, false>(a, fl, out, stride, grid, s);
    }
}

}  // namespace vbtb
