// point_query.cuh -- (c) batched (x, y, z, t) point queries.  Included by kernels.cu.
//
// A query reads the eight corner controls of one cell (eight more of a FINE6 leaf or of a residual
// grid, one shell control of a Mode2 leaf, one event of a scientific leaf), each a short chain of
// dependent reads.  With one thread per query those chains run one after the other and lanes of
// different leaf kinds wait for each other; with eight lanes per query the set-up is done eight
// times.  So a warp takes up to 32 queries through three steps: each lane prepares its own query
// (leaf, cell, time bin) and leaves what the corners need in shared memory; the warp then decodes
// all corners of all queries, eight lanes to a query, streams of one kind together; and each lane
// forms its own query's lerps from the corner values, in the reference's order.  No step repeats
// another's work, and a batch of a few queries is still only one chain long.
// Bound by instruction issue (67 % of the slots, 63 warp instructions per query on a scientific
// field), then by L1/L2 latency; DRAM is idle.  On a B200: 1,000,000 random queries of a 256^3 x 96 plume
// 50 us, of a dense 128 x 128 x 192 x 40 fire 133, of a 128^3 x 64 scientific field 83; 1,000 queries 6.2 (one
// thread per query 138, 355, 203 and 34; eight lanes to a query from start to end 79, 226, 165).
#pragma once

namespace vbtb {

// Eight CTAs per SM: at most 64 registers (the kernels with scientific queries spill some set-up values) and 32
// warps, which hide the reads better than 24 warps at 80 registers (fire 175 us against 153 in the kernel for
// both kinds; 40 warps at 48 registers 143, but the plume 74 against 66).
// Events of a batch that eight lanes each look up in turn; more go to their own lanes.
constexpr int kPqEvents = 8;
constexpr int kPqWarps = 4, kPqCtas = 8, kPqThreads = 32 * kPqWarps, kPqBatch = 32;

// The general decode of one scientific query (src: decodeScientificValueAtCpu,
// render/src/scientific_decode.cpp:335-359) by one thread: sections that leave the payload.
__device__ __noinline__ float sci_point_general(const DeviceAsset& a, LeafEntry e, uint32_t lx, uint32_t ly, uint32_t lz,
                                                uint32_t t, bool* oob_out)
{
    SciReader rd{a.payload, a.g.payload_words, false};
    const uint64_t base = 4ull * e.word_off;
    const uint32_t hdr = e.header;
    const int keep = (int)((hdr >> 2) & 0x3Fu) + 1;
    const float* brow = a.basis + (uint64_t)t * 64u;
    const AxisWeight ax = c_sci_axis[0][lx], ay = c_sci_axis[0][ly], az = c_sci_axis[0][lz];
    auto at = [&](int cx, int cy, int cz) { return sci_control(a, rd, base, keep, (cz * 4 + cy) * 4 + cx, brow); };
    const float c00 = lerp_ref(at(ax.i0, ay.i0, az.i0), at(ax.i1, ay.i0, az.i0), ax.t, ax.omt);
    const float c01 = lerp_ref(at(ax.i0, ay.i0, az.i1), at(ax.i1, ay.i0, az.i1), ax.t, ax.omt);
    const float c10 = lerp_ref(at(ax.i0, ay.i1, az.i0), at(ax.i1, ay.i1, az.i0), ax.t, ax.omt);
    const float c11 = lerp_ref(at(ax.i0, ay.i1, az.i1), at(ax.i1, ay.i1, az.i1), ax.t, ax.omt);
    const float coarse = lerp_ref(lerp_ref(c00, c10, ay.t, ay.omt), lerp_ref(c01, c11, ay.t, ay.omt), az.t, az.omt);
    const uint32_t mode = hdr & 3u;
    float r = 0.0f;
    if (mode == 1u) {
        r = sci_sparse(rd, base, hdr, keep, (lz * 8u + ly) * 8u + lx, t);
    } else if (mode >= 2u) {
        const int res = mode == 2u ? 3 : 4;
        const int bits = (int)((hdr >> 8) & 0xFu);
        const uint32_t sub = (hdr >> 12) & 7u;
        const int per = res * res * res;
        const uint64_t scales = base + 4u + (uint64_t)(64 * (keep + 1));
        const int gi = mode == 2u ? 1 : 2;
        const AxisWeight dx = c_sci_axis[gi][lx], dy = c_sci_axis[gi][ly], dz = c_sci_axis[gi][lz];
        auto tri = [&](uint64_t data, float sc) {
            auto S = [&](int cx, int cy, int cz) { return bfp_sample(rd, data, res, bits, sc, (cz * res + cy) * res + cx); };
            const float d00 = lerp_ref(S(dx.i0, dy.i0, dz.i0), S(dx.i1, dy.i0, dz.i0), dx.t, dx.omt);
            const float d01 = lerp_ref(S(dx.i0, dy.i0, dz.i1), S(dx.i1, dy.i0, dz.i1), dx.t, dx.omt);
            const float d10 = lerp_ref(S(dx.i0, dy.i1, dz.i0), S(dx.i1, dy.i1, dz.i0), dx.t, dx.omt);
            const float d11 = lerp_ref(S(dx.i0, dy.i1, dz.i1), S(dx.i1, dy.i1, dz.i1), dx.t, dx.omt);
            return lerp_ref(lerp_ref(d00, d10, dy.t, dy.omt), lerp_ref(d01, d11, dy.t, dy.omt), dz.t, dz.omt);
        };
        if (sub == 1u) {
            const int tkeep = (int)((hdr >> 15) & 0xFu) + 1;
            if (bits > 0) {
                const int bbytes = (per * bits + 7) / 8;
                const uint64_t data = scales + (uint64_t)(tkeep * 2);
                for (int k = 0; k < tkeep; ++k) {
                    const float sc = half_bits_to_float(rd.u16(scales + (uint64_t)(k * 2)));
                    r = __fadd_rn(r, __fmul_rn(tri(data + (uint64_t)(k * bbytes), sc), __ldg(brow + k)));
                }
            }
        } else {
            const int fbytes = (per * bits + 7) / 8;
            const float sc = half_bits_to_float(rd.u16(scales + t * 2u));
            r = tri(scales + (uint64_t)a.g.frames * 2u + (uint64_t)t * fbytes, sc);
        }
    }
    *oob_out = rd.oob;
    return __fadd_rn(coarse, r);
}

// The residual of voxel li at frame t in a SparseEvents leaf (section at byte sb, inside the payload)
// with kFlagSorted, by eight lanes (`sub` = 0..7 of lane mask `mask`).  The reference's binary search finds a key exactly
// when it is present there, so each lane looks at one word of two keys: a bin holds about ten
// events, one step instead of the search's four dependent ones.
__device__ __forceinline__ float sci_event(const uint32_t* __restrict__ lw, uint32_t sb, uint32_t hdr, uint32_t cap,
                                           uint32_t li, uint32_t t, uint32_t sub, uint32_t mask)
{
    const uint32_t count = (hdr >> 16) & 0x0FFFu;
    const uint32_t fpb = ((hdr >> 10) & 0xFu) + 1u;
    // min(15, t / fpb): (t + 1/2) / fpb is at least 1/32 from a whole number, far above the quotient's error
    const uint32_t bin = t >= 15u * fpb ? 15u : (uint32_t)__fdividef((float)t + 0.5f, (float)fpb);
    const uint32_t sw = sb >> 2;
    const float es = __uint_as_float(__ldg(lw + sw));
    const uint32_t mw = __ldg(lw + sw + 1u + (li >> 5));
    const uint32_t bw = sw + 17u + (bin >> 1);
    const uint32_t b0 = __ldg(lw + bw), b1 = __ldg(lw + bw + 1u);
    if (!(es > 0.0f) || ((mw >> (li & 31u)) & 1u) == 0u) return 0.0f;
    const uint32_t se = bin & 1u ? __funnelshift_r(b0, b1, 16) : b0;
    uint32_t lo = se & 0xFFFFu, hi = bin < 15u ? se >> 16 : count;
    const uint32_t target = ((((t - bin * fpb) & 0xFFu) << 9) | li) & 0xFFFFu;
    const uint32_t kw = sw + 25u, rw = kw + cap / 2u;
    while (hi > lo + 32u) {   // keep the target's place in [lo, hi)
        const uint32_t mid = (lo + hi) >> 1;
        const uint32_t key = (__ldg(lw + kw + (mid >> 1)) >> ((mid & 1u) * 16u)) & 0xFFFFu;
        if (key <= target) lo = mid;
        else hi = mid;
    }
    uint32_t found = 0u;   // the event's index + 1
    for (uint32_t i = (lo & ~1u) + 2u * sub; i < hi; i += 16u) {
        const uint32_t keys = __ldg(lw + kw + (i >> 1));
        if (i >= lo && (keys & 0xFFFFu) == target) found = i + 1u;
        if (i + 1u < hi && (keys >> 16) == target) found = i + 2u;
    }
    found = __reduce_or_sync(mask, found);   // at most one lane found it
    if (found == 0u) return 0.0f;
    const uint32_t i = found - 1u;
    int q = (int)((__ldg(lw + rw + (i >> 3)) >> ((i & 7u) * 4u)) & 0xFu);
    if (q & 8) q -= 16;
    return __fmul_rn((float)q, es);
}

// Axis weights of the common grids, [render 4^3, render 6^3, scientific 4^3, 3^3][position] = {t, i0}
// (i1 is i0 + 1); a position inside a cropped leaf has the weights it has in a whole one.
struct CellAxis {
    uint32_t i0;
    float t, omt;
};

// The same by one thread with the reference's search: keys in any order.  Also the events of a batch with many
// of them: eight lanes to an event take a batch's events in turn, four at a time.
__device__ __noinline__ float sci_event_alone(const DeviceAsset& a, LeafEntry e, uint32_t li, uint32_t t, bool* oob)
{
    SciReader rd{a.payload, a.g.payload_words, false};
    const SparseLeaf sp = sparse_leaf(rd, 4ull * e.word_off, e.header, (int)((e.header >> 2) & 0x3Fu) + 1);
    const float r = sp.es > 0.0f ? sparse_at(rd, sp, li, t) : 0.0f;
    *oob = rd.oob;
    return r;
}

// sci_control_fast for a record of any length.
__device__ __noinline__ float sci_control_long(const uint32_t* __restrict__ w, uint32_t cb, uint32_t keep,
                                               const float* __restrict__ brow, const float* __restrict__ scales)
{
    const uint32_t* p = w + (cb >> 2);
    const uint32_t sh = (cb & 3u) * 8u;
    uint32_t x = __ldg(p), y = __ldg(p + 1);
    double sum = (double)half_to_float_exact(__funnelshift_r(x, y, sh) & 0xFFFFu) * (double)__ldg(brow);
    for (uint32_t k0 = 0;; k0 += 4u) {   // record bytes k0 .. k0 + 3: the coefficients from k0 - 1 on
        const uint32_t r = __funnelshift_r(x, y, sh);
#pragma unroll
        for (uint32_t i = 0; i < 4u; ++i) {
            const uint32_t k = k0 + i - 1u;
            if (k0 + i >= 2u && k < keep)
                sum = __fma_rn((double)__fmul_rn(byte_to_float(r, i), __ldg(scales + k - 1u)), (double)__ldg(brow + k), sum);
        }
        if (k0 + 3u >= keep) return (float)sum;
        x = y;
        y = __ldg(p + 2u + (k0 >> 2));
    }
}

// The temporal-basis residual of a query by eight lanes (`sub` = its corner of the cell, lane mask `mask`): of
// each basis grid the lanes' samples, their trilinear by three exchanges, times the frame's basis value
// (render/src/scientific_decode.cpp:177-233).  Codes of R^3 grids from byte `sb` of the leaf on.
__device__ __noinline__ float sci_basis_residual(const uint32_t* __restrict__ lw, uint32_t sb, uint32_t hdr, uint32_t ci,
                                                 CellAxis ax, CellAxis ay, CellAxis az,
                                                 const float* __restrict__ brow, uint32_t sub, uint32_t mask)
{
    const uint32_t per = (hdr & 3u) == 2u ? 27u : 64u, bits = (hdr >> 8) & 0xFu, tkeep = ((hdr >> 15) & 0xFu) + 1u;
    const uint32_t bo = ci * bits, bytes = (per * bits + 7u) / 8u;
    float r = 0.0f;
    for (uint32_t k = 0; bits != 0u && k < tkeep; ++k) {
        const uint32_t code = ((pay_u32(lw, sb + 2u * tkeep + k * bytes + (bo >> 3)) & 0xFFFFu) >> (bo & 7u)) & ((1u << bits) - 1u);
        float v = decode_bfp(code, half_to_float_exact(pay_u32(lw, sb + 2u * k) & 0xFFFFu), (int)bits);
        auto along = [&](const CellAxis& w, uint32_t bit) {
            const float o = __shfl_xor_sync(mask, v, (int)bit);
            v = lerp_ref(sub & bit ? o : v, sub & bit ? v : o, w.t, w.omt);
        };
        along(ax, 1u);
        along(ay, 2u);
        along(az, 4u);
        r = __fadd_rn(r, __fmul_rn(v, __ldg(brow + k)));
    }
    return r;
}

// What the corner step needs of a query.  Render leaves: `grids` = coarse corner 0 | R << 9 | fine
// corner 0 << 12 | R << 21 | bin << 24 | sorted << 27 | FP32 codecs << 28, 29; `kf`, the fine
// stream's byte offset in `at`, the frame in `t`.  Scientific leaves: corner 0 |
// residual corner 0 << 12 | residual R << 21 | keep << 24, the header in `kf`, the residual grid's (or the event or
// temporal-basis section's) byte offset in `at`, the frame in `t`.
struct __align__(16) QueryCell {
    const uint32_t* lw;    // the leaf block
    const float* brow;     // scientific: basis row of the frame
    const float* scales;   // scientific: AC scales
    uint32_t grids, kf, at, t, voxel, scale;
};

struct QueryShared {
    QueryCell cell[kPqBatch];
    float val[kPqBatch * 17];   // per query: 8 corners, 8 of the second grid, the event or temporal-basis residual
    uint16_t list[2 * kPqBatch];
    uint8_t second[kPqBatch], residuals[kPqBatch];
};

__device__ __forceinline__ CellAxis cell_axis(const float2* table, int grid, uint32_t res, uint32_t pos)
{
    float2 w;
    if (grid >= 0) {
        w = table[grid * 8 + pos];
    } else {
        const AxisWeight aw = g_axis[axis_index((int)res, 8, (int)pos)];
        w = make_float2(aw.t, __uint_as_float((uint32_t)aw.i0));
    }
    return CellAxis{__float_as_uint(w.y), w.x, __fsub_rn(1.0f, w.x)};
}
__device__ __forceinline__ int render_grid(uint32_t res) { return res == 4u ? 0 : res == 6u ? 1 : -1; }

// Corner 0 of the cell of (lx, ly, lz), and its trilinear from the eight corner values v.
__device__ __forceinline__ uint32_t cell_corner(const float2* table, int grid, uint32_t res, uint32_t lx, uint32_t ly,
                                                uint32_t lz)
{
    if (res < 2u) return 0u;
    return (cell_axis(table, grid, res, lz).i0 * res + cell_axis(table, grid, res, ly).i0) * res +
           cell_axis(table, grid, res, lx).i0;
}
__device__ __forceinline__ float cell_value(const float2* table, int grid, uint32_t res, uint32_t lx, uint32_t ly,
                                            uint32_t lz, const float* v)
{
    if (res < 2u) return res == 1u ? v[0] : 0.0f;
    const CellAxis ax = cell_axis(table, grid, res, lx), ay = cell_axis(table, grid, res, ly),
                   az = cell_axis(table, grid, res, lz);
    const float c00 = lerp_ref(v[0], v[1], ax.t, ax.omt), c10 = lerp_ref(v[2], v[3], ax.t, ax.omt);
    const float c01 = lerp_ref(v[4], v[5], ax.t, ax.omt), c11 = lerp_ref(v[6], v[7], ax.t, ax.omt);
    return lerp_ref(lerp_ref(c00, c10, ay.t, ay.omt), lerp_ref(c01, c11, ay.t, ay.omt), az.t, az.omt);
}
// Corner k of a cell: its offset from corner 0 (a grid of one control has one corner).
__device__ __forceinline__ uint32_t corner_step(uint32_t k, uint32_t res)
{
    return res < 2u ? 0u : (k & 1u) + ((k >> 1) & 1u) * res + (k >> 2) * res * res;
}

// The queries of a launch: of render files, of scientific files, or of both (a serving step).  A kernel for one
// kind has no registers spilled for the other: against the kernel for both, 1,000,000 queries of the plume 57 -> 50
// us, of the field 86 -> 83, a thousand 6.8 -> 6.2.
enum : int { kRenderOnly, kSciOnly, kBoth };

// Up to 32 queries, one per lane (`on`): value and where to put it are the lane's own.
template <class Resolve>
__device__ __forceinline__ void query_batch(QueryShared& sh, const float2* table, uint32_t batch, bool on, uint64_t i,
                                            const uint4* __restrict__ q, const Resolve& resolve)
{
    const uint32_t lane = threadIdx.x & 31u, sub = lane & 7u, group = lane >> 3, gmask = 0xFFu << (8u * group);
    enum : uint32_t { kNone, kRender, kSci, kSciGeneral };
    uint32_t kind = kNone, leaf = 0, place = 0;   // place: lx | ly << 3 | lz << 6
    bool second = false, event = false, alone = false, tbasis = false;
    const auto r = resolve.request(on ? i : 0);
    const DeviceAsset& a = resolve.asset(r);
    constexpr bool kRt = Resolve::kFamily != kSciOnly, kSc = Resolve::kFamily != kRenderOnly;   // kinds that occur
    const bool sci = !kRt || (kSc && a.g.profile == 2u);
    // 1. the lane's query
    if (on) {
        const uint4 qq = q[i];
        uint32_t lx = 0, ly = 0, lz = 0;
        // leaf lookup as render/src/vbt_file.cpp:250-262 leafIndexForVoxel (clamped leaf coordinates)
        const uint32_t bx = min(a.g.lcx - 1u, qq.x >> 3), by = min(a.g.lcy - 1u, qq.y >> 3),
                       bz = min(a.g.lcz - 1u, qq.z >> 3);
        leaf = (bz * a.g.lcy + by) * a.g.lcx + bx;
        const uint32_t t = qq.w;
        const LeafEntry e = a.entries[leaf];
        const uint32_t st = entry_status(e);
        QueryCell c{};
        c.lw = a.payload + e.word_off;
        if (st != kOk) {
            record_error(resolve.err(r), leaf, st);
        } else if (sci) {
            lx = qq.x & 7u, ly = qq.y & 7u, lz = qq.z & 7u;
            if (t >= a.g.frames) {   // the reference indexes its per-frame tables out of range here
                record_error(resolve.err(r), leaf, kErrDecodeOob);
            } else {
                // bytes of the payload from the leaf on: a section inside them is read unchecked
                const uint64_t room = 4ull * (a.g.payload_words - e.word_off);
                const uint32_t lim = room < 0xFFFFFFFFull ? (uint32_t)room : 0xFFFFFFFFu;
                const uint32_t hdr = e.header, mode = hdr & 3u, keep = ((hdr >> 2) & 0x3Fu) + 1u;
                const uint32_t sb = 4u + 64u * (keep + 1u);
                bool plain = sb + 4u <= lim;
                c.brow = a.basis + (uint64_t)t * 64u;
                c.scales = a.scales;
                c.grids = cell_corner(table, 2, 4u, lx, ly, lz) | (keep << 24);
                c.kf = hdr;
                c.t = t;
                c.voxel = (lz * 8u + ly) * 8u + lx;
                if (mode == 1u && ((hdr >> 16) & 0x0FFFu) != 0u) {
                    const uint32_t tier = (hdr >> 8) & 3u;
                    const uint32_t cap = tier == 0u ? 64u : tier == 1u ? 256u : tier == 2u ? 768u : 1024u;
                    plain = plain && sb + 100u + 2u * cap + cap / 2u <= lim;
                    alone = (e.info & kFlagSorted) == 0u;
                    c.at = sb;
                    c.scale = cap;
                    event = plain && ((__ldg(c.lw + (sb >> 2) + 1u + (c.voxel >> 5)) >> (c.voxel & 31u)) & 1u) != 0u;
                } else if (mode >= 2u) {
                    const uint32_t res = mode == 2u ? 3u : 4u, bits = (hdr >> 8) & 0xFu;
                    const uint32_t bytes = (res * res * res * bits + 7u) / 8u;
                    tbasis = ((hdr >> 12) & 7u) == 1u;
                    const uint32_t grids = tbasis ? ((hdr >> 15) & 0xFu) + 1u : a.g.frames;
                    const uint64_t data = (uint64_t)sb + 2ull * grids + (tbasis ? 0ull : (uint64_t)t * bytes);
                    plain = plain && data + (tbasis ? (uint64_t)grids : 1ull) * bytes <= lim;
                    c.at = tbasis ? sb : (uint32_t)data;
                    c.scale = sb + 2u * t;
                    c.grids |= (cell_corner(table, mode == 2u ? 3 : 2, res, lx, ly, lz) << 12) | (res << 21);
                    second = plain && !tbasis;
                    tbasis = plain && tbasis;
                }
                kind = plain ? kSci : kSciGeneral;
            }
        } else if ((e.header & 3u) != kModeEmpty) {
            lx = qq.x - 8u * bx, ly = qq.y - 8u * by, lz = qq.z - 8u * bz;
            // outside the volume: no such voxel in any frame
            if (lx < 8u && ly < 8u && lz < 8u && qq.x < a.g.width && qq.y < a.g.height && qq.z < a.g.depth) {
                kind = kRender;
                const int frame = clamp_frame((int)t, (int)a.g.frames);
                const uint32_t cres = (e.header >> 6) & 7u, fres = (e.header >> 9) & 7u;
                second = (e.info & kFlagFine) != 0u;
                c.grids = cell_corner(table, render_grid(cres), cres, lx, ly, lz) | (cres << 9) | (fres << 21) |
                          (time_bin(frame, 8u, (int)a.g.frames) << 24) | (e.info & kFlagSorted ? 1u << 27 : 0u) |
                          (((e.header >> 2) & 3u) == 1u ? 1u << 28 : 0u) | (((e.header >> 4) & 3u) == 1u ? 1u << 29 : 0u);
                if (second) c.grids |= cell_corner(table, render_grid(fres), fres, lx, ly, lz) << 12;
                c.kf = e.kf;
                c.at = 8u + e.coarse_bytes;
                c.t = (uint32_t)frame;
            }
        }
        place = lx | (ly << 3) | (lz << 6);
        sh.cell[lane] = c;
    }
    const uint32_t m1 = __ballot_sync(0xFFFFFFFFu, kind == kRender || kind == kSci);
    const uint32_t m2 = __ballot_sync(0xFFFFFFFFu, second);
    // a batch's events: eight lanes to each, or, when they are many, each lane its own
    const uint32_t me = __ballot_sync(0xFFFFFFFFu, event);
    alone = alone || __popc(me) > kPqEvents;
    const bool residual = tbasis || (event && !alone);
    const uint32_t m3 = __ballot_sync(0xFFFFFFFFu, residual);
    const uint32_t below = (1u << lane) - 1u;
    const uint32_t msci = !kRt ? 0xFFFFFFFFu : !kSc ? 0u : __ballot_sync(0xFFFFFFFFu, on && sci);
    if (second) sh.second[__popc(m2 & below)] = (uint8_t)lane;
    if (residual) sh.residuals[__popc(m3 & below)] = (uint8_t)lane;
    __syncwarp();
    // 2. the corners: four queries at a time
    for (uint32_t s0 = 0; s0 < batch; s0 += 4u) {
        const uint32_t s = s0 + group;
        if (s >= batch || ((m1 >> s) & 1u) == 0u) continue;
        const QueryCell& c = sh.cell[s];
        const uint32_t g = c.grids;
        float v = 0.0f;
        if ((msci >> s) & 1u) {
            const uint32_t keep = g >> 24, cb = 4u + ((g & 0x1FFu) + corner_step(sub, 4u)) * (keep + 1u);
            v = keep <= 7u ? sci_control_fast(c.lw, cb, (int)keep, c.brow, c.scales)
                           : sci_control_long(c.lw, cb, keep, c.brow, c.scales);
        } else {
            const uint32_t R = (g >> 9) & 7u;
            if (R != 0u)
                v = control_at(LeafStream{c.lw, 8u, R * R * R, 8u, c.kf & 0xFFFFu}, (g >> 28) & 1u,
                               (g & 0x1FFu) + corner_step(sub, R), (int)c.t, (g >> 24) & 7u, ((g >> 27) & 1u) != 0u);
        }
        sh.val[s * 17u + sub] = v;
    }
    const uint32_t n2 = (uint32_t)__popc(m2), n3 = kSc ? (uint32_t)__popc(m3) : 0u;
    for (uint32_t k = group; k < n2; k += 4u) {
        const uint32_t s = sh.second[k];
        const QueryCell& c = sh.cell[s];
        const uint32_t g = c.grids, R = (g >> 21) & 7u, ci = ((g >> 12) & 0x1FFu) + corner_step(sub, R);
        float v = 0.0f;
        if ((msci >> s) & 1u) {   // bfp_sample at bit ci * bits of the frame's grid
            const uint32_t bits = (c.kf >> 8) & 0xFu, bo = ci * bits;
            const uint32_t code = ((pay_u32(c.lw, c.at + (bo >> 3)) & 0xFFFFu) >> (bo & 7u)) & ((1u << bits) - 1u);
            v = decode_bfp(code, half_to_float_exact(pay_u32(c.lw, c.scale) & 0xFFFFu), (int)bits);
        } else if (R != 0u) {
            v = control_at(LeafStream{c.lw, c.at, R * R * R, 8u, c.kf >> 16}, (g >> 29) & 1u, ci, (int)c.t,
                           (g >> 24) & 7u, ((g >> 27) & 1u) != 0u);
        }
        sh.val[s * 17u + 8u + sub] = v;
    }
    for (uint32_t k = group; k < n3; k += 4u) {
        const uint32_t s = sh.residuals[k];
        const QueryCell& c = sh.cell[s];
        float v;
        if ((c.kf & 3u) == 1u) {
            v = sci_event(c.lw, c.at, c.kf, c.scale, c.voxel, c.t, sub, gmask);
        } else {
            const uint32_t R = (c.grids >> 21) & 7u;
            const int grid = R == 3u ? 3 : 2;
            v = sci_basis_residual(c.lw, c.at, c.kf, ((c.grids >> 12) & 0x1FFu) + corner_step(sub, R),
                                   cell_axis(table, grid, R, c.voxel & 7u), cell_axis(table, grid, R, (c.voxel >> 3) & 7u),
                                   cell_axis(table, grid, R, c.voxel >> 6), c.brow, sub, gmask);
        }
        if (sub == 0u) sh.val[s * 17u + 16u] = v;
    }
    __syncwarp();
    // 3. the lane's own value
    if (on) {
        const float* v = sh.val + lane * 17u;
        const uint32_t lx = place & 7u, ly = (place >> 3) & 7u, lz = place >> 6;
        float out = 0.0f;
        if (kRt && kind == kRender) {
            const LeafEntry e = a.entries[leaf];   // again, so that it holds no registers meanwhile
            const uint32_t cres = (e.header >> 6) & 7u, fres = (e.header >> 9) & 7u;
            out = cell_value(table, render_grid(cres), cres, lx, ly, lz, v);
            bool in_occ = false;
            uint64_t mask = 0;
            const uint32_t* lw = a.payload + e.word_off;
            const uint32_t ow = (8u + e.coarse_bytes) >> 2, bit = ly * 8u + lx;   // occupancy: mask[lz], then prefix[lz]
            if (e.info & kFlagOccClamp) {
                mask = ((uint64_t)__ldg(lw + ow + 2u * lz + 1u) << 32) | __ldg(lw + ow + 2u * lz);
                in_occ = (mask >> bit) & 1ull;
            }
            if (second) {
                out = __fadd_rn(out, cell_value(table, render_grid(fres), fres, lx, ly, lz, v + 8));
            } else if ((e.info & kFlagShell) && in_occ) {
                const uint32_t pref = (__ldg(lw + ow + 16u + (lz >> 1)) >> ((lz & 1u) * 16u)) & 0xFFFFu;
                const uint32_t di = (pref + __popcll(mask & ((1ull << bit) - 1ull))) & 0xFFFFu;
                const int frame = (int)sh.cell[lane].t;
                out = __fadd_rn(out, control_at(LeafStream{lw, e.shell_off, entry_shell_active(e), 4u, e.kf >> 16},
                                                (e.header >> 4) & 3u, di, frame, time_bin(frame, 4u, (int)a.g.frames),
                                                (e.info & kFlagSorted) != 0u));
            }
            if ((e.info & kFlagOccClamp) && !in_occ && out < 0.0f) out = 0.0f;
        } else if (kSc && kind == kSci) {
            const float coarse = cell_value(table, 2, 4u, lx, ly, lz, v);
            float res = residual ? v[16] : 0.0f;
            if (event && alone) {
                bool oob = false;
                res = sci_event_alone(a, a.entries[leaf], (lz * 8u + ly) * 8u + lx, sh.cell[lane].t, &oob);
                if (oob) record_error(resolve.err(r), leaf, kErrDecodeOob);
            }
            if (second) res = (sh.cell[lane].kf & 3u) == 2u ? cell_value(table, 3, 3u, lx, ly, lz, v + 8)
                                                    : cell_value(table, 2, 4u, lx, ly, lz, v + 8);
            out = __fadd_rn(coarse, res);
        } else if (kSc && kind == kSciGeneral) {
            bool oob = false;
            out = sci_point_general(a, a.entries[leaf], lx, ly, lz, sh.cell[lane].t, &oob);
            if (oob) record_error(resolve.err(r), leaf, kErrDecodeOob);
        }
        resolve.put(r, i, out);
    }
    __syncwarp();
}

// True when a query decodes to 0 without any decoding and without recording an error: a
// render-temporal query in an EMPTY leaf or outside the volume.
__device__ __forceinline__ bool point_trivial(const DeviceAsset& a, uint4 qq)
{
    if (a.g.profile == 2u) return false;
    const uint32_t bx = min(a.g.lcx - 1u, qq.x >> 3), by = min(a.g.lcy - 1u, qq.y >> 3), bz = min(a.g.lcz - 1u, qq.z >> 3);
    const uint32_t leaf = (bz * a.g.lcy + by) * a.g.lcx + bx;
    const uint32_t info = __ldg(&a.entries[leaf].info), header = __ldg(&a.entries[leaf].header);
    if (((info >> 16) & 0xFFu) != kOk) return false;   // query_batch records the status
    return (header & 3u) == kModeEmpty || qq.x >= a.g.width || qq.y >= a.g.height || qq.z >= a.g.depth;
}

// A warp's queries [base, base + chunk).  In a chunk of a sparse volume the trivial queries are
// answered on the way and the others queued until they fill a batch -- most random queries there
// are trivial; chunks of other volumes go through as they are.
template <class Resolve>
__device__ __forceinline__ void query_chunk(uint64_t n, uint32_t chunk, const uint4* __restrict__ q, const Resolve& resolve)
{
    __shared__ QueryShared s_all[kPqWarps];
    __shared__ float2 s_axis[32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (threadIdx.x < 32u) {
        const int g = (int)(lane >> 3), p = (int)(lane & 7u);
        const AxisWeight w = g < 2 ? g_axis[axis_index(g == 0 ? 4 : 6, 8, p)] : g_sci_axis[g - 2][p];
        s_axis[lane] = make_float2(w.t, __uint_as_float((uint32_t)w.i0));
    }
    __syncthreads();
    QueryShared& sh = s_all[warp];
    const uint64_t base = ((uint64_t)blockIdx.x * kPqWarps + warp) * chunk;
    if (base >= n) return;
    const uint32_t cnt = n - base < (uint64_t)chunk ? (uint32_t)(n - base) : chunk;
    if (!resolve.sparse(base)) {
        for (uint32_t j0 = 0; j0 < cnt; j0 += kPqBatch) {
            const uint32_t batch = cnt - j0 < (uint32_t)kPqBatch ? cnt - j0 : (uint32_t)kPqBatch;
            query_batch(sh, s_axis, batch, lane < batch, base + j0 + lane, q, resolve);
        }
        return;
    }
    uint32_t queued = 0, j0 = 0;
    while (j0 < cnt || queued != 0u) {
        while (queued < (uint32_t)kPqBatch && j0 < cnt) {
            const uint32_t j = j0 + lane;
            bool need = false;
            if (j < cnt) {
                const auto r = resolve.request(base + j);
                need = !point_trivial(resolve.asset(r), q[base + j]);
                if (!need) resolve.put(r, base + j, 0.0f);
            }
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, need);
            if (need) sh.list[queued + (uint32_t)__popc(m & ((1u << lane) - 1u))] = (uint16_t)j;
            queued += (uint32_t)__popc(m);
            j0 += 32u;
        }
        __syncwarp();
        if (queued == 0u) break;
        const uint32_t batch = queued < (uint32_t)kPqBatch ? queued : (uint32_t)kPqBatch;
        query_batch(sh, s_axis, batch, lane < batch, base + (lane < batch ? sh.list[lane] : 0u), q, resolve);
        queued -= batch;
        const uint16_t rest = lane < queued ? sh.list[kPqBatch + lane] : (uint16_t)0;
        __syncwarp();
        if (lane < queued) sh.list[lane] = rest;
        __syncwarp();
    }
}

// Queries per warp: at most `top`, and few enough that every SM has 16 warps' worth (a small batch
// is bound by its longest chain, so it spreads as far as four queries per warp, one corner step).
static uint32_t query_chunk_size(uint64_t n, uint32_t top)
{
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    }
    uint32_t chunk = top;
    while (chunk > 4u && (n + chunk - 1) / chunk < 16ull * (uint64_t)(sms > 0 ? sms : 1)) chunk >>= 1;
    return chunk;
}
// A batch per warp where every query is decoded (more only lengthens the last wave); eight where most
// are answered on the way, so that the queue fills whole batches (128 queries: plume 70 us).
constexpr uint32_t kPqDenseChunk = 32, kPqSparseChunk = 256;

static unsigned query_blocks(uint64_t n, uint32_t chunk)
{
    const uint64_t per = (uint64_t)chunk * kPqWarps;
    return (unsigned)((n + per - 1) / per);
}

template <int FAMILY>
struct OneAssetQueries {
    static constexpr int kFamily = FAMILY;
    const DeviceAsset& a;
    float* __restrict__ out;
    __device__ __forceinline__ bool sparse(uint64_t) const { return a.g.sparse != 0u; }
    __device__ __forceinline__ int request(uint64_t) const { return 0; }
    __device__ __forceinline__ const DeviceAsset& asset(int) const { return a; }
    __device__ __forceinline__ unsigned long long* err(int) const { return a.err; }
    __device__ __forceinline__ void put(int, uint64_t i, float v) const { out[i] = v; }
};

template <int FAMILY>
__global__ void __launch_bounds__(kPqThreads, kPqCtas) query_points_kernel(const __grid_constant__ DeviceAsset a,
                                                                  const uint4* __restrict__ q, uint64_t n,
                                                                  uint32_t chunk, float* __restrict__ out)
{
    query_chunk(n, chunk, q, OneAssetQueries<FAMILY>{a, out});
}

// Point queries of several requests over several resident assets in one launch.  The segment
// table holds starts[0..k] (each request's first query; starts[k] = n), asset[k] (request r reads
// assets[asset[r]]) and, 8-byte aligned after them, outs[k] (request r's result array).  Request
// r's decode errors go to errs[r].
struct BatchQueries {
    static constexpr int kFamily = kBoth;
    const DeviceAsset* __restrict__ assets;
    const uint32_t* __restrict__ seg;
    uint32_t k;
    unsigned long long* errs;
    __device__ __forceinline__ int request(uint64_t i) const
    {
        int lo = 0, hi = (int)k - 1;
        while (lo < hi) {   // the last request whose first query is at or before i
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(seg + mid) <= (uint32_t)i) lo = mid;
            else hi = mid - 1;
        }
        return lo;
    }
    __device__ __forceinline__ const DeviceAsset& asset(int r) const { return assets[__ldg(seg + k + 1 + r)]; }
    __device__ __forceinline__ unsigned long long* err(int r) const { return errs + r; }
    // the chunk starting at query i takes the compacting path when its first query's asset is sparse
    __device__ __forceinline__ bool sparse(uint64_t i) const { return asset(request(i)).g.sparse != 0u; }
    __device__ __forceinline__ void put(int r, uint64_t i, float v) const
    {
        const unsigned long long* outs = reinterpret_cast<const unsigned long long*>(seg + ((2u * k + 2u) & ~1u));
        reinterpret_cast<float*>(__ldg(outs + r))[i - __ldg(seg + r)] = v;
    }
};

__global__ void __launch_bounds__(kPqThreads, kPqCtas) query_points_batch_kernel(const DeviceAsset* __restrict__ assets,
                                                                        const uint32_t* __restrict__ seg, uint32_t k,
                                                                        const uint4* __restrict__ q, uint64_t n,
                                                                        uint32_t chunk, unsigned long long* errs)
{
    query_chunk(n, chunk, q, BatchQueries{assets, seg, k, errs});
}

void launch_query_points_batch(const DeviceAsset* assets, const uint32_t* seg, uint32_t k, const uint4* q, uint64_t n,
                               unsigned long long* errs, int sparse, cudaStream_t s)
{
    if (n == 0 || k == 0) return;
    const uint32_t chunk = query_chunk_size(n, sparse == 2 ? kPqSparseChunk : sparse ? 2u * kPqDenseChunk : kPqDenseChunk);
    query_points_batch_kernel<<<query_blocks(n, chunk), kPqThreads, 0, s>>>(assets, seg, k, q, n, chunk, errs);
}

void launch_query_points(const DeviceAsset& a, const uint32_t* q, uint64_t n, float* out, bool sparse, cudaStream_t s)
{
    if (n == 0) return;
    const uint32_t chunk = query_chunk_size(n, sparse ? kPqSparseChunk : kPqDenseChunk);
    const auto kernel = a.g.profile == 2u ? query_points_kernel<kSciOnly> : query_points_kernel<kRenderOnly>;
    kernel<<<query_blocks(n, chunk), kPqThreads, 0, s>>>(a, reinterpret_cast<const uint4*>(q), n, chunk, out);
}

}  // namespace vbtb
