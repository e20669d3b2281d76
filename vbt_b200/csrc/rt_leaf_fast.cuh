// rt_leaf_fast.cuh -- the render decode kernel's specialised paths for the leaf shapes that make up
// nearly every render-temporal asset: GRID4 (a 4^3 coarse grid), FINE6 (4^3 coarse + 6^3 fine) and
// Mode2 (4^3 coarse + shell), FP16 key frames that strictly increase, over a timeline (frames stepping
// by 0 or 1).
// Included by rt_kernel_leaf.cuh; the general leaf_decode there covers every other leaf.
//
// Same arithmetic as the general path, operation for operation (so the same bits):
//  - controls: the streaming cursor of rt_staged.cuh (m_control_stream), but each cursor is set
//    up once per launch and then carried in registers across the frame batches.  A unit is one
//    control and one contiguous part of the launch's frames: GRID4 splits each of its 64 controls
//    into 4 parts (256 units), FINE6 keeps its 280 controls whole (one unit per thread of the
//    288).  A batch takes the next frames of every part, as many as the control buffer holds.
//    Key reads are byte offsets into the staged leaf (32-bit arithmetic), and the FP16 value is
//    the hardware conversion, exact for every value but NaN -- such leaves (kFlagHalfPlain
//    unset) take the general path, which keeps the reference's NaN payloads.  Key spans are
//    below 256 frames (u8 frames), so RN(1/span) always comes from the table.
//  - voxels: the separable trilinear with the grid resolution a compile-time constant, a lane's y rows
//    in registers for its z lerps, weights as 16-byte rows per lane: about half the shared-memory
//    instructions of y rows passed through shared memory (waits on it were the first stall), 32
//    frames of a 128 x 128 x 192 fire 294 -> 269 us, dense 372 -> 323, of a 256^3 plume 221 -> 203.
#pragma once

namespace vbtb {

// A cursor over one control's keys: k = first key with frame > t (0..kc), [fp, fn) the key
// interval around t with values vp, vn, the key after it prefetched (fnn, vnn), and per interval
// bf = span, y = RN(1/span), d = vn - vp.
struct KeyCursor {
    uint32_t kb;   // stage byte offset of the control's first key
    int k, kc;
    int fp, fn, fnn;
    float vp, vn, vnn;
    float bf, y, d;
};

// Key i of an FP16 stream at stage byte offset `off`: frame byte and binary16 value (hardware
// conversion; the leaf holds no NaN key).  The stage is padded, so the second word always exists.
__device__ __forceinline__ void fast_key(const uint8_t* __restrict__ st, uint32_t off, int& frame, float& value)
{
    const uint32_t* w = reinterpret_cast<const uint32_t*>(st + (off & ~3u));
    const uint32_t k = __funnelshift_r(w[0], w[1], (off & 3u) * 8u);
    frame = (int)(k & 0xFFu);
    value = __half2float(__ushort_as_half((unsigned short)(k >> 8)));
}

__device__ __forceinline__ void fast_interval(KeyCursor& cu, const float* __restrict__ rcp)
{
    const int b = cu.fn - cu.fp;
    cu.bf = (float)b;
    cu.y = rcp[b & 255];   // outside 0 < k < kc the interval is never selected
    cu.d = __fsub_rn(cu.vn, cu.vp);
}

// Set the cursor of control ci of the stream at stage offset sbase (C controls, `bins` = 8 or 4 time
// bins, kf keys in its pool) for first frame t0 in time bin bin0: the start of m_control_stream.
__device__ __forceinline__ void fast_cursor_init(const uint8_t* __restrict__ st, uint32_t sbase, uint32_t C, uint32_t bins,
                                                 uint32_t ci, uint32_t kf, int t0, uint32_t bin0,
                                                 const float* __restrict__ rcp, KeyCursor& cu)
{
    cu.k = 0;
    cu.kc = 0;
    cu.fp = cu.fn = cu.fnn = 0;
    cu.vp = cu.vn = cu.vnn = 0.0f;
    cu.bf = cu.y = 1.0f;
    cu.d = 0.0f;
    cu.kb = 0u;
    const uint32_t desc = *reinterpret_cast<const uint32_t*>(st + sbase + 4u * ci);
    const uint32_t kc = (desc >> 16) & 0xFFu, ks = desc & 0xFFFFu;
    if (kc == 0u || ks + kc > kf) return;   // decodes to 0 (see decode_control, rt_search.cuh)
    cu.kc = (int)kc;
    cu.kb = sbase + (4u + bins) * C + 3u * ks;   // descriptors (4 C) + bin rows (bins C, 4-aligned)
    const uint32_t hb = st[sbase + 4u * C + bins * ci + bin0];
    uint32_t k = hb < kc - 1u ? hb : kc - 1u;
    if ((int)st[cu.kb + 3u * k] > t0) {
        uint32_t lo = 0, hi = k;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if ((int)st[cu.kb + 3u * mid] > t0) hi = mid;
            else lo = mid + 1u;
        }
        k = lo;
    } else {
        ++k;
        while (k < kc && (int)st[cu.kb + 3u * k] <= t0) ++k;
    }
    cu.k = (int)k;
    if (k > 0u) fast_key(st, cu.kb + 3u * (k - 1u), cu.fp, cu.vp);
    if (k < kc) fast_key(st, cu.kb + 3u * k, cu.fn, cu.vn);
    if (k + 1u < kc) fast_key(st, cu.kb + 3u * (k + 1u), cu.fnn, cu.vnn);
    fast_interval(cu, rcp);
}

// The control's value at frame t (t >= the previous call's t, by at most one frame).
__device__ __forceinline__ float fast_cursor_step(KeyCursor& cu, const uint8_t* __restrict__ st, int t,
                                                  const float* __restrict__ rcp)
{
    if (cu.k < cu.kc && cu.fn <= t) {
        cu.fp = cu.fn;
        cu.vp = cu.vn;
        cu.fn = cu.fnn;
        cu.vn = cu.vnn;
        ++cu.k;
        if (cu.k + 1 < cu.kc) fast_key(st, cu.kb + 3u * (uint32_t)(cu.k + 1), cu.fnn, cu.vnn);
        fast_interval(cu, rcp);
    }
    const int ai = t - cu.fp;
    const float lerp = __fadd_rn(cu.vp, __fmul_rn(div_small_rn((float)ai, cu.bf, cu.y), cu.d));
    return cu.k == 0 ? cu.vn : ((cu.k == cu.kc || ai == 0) ? cu.vp : lerp);
}

// Axis weights as 16-byte rows {t, 1 - t, i0, i1} (a shared table [grid][axis][position], rt_frames.cuh):
// one 128-bit shared load per weight, read right where it is used.
__device__ __forceinline__ void axis_row(const float4* __restrict__ w16, int axis, int pos, float& t, float& omt,
                                         int& i0, int& i1)
{
    const float4 r = w16[axis * 8 + pos];
    t = r.x;
    omt = r.y;
    i0 = __float_as_int(r.z);
    i1 = __float_as_int(r.w);
}

// The x- and y-phases of trilinear_quads_ptr (rt_staged.cuh) for a compile-time even resolution R:
// the same lerps on the same operands in the same order, item loops unrolled.  x-lerps go to x2
// ([control row z*R + y][lx pair]), y-lerps to y4 ([control row z][ly][lx quad]).
template <int R>
__device__ __forceinline__ void trilinear_xy(const float4* __restrict__ w16, float2* x2, float4* y4,
                                             const float* __restrict__ g, int lane)
{
    static_assert(R % 2 == 0 && R >= 2 && R <= 6, "even resolutions up to 6");
    constexpr int NX = R * R * 4;
    {
        const int p = lane & 3;
        float ta, oa, tb, ob;
        int a0, a1, b0, b1;
        axis_row(w16, 0, 2 * p, ta, oa, a0, a1);
        axis_row(w16, 0, 2 * p + 1, tb, ob, b0, b1);
#pragma unroll
        for (int m = 0; m < (NX + 31) / 32; ++m) {
            const int row = (lane >> 2) + 8 * m;
            if (NX % 32 == 0 || row < R * R) {
                const float* gr = g + row * R;
                const float2 A = make_float2(gr[a0], gr[b0]);
                const float2 B = make_float2(gr[a1], gr[b1]);
                x2[lane + 32 * m] = lerp2(A, B, make_float2(ta, tb), make_float2(oa, ob));
            }
        }
    }
    __syncwarp();
    const int k = lane & 1;
    float t, o;
    int i0, i1;
    axis_row(w16, 1, (lane >> 1) & 7, t, o, i0, i1);
    const float2 ty = make_float2(t, t), oy = make_float2(o, o);
#pragma unroll
    for (int m = 0; m < R / 2; ++m) {   // R * 16 y items
        const int z = (lane >> 4) + 2 * m;
        const float4 a = *reinterpret_cast<const float4*>(x2 + (z * R + i0) * 4 + 2 * k);
        const float4 b = *reinterpret_cast<const float4*>(x2 + (z * R + i1) * 4 + 2 * k);
        const float2 lo2 = lerp2(make_float2(a.x, a.y), make_float2(b.x, b.y), ty, oy);
        const float2 hi2 = lerp2(make_float2(a.z, a.w), make_float2(b.z, b.w), ty, oy);
        y4[lane + 32 * m] = make_float4(lo2.x, lo2.y, hi2.x, hi2.y);
    }
    __syncwarp();
}

// The z-phase of trilinear_quads_ptr for the lane's quad i (voxels 4 (lane + 32 i) .. + 3).
__device__ __forceinline__ float4 trilinear_z(const float4* __restrict__ w16, const float4* y4, int lane, int i)
{
    const int k = lane & 1, ly = (lane >> 1) & 7;
    float tz, oz;
    int i0, i1;
    axis_row(w16, 2, 2 * i + (lane >> 4), tz, oz, i0, i1);
    const float4 A = y4[(i0 * 8 + ly) * 2 + k];
    const float4 B = y4[(i1 * 8 + ly) * 2 + k];
    const float2 t = make_float2(tz, tz), omt = make_float2(oz, oz);
    const float2 lo2 = lerp2(make_float2(A.x, A.y), make_float2(B.x, B.y), t, omt);
    const float2 hi2 = lerp2(make_float2(A.z, A.w), make_float2(B.z, B.w), t, omt);
    return make_float4(lo2.x, lo2.y, hi2.x, hi2.y);
}

// The weights of a grid's lanes: x quad first / second by the half lane & 1, z rows first / second by the half
// lane >> 4 (both in mirrored order for the upper half), {y t, y 1 - t, y control} by (lane >> 1) & 7.  Rows
// per half instead of per lane leave 4.5 KB more of the shared memory to the leaf stage: a 256^3 plume whose
// largest leaves lie there 512 -> 460 us (96 frames), one staged either way 466 -> 457.
struct LaneWeights {
    float4 xf[2], xs[2], zf[2], zs[2], y[8];
};
static_assert(2 * sizeof(LaneWeights) == 512, "their place in the leaf kernel's layout");

__device__ __forceinline__ void fill_lane_weights(LaneWeights* w)   // a barrier follows
{
    const int i = (int)threadIdx.x;
    if (i < 32) {   // grid, axis (x, z), half, position
        const int g = i >> 4, up = (i >> 2) & 1, k = i & 3;
        const AxisWeight aw = g_axis[axis_index(g == 0 ? 4 : 6, 8, up ? 7 - k : k)];
        float4* f = (i >> 3) & 1 ? w[g].zf : w[g].xf;
        float4* s = (i >> 3) & 1 ? w[g].zs : w[g].xs;
        reinterpret_cast<float*>(f + up)[k] = up ? aw.t : aw.omt;
        reinterpret_cast<float*>(s + up)[k] = up ? aw.omt : aw.t;
    } else if (i < 48) {
        const int g = (i >> 3) & 1, p = i & 7;
        const AxisWeight ay = g_axis[axis_index(g == 0 ? 4 : 6, 8, p)];
        w[g].y[p] = make_float4(ay.t, ay.omt, __int_as_float((int)ay.i0), 0.0f);
    }
}

// The separable trilinear of an R^3 grid (R = 4 or 6) with one lane's rows in registers.  Positions 0..3
// of an axis (7..4, mirrored, in its upper half) lie between controls 0,1 / 0,1 / 0,1 / 1,2 of the
// half for R = 4 and 0,1 / 0,1 / 1,2 / 2,3 for R = 6 (the axis table's first controls are
// 0 0 0 1 1 2 2 2 and 0 0 1 2 2 3 4 4).  In mirrored order a (1 - t) + b t is b t + a (1 - t): the same
// products and the same sum, and the controls of both halves have the same register names.

// x: every control row's 8 positions into x[8 * row ..]; g 16-byte (R = 4) or 8-byte (R = 6) aligned.
template <int R>
__device__ __forceinline__ void grid_x(const LaneWeights& w, const float* __restrict__ g, float* __restrict__ x, int lane)
{
    const bool up = (lane & 1) != 0;
    const float4 f = w.xf[lane & 1], s = w.xs[lane & 1];
#pragma unroll
    for (int m = 0; m < (R == 4 ? 1 : 3); ++m) {
        const int row = (lane >> 1) + 16 * m;
        if (R == 4 || row < 36) {
            float n0, n1, n2, n3 = 0.0f;
            if (R == 4) {
                const float4 c = *reinterpret_cast<const float4*>(g + 4 * row);
                n0 = up ? c.w : c.x;
                n1 = up ? c.z : c.y;
                n2 = up ? c.y : c.z;
            } else {
                const float2* p = reinterpret_cast<const float2*>(g + 6 * row + (up ? 2 : 0));
                const float2 a = p[0], b = p[1];
                n0 = up ? b.y : a.x;
                n1 = up ? b.x : a.y;
                n2 = up ? a.y : b.x;
                n3 = up ? a.x : b.y;
            }
            const float o0 = lerp_fs(n0, n1, f.x, s.x), o1 = lerp_fs(n0, n1, f.y, s.y);
            const float o2 = R == 4 ? lerp_fs(n0, n1, f.z, s.z) : lerp_fs(n1, n2, f.z, s.z);
            const float o3 = R == 4 ? lerp_fs(n1, n2, f.w, s.w) : lerp_fs(n2, n3, f.w, s.w);
            *reinterpret_cast<float4*>(x + 8 * row + 4 * (lane & 1)) =
                up ? make_float4(o3, o2, o1, o0) : make_float4(o0, o1, o2, o3);
        }
    }
}

// y: the lane's row (lane >> 1) & 7, quad lane & 1, in the control planes of its half (3 of 4, 4 of 6).
template <int R>
constexpr int kGridRows = R == 4 ? 3 : 4;
template <int R>
__device__ __forceinline__ void grid_y(const LaneWeights& w, const float* __restrict__ x, int lane, float4 (&y)[kGridRows<R>])
{
    const float4 wy = w.y[(lane >> 1) & 7];
    const float* r0 = x + 8 * __float_as_int(wy.z) + 4 * (lane & 1);
#pragma unroll
    for (int n = 0; n < kGridRows<R>; ++n) {
        const float* r = r0 + 8 * R * (lane >= 16 ? R - 1 - n : n);
        y[n] = lerp4(*reinterpret_cast<const float4*>(r), *reinterpret_cast<const float4*>(r + 8), wy.y, wy.x);
    }
}

// z: layer i (lanes 0-15) or 7 - i.
template <int R>
__device__ __forceinline__ float4 grid_z(const LaneWeights& w, const float4 (&y)[kGridRows<R>], int lane, int i)
{
    const float f = reinterpret_cast<const float*>(&w.zf[lane >> 4])[i], s = reinterpret_cast<const float*>(&w.zs[lane >> 4])[i];
    const int n = R == 4 ? (i == 3 ? 1 : 0) : (i == 3 ? 2 : i == 2 ? 1 : 0);
    return lerp4(y[n], y[n + 1], f, s);
}

// The specialised path of a leaf, if it has one.  (Staged, timeline frames, strictly increasing FP16 keys
// without NaN, coarse resolution 4, and alone, with a fine stream of resolution 6, or with a Mode2
// occupancy and its shell.)
enum : int { kFastNone, kFastGrid4, kFastFine6, kFastShell };
__device__ __forceinline__ int fast_leaf_shape(const LeafEntry& e, bool steps01)
{
    const uint32_t need = kFlagSorted | kFlagHalfPlain;
    if (!steps01 || (e.info & need) != need || ((e.header >> 6) & 7u) != 4u || ((e.header >> 2) & 3u) == 1u) return kFastNone;
    const bool fcodec_ok = ((e.header >> 4) & 3u) != 1u;
    if (e.info & kFlagOccClamp) return (e.info & kFlagFine) == 0u && ((e.info & kFlagShell) == 0u || fcodec_ok) ? kFastShell : kFastNone;
    if ((e.info & kFlagFine) == 0u) return (e.info & kFlagShell) == 0u ? kFastGrid4 : kFastNone;
    return ((e.header >> 9) & 7u) == 6u && fcodec_ok ? kFastFine6 : kFastNone;
}

// Decode one staged leaf of the fast shape for all nframes frames of the launch (NW warps; the
// leaf's bytes start at stage offset lb).  Quads go to sink(frame index, lz, ly, lx0, values).
// Per lane and slot the voxel phase holds one quad at a time.
template <bool FINE, int NW, class Sink>
__device__ __forceinline__ void leaf_decode_fast(const uint8_t* __restrict__ st, uint32_t lb, const LeafSmem& s,
                                                 const LeafEntry& e, int nframes, const LeafGeom& G,
                                                 const Sink& sink)
{
    constexpr int CC = 64, CT = FINE ? 64 + 216 : 64;
    constexpr int P = FINE ? 1 : 4;   // parts per control
    static_assert(CT * P <= 32 * NW, "one unit per thread");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int Lp = (nframes + P - 1) / P;   // frames per part
    int m = kLeafCtrlBudget / (CT * P);     // frames per part per batch
    if (m > Lp) m = Lp;
    if (P == 1 && m > NW) m -= m % NW;      // whole voxel rounds
    // this thread's unit
    const bool unit = tid < CT * P;
    const int c = FINE ? tid : (tid & 63);
    const int p = FINE ? 0 : (tid >> 6);
    const bool is_fine = FINE && c >= CC;
    const uint32_t C = is_fine ? 216u : 64u;
    const uint32_t ci = (uint32_t)(is_fine ? c - CC : c);
    const int f_lo = p * Lp, f_hi = min(nframes, f_lo + Lp);
    KeyCursor cu;
    if (unit && f_lo < f_hi) {
        const uint32_t sbase = lb + 8u + (is_fine ? e.coarse_bytes : 0u);
        const uint32_t kf = is_fine ? (e.kf >> 16) : (e.kf & 0xFFFFu);
        fast_cursor_init(st, sbase, C, 8u, ci, kf, s.fr[f_lo], s.b8[f_lo], s.rcp, cu);
    }
    const bool plain = G.w == 8 && G.h == 8 && G.d == 8;
    float* xc = reinterpret_cast<float*>(s.x2 + warp * 196);   // x rows: 128 floats, and 288 in the y rows' place
    float* xf = reinterpret_cast<float*>(s.y4 + warp * 112);
    for (int b0 = 0; b0 < Lp; b0 += m) {
        const int mb = min(m, Lp - b0);
        // 1. controls: slot p * mb + j holds frame f_lo + b0 + j
        if (unit) {
            float* dst = s.ctrl + (p * mb) * CT + c;
            for (int j = 0; j < mb; ++j) {
                const int fi = f_lo + b0 + j;
                if (fi >= f_hi) break;
                dst[j * CT] = fast_cursor_step(cu, st, s.fr[fi], s.rcp);
            }
        }
        __syncthreads();
        // 2. voxels, one slot (frame) per warp
        for (int slot = warp; slot < P * mb; slot += NW) {
            const int pp = P == 1 ? 0 : slot / mb, j = slot - pp * mb;
            const int fi = pp * Lp + b0 + j;
            if (fi >= min(nframes, (pp + 1) * Lp)) continue;
            const float* g = s.ctrl + slot * CT;
            grid_x<4>(s.lanes[0], g, xc, lane);
            if (FINE) grid_x<6>(s.lanes[1], g + CC, xf, lane);
            __syncwarp();
            float4 yc[kGridRows<4>], yf[kGridRows<6>];
            grid_y<4>(s.lanes[0], xc, lane, yc);
            if (FINE) grid_y<6>(s.lanes[1], xf, lane, yf);
            const int ly = (lane >> 1) & 7, lx0 = 4 * (lane & 1);
#pragma unroll
            for (int i = 0; i < 4; ++i) {   // coarse + fine, rounded once (the reference's sum)
                float4 v = grid_z<4>(s.lanes[0], yc, lane, i);
                if (FINE) {
                    const float4 f = grid_z<6>(s.lanes[1], yf, lane, i);
                    v = make_float4(__fadd_rn(v.x, f.x), __fadd_rn(v.y, f.y), __fadd_rn(v.z, f.z), __fadd_rn(v.w, f.w));
                }
                const int lz = lane >= 16 ? 7 - i : i;
                if (!plain) {
                    const bool row_in = ly < G.h && lz < G.d;
                    if (!row_in || lx0 >= G.w) v.x = 0.0f;
                    if (!row_in || lx0 + 1 >= G.w) v.y = 0.0f;
                    if (!row_in || lx0 + 2 >= G.w) v.z = 0.0f;
                    if (!row_in || lx0 + 3 >= G.w) v.w = 0.0f;
                }
                sink(fi, lz, ly, lx0, v);
            }
            __syncwarp();   // the tables are read before the next slot overwrites them
        }
        __syncthreads();
    }
}

// The same for a Mode2 leaf: 64 coarse and up to 512 shell controls, one or two cursors per thread, carried
// across the batches as above (the general path started every control's cursor anew for each batch of
// some eight frames; 32 frames of a 128^3 level set 246 -> 186 us).  A lane's four quads of occupancy do not change from frame to frame: the four
// bits of a quad and the index of its first shell control are one register.
template <int NW, class Sink>
__device__ __forceinline__ void leaf_decode_shell(const uint8_t* __restrict__ st, uint32_t lb, const LeafSmem& s,
                                                  const LeafEntry& e, int nframes, const LeafGeom& G, const Sink& sink)
{
    static_assert(64 + 512 <= 2 * 32 * NW, "two controls per thread");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool shell = (e.info & kFlagShell) != 0u;
    const uint32_t C2 = shell ? entry_shell_active(e) : 0u;
    const int CT = 64 + (int)C2, Cs = (CT + 3) & ~3;
    int m = min(kLeafCtrlBudget / Cs, nframes);   // frames per batch
    if (m > NW) m -= m % NW;                      // whole voxel rounds
    const int c1 = tid + 32 * NW;
    const bool on0 = tid < CT, on1 = c1 < CT;
    KeyCursor u0, u1;
    auto init = [&](int c, KeyCursor& cu) {
        const bool first = c < 64;
        fast_cursor_init(st, lb + (first ? 8u : e.shell_off), first ? 64u : C2, first ? 8u : 4u,
                         (uint32_t)(first ? c : c - 64), first ? e.kf & 0xFFFFu : e.kf >> 16, s.fr[0],
                         first ? s.b8[0] : s.b4[0], s.rcp, cu);
    };
    if (on0) init(tid, u0);
    if (on1) init(c1, u1);
    const bool plain = G.w == 8 && G.h == 8 && G.d == 8;
    const int ly = (lane >> 1) & 7, lx0 = 4 * (lane & 1);
    uint32_t occ[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {   // mask[lz], then prefix[lz], of the occupancy after the coarse stream
        const int lz = lane >= 16 ? 7 - i : i;
        const uint8_t* ob = st + lb + 8u + e.coarse_bytes;
        const uint32_t* mw = reinterpret_cast<const uint32_t*>(ob + 8 * lz);
        const uint64_t mask = ((uint64_t)mw[1] << 32) | mw[0];
        const uint32_t pref = (*reinterpret_cast<const uint32_t*>(ob + 64 + 4 * (lz >> 1)) >> ((lz & 1) * 16)) & 0xFFFFu;
        const uint32_t bit = (uint32_t)(8 * ly + lx0);
        occ[i] = ((uint32_t)(mask >> bit) & 15u) << 16 | (64u + pref + (uint32_t)__popcll(mask & ((1ull << bit) - 1ull)));
    }
    float* xc = reinterpret_cast<float*>(s.x2 + warp * 196);
    for (int b0 = 0; b0 < nframes; b0 += m) {
        const int mb = min(m, nframes - b0);
        if (on0)
            for (int j = 0; j < mb; ++j) s.ctrl[j * Cs + tid] = fast_cursor_step(u0, st, s.fr[b0 + j], s.rcp);
        if (on1)
            for (int j = 0; j < mb; ++j) s.ctrl[j * Cs + c1] = fast_cursor_step(u1, st, s.fr[b0 + j], s.rcp);
        __syncthreads();
        for (int j = warp; j < mb; j += NW) {
            const float* g = s.ctrl + j * Cs;
            grid_x<4>(s.lanes[0], g, xc, lane);
            __syncwarp();
            float4 y[kGridRows<4>];
            grid_y<4>(s.lanes[0], xc, lane, y);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 z = grid_z<4>(s.lanes[0], y, lane, i);
                float q[4] = {z.x, z.y, z.z, z.w};
                const float* v = g + (occ[i] & 0xFFFFu);
                const int lz = lane >= 16 ? 7 - i : i;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if ((occ[i] >> (16 + k)) & 1u) {
                        if (shell) q[k] = __fadd_rn(q[k], *v++);
                    } else if (q[k] < 0.0f) {
                        q[k] = 0.0f;
                    }
                    if (!plain && (ly >= G.h || lz >= G.d || lx0 + k >= G.w)) q[k] = 0.0f;
                }
                sink(b0 + j, lz, ly, lx0, make_float4(q[0], q[1], q[2], q[3]));
            }
            __syncwarp();   // the x rows are read before the next frame overwrites them
        }
        __syncthreads();
    }
}

}  // namespace vbtb
