// rt_frames.cuh -- single frames and slices of render-temporal leaves, one warp per leaf and frame.
// Included by kernels.cu.
//
// The launch that streams many frames of a leaf (rt_kernel_leaf.cuh) first brings the whole leaf into
// shared memory; for one frame, or a few, that reads 10 to 50 KB where the frame needs two keys of
// each control.  Here a warp reads just those from the payload (control_sorted: descriptor, hint and
// one window of keys), and makes the voxels with the specialised path's separable trilinear.  A slice
// decodes only the two planes of controls on either side of it.  Bound by the latency of the control
// reads, which many resident warps hide, then by instruction issue.  On a B200, files not in L2: one
// frame of a 125 x 131 x 190 fire 79 -> 26 us on the device, a 16-frame slice of a 128 x 128 x 192 one
// 42 -> 11; a FINE6 leaf's controls one at a time instead of three in flight: 46 us.
#pragma once

namespace vbtb {

// Shared floats of a warp: controls (64 coarse, then 216 fine or up to 512 shell values), x rows, y rows;
// leaves of no common shape use them as rt_decode_controls' slots.
constexpr int kRtCtrl = 64 + 512, kRtX = 384, kRtY = 384, kRtWarpFloats = kRtCtrl + kRtX + kRtY;
static_assert(kRtWarpFloats >= kCtrlSlots && kRtWarpFloats % 4 == 0, "room for the general slots, 16-byte rows");

// Controls of a lane whose reads are in flight together: a FINE6 leaf's 280 are three rounds of reads.
constexpr int kRtBatch = 3;

// The axis weights of whole leaves for 4 and 6 controls, as leaf_decode_fast reads them; a position
// inside a cropped leaf has the weights it has in a whole one.
__device__ __forceinline__ void fill_axis_rows(float4* w16)
{
    for (int i = (int)threadIdx.x; i < 48; i += (int)blockDim.x) {
        const AxisWeight aw = g_axis[axis_index(i < 24 ? 4 : 6, 8, i & 7)];
        w16[i] = make_float4(aw.t, aw.omt, __int_as_float((int)aw.i0), __int_as_float((int)aw.i1));
    }
    __syncthreads();
}

// A leaf with ordered FP16 keys, none of them NaN, and a 4^3 coarse grid, alone (GRID4), with a 6^3 fine grid (FINE6) or
// with a Mode2 shell.
__device__ __forceinline__ bool rt_common_shape(const LeafEntry& e)
{
    const uint32_t hdr = e.header, need = kFlagSorted | kFlagHalfPlain;
    if ((e.info & need) != need || ((hdr >> 6) & 7u) != 4u || ((hdr >> 2) & 3u) == 1u) return false;
    if (e.info & kFlagFine) return (e.info & kFlagOccClamp) == 0u && ((hdr >> 9) & 7u) == 6u && ((hdr >> 4) & 3u) != 1u;
    return (e.info & kFlagShell) == 0u || ((hdr >> 4) & 3u) != 1u;
}

// Mode2: voxels bit0 .. bit0 + 3 of a layer with occupancy `mask` add their shell values (shell[0] =
// the layer's first); the others are clamped at 0 from below.
__device__ __forceinline__ float4 shell_quad(float4 v, uint64_t mask, uint32_t bit0, const float* shell)
{
    float q[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (uint32_t k = 0; k < 4u; ++k) {
        const uint32_t bit = bit0 + k;
        if ((mask >> bit) & 1ull) {
            if (shell) q[k] = __fadd_rn(q[k], shell[__popcll(mask & ((1ull << bit) - 1ull))]);
        } else if (q[k] < 0.0f) {
            q[k] = 0.0f;
        }
    }
    return make_float4(q[0], q[1], q[2], q[3]);
}

// All voxels of one valid, non-EMPTY leaf at clamped frame `frame`: put(ly, lz, lx0, quad).
template <class Put>
__device__ __forceinline__ void rt_leaf_frame(const DeviceAsset& a, const LeafEntry& e, int frame, int w, int h, int d,
                                              float* sm, const float4* w16, const Put& put)
{
    const int lane = threadIdx.x & 31;
    if (!rt_common_shape(e)) {
        rt_decode_controls(a, e, frame, sm, lane);
        __syncwarp();
        for (int r = lane; r < 64; r += 32) {
            float v[8];
            rt_row(a, e, sm, w, h, d, r & 7, r >> 3, v);
            put(r & 7, r >> 3, 0, make_float4(v[0], v[1], v[2], v[3]));
            put(r & 7, r >> 3, 4, make_float4(v[4], v[5], v[6], v[7]));
        }
        __syncwarp();
        return;
    }
    const uint32_t* __restrict__ lw = a.payload + e.word_off;
    const bool fine = (e.info & kFlagFine) != 0u, shell = (e.info & kFlagShell) != 0u, occ = (e.info & kFlagOccClamp) != 0u;
    const uint32_t bin8 = time_bin(frame, 8u, (int)a.g.frames), fine_at = 8u + e.coarse_bytes;
    const LeafStream cs{lw, 8u, 64u, 8u, e.kf & 0xFFFFu};
    // coarse and fine controls in one run of units, so that no lane waits between the streams
    const LeafStream fs{lw, fine ? fine_at : e.shell_off, fine ? 216u : entry_shell_active(e), fine ? 8u : 4u, e.kf >> 16};
    const uint32_t n2 = fine || shell ? fs.controls : 0u;
    const uint32_t bin2 = fine ? bin8 : time_bin(frame, 4u, (int)a.g.frames);
    const uint32_t total = 64u + n2;
#pragma unroll 1
    for (uint32_t c0 = (uint32_t)lane; c0 < total; c0 += 32u * kRtBatch) {
        uint32_t desc[kRtBatch], hint[kRtBatch];
        KeyWindow k[kRtBatch];
#pragma unroll
        for (int i = 0; i < kRtBatch; ++i) {
            const uint32_t c = c0 + 32u * (uint32_t)i;
            desc[i] = hint[i] = 0u;
            if (c < 64u) {
                desc[i] = __ldg(lw + 2u + c);
                hint[i] = hint_word(cs, c, bin8);
            } else if (c < total) {
                desc[i] = __ldg(lw + (fs.base >> 2) + c - 64u);
                hint[i] = hint_word(fs, c - 64u, bin2);
            }
        }
#pragma unroll
        for (int i = 0; i < kRtBatch; ++i) {
            const uint32_t c = c0 + 32u * (uint32_t)i;
            k[i] = c < 64u ? key_start(cs, desc[i], hint[i], bin8) : key_start(fs, desc[i], hint[i], bin2);
            if (k[i].kc) key_window(lw, k[i]);
        }
#pragma unroll
        for (int i = 0; i < kRtBatch; ++i) {
            const uint32_t c = c0 + 32u * (uint32_t)i;
            if (c < total) sm[c] = key_value_at<true>(lw, k[i], frame);
        }
    }
    __syncwarp();
    float2* x2 = reinterpret_cast<float2*>(sm + kRtCtrl);
    float4* y4 = reinterpret_cast<float4*>(sm + kRtCtrl + kRtX);
    float4* yc = fine ? reinterpret_cast<float4*>(x2 + 64) : y4;
    if (fine) trilinear_xy<6>(w16 + 24, x2, y4, sm + 64, lane);
    trilinear_xy<4>(w16, x2, yc, sm, lane);
    const int ly = (lane >> 1) & 7, lx0 = 4 * (lane & 1);
    const uint32_t ow = fine_at >> 2;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float4 v = trilinear_z(w16, yc, lane, i);
        const int lz = 2 * i + (lane >> 4);
        if (fine) {
            v = add4(v, trilinear_z(w16 + 24, y4, lane, i));
        } else if (occ) {
            const uint64_t mask = ((uint64_t)__ldg(lw + ow + 2 * lz + 1) << 32) | __ldg(lw + ow + 2 * lz);
            const uint32_t pref = (__ldg(lw + ow + 16 + (lz >> 1)) >> ((lz & 1) * 16)) & 0xFFFFu;
            v = shell_quad(v, mask, (uint32_t)(ly * 8 + lx0), shell ? sm + 64 + pref : nullptr);
        }
        put(ly, lz, lx0, v);
    }
    __syncwarp();   // the rows are read before the next frame overwrites them
}

// The rows of layer lz of one valid, non-EMPTY leaf at clamped frame `frame`: put(ly, lx0, quad).
template <class Put>
__device__ __forceinline__ void rt_leaf_layer(const DeviceAsset& a, const LeafEntry& e, int frame, int w, int h, int d,
                                              int lz, float* sm, const float4* w16, const Put& put)
{
    const int lane = threadIdx.x & 31;
    if (!rt_common_shape(e)) {
        rt_decode_controls(a, e, frame, sm, lane);
        __syncwarp();
        if (lane < 16) {
            float v[4];
            rt_voxels<4>(a, e, sm, w, h, d, 4 * (lane & 1), lane >> 1, lz, v);
            put(lane >> 1, 4 * (lane & 1), make_float4(v[0], v[1], v[2], v[3]));
        }
        __syncwarp();
        return;
    }
    const uint32_t* __restrict__ lw = a.payload + e.word_off;
    const bool fine = (e.info & kFlagFine) != 0u, shell = (e.info & kFlagShell) != 0u, occ = (e.info & kFlagOccClamp) != 0u;
    const uint32_t bin8 = time_bin(frame, 8u, (int)a.g.frames), fine_at = 8u + e.coarse_bytes;
    float tc, oc, tf, of;
    int zc, zf, z1;
    axis_row(w16, 2, lz, tc, oc, zc, z1);
    axis_row(w16 + 24, 2, lz, tf, of, zf, z1);
    float* const layer = sm + 128;   // the layer's shell values
    uint64_t mask = 0;
    uint32_t n2 = 0, c2 = 0;   // second stream: its controls of this layer, from control c2 on
    LeafStream fs{lw, fine_at, 216u, 8u, e.kf >> 16};
    if (occ) {
        const uint32_t ow = fine_at >> 2;
        mask = ((uint64_t)__ldg(lw + ow + 2 * lz + 1) << 32) | __ldg(lw + ow + 2 * lz);
        if (shell) {
            c2 = (__ldg(lw + ow + 16 + (lz >> 1)) >> ((lz & 1) * 16)) & 0xFFFFu;
            n2 = (uint32_t)__popcll(mask);
            fs = LeafStream{lw, e.shell_off, entry_shell_active(e), 4u, e.kf >> 16};
        }
    } else if (fine) {
        c2 = 36u * (uint32_t)zf;
        n2 = 72u;
    }
    const uint32_t bin2 = fine ? bin8 : time_bin(frame, 4u, (int)a.g.frames);
#pragma unroll 1
    for (uint32_t c = (uint32_t)lane; c < 32u + n2; c += 32u) {   // 32 coarse controls: planes zc, zc + 1
        const bool first = c < 32u;
        const LeafStream s{lw, first ? 8u : fs.base, first ? 64u : fs.controls, first ? 8u : fs.bins,
                           first ? e.kf & 0xFFFFu : fs.kf};
        const float v = control_sorted<true>(s, first ? 16u * (uint32_t)zc + c : c2 + c - 32u, frame, first ? bin8 : bin2);
        if (first) sm[c] = v;
        else if (fine) sm[c] = v;
        else layer[c - 32u] = v;
    }
    __syncwarp();
    // x rows of the two planes of each grid ([plane][row][pair]), then the lane's y and z lerps
    float2* xc = reinterpret_cast<float2*>(sm + kRtCtrl);
    float2* xf = xc + 32;
    float ta, oa, tb, ob;
    int a0, a1, b0, b1;
    axis_row(w16, 0, 2 * (lane & 3), ta, oa, a0, a1);
    axis_row(w16, 0, 2 * (lane & 3) + 1, tb, ob, b0, b1);
    {
        const float* g = sm + 4 * (lane >> 2);
        xc[lane] = lerp2(make_float2(g[a0], g[b0]), make_float2(g[a1], g[b1]), make_float2(ta, tb), make_float2(oa, ob));
    }
    if (fine) {
        axis_row(w16 + 24, 0, 2 * (lane & 3), ta, oa, a0, a1);
        axis_row(w16 + 24, 0, 2 * (lane & 3) + 1, tb, ob, b0, b1);
        for (int i = lane; i < 48; i += 32) {
            const float* g = sm + 32 + 6 * (i >> 2);
            xf[i] = lerp2(make_float2(g[a0], g[b0]), make_float2(g[a1], g[b1]), make_float2(ta, tb), make_float2(oa, ob));
        }
    }
    __syncwarp();
    if (lane < 16) {
        const int ly = lane >> 1, k = lane & 1, lx0 = 4 * k;
        auto quad = [&](const float2* x, int rows, int grid, float t, float o) {
            float ty, oy;
            int i0, i1;
            axis_row(w16 + grid, 1, ly, ty, oy, i0, i1);
            float4 p[2];
#pragma unroll
            for (int z = 0; z < 2; ++z) {
                const float4 A = *reinterpret_cast<const float4*>(x + (z * rows + i0) * 4 + 2 * k);
                const float4 B = *reinterpret_cast<const float4*>(x + (z * rows + i1) * 4 + 2 * k);
                p[z] = make_float4(lerp_ref(A.x, B.x, ty, oy), lerp_ref(A.y, B.y, ty, oy), lerp_ref(A.z, B.z, ty, oy),
                                   lerp_ref(A.w, B.w, ty, oy));
            }
            return make_float4(lerp_ref(p[0].x, p[1].x, t, o), lerp_ref(p[0].y, p[1].y, t, o),
                               lerp_ref(p[0].z, p[1].z, t, o), lerp_ref(p[0].w, p[1].w, t, o));
        };
        float4 v = quad(xc, 4, 0, tc, oc);
        if (fine) v = add4(v, quad(xf, 6, 24, tf, of));
        else if (occ) v = shell_quad(v, mask, (uint32_t)(ly * 8 + lx0), shell ? layer : nullptr);
        put(ly, lx0, v);
    }
    __syncwarp();
}

// Four floats of a row that has w from lx0 on inside the volume.
__device__ __forceinline__ void store_row_quad(float* o, int lx0, int w, float4 v)
{
    if (lx0 + 4 <= w && (reinterpret_cast<uintptr_t>(o) & 15u) == 0u) {
        *reinterpret_cast<float4*>(o) = v;
    } else {
        if (lx0 < w) o[0] = v.x;
        if (lx0 + 1 < w) o[1] = v.y;
        if (lx0 + 2 < w) o[2] = v.z;
        if (lx0 + 3 < w) o[3] = v.w;
    }
}

constexpr int kRtWarps = 4, kRtCtas = 6;

// The launch's frames (grid.y) of every active leaf into the cache, or of every leaf into dense frames
// (zeros for EMPTY ones).
template <bool DENSE>
__global__ void __launch_bounds__(kRtWarps * 32, kRtCtas) rt_frames_kernel(DeviceAsset a, FrameList fl,
                                                                          float* __restrict__ out, uint64_t frame_stride)
{
    __shared__ __align__(16) float s_all[kRtWarps][kRtWarpFloats];
    __shared__ float4 s_w16[48];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t n_leaves = DENSE ? a.g.leaf_count : *(volatile const uint32_t*)a.counters;
    if ((uint64_t)blockIdx.x * kRtWarps >= n_leaves) return;
    fill_axis_rows(s_w16);
    const int frame = clamp_frame(fl.f[blockIdx.y], (int)a.g.frames);
    float* const fo = out + (uint64_t)blockIdx.y * frame_stride;
    for (uint64_t at = (uint64_t)blockIdx.x * kRtWarps + warp; at < n_leaves; at += (uint64_t)gridDim.x * kRtWarps) {
        const uint32_t leaf = DENSE ? (uint32_t)at : __ldg(a.active_list + at);
        const LeafEntry e = a.entries[leaf];
        uint32_t bx, by, bz;
        int w, h, d;
        leaf_extent(a.g, leaf, bx, by, bz, w, h, d);
        auto put = [&](int ly, int lz, int lx0, float4 v) {
            if (DENSE) {
                if (ly < h && lz < d)
                    store_row_quad(fo + ((uint64_t)(bz * 8u + (uint32_t)lz) * a.g.height + (by * 8u + (uint32_t)ly)) * a.g.width +
                                       bx * 8u + (uint32_t)lx0, lx0, w, v);
            } else {
                const bool in = ly < h && lz < d;
                if (!in || lx0 >= w) v.x = 0.0f;
                if (!in || lx0 + 1 >= w) v.y = 0.0f;
                if (!in || lx0 + 2 >= w) v.z = 0.0f;
                if (!in || lx0 + 3 >= w) v.w = 0.0f;
                *reinterpret_cast<float4*>(fo + at * 512u + (uint32_t)(64 * lz + 8 * ly + lx0)) = v;
            }
        };
        const uint32_t st = entry_status(e);
        if (st != kOk || (e.header & 3u) == kModeEmpty) {
            if (st != kOk && lane == 0 && blockIdx.y == 0) record_error(a.err, leaf, st);
            for (int r = lane; r < 128; r += 32) put((r >> 1) & 7, r >> 4, 4 * (r & 1), make_float4(0.f, 0.f, 0.f, 0.f));
            continue;
        }
        rt_leaf_frame(a, e, frame, w, h, d, s_all[warp], s_w16, put);
    }
}

static int rt_frames_full()
{
    static int full = 0;
    if (!full) {
        int dev = 0, sms = 0, per = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, rt_frames_kernel<false>, kRtWarps * 32, 0);
        full = sms * (per > 0 ? per : 1);
    }
    return full;
}

template <bool DENSE>
static void launch_rt_frames(const DeviceAsset& a, const FrameList& fl, float* out, uint64_t stride, int grid, cudaStream_t s)
{
    // a CTA per four leaves, so that the leaves spread as CTAs finish, up to four waves (the active count
    // is not known here; CTAs past it end at once)
    const uint32_t most = (a.g.leaf_count + kRtWarps - 1) / kRtWarps;
    const uint32_t g = grid > 0 ? (uint32_t)grid : 4u * (uint32_t)rt_frames_full();
    rt_frames_kernel<DENSE><<<dim3(most < g ? most : g, (unsigned)fl.n), kRtWarps * 32, 0, s>>>(a, fl, out, stride);
}

}  // namespace vbtb
