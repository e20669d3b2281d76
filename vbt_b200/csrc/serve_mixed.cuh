// serve_mixed.cuh -- one persistent launch over the slice and frame requests a serving step
// admitted, of any resident assets, mixed.  Included by kernels.cu (it uses that file's decode
// helpers).  (The step's point requests go to the multi-asset point kernel beside it: a point is a
// chain of dependent loads that wants every thread an SM can hold in flight, while a leaf tile
// needs this kernel's 128 registers per thread.)
//
// The requests form a table (MixedReq, in device memory) with a running count of tiles.  A tile is
// one warp's piece of work:
//   slice   one (leaf of the z layer, frame): slice_tile, as query_slice_kernel;
//   frames  one (leaf, frame) of a dense frame (zeros for an EMPTY leaf): rt_leaf_frame, as
//           rt_frames_kernel, or the scientific per-frame functions.
// Warps take tiles kTileGrab at a time from a work counter (zeroed before the launch), so the
// tiles of large and small requests spread over the GPU as they come.  Each request has its own
// result array and error word; the values are those of the per-request kernels, bit for bit.
#pragma once

namespace vbtb {

constexpr uint32_t kTileGrab = 4;

// Tiles of one request (the host's count: same arithmetic).
__host__ __device__ __forceinline__ uint64_t mixed_tiles(const MixedReq& r, const AssetGeom& g)
{
    return r.kind == kMixedSlice ? (uint64_t)g.lcx * g.lcy * (uint64_t)(r.t1 - r.t0) : (uint64_t)g.leaf_count * r.n;
}

// Frame tile: all voxels of `leaf` at frame index `fr` (as given) into the dense frame `fb`.
__device__ __forceinline__ void mixed_frame_tile(const DeviceAsset& a, uint32_t leaf, int fr, float* __restrict__ fb,
                                                 float* __restrict__ sm, const float4* w16, unsigned long long* err)
{
    const int lane = threadIdx.x & 31;
    const LeafEntry e = a.entries[leaf];
    uint32_t bx, by, bz;
    int w, h, d;
    leaf_extent(a.g, leaf, bx, by, bz, w, h, d);
    const bool sci = a.g.profile == 2u;
    const uint32_t st = entry_status(e);
    if (st != kOk && lane == 0) record_error(err, leaf, st);
    float* const dst = fb + ((uint64_t)(bz * 8u) * a.g.height + by * 8u) * a.g.width + bx * 8u;
    auto put = [&](int ly, int lz, int lx0, float4 v) {
        if (ly < h && lz < d)
            store_row_quad(dst + ((uint64_t)((uint32_t)lz) * a.g.height + (uint32_t)ly) * a.g.width + (uint32_t)lx0, lx0, w, v);
    };
    if (st != kOk || (!sci && (e.header & 3u) == kModeEmpty)) {
        for (int r = lane; r < 128; r += 32) put((r >> 1) & 7, r >> 4, 4 * (r & 1), make_float4(0.f, 0.f, 0.f, 0.f));
        return;
    }
    if (!sci) {
        rt_leaf_frame(a, e, clamp_frame(fr, (int)a.g.frames), w, h, d, sm, w16, put);
        return;
    }
    const bool scatter = (e.header & 3u) == 1u && (e.info & kFlagSorted) != 0u;
    bool oob = false;
    sci_decode_controls(a, e, (uint32_t)fr, sm, lane, oob);
    __syncwarp();
    for (int r = lane; r < 64; r += 32) {
        float v[8];
        sci_row(a, e, sm, (uint32_t)fr, w, h, d, r & 7, r >> 3, v, oob, scatter);
        put(r & 7, r >> 3, 0, make_float4(v[0], v[1], v[2], v[3]));
        put(r & 7, r >> 3, 4, make_float4(v[4], v[5], v[6], v[7]));
    }
    if (scatter && (uint32_t)fr < a.g.frames) {
        __syncwarp();   // the rows written by the other lanes are visible
        sci_scatter_frame(a, e, (uint32_t)fr, w, h, d, lane,
                          [&](uint32_t li) {
                              return dst + ((uint64_t)(li >> 6) * a.g.height + ((li >> 3) & 7u)) * a.g.width + (li & 7u);
                          },
                          oob);
    }
    if (__any_sync(0xFFFFFFFFu, oob) && lane == 0) record_error(err, leaf, kErrDecodeOob);
    __syncwarp();
}

constexpr int kMixedWarps = 8;

__global__ void __launch_bounds__(kMixedWarps * 32, 3) serve_mixed_kernel(const DeviceAsset* __restrict__ assets,
                                                                       const MixedReq* __restrict__ reqs, uint32_t k,
                                                                       uint64_t n_tiles, unsigned long long* counter,
                                                                       unsigned long long* errs)
{
    __shared__ __align__(16) float s_all[kMixedWarps][kRtWarpFloats];
    __shared__ float4 s_w16[48];
    __shared__ uint64_t s_first[kMaxMixedReqs + 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (uint32_t i = (uint32_t)tid; i < k; i += blockDim.x) s_first[i] = reqs[i].first;
    if (tid == 0) s_first[k] = n_tiles;
    fill_axis_rows(s_w16);   // and the table of first tiles is complete
    float* sm = s_all[warp];
    for (;;) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(counter, (unsigned long long)kTileGrab);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if (base >= n_tiles) break;   // the counter only grows: every later grab is past the end too
        for (uint32_t j = 0; j < kTileGrab; ++j) {
            const uint64_t tile = base + j;
            if (tile >= n_tiles) break;
            int lo = 0, hi = (int)k - 1;
            while (lo < hi) {   // the last request whose first tile is at or before this one
                const int mid = (lo + hi + 1) >> 1;
                if (s_first[mid] <= tile) lo = mid;
                else hi = mid - 1;
            }
            const MixedReq rq = reqs[lo];
            const DeviceAsset& a = assets[rq.asset];
            const uint64_t u = tile - rq.first;
            unsigned long long* err = errs + lo;
            if (rq.kind == kMixedSlice) {
                const uint32_t layer = a.g.lcx * a.g.lcy;
                const uint32_t li = (uint32_t)(u % layer), f = (uint32_t)(u / layer);
                const uint32_t bz = min(a.g.lcz - 1u, rq.a0 >> 3);
                float* dst = reinterpret_cast<float*>(rq.out) +
                             ((uint64_t)f * a.g.height + li / a.g.lcx * 8u) * a.g.width + li % a.g.lcx * 8u;
                slice_tile(a, bz * layer + li, rq.a0, rq.t0 + (int)f, dst, sm, s_w16, err);
            } else {
                const uint32_t L = a.g.leaf_count;
                const uint64_t fi = u / L;
                const int fr = reinterpret_cast<const int*>(rq.in)[fi];
                float* fb = reinterpret_cast<float*>(rq.out) + fi * ((uint64_t)a.g.width * a.g.height * a.g.depth);
                mixed_frame_tile(a, (uint32_t)(u % L), fr, fb, sm, s_w16, err);
            }
        }
    }
}

static int mixed_grid(uint64_t n_tiles)
{
    static int full = 0;
    if (!full) {
        int dev = 0, sms = 0, per = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, serve_mixed_kernel, kMixedWarps * 32, 0);
        full = sms * (per > 0 ? per : 1);
    }
    const uint64_t want = (n_tiles + (uint64_t)kTileGrab * kMixedWarps - 1) / ((uint64_t)kTileGrab * kMixedWarps);
    return (int)(want < (uint64_t)full ? (want > 0 ? want : 1) : (uint64_t)full);
}

}  // namespace vbtb
