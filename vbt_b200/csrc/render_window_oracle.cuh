// render_window_oracle.cuh -- the FP64 error oracle of render-temporal windows.  Included by kernels.cu after
// sci_window_oracle.cuh.  A window is a run of frames of the cache, and its decode is the cache's
// (launch_decode_cache).
#pragma once

namespace vbtb {

// Exact-arithmetic trilinear of one control grid (resolution R) at voxel (lx, ly, lz): the
// reference's nested lerps with its FP32 weights t and 1 - t, expanded without rounding.
__device__ __forceinline__ double trilinear_f64(const AxisWeight (*w)[8], const double* g, int R, int lx, int ly,
                                                int lz)
{
    if (R < 2) return R == 1 ? g[0] : 0.0;
    const AxisWeight ax = w[0][lx], ay = w[1][ly], az = w[2][lz];
    double v = 0.0;
    for (int cz = 0; cz < 2; ++cz)
        for (int cy = 0; cy < 2; ++cy)
            for (int cx = 0; cx < 2; ++cx) {
                const int ci = ((cz ? az.i1 : az.i0) * R + (cy ? ay.i1 : ay.i0)) * R + (cx ? ax.i1 : ax.i0);
                v += (double)(cx ? ax.t : ax.omt) * (double)(cy ? ay.t : ay.omt) * (double)(cz ? az.t : az.omt) * g[ci];
            }
    return v;
}

// FP64 error oracle of any render-temporal cache of frames [t0, t0 + n) (cache layout, active
// ranks of the current page table): per voxel and frame the reference composition
// (render_smoke_vbt_bench_main.cpp:277-387) evaluated in double without intermediate rounding --
// controls from the bracket the reference's search selects, interpolated exactly; the trilinear
// with the reference's FP32 weights; fine grid or Mode2 shell residual; Mode2's clamp of negatives
// outside the occupancy -- reduced as sci_window_oracle_kernel reduces.
__global__ void __launch_bounds__(256) render_window_oracle_kernel(DeviceAsset a, int t0, int n,
                                                                   const float* __restrict__ vals,
                                                                   uint64_t frame_stride, unsigned long long* stats)
{
    __shared__ double s_ctrl[343 + 512];
    __shared__ AxisWeight s_w[2][3][8];
    __shared__ double s_max[8], s_sum[8];
    __shared__ unsigned long long s_lo[8], s_hi[8];
    const int tid = threadIdx.x;
    const int total = (int)a.g.frames;
    double my_max = 0.0, my_sum = 0.0;
    unsigned long long my_lo = ~0ull, my_hi = 0ull;
    const GlobalWords m{a.payload};
    const uint32_t n_leaves = *(volatile const uint32_t*)a.counters;
    for (uint32_t rank = blockIdx.x; rank < n_leaves; rank += gridDim.x) {
        const uint32_t leaf = __ldg(a.active_list + rank);
        const LeafEntry e = a.entries[leaf];
        int ew, eh, ed;
        uint32_t gx, gy, gz;
        leaf_extent(a.g, leaf, gx, gy, gz, ew, eh, ed);
        const float* row0 = vals + (uint64_t)rank * 512u;
        if (entry_status(e) != kOk || (e.header & 3u) == kModeEmpty) {   // the cache holds 0
            for (int i = tid; i < n * 512; i += 256)
                my_max = fmax(my_max, fabs((double)row0[(uint64_t)(i >> 9) * frame_stride + (i & 511)]));
            continue;
        }
        const uint64_t base = 4ull * e.word_off;
        const int cres = (int)((e.header >> 6) & 7u), fres = (int)((e.header >> 9) & 7u);
        const bool fine = (e.info & kFlagFine) != 0u, shell = (e.info & kFlagShell) != 0u;
        const bool occ = (e.info & kFlagOccClamp) != 0u;
        const StreamRef cs{base + 8u, (uint32_t)(cres * cres * cres), 8u, e.kf & 0xFFFFu, (e.header >> 2) & 3u};
        const StreamRef fs{base + 8u + e.coarse_bytes, (uint32_t)(fres * fres * fres), 8u, e.kf >> 16,
                           (e.header >> 4) & 3u};
        const StreamRef ss{base + e.shell_off, entry_shell_active(e), 4u, e.kf >> 16, (e.header >> 4) & 3u};
        const int Cc = (int)cs.controls;
        const int Cf = fine ? (int)fs.controls : (shell ? (int)ss.controls : 0);
        if (tid < 48) {
            const int ws = tid / 24, axis = (tid % 24) >> 3, p = tid & 7;
            const int R = ws == 0 ? cres : fres;
            const int ext = axis == 0 ? ew : (axis == 1 ? eh : ed);
            s_w[ws][axis][p] = g_axis[axis_index(R, ext, p)];
        }
        for (int f = 0; f < n; ++f) {
            const int t = t0 + f;
            for (int c = tid; c < Cc + Cf; c += 256) {
                const StreamRef& st = c < Cc ? cs : (fine ? fs : ss);
                const uint32_t ci = (uint32_t)(c < Cc ? c : c - Cc);
                s_ctrl[c] = m_control_value_f64(m, st, ci, t, time_bin(t, st.bins, total));
            }
            __syncthreads();
            for (int v = tid; v < 512; v += 256) {
                const int lx = v & 7, ly = (v >> 3) & 7, lz = v >> 6;
                double ref = 0.0;
                if (lx < ew && ly < eh && lz < ed) {
                    ref = trilinear_f64(s_w[0], s_ctrl, cres, lx, ly, lz);
                    if (fine) ref += trilinear_f64(s_w[1], s_ctrl + Cc, fres, lx, ly, lz);
                    if (occ) {
                        const uint64_t ob = base + 8u + e.coarse_bytes;
                        const uint32_t g = (uint32_t)v >> 6, bit = (uint32_t)v & 63u;
                        const uint64_t mk = ((uint64_t)m((uint32_t)((ob + 8u * g + 4u) >> 2)) << 32) |
                                            m((uint32_t)((ob + 8u * g) >> 2));
                        const uint32_t pref = (m((uint32_t)((ob + 64u + 2u * g) >> 2)) >> ((g & 1u) * 16u)) & 0xFFFFu;
                        const bool in_occ = ((mk >> bit) & 1ull) != 0ull;
                        if (shell && in_occ) {
                            const uint32_t di = (pref + (uint32_t)__popcll(mk & ((1ull << bit) - 1ull))) & 0xFFFFu;
                            ref += s_ctrl[Cc + (int)di];
                        }
                        if (!in_occ && ref < 0.0) ref = 0.0;
                    }
                }
                const double got = (double)row0[(uint64_t)f * frame_stride + v];
                const double err = fabs(got - ref);
                my_max = fmax(my_max, err);
                my_sum += err * err;
                const unsigned long long o = win_ordered(ref);
                my_lo = o < my_lo ? o : my_lo;
                my_hi = o > my_hi ? o : my_hi;
            }
            __syncthreads();
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        my_max = fmax(my_max, __shfl_down_sync(0xFFFFFFFFu, my_max, o));
        my_sum += __shfl_down_sync(0xFFFFFFFFu, my_sum, o);
        const unsigned long long lo2 = __shfl_down_sync(0xFFFFFFFFu, my_lo, o);
        const unsigned long long hi2 = __shfl_down_sync(0xFFFFFFFFu, my_hi, o);
        my_lo = lo2 < my_lo ? lo2 : my_lo;
        my_hi = hi2 > my_hi ? hi2 : my_hi;
    }
    const int warp = tid >> 5, lane = tid & 31;
    if (lane == 0) {
        s_max[warp] = my_max;
        s_sum[warp] = my_sum;
        s_lo[warp] = my_lo;
        s_hi[warp] = my_hi;
    }
    __syncthreads();
    if (tid == 0) {
        double mx = 0.0, sm = 0.0;
        unsigned long long lo = ~0ull, hi = 0ull;
        for (int w = 0; w < 8; ++w) {
            mx = fmax(mx, s_max[w]);
            sm += s_sum[w];
            lo = s_lo[w] < lo ? s_lo[w] : lo;
            hi = s_hi[w] > hi ? s_hi[w] : hi;
        }
        atomicMax(stats + 0, (unsigned long long)__double_as_longlong(mx));
        atomicAdd(reinterpret_cast<double*>(stats + 1), sm);
        atomicMin(stats + 2, lo);
        atomicMax(stats + 3, hi);
    }
}

void launch_render_window_oracle(const DeviceAsset& a, int t0, int n, const float* vals, uint64_t frame_stride,
                                 unsigned long long* stats, cudaStream_t s)
{
    cudaMemsetAsync(stats, 0, 4 * sizeof(unsigned long long), s);
    cudaMemsetAsync(stats + 2, 0xFF, sizeof(unsigned long long), s);
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    render_window_oracle_kernel<<<4 * sms, 256, 0, s>>>(a, t0, n, vals, frame_stride, stats);
}

}  // namespace vbtb
