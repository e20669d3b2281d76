// sci_window_oracle.cuh -- the FP64 error oracle of scientific windows (and of any cache of scientific frames).
// Included by kernels.cu (it uses that file's scientific helpers).  The windows themselves are decoded by the
// frames kernel (sci_frames.cuh).
#pragma once

namespace vbtb {

// FP64 error oracle of a window (any scientific output of frames [t0, t0 + n) in the cache
// layout; voxels outside a boundary leaf's extent must be 0): per voxel and frame the reference
// model evaluated in double -- the coarse controls
// as sum_k q_k b_k(t) over the same FP32 coefficients and basis values, the trilinear weights as
// the reference's FP32 t and 1 - t, both without rounding, plus the FP32 sparse residual -- and
// the reduction stats[0] = max |value - oracle| (as ordered bits), stats[1] = sum of squares,
// stats[2] / stats[3] = oracle min / max (as ordered bits), in double.
__device__ __forceinline__ unsigned long long win_ordered(double x)
{
    const unsigned long long b = __double_as_longlong(x);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

// The DenseGrid residual of voxel (lx, ly, lz) at frame t in double without intermediate rounding:
// the decoded BFP samples and the reference's FP32 axis weights, the per-frame grid or the sum of
// the temporal-basis grids times the basis values (render/src/scientific_decode.cpp:125-233).
__device__ double dense_residual_f64(const DeviceAsset& a, SciReader& rd, uint64_t base, uint32_t hdr, int keep,
                                     uint32_t lx, uint32_t ly, uint32_t lz, uint32_t t)
{
    const uint32_t mode = hdr & 3u;
    const int res = mode == 2u ? 3 : 4, per = res * res * res;
    const int bits = (int)((hdr >> 8) & 0xFu);
    const uint32_t sub = (hdr >> 12) & 7u;
    const int tkeep = (int)((hdr >> 15) & 0xFu) + 1;
    const int sel = mode == 2u ? 1 : 2;
    const AxisWeight ax = c_sci_axis[sel][lx], ay = c_sci_axis[sel][ly], az = c_sci_axis[sel][lz];
    const uint64_t scales = base + 4u + (uint64_t)(64 * (keep + 1));
    auto tri = [&](uint64_t data, float sc) {
        double r = 0.0;
        for (int cz = 0; cz < 2; ++cz)
            for (int cy = 0; cy < 2; ++cy)
                for (int cx = 0; cx < 2; ++cx) {
                    const int ci = ((cz ? az.i1 : az.i0) * res + (cy ? ay.i1 : ay.i0)) * res + (cx ? ax.i1 : ax.i0);
                    const double w = (double)(cx ? ax.t : ax.omt) * (double)(cy ? ay.t : ay.omt) *
                                     (double)(cz ? az.t : az.omt);
                    r += w * (double)bfp_sample(rd, data, res, bits, sc, ci);
                }
        return r;
    };
    if (sub == 1u) {
        if (bits <= 0) return 0.0;
        const int bbytes = (per * bits + 7) / 8;
        const uint64_t data = scales + (uint64_t)(tkeep * 2);
        const float* brow = a.basis + (uint64_t)t * 64u;
        double r = 0.0;
        for (int k = 0; k < tkeep; ++k)
            r += tri(data + (uint64_t)(k * bbytes), half_bits_to_float(rd.u16(scales + (uint64_t)(k * 2)))) *
                 (double)__ldg(brow + k);
        return r;
    }
    const int fbytes = (per * bits + 7) / 8;
    return tri(scales + (uint64_t)a.g.frames * 2u + (uint64_t)t * fbytes, half_bits_to_float(rd.u16(scales + t * 2u)));
}

__global__ void __launch_bounds__(256) sci_window_oracle_kernel(DeviceAsset a, int t0, int n,
                                                                const float* __restrict__ vals, uint64_t frame_stride,
                                                                unsigned long long* stats)
{
    __shared__ double s_max[8], s_sum[8];
    __shared__ unsigned long long s_lo[8], s_hi[8];
    double my_max = 0.0, my_sum = 0.0;
    unsigned long long my_lo = ~0ull, my_hi = 0ull;
    const uint64_t items = (uint64_t)a.g.leaf_count * 512u;
    for (uint64_t it = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; it < items;
         it += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t leaf = (uint32_t)(it >> 9), v = (uint32_t)(it & 511u);
        const LeafEntry e = a.entries[leaf];
        const uint32_t hdr = e.header, mode = hdr & 3u;
        if (entry_status(e) != kOk) continue;
        const int keep = (int)((hdr >> 2) & 0x3Fu) + 1;
        const uint64_t base = 4ull * e.word_off;
        SciReader rd{a.payload, a.g.payload_words, false};
        const uint32_t lx = v & 7u, ly = (v >> 3) & 7u, lz = v >> 6;
        uint32_t gx, gy, gz;
        int ew, eh, ed;
        leaf_extent(a.g, leaf, gx, gy, gz, ew, eh, ed);
        if ((int)lx >= ew || (int)ly >= eh || (int)lz >= ed) {   // outside the volume: the cache holds 0
            for (int f = 0; f < n; ++f)
                my_max = fmax(my_max, fabs((double)vals[(uint64_t)f * frame_stride + (uint64_t)leaf * 512u + v]));
            continue;
        }
        const AxisWeight ax = c_sci_axis[0][lx], ay = c_sci_axis[0][ly], az = c_sci_axis[0][lz];
        for (int f = 0; f < n; ++f) {
            const uint32_t t = (uint32_t)(t0 + f);
            const float* brow = a.basis + (uint64_t)t * 64u;
            double ref = 0.0;
            for (int cz = 0; cz < 2; ++cz)
                for (int cy = 0; cy < 2; ++cy)
                    for (int cx = 0; cx < 2; ++cx) {
                        const int ci = ((cz ? az.i1 : az.i0) * 4 + (cy ? ay.i1 : ay.i0)) * 4 + (cx ? ax.i1 : ax.i0);
                        const double w = (double)(cx ? ax.t : ax.omt) * (double)(cy ? ay.t : ay.omt) *
                                         (double)(cz ? az.t : az.omt);
                        const uint64_t cb = base + 4u + (uint64_t)ci * (keep + 1);
                        double c = (double)half_bits_to_float(rd.u16(cb)) * (double)__ldg(brow);
                        for (int k = 1; k < keep; ++k) {
                            const float q = __fmul_rn((float)(int8_t)rd.byte(cb + 2u + (k - 1)), __ldg(a.scales + k - 1));
                            c += (double)q * (double)__ldg(brow + k);
                        }
                        ref += w * c;
                    }
            if (mode == 1u) ref += (double)sci_sparse(rd, base, hdr, keep, v, t);
            else if (mode >= 2u) ref += dense_residual_f64(a, rd, base, hdr, keep, lx, ly, lz, t);
            const double got = (double)vals[(uint64_t)f * frame_stride + (uint64_t)leaf * 512u + v];
            const double err = fabs(got - ref);
            my_max = fmax(my_max, err);
            my_sum += err * err;
            const unsigned long long o = win_ordered(ref);
            my_lo = o < my_lo ? o : my_lo;
            my_hi = o > my_hi ? o : my_hi;
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
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
        s_max[warp] = my_max;
        s_sum[warp] = my_sum;
        s_lo[warp] = my_lo;
        s_hi[warp] = my_hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double mx = 0.0, sm = 0.0;
        unsigned long long lo = ~0ull, hi = 0ull;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            mx = fmax(mx, s_max[w]);
            sm += s_sum[w];
            lo = s_lo[w] < lo ? s_lo[w] : lo;
            hi = s_hi[w] > hi ? s_hi[w] : hi;
        }
        atomicMax(stats + 0, (unsigned long long)__double_as_longlong(mx));   // non-negative: bits order
        atomicAdd(reinterpret_cast<double*>(stats + 1), sm);
        atomicMin(stats + 2, lo);
        atomicMax(stats + 3, hi);
    }
}

void launch_sci_window_oracle(const DeviceAsset& a, int t0, int n, const float* vals, uint64_t frame_stride,
                              unsigned long long* stats, cudaStream_t s)
{
    cudaMemsetAsync(stats, 0, 4 * sizeof(unsigned long long), s);       // max, sum (0.0), -, max
    cudaMemsetAsync(stats + 2, 0xFF, sizeof(unsigned long long), s);   // min starts at the top
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    sci_window_oracle_kernel<<<4 * sms, 256, 0, s>>>(a, t0, n, vals, frame_stride, stats);
}

}  // namespace vbtb
