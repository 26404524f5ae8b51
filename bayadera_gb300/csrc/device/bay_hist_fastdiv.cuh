// bay_hist_fastdiv.cuh -- histogram bin counts with the reference's division flavour.
//
// The reference builds its estimate kernels with NVRTC and -use_fast_math, the bin count
// being the compile-time WGS (nvidia_gtx.clj:614-616), and bins a value by
// (uint)((x - lo) / (hi - lo) * WGS) clamped to WGS - 1 (nvidia-gtx-estimate.cu:22-23):
// the division there is the compiler's fast division.  The library compiles this file the
// same way (-use_fast_math, BAY_HIST_BINS a compile-time constant) so the same expression
// gets the same division; bay_estimates.cu's hist_count is the IEEE-division default.
//
// Layout, split and counting as hist_count: values point-major (xs[w * D + d]), a CTA the
// dimension tile blockIdx.x / gx and share blockIdx.x % gx of the rows, thread t dimension
// t % dt, per-CTA shared-memory counts, one global atomic per non-empty bin.

extern "C" __global__ void __launch_bounds__(256)
bay_hist_count_fastdiv(const float* xs, unsigned int D, unsigned long long W, unsigned int gx,
                       unsigned int tile, const float* limits, unsigned int* counts) {
    extern __shared__ unsigned int h[];
    const unsigned int by = blockIdx.x / gx, bx = blockIdx.x - by * gx;
    const unsigned int d0 = by * tile, dt = D - d0 < tile ? D - d0 : tile;
    const unsigned int rp = 256u / dt, rl = threadIdx.x / dt, dl = threadIdx.x - rl * dt;
    for (unsigned int b = threadIdx.x; b < dt * BAY_HIST_BINS; b += 256u) h[b] = 0u;
    __syncthreads();
    if (rl < rp) {
        const float lower = limits[2ull * (d0 + dl)];
        const float upper = limits[2ull * (d0 + dl) + 1];
        for (unsigned long long w = (unsigned long long)bx * rp + rl; w < W;
             w += (unsigned long long)gx * rp) {
            const float x = xs[w * D + d0 + dl];
            unsigned int bin = (unsigned int)((x - lower) / (upper - lower) * BAY_HIST_BINS);
            bin = (bin < BAY_HIST_BINS) ? bin : BAY_HIST_BINS - 1;
            atomicAdd(&h[dl * BAY_HIST_BINS + bin], 1u);
        }
    }
    __syncthreads();
    for (unsigned int b = threadIdx.x; b < dt * BAY_HIST_BINS; b += 256u)
        if (h[b]) atomicAdd(&counts[(unsigned long long)d0 * BAY_HIST_BINS + b], h[b]);
}
