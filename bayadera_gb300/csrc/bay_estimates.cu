// bay_estimates.cu -- per-dimension estimates of a walker-major (point-major) matrix
// x[w * D + d], W points of D coordinates: FP64 moments, limits, the integer histogram with
// its bitonic ranks.  Used on a sampler's walkers and on data matrices alike.
//
// Every kernel reads x where it lies, once a pass, in the flat order: a CTA owns a tile of
// dt dimensions (at most 64 for the sums and limits) and rp = 256 / dt rows a pass, thread t
// working for dimension t % dt on row t / dt, so a warp's loads are consecutive words and a
// thread's dimension never changes.  gx CTAs share a dimension tile's rows (about 4 CTAs an SM over the grid,
// at least 16 elements a thread); their partial results go to the context's workspace and
// the tile's last CTA (a ticket, reset for the next launch) combines them in CTA order, so
// the result does not depend on which CTA that is.
// The earlier kernels took a dimension-major copy of the matrix (a transpose per call, as
// large as the data) and ran one CTA a dimension: 4,194,315 x 6 values took 7,546 us for the
// moments and 3,297 us for the limits (6 of 152 SMs at work), and 222 us a transpose.
#include "bay_kernels.cuh"

namespace {

constexpr uint32_t kThreads = 256;
constexpr uint32_t kBatch = 16;         // elements a thread has in flight, and sums in fp32

// The CTA's place: dimension tile [d0, d0 + dt) and share bx of gx of the rows; the thread's
// dimension d0 + dl and first row r0, the next ones `stride` rows on.
struct Place {
    uint32_t d0, dt, dl, bx, by;
    uint32_t rp, rl;
    uint64_t r0, stride;
    bool on;
};
__device__ __forceinline__ Place place_of(uint32_t D, uint32_t gx, uint32_t tile) {
    Place p;
    p.by = blockIdx.x / gx;
    p.bx = blockIdx.x - p.by * gx;
    p.d0 = p.by * tile;
    p.dt = D - p.d0 < tile ? D - p.d0 : tile;
    p.rp = kThreads / p.dt;
    p.rl = threadIdx.x / p.dt;
    p.dl = threadIdx.x - p.rl * p.dt;
    p.on = p.rl < p.rp;
    p.r0 = (uint64_t)p.bx * p.rp + p.rl;
    p.stride = (uint64_t)gx * p.rp;
    return p;
}

// The thread's kBatch values from row r on (`none` past the last row), all loads in flight.
__device__ __forceinline__ void load_batch(float (&v)[kBatch], const float* col, uint64_t r,
                                           uint64_t stride, uint64_t W, uint32_t D, float none) {
    if (r + (kBatch - 1) * stride < W) {
        const float* q = col + r * D;
        const uint64_t step = stride * D;
#pragma unroll
        for (uint32_t i = 0; i < kBatch; ++i) v[i] = __ldg(q + i * step);
    } else {
#pragma unroll
        for (uint32_t i = 0; i < kBatch; ++i) v[i] = r + i * stride < W ? __ldg(col + (r + i * stride) * D) : none;
    }
}

// red[thread] summed over the rows of each dimension in a fixed tree; the sum of dimension
// dl is in red[dl].
__device__ __forceinline__ void rows_sum(const Place& p, double* red) {
    uint32_t o = 1;
    while (o < p.rp) o <<= 1;
    for (o >>= 1; o > 0; o >>= 1) {
        __syncthreads();
        if (p.on && p.rl < o && p.rl + o < p.rp) red[threadIdx.x] += red[threadIdx.x + o * p.dt];
    }
    __syncthreads();
}

// Whether this CTA is the last of its tile's gx to get here (every CTA's earlier writes are
// then visible to it); the ticket is left at 0 for the next launch.
__device__ __forceinline__ bool last_of_tile(uint32_t* ticket, uint32_t gx) {
    __shared__ uint32_t s_last;
    if (gx == 1) return true;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        s_last = atomicAdd(ticket, 1u) == gx - 1u ? 1u : 0u;
        if (s_last) *ticket = 0u;
    }
    __syncthreads();
    __threadfence();
    return s_last != 0u;
}

// s + x as a sum and its exact rounding error (Knuth's TwoSum), the error into e.
__device__ __forceinline__ void two_sum(float& s, float& e, float x) {
    const float t = __fadd_rn(s, x);
    const float b = __fsub_rn(t, s);
    e = __fadd_rn(e, __fadd_rn(__fsub_rn(s, __fsub_rn(t, b)), __fsub_rn(x, b)));
    s = t;
}

// Pass MODE of the moments: 0 sums x (mean[d] = sum / W), 1 sums (x - c)^2 and x - c about
// c, the mean rounded to fp32: var[d] = sum (x - c)^2 / W - (sum (x - c) / W)^2, the
// population variance (c is the float next to the mean: the subtrahend never exceeds about
// the variance itself, and is some 2^-48 mean^2).
// FP64 issue is 1/64 of fp32 here (1.9 operations a clock an SM), and an FP64 conversion and
// addition an element held the pass to 0.83 elements a clock an SM, a sixth of what HBM
// delivers.  So the sums are fp32 words with their exact rounding errors beside them
// (fp_sum), flushed to the FP64 accumulators every kFlush elements: 6 or 10 FP64 operations
// per 64 elements.  Variances of 1,000 to 4,194,304 values against 128 bits: 2.3e-16 off at
// most, a run of FP64 additions 5.3e-16.  Batches that fp32 cannot hold (largest |x - c|
// outside [1e-12, 1e15], an infinity, NaN, an overflow) take FP64 throughout.
// 4,194,315 x 6 values: some 40 us the sum and 65 us the squares, against 7,546 us for both with
// one CTA a dimension and FP64 throughout.
constexpr uint32_t kFlush = 64;
struct fp_sum {
    float s = 0.0f;                             // sum
    float e = 0.0f, l = 0.0f;                   // errors of s and of the products, and of e
    float s1 = 0.0f, e1 = 0.0f;                 // MODE 1: sum of x - c, its errors
    template <int MODE>
    __device__ __forceinline__ void add(float x, float c, float& top) {
        if (MODE == 0) {
            float d = 0.0f;
            two_sum(s, d, x);
            two_sum(e, l, d);
            return;
        }
        float t = x, te = 0.0f;
        two_sum(t, te, -c);                     // t + te = x - c, exactly
        top = fmaxf(top, fabsf(t));
        two_sum(s1, e1, t);
        e1 = __fadd_rn(e1, te);
        // (t + te)^2 = q + qe + p + pe + te^2, the first four exact
        const float q = __fmul_rn(t, t), qe = __fmaf_rn(t, t, -q);
        const float t2 = __fadd_rn(t, t), p = __fmul_rn(t2, te), pe = __fmaf_rn(t2, te, -p);
        // (the errors of s go to e as well: a plain fp32 sum of them would be 2^-49 of s off,
        // all one way for a skewed column)
        float d = 0.0f;
        two_sum(s, d, q);
        two_sum(e, l, d);
        two_sum(e, l, qe);
        two_sum(e, l, p);
        l = __fadd_rn(l, __fmaf_rn(te, te, pe));
    }
    template <int MODE>
    __device__ __forceinline__ bool good(float top) const {
        const float f = MODE == 0 ? s + e : (s + e) + (s1 + e1);
        return isfinite(f) && (MODE == 0 || top == 0.0f || (top >= 1e-12f && top <= 1e15f));
    }
    template <int MODE>
    __device__ __forceinline__ void flush(double* acc) {
        acc[0] += (double)s;
        acc[0] += (double)e;
        acc[0] += (double)l;
        if (MODE == 1) {
            acc[MODE] += (double)s1;
            acc[MODE] += (double)e1;
        }
        *this = fp_sum();
    }
};

// The CTA's sums of its share of dimension p.dl, in `total` of every thread of that dimension:
// MODE 0 of x, MODE 1 of (x - c)^2 and x - c.
template <int MODE>
__device__ __forceinline__ void moments_share(const Place& p, const float* __restrict__ x, uint32_t D,
                                              uint64_t W, float c, double* red,
                                              double (&total)[MODE + 1]) {
    double acc[MODE + 1] = {};
    if (p.on) {
        const float* col = x + p.d0 + p.dl;
        fp_sum f;
        uint32_t held = 0;
        float ahead[kBatch];
        load_batch(ahead, col, p.r0, p.stride, W, D, c);
        for (uint64_t r = p.r0; r < W; r += kBatch * p.stride) {
            float v[kBatch];
#pragma unroll
            for (uint32_t i = 0; i < kBatch; ++i) v[i] = ahead[i];
            load_batch(ahead, col, r + kBatch * p.stride, p.stride, W, D, c);
            const fp_sum before = f;
            float top = 0.0f;
#pragma unroll
            for (uint32_t i = 0; i < kBatch; ++i) f.add<MODE>(v[i], c, top);
            if (!f.good<MODE>(top)) {
                f = before;
#pragma unroll 1
                for (uint32_t i = 0; i < kBatch && r + i * p.stride < W; ++i) {
                    const double t = (double)__ldg(col + (r + i * p.stride) * D) - (double)c;
                    acc[0] += MODE == 0 ? t : t * t;
                    if (MODE == 1) acc[MODE] += t;
                }
            }
            held += kBatch;
            if (held >= kFlush) {
                f.flush<MODE>(acc);
                held = 0;
            }
        }
        f.flush<MODE>(acc);
    }
#pragma unroll
    for (int q = 0; q <= MODE; ++q) {
        red[threadIdx.x] = acc[q];
        rows_sum(p, red);
        total[q] = red[p.dl];
        __syncthreads();
    }
}

__device__ __forceinline__ double variance_of(const double (&total)[2], uint64_t W) {
    const double m = total[0] / (double)W, u = total[1] / (double)W;
    const double v = m - u * u;
    return v < 0.0 ? 0.0 : v;
}

template <int MODE>
__global__ void __launch_bounds__(kThreads)
moments_pass(const float* __restrict__ x, uint32_t D, uint64_t W, uint32_t gx, uint32_t tile,
             double* mean, double* var, double* part, uint32_t* tickets) {
    __shared__ double red[kThreads];
    const Place p = place_of(D, gx, tile);
    const float c = MODE == 1 && p.on ? (float)mean[p.d0 + p.dl] : 0.0f;
    double total[MODE + 1];
    moments_share<MODE>(p, x, D, W, c, red, total);
    if (gx > 1) {
        double* mine = part + ((uint64_t)p.d0 + p.dl) * gx * (MODE + 1);   // [dim][CTA][sum]
        if (p.on && p.rl == 0)
#pragma unroll
            for (int q = 0; q <= MODE; ++q) mine[(uint64_t)p.bx * (MODE + 1) + q] = total[q];
        if (!last_of_tile(&tickets[p.by], gx)) return;
#pragma unroll
        for (int q = 0; q <= MODE; ++q) {
            double a = 0.0;
            if (p.on)
                for (uint32_t b = p.rl; b < gx; b += kBatch * p.rp) {
                    double w[kBatch];       // their loads all in flight: this tail is alone
#pragma unroll
                    for (uint32_t i = 0; i < kBatch; ++i)
                        w[i] = b + i * p.rp < gx ? __ldcg(&mine[(uint64_t)(b + i * p.rp) * (MODE + 1) + q]) : 0.0;
#pragma unroll
                    for (uint32_t i = 0; i < kBatch; ++i) a += w[i];
                }
            red[threadIdx.x] = a;
            rows_sum(p, red);
            total[q] = red[p.dl];
            __syncthreads();
        }
    }
    if (p.on && p.rl == 0) {
        if constexpr (MODE == 0) mean[p.d0 + p.dl] = total[0] / (double)W;
        else var[p.d0 + p.dl] = variance_of(total, W);
    }
}

// Both passes where a CTA has all rows of its dimensions.
__global__ void __launch_bounds__(kThreads)
moments_both(const float* __restrict__ x, uint32_t D, uint64_t W, uint32_t tile, double* mean, double* var) {
    __shared__ double red[kThreads];
    const Place p = place_of(D, 1u, tile);
    double sum[1], sq[2];
    moments_share<0>(p, x, D, W, 0.0f, red, sum);
    const double mu = sum[0] / (double)W;
    moments_share<1>(p, x, D, W, (float)mu, red, sq);
    if (p.on && p.rl == 0) {
        mean[p.d0 + p.dl] = mu;
        var[p.d0 + p.dl] = variance_of(sq, W);
    }
}

// Limits [min, max] of every dimension (NaN values are passed over, a column of NaN alone
// gives NaN); zero_fold folds 0.0 in (reference Q7).  counts, when given, is set to `start`.
__global__ void __launch_bounds__(kThreads)
limits_pass(const float* __restrict__ x, uint32_t D, uint64_t W, uint32_t gx, uint32_t tile,
            int zero_fold, float* limits, float2* part, uint32_t* tickets, uint32_t* counts,
            uint64_t n_counts, uint32_t start, uint32_t n_limits) {
    __shared__ float2 red[kThreads];
    for (uint64_t i = blockIdx.x * (uint64_t)kThreads + threadIdx.x; i < n_counts;
         i += (uint64_t)gridDim.x * kThreads)
        counts[i] = start;
    if (blockIdx.x >= n_limits) return;      // there for the counts alone
    const Place p = place_of(D, gx, tile);
    const float nan = __int_as_float(0x7fc00000);
    float mn = nan, mx = nan;
    if (p.on) {
        const float* col = x + p.d0 + p.dl;
        float ahead[kBatch];
        load_batch(ahead, col, p.r0, p.stride, W, D, nan);
        for (uint64_t r = p.r0; r < W; r += kBatch * p.stride) {
            float v[kBatch];
#pragma unroll
            for (uint32_t i = 0; i < kBatch; ++i) v[i] = ahead[i];
            load_batch(ahead, col, r + kBatch * p.stride, p.stride, W, D, nan);
#pragma unroll
            for (uint32_t i = 0; i < kBatch; ++i) {
                mn = fminf(mn, v[i]);
                mx = fmaxf(mx, v[i]);
            }
        }
    }
    for (int level = 0; level < 2; ++level) {
        red[threadIdx.x] = make_float2(mn, mx);
        uint32_t o = 1;
        while (o < p.rp) o <<= 1;
        for (o >>= 1; o > 0; o >>= 1) {
            __syncthreads();
            if (p.on && p.rl < o && p.rl + o < p.rp) {
                const float2 a = red[threadIdx.x], b = red[threadIdx.x + o * p.dt];
                red[threadIdx.x] = make_float2(fminf(a.x, b.x), fmaxf(a.y, b.y));
            }
        }
        __syncthreads();
        if (level == 1 || gx == 1) break;
        if (p.on && p.rl == 0) part[(uint64_t)p.bx * D + p.d0 + p.dl] = red[p.dl];
        if (!last_of_tile(&tickets[p.by], gx)) return;
        mn = mx = nan;
        if (p.on)
            for (uint32_t b = p.rl; b < gx; b += kBatch * p.rp) {
                float2 q[kBatch];
#pragma unroll
                for (uint32_t i = 0; i < kBatch; ++i)
                    q[i] = __ldcg(&part[(uint64_t)(b + i * p.rp < gx ? b + i * p.rp : b) * D + p.d0 + p.dl]);
#pragma unroll
                for (uint32_t i = 0; i < kBatch; ++i) {
                    mn = fminf(mn, q[i].x);
                    mx = fmaxf(mx, q[i].y);
                }
            }
    }
    if (p.on && p.rl == 0) {
        const float2 q = red[p.dl];
        limits[2 * (uint64_t)(p.d0 + p.dl)] = zero_fold ? fminf(q.x, 0.0f) : q.x;
        limits[2 * (uint64_t)(p.d0 + p.dl) + 1] = zero_fold ? fmaxf(q.y, 0.0f) : q.y;
    }
}

// histogram (nvidia-gtx-estimate.cu:5-32): bin = (uint)((x - lo)/(hi - lo) * bins) with
// IEEE division and the saturating float->uint conversion, clamped to bins - 1.
// The CTA's dimension tile has dt * bins shared-memory counts (12,288 at most, 48 KB), in
// `copies` copies over the warps where they are few; one global atomic per non-empty bin.
__global__ void __launch_bounds__(kThreads)
hist_count(const float* __restrict__ x, uint32_t D, uint64_t W, uint32_t gx, uint32_t tile,
           uint32_t bins, uint32_t copies, const float* limits, uint32_t* counts) {
    extern __shared__ uint32_t h[];
    const Place p = place_of(D, gx, tile);
    const uint32_t nh = p.dt * bins;
    for (uint32_t b = threadIdx.x; b < nh * copies; b += kThreads) h[b] = 0;
    __syncthreads();
    if (p.on) {
        const float lo = limits[2 * (uint64_t)(p.d0 + p.dl)], hi = limits[2 * (uint64_t)(p.d0 + p.dl) + 1];
        const float range = __fsub_rn(hi, lo);
        const float fb = (float)bins;
        uint32_t* mine = h + ((threadIdx.x >> 5) % copies) * nh + p.dl * bins;
        const float* col = x + p.d0 + p.dl;
        float ahead[kBatch];
        load_batch(ahead, col, p.r0, p.stride, W, D, 0.0f);
        for (uint64_t r = p.r0; r < W; r += kBatch * p.stride) {
            float v[kBatch];
            const bool full = r + (kBatch - 1) * p.stride < W;
#pragma unroll
            for (uint32_t i = 0; i < kBatch; ++i) v[i] = ahead[i];
            load_batch(ahead, col, r + kBatch * p.stride, p.stride, W, D, 0.0f);
#pragma unroll
            for (uint32_t i = 0; i < kBatch; ++i) {
                const float q = __fmul_rn(__fdiv_rn(__fsub_rn(v[i], lo), range), fb);
                uint32_t b = __float2uint_rz(q);
                b = b < bins ? b : bins - 1;
                if (full || r + i * p.stride < W) atomicAdd(&mine[b], 1u);
            }
        }
    }
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < nh; b += kThreads) {
        uint32_t n = 0;
        for (uint32_t k = 0; k < copies; ++k) n += h[k * nh + b];
        if (n) atomicAdd(&counts[(uint64_t)p.d0 * bins + b], n);
    }
}

// uint_to_real (nvidia-gtx-estimate.cu:34-44) and bitonic_local (:117-147): the
// reference's compare-exchange network over (bin, pdf) pairs, decreasing pdf; equal
// pdfs count as "smaller" when the partner position j is below lid.
__global__ void hist_finish(const uint32_t* counts, const float* limits, uint32_t bins,
                            float alpha, float* pdf, float* ranks) {
    extern __shared__ float2 aux[];
    const uint32_t d = blockIdx.x, lid = threadIdx.x;
    const float c = __fdiv_rn(alpha, __fsub_rn(limits[2 * d + 1], limits[2 * d]));
    const float p = __fmul_rn(c, (float)counts[(uint64_t)d * bins + lid]);
    pdf[(uint64_t)d * bins + lid] = p;
    float2 v = make_float2((float)lid, p);
    aux[lid] = v;
    __syncthreads();
    for (uint32_t length = 1; length < bins; length <<= 1) {
        const bool direction = (lid & (length << 1)) != 0;
        for (uint32_t inc = length; inc > 0; inc >>= 1) {
            const uint32_t j = lid ^ inc;
            const float2 o = aux[j];
            const bool smaller = (v.y < o.y) || (o.y == v.y && j < lid);
            const bool swap = smaller ^ (j < lid) ^ direction;
            v = swap ? o : v;
            __syncthreads();
            aux[lid] = v;
            __syncthreads();
        }
    }
    ranks[(uint64_t)d * bins + lid] = v.x;
}

}  // namespace

namespace bay {

// tiles of at most tile_max dimensions, shares of at least rows_min rows
est_plan est_plan_of(uint32_t D, uint64_t W, uint32_t tile_max, uint64_t rows_min) {
    est_plan p;
    uint32_t tile = tile_max < kThreads ? tile_max : kThreads;
    if (tile < 1) tile = 1;
    const uint32_t gy = (uint32_t)(((uint64_t)D + tile - 1) / tile);
    p.tile = (uint32_t)(((uint64_t)D + gy - 1) / gy);      // equal tiles
    p.gy = (uint32_t)(((uint64_t)D + p.tile - 1) / p.tile);
    const uint64_t rp = kThreads / p.tile;
    uint64_t per = rp * kBatch;                            // rows a CTA has at least
    if (per < rows_min) per = rows_min;
    const uint64_t gx = (W + per - 1) / per;
    const uint64_t most = p.gy >= kEstCtas ? 1 : kEstCtas / p.gy;   // 4 CTAs an SM
    p.gx = (uint32_t)(gx < most ? (gx < 1 ? 1 : gx) : most);
    return p;
}

constexpr uint64_t kAlone = 64 * kThreads;     // values that a CTA takes alone: 64 a thread

// The moments' and limits' plan.  A CTA's last one of a tile adds up gx partial results a
// dimension (FP64 issue: 2,048 of them take 0.6 us, and it is alone then), so with many CTAs the
// tiles are as narrow as keeps gx * tile below that (8 dimensions, a 32-byte sector, to 64); with
// few, so narrow that one CTA has all rows of its dimensions and no others to wait for, at up to
// 64 values a thread.  Moments
// of 4,096 x 256, 65,536 x 100 and 1,000 x 20 values on the device, in tiles of up to 256
// dimensions 100, 102 and 51 us a call, now 53, 77 and 38.
est_plan sums_plan_of(uint32_t D, uint64_t W) {
    // CTAs, of a batch a thread at least
    uint64_t n = W > (uint64_t)kEstCtas * kThreads * kBatch ? kEstCtas : W * D / (kThreads * kBatch) + 1;
    if (n > kEstCtas) n = kEstCtas;
    uint64_t tile = 8;
    if (n <= kEstCtas / 4) {
        tile = (D + n - 1) / n;
        if (tile > 64) tile = 64;
        while (tile > 1 && W * tile > kAlone) tile = (tile + 1) / 2;
        return est_plan_of(D, W, (uint32_t)tile, W * tile <= kAlone ? W : 0);
    }
    while (tile < 64 && n * (tile + 8) * (tile + 8) <= 2048ull * D) tile += 8;
    return est_plan_of(D, W, (uint32_t)tile, 0);
}

size_t est_workspace(uint32_t D, uint64_t W) {
    const est_plan p = sums_plan_of(D, W);
    return kEstTickets * sizeof(uint32_t) + 2 * sizeof(double) * (size_t)p.gx * D;
}

cudaError_t launch_moments(const float* x, uint32_t D, uint64_t W, double* mean, double* var,
                           void* ws, cudaStream_t s) {
    const est_plan p = sums_plan_of(D, W);
    uint32_t* tickets = static_cast<uint32_t*>(ws);
    double* part = reinterpret_cast<double*>(tickets + kEstTickets);
    if (var && p.gx == 1) {
        moments_both<<<p.gy, kThreads, 0, s>>>(x, D, W, p.tile, mean, var);
        count_launches(1);
        return cudaGetLastError();
    }
    moments_pass<0><<<p.gx * p.gy, kThreads, 0, s>>>(x, D, W, p.gx, p.tile, mean, var, part, tickets);
    count_launches(1);
    if (var) {
        moments_pass<1><<<p.gx * p.gy, kThreads, 0, s>>>(x, D, W, p.gx, p.tile, mean, var, part, tickets);
        count_launches(1);
    }
    return cudaGetLastError();
}

cudaError_t launch_limits(const float* x, uint32_t D, uint64_t W, int zero_fold, float* limits,
                          uint32_t* counts, uint64_t n_counts, uint32_t start, void* ws,
                          cudaStream_t s) {
    const est_plan p = sums_plan_of(D, W);
    uint32_t* tickets = static_cast<uint32_t*>(ws);
    // 16 counts a thread at least, by CTAs of their own where the limits' are too few
    uint64_t ctas = (n_counts + kThreads * 16 - 1) / (kThreads * 16);
    if (ctas > kEstCtas) ctas = kEstCtas;
    if (ctas < (uint64_t)p.gx * p.gy) ctas = (uint64_t)p.gx * p.gy;
    limits_pass<<<(uint32_t)ctas, kThreads, 0, s>>>(x, D, W, p.gx, p.tile, zero_fold, limits,
                                                    reinterpret_cast<float2*>(tickets + kEstTickets),
                                                    tickets, counts, n_counts, start, p.gx * p.gy);
    count_launches(1);
    return cudaGetLastError();
}

est_plan hist_plan_of(uint32_t D, uint64_t W, uint32_t bins) {
    // a CTA's rows are at least eight times its bins, so that the counts it adds at the end
    // are few beside the values it bins; where that leaves fewer than two CTAs an SM, narrower
    // tiles of dimensions (down to a 32-byte sector) make more.  12,290 x 37 values into 256
    // bins: 8.6 us against 17.8 us in one tile of 37 and 24 row shares
    uint32_t tile = kHistCounts / bins;
    est_plan p = est_plan_of(D, W, tile, 8ull * bins);
    while (p.gx * p.gy < kEstCtas / 2 && p.tile > 8) {
        tile = (p.tile + 1) / 2;
        p = est_plan_of(D, W, tile, 8ull * bins);
    }
    const uint32_t room = kHistCounts / (p.tile * bins);
    p.copies = room < 1 ? 1 : room < kThreads / 32 ? room : kThreads / 32;
    return p;
}

cudaError_t launch_hist_count(const float* x, uint32_t D, uint64_t W, uint32_t bins,
                              const float* limits, uint32_t* counts, cudaStream_t s) {
    const est_plan p = hist_plan_of(D, W, bins);
    hist_count<<<p.gx * p.gy, kThreads, sizeof(uint32_t) * p.tile * bins * p.copies, s>>>(
        x, D, W, p.gx, p.tile, bins, p.copies, limits, counts);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_hist_finish(const uint32_t* counts, const float* limits, uint32_t D,
                               uint32_t bins, uint64_t n, float* pdf, float* ranks,
                               cudaStream_t s) {
    const float alpha = (float)((double)bins / (double)n);
    hist_finish<<<D, bins, bins * sizeof(float2), s>>>(counts, limits, bins, alpha, pdf, ranks);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace bay
