// bay_kernels.cu -- nvcc-compiled kernels of the stretch-move engine: walker init, the GEMM
// forms' matrix layouts, per-step means, acor, and the device-resident control block.  The
// estimates are in bay_estimates.cu, the per-model fused stretch kernels in
// device/bay_stretch.cuh (NVRTC).
#include <cooperative_groups.h>

#include <atomic>

#include "bay_kernels.cuh"
#include "device/bay_normal.cuh"
#include "device/bay_rng.cuh"

namespace {

constexpr unsigned FULL = 0xffffffffu;

// Fixed-order block sum of a double (deterministic); all threads get the result.
__device__ double block_sum_d(double v, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(FULL, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
        red[32] = s;
    }
    __syncthreads();
    const double r = red[32];
    __syncthreads();
    return r;
}

__global__ void ctl_apply(bay_ctl* c, bay_ctl_op op) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const unsigned m = op.mask;
    if (m & BAY_CTL_SET_STEP0) c->step[0] = op.step[0];
    if (m & BAY_CTL_SET_STEP1) c->step[1] = op.step[1];
    if (m & BAY_CTL_ADD_STEP0) c->step[0] += op.step[0];
    if (m & BAY_CTL_ADD_STEP1) c->step[1] += op.step[1];
    if (m & BAY_CTL_SET_SEED0) c->seed[0] = op.seed[0];
    if (m & BAY_CTL_SET_SEED1) c->seed[1] = op.seed[1];
    if (m & BAY_CTL_SET_A) c->a = op.a;
    if (m & BAY_CTL_SET_BETA) c->beta = op.beta;
    if (m & BAY_CTL_RESET_ACCEPTED) c->accepted = 0ull;
    if (m & BAY_CTL_RESET_TICKETS) {
        c->ticket[0] = 0u;
        c->ticket[1] = 0u;
    }
}

// mix!'s a-adaptation probes (mcmc.clj:84-91): init-move! before the probe's accu step,
// the loop's rule after it.  The rule runs in FP64 with explicit IEEE operations (no fused
// multiply-add), so a follows the same sequence as the host loop.
__global__ void mix_begin(bay_ctl* c, const bay_mix_state* st) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    c->seed[1] += 2u;
    c->step[1] = 0u;
    c->a = (float)st->a;
    c->accepted = 0ull;
    c->ticket[0] = 0u;
    c->ticket[1] = 0u;
}

__global__ void mix_end(bay_ctl* c, bay_mix_state* st, unsigned long long W, unsigned int step,
                        double min_acc, double max_acc, cudaGraphConditionalHandle cont) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    c->step[1] += 1u;                                   // the probe's one accu step
    const double r = __ddiv_rn((double)c->accepted, (double)W);
    const double target = __ddiv_rn(__dadd_rn(max_acc, min_acc), 2.0);
    st->rate = r;
    st->probes += 1u;
    unsigned int go = 0u;
    if (!(step < st->i)) {
        if (r < min_acc) {
            st->a = __dadd_rn(1.0, __dmul_rn(__dsub_rn(st->a, 1.0), __ddiv_rn(r, target)));
            go = 1u;
        } else if (max_acc < r) {
            st->a = __dmul_rn(st->a, __ddiv_rn(r, target));
            go = 1u;
        }
        if (go) st->i += 1u;
        if (go && !((float)st->a > 1.0f)) {
            st->bad = 1u;
            go = 0u;
        }
    }
    cudaGraphSetConditional(cont, go);
}

// init_walkers (nvidia-gtx-mcmc-stretch.cu:158-195): element e = w*D + d (the
// reference's AoS index) takes word e%4 of Philox(ctr {e/4, 0xf00dcafe, 0xdeadbeef,
// 0xbeeff00d}, key {seed, 0xdecafaaa}); x = u*hi + (1-u)*lo, first product fused.
// The walker state is walker-major, so element e is written at xs[e] (coalesced).
__global__ void init_uniform(float* xs, uint32_t D, uint64_t W, uint32_t seed,
                             const float* limits) {
    const uint64_t n = (uint64_t)D * W;
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < n;
         e += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t d = e % D;
        bay_u4 c;
        c.x = (unsigned)(e >> 2);
        c.y = 0xf00dcafeu;
        c.z = 0xdeadbeefu;
        c.w = 0xbeeff00du;
        const bay_u4 r = bay_philox4x32_10(c, seed, 0xdecafaaau);
        const unsigned word = (e & 3) == 0 ? r.x : (e & 3) == 1 ? r.y : (e & 3) == 2 ? r.z : r.w;
        const float u = bay_u01(word);
        const float lo = limits[2 * d], hi = limits[2 * d + 1];
        xs[e] = __fmaf_rn(u, hi, __fmul_rn(__fsub_rn(1.0f, u), lo));
    }
}

// N(mean, sd^2) init: element e = w*D + d uses pair p = e/2, Philox(ctr {p, 0x6e6f726d,
// 0x77616c6b, 0xbeeff00d}, key {seed, 0x9a55a9e5}); Box-Muller in FP64 on words 0, 1, the
// even element the cosine's.  A thread makes a pair, in pairs of floats where their bound
// settles the rounding (device/bay_normal.cuh), else in FP64, whose issue bounded the kernel:
// 3,276,800 elements 263 us (500 us one element a thread), now 27.  Members (off, count,
// seed): blockIdx.y's block of count values at off, so that a batch of samplers is one launch.
__device__ __forceinline__ void normal_pairs(float* xs, uint64_t n, uint32_t seed, float mean,
                                             float sd) {
    for (uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; 2 * p < n;
         p += (uint64_t)gridDim.x * blockDim.x) {
        bay_u4 ctr;
        ctr.x = (unsigned)p;
        ctr.y = 0x6e6f726du;
        ctr.z = 0x77616c6bu;
        ctr.w = 0xbeeff00du;
        const bay_u4 r = bay_philox4x32_10(ctr, seed, 0x9a55a9e5u);
        const float u0 = bay_u01(r.x), u1 = bay_u01(r.y);
        const bay_df radius = bay_df_radius(u1);
        bay_df c, s;
        bay_df_circle(u0, c, s);
        float x0, x1;
        const bool ok0 = bay_df_normal(mean, sd, radius, c, &x0);
        const bool ok1 = bay_df_normal(mean, sd, radius, s, &x1);
        if (!(ok0 && ok1)) {
            const double rr = sqrt(-2.0 * log((double)u1));
            const double t = 6.283185307179586 * (double)u0;
            x0 = (float)((double)mean + (double)sd * (rr * cos(t)));
            x1 = (float)((double)mean + (double)sd * (rr * sin(t)));
        }
        xs[2 * p] = x0;
        if (2 * p + 1 < n) xs[2 * p + 1] = x1;
    }
}
__global__ void init_normal(float* xs, uint64_t n, uint32_t seed, float mean, float sd) {
    normal_pairs(xs, n, seed, mean, sd);
}
__global__ void init_normal_members(float* xs, const bay_init_member* mem, float mean, float sd) {
    const bay_init_member m = mem[blockIdx.y];
    normal_pairs(xs + m.off, m.count, m.seed, mean, sd);
}

// One CTA per (step, dim): the 2 x G per-CTA sums part[((t*2 + h)*D + d)*G + b] read
// coalesced along b, summed in FP64 in a fixed order.
__global__ void reduce_means(const bay_ctl* ctl, const float* part, float* means,
                             uint32_t means_cap, uint32_t G, uint32_t D, double inv_W) {
    __shared__ double red[33];
    const uint32_t t = blockIdx.x, d = blockIdx.y;
    const uint32_t step = ctl->step[1] + t;
    double s = 0.0;
    for (uint32_t h = 0; h < 2; ++h) {
        const float* p = part + (((size_t)t * 2 + h) * D + d) * G;
        for (uint32_t b = threadIdx.x; b < G; b += blockDim.x) s += (double)p[b];
    }
    s = block_sum_d(s, red);
    if (threadIdx.x == 0 && step < means_cap) means[(size_t)step * D + d] = (float)(s * inv_W);
}

// The GEMM form's matrix laid out once per sampler: lay[f*NP + r] = A[r][f] (rows past
// `rows` zero), then lay[F*NP + r*auxs + c] = A[r][aux_col + c].
__global__ void gemm_layout(const float* A, uint64_t ld, uint32_t rows, uint32_t F, uint32_t NP,
                            uint32_t aux_col, uint32_t aux_len, uint32_t auxs, float* lay) {
    const uint64_t nA = (uint64_t)F * NP;
    const uint64_t n = nA + (uint64_t)NP * auxs;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        float v = 0.0f;
        if (i < nA) {
            const uint64_t f = i / NP, r = i % NP;
            if (r < rows) v = A[r * ld + f];
        } else {
            const uint64_t e = i - nA, r = e / auxs, c = e % auxs;
            if (r < rows && c < aux_len) v = A[r * ld + aux_col + c];
        }
        lay[i] = v;
    }
}

// bf16 of a float rounded to nearest even, as its 16 bits (NaN stays a quiet NaN)
__device__ __forceinline__ unsigned short bf16_rn(float x) {
    unsigned int u = __float_as_uint(x);
    if ((u & 0x7fffffffu) > 0x7f800000u) return (unsigned short)((u >> 16) | 0x40u);
    u += 0x7fffu + ((u >> 16) & 1u);
    return (unsigned short)(u >> 16);
}

// Tensor-core GEMM form: the matrix as bf16 hi + lo, row-major [rows_pad][Fp] (features
// past F and rows past `rows` zero), and the rows' aux values [rows_pad][auxs].
__global__ void gemm_split(const float* A, uint64_t ld, uint32_t rows, uint32_t F, uint32_t Fp,
                           uint64_t rows_pad, uint32_t aux_col, uint32_t aux_len, uint32_t auxs,
                           unsigned short* hi, unsigned short* lo, float* aux) {
    const uint64_t nA = rows_pad * Fp, n = nA + rows_pad * auxs;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        if (i < nA) {
            const uint64_t r = i / Fp, f = i % Fp;
            const float v = (r < rows && f < F) ? A[r * ld + f] : 0.0f;
            const unsigned short h = bf16_rn(v);
            hi[i] = h;
            lo[i] = bf16_rn(__fsub_rn(v, __uint_as_float((unsigned int)h << 16)));
        } else {
            const uint64_t e = i - nA, r = e / auxs, c = e % auxs;
            aux[e] = (r < rows && c < aux_len) ? A[r * ld + aux_col + c] : 0.0f;
        }
    }
}

// Resident tensor-core GEMM form: the matrix as the MMA's B operand -- bf16 hi atoms then
// lo atoms, each atom [NP rows][64 features] in 128-byte rows with 16-byte unit u of row r
// stored at unit u ^ (r % 8) -- followed by the rows' aux values [NP][auxs]; rows past
// `rows` and features past F are zero.
__global__ void gemm_tc_image(const float* A, uint64_t ld, uint32_t rows, uint32_t F, uint32_t KC,
                              uint32_t NP, uint32_t aux_col, uint32_t aux_len, uint32_t auxs,
                              unsigned char* img) {
    const uint64_t n_units = (uint64_t)KC * NP * 8;      // 16-byte units per hi (or lo) block
    const uint64_t n = n_units + (uint64_t)NP * auxs;
    const uint64_t lo_off = n_units * 16;
    float* aux = reinterpret_cast<float*>(img + 2 * lo_off);
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        if (i < n_units) {
            const uint32_t c = (uint32_t)(i / ((uint64_t)NP * 8));
            const uint32_t rem = (uint32_t)(i - (uint64_t)c * NP * 8);
            const uint32_t r = rem >> 3, u = rem & 7u;
            unsigned int hw[4], lw[4];
            for (int q = 0; q < 4; ++q) {
                unsigned int hh[2], ll[2];
                for (int j = 0; j < 2; ++j) {
                    const uint32_t f = c * 64u + u * 8u + 2u * q + j;
                    const float v = (r < rows && f < F) ? A[(uint64_t)r * ld + f] : 0.0f;
                    const unsigned short h = bf16_rn(v);
                    hh[j] = h;
                    ll[j] = bf16_rn(__fsub_rn(v, __uint_as_float((unsigned int)h << 16)));
                }
                hw[q] = hh[0] | (hh[1] << 16);
                lw[q] = ll[0] | (ll[1] << 16);
            }
            const uint64_t off = (uint64_t)c * NP * 128 + (uint64_t)r * 128 + ((u ^ (r & 7u)) << 4);
            *reinterpret_cast<uint4*>(img + off) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
            *reinterpret_cast<uint4*>(img + lo_off + off) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
        } else {
            const uint64_t e = i - n_units, r = e / auxs, cc = e % auxs;
            aux[e] = (r < rows && cc < aux_len) ? A[r * ld + aux_col + cc] : 0.0f;
        }
    }
}

__global__ void fill_bytes(uint4* p, uint64_t n16, unsigned int v) {
    const uint4 q = make_uint4(v, v, v, v);
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n16;
         i += (uint64_t)gridDim.x * blockDim.x)
        p[i] = q;
}

// acor (nvidia-gtx-acor.cu:116-168 + nvidia_gtx.clj:240-278), a cluster of C CTAs a
// dimension, no dynamic parallelism: mean, centring, the first pass, then pairwise halving
// while 10 < lag2 and lag2 < 5 tau; tau = D (n - lag) / (stride (n2 - lag2) C0_first),
// sigma = sqrt(D / (stride (n2 - lag2) n)).
// FP64 issue bounds it (1.9 operations a clock an SM).  A pass needs, for every t with
// t + lag < n, x_t^2 and x_t times the sum of the lag entries after t: adding those up for
// each t is n lag additions.  A thread here takes a run of R consecutive t from a tile in
// shared memory, puts the first window together from the runs' sums and slides it: about
// 1.3 + 2 additions a t at R = 16, lag = 64.  C grows with the series to 16 CTAs (a cluster of that size is opt-in; 8 otherwise),
// whose partial sums meet in distributed shared memory: a barrier of a cluster costs some
// hundred ns, a grid's over a us, and the decision to halve needs two for every level.
// 8 x 200,003 values: 191 us; 7,975 us with one 256-thread CTA a dimension and full windows.
constexpr uint32_t kAcorThreads = 256;
constexpr uint32_t kAcorRun = 16;                          // longest run of a thread
constexpr uint32_t kAcorMaxLag = 64;
constexpr uint32_t kAcorTile = kAcorThreads * kAcorRun + kAcorMaxLag;
constexpr uint32_t kAcorCluster = 16;

// a padded slot an entry: runs of 16 start in different banks
__device__ __forceinline__ uint32_t acor_slot(uint32_t i) { return i + (i >> 4); }

struct acor_shared {
    double tile[kAcorTile + kAcorTile / 16 + 1];
    double runs[kAcorThreads + kAcorMaxLag / kAcorRun];   // sums of the tile's runs of 16
    double tail[2 * kAcorMaxLag];                          // the series' last entries
    double red[2][kAcorThreads];
    double got[2][kAcorCluster];       // the CTAs' partial sums, written by each of them
};

__device__ __forceinline__ void cluster_sync(cooperative_groups::cluster_group& cl) {
    if (cl.num_blocks() == 1) __syncthreads();
    else cl.sync();
}

// The cluster's sums of the N values, in lane, warp and CTA order; a barrier of the cluster.
// (An FP64 instruction takes a warp 17 clocks of the SM here, however many lanes it has: the
// first levels go over shared memory, where a warp adds up four warps' values.)
template <int N>
__device__ __forceinline__ void cluster_sum(cooperative_groups::cluster_group& cl, acor_shared& sh,
                                            double (&v)[N]) {
    const uint32_t C = cl.num_blocks(), me = cl.block_rank(), tid = threadIdx.x;
#pragma unroll
    for (int k = 0; k < N; ++k) sh.red[k][tid] = v[k];
    __syncthreads();
    if (tid < 32) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            double a = sh.red[k][tid];
#pragma unroll
            for (uint32_t w = 1; w < kAcorThreads / 32; ++w) a += sh.red[k][tid + 32 * w];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(FULL, a, o);
            if (tid < C) {
                if (C == 1) sh.got[k][0] = a;
                else *cl.map_shared_rank(&sh.got[k][me], tid) = a;
            }
        }
    }
    cluster_sync(cl);
#pragma unroll
    for (int k = 0; k < N; ++k) {
        double a = sh.got[k][0];
        for (uint32_t r = 1; r < C; ++r) a += sh.got[k][r];
        v[k] = a;
    }
}

// One pass (nvidia-gtx-acor.cu:40-103) in FP64: x_t = m[t*stride] for t + lag < n; the lag
// window of t reads x (zeroed past n - lag) inside t's block of B = min(wgs, n) entries and
// raw m across the block edge, as the reference's shared-memory window does.  So only the
// windows of the last lag t's that reach past n - lag differ from raw ones; those are
// added up one by one, on the last CTA.
__device__ void acor_pass(cooperative_groups::cluster_group& cl, acor_shared& sh, const double* m,
                          uint64_t stride, uint32_t n, uint32_t wgs, uint32_t lag, uint32_t R,
                          double* c0_out, double* d_out) {
    const uint32_t C = cl.num_blocks(), me = cl.block_rank(), tid = threadIdx.x;
    const uint32_t plain = n > 2u * lag ? n - 2u * lag : 0u;      // t below: raw windows
    const uint32_t per = kAcorThreads * R;
    double c0 = 0.0, dd = 0.0;
    if (me == C - 1 && plain + tid < n && tid < 2u * lag)
        sh.tail[tid] = __ldcg(&m[(uint64_t)(plain + tid) * stride]);
    for (uint64_t t0 = (uint64_t)me * per; t0 < plain; t0 += (uint64_t)C * per) {
        const uint32_t have = (uint32_t)(n - t0 < per + lag ? n - t0 : per + lag);
        __syncthreads();
        for (uint32_t i = tid; i < have; i += kAcorThreads)
            sh.tile[acor_slot(i)] = __ldcg(&m[(t0 + i) * stride]);
        __syncthreads();
        const uint32_t i0 = tid * R;
        const bool by_runs = R == kAcorRun && lag + 1 >= kAcorRun;
        if (by_runs) {      // entries past `have` are read (not used by any window): in the tile
            for (uint32_t j = tid; j < kAcorThreads + kAcorMaxLag / kAcorRun; j += kAcorThreads) {
                double q = 0.0;
#pragma unroll
                for (uint32_t i = 0; i < kAcorRun; ++i) q += sh.tile[acor_slot(j * kAcorRun + i)];
                sh.runs[j] = q;
            }
            __syncthreads();
        }
        if (t0 + i0 < plain) {
            const uint32_t i1 = plain - t0 < i0 + R ? (uint32_t)(plain - t0) : i0 + R;
            double acc = 0.0;
            uint32_t s = 1;
            if (by_runs) {
#pragma unroll
                for (; s < kAcorRun; ++s) acc += sh.tile[acor_slot(i0 + s)];
                for (; s + kAcorRun <= lag + 1; s += kAcorRun) acc += sh.runs[tid + s / kAcorRun];
            }
            double part[4] = {};                        // (shorter chains of additions)
            for (; s + 3 <= lag; s += 4)
#pragma unroll
                for (uint32_t q = 0; q < 4; ++q) part[q] += sh.tile[acor_slot(i0 + s + q)];
            for (; s <= lag; ++s) acc += sh.tile[acor_slot(i0 + s)];
            acc += (part[0] + part[1]) + (part[2] + part[3]);
            double x = sh.tile[acor_slot(i0)];
            for (uint32_t i = i0;;) {
                c0 += x * x;
                dd += x * (x + 2.0 * acc);
                if (++i >= i1) break;
                x = sh.tile[acor_slot(i)];
                acc += sh.tile[acor_slot(i + lag)] - x;
            }
        }
    }
    if (me == C - 1) {
        // t in [plain, n - lag), the last threads first: in a short series those have no run,
        // so both parts go on at once
        const uint32_t B = wgs < n ? wgs : n;
        if ((uint64_t)me * per >= plain) __syncthreads();   // no tile: the staged entries' barrier
        const uint64_t t = (uint64_t)plain + (kAcorThreads - 1u - tid);
        if (t + lag < n) {                              // fewer than 2 lag <= 128 of them
            const double x = sh.tail[t - plain];
            const uint64_t blk_end = (t / B + 1) * B;
            double part[4] = {};
            for (uint64_t u = t + 1; u <= t + lag; u += 4)
#pragma unroll
                for (uint32_t q = 0; q < 4; ++q)
                    if (u + q <= t + lag && (u + q >= blk_end || u + q + lag < n))
                        part[q] += sh.tail[u + q - plain];
            const double acc = (part[0] + part[1]) + (part[2] + part[3]);
            c0 += x * x;
            dd += x * (x + 2.0 * acc);
        }
    }
    double both[2] = {c0, dd};
    cluster_sum(cl, sh, both);
    *c0_out = both[0];
    *d_out = both[1];
}

__global__ void __launch_bounds__(kAcorThreads)
acor_kernel(const float* series, uint32_t n, uint64_t st, uint64_t sd, uint32_t wgs, uint32_t lag,
            double* work, double* tau_out, double* mean_out, double* sigma_out) {
    __shared__ acor_shared sh;
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const uint32_t C = cl.num_blocks(), me = cl.block_rank();
    const uint32_t d = blockIdx.x / C;
    double* m = work + (uint64_t)d * n;
    cluster_sync(cl);                                 // every CTA's shared memory is there
    const uint64_t step = (uint64_t)C * kAcorThreads, first = (uint64_t)me * kAcorThreads + threadIdx.x;
    constexpr uint32_t U = 8;                         // loads in flight
    double sum[1] = {};
    for (uint64_t t = first; t < n; t += U * step) {
        float v[U];
#pragma unroll
        for (uint32_t i = 0; i < U; ++i) v[i] = t + i * step < n ? __ldg(&series[(t + i * step) * st + d * sd]) : 0.0f;
#pragma unroll
        for (uint32_t i = 0; i < U; ++i)
            if (t + i * step < n) sum[0] += (double)v[i];
    }
    cluster_sum(cl, sh, sum);
    const double mu = sum[0] / (double)n;
    for (uint64_t t = first; t < n; t += U * step) {
        float v[U];
#pragma unroll
        for (uint32_t i = 0; i < U; ++i) v[i] = t + i * step < n ? __ldg(&series[(t + i * step) * st + d * sd]) : 0.0f;
#pragma unroll
        for (uint32_t i = 0; i < U; ++i)
            if (t + i * step < n) m[t + i * step] = (double)v[i] - mu;
    }
    cluster_sync(cl);
    // shorter runs while the threads outnumber the entries
    const uint32_t R = n / (C * kAcorThreads) >= 8u ? kAcorRun : 4u;
    double c0a, da;
    acor_pass(cl, sh, m, 1, n, wgs, lag, R, &c0a, &da);
    const double c0 = c0a;
    double tau = da / c0;
    uint32_t lag2 = lag, n2 = n;
    uint64_t stride = 1;
    while (10u < lag2 && (double)lag2 < tau * 5.0) {
        n2 /= 2;
        lag2 = (lag * 5u < n2) ? lag : ((n2 / 5u) > 10u ? n2 / 5u : 10u);
        const double c0prev = c0a;
        for (uint64_t g = first; g < n2; g += U * step) {
            double v[U], w[U];
#pragma unroll
            for (uint32_t i = 0; i < U; ++i) {
                const uint64_t h = g + i * step < n2 ? g + i * step : g;
                v[i] = __ldcg(&m[2 * h * stride]);
                w[i] = __ldcg(&m[(2 * h + 1) * stride]);
            }
#pragma unroll
            for (uint32_t i = 0; i < U; ++i)
                if (g + i * step < n2) m[2 * (g + i * step) * stride] = v[i] + w[i];
        }
        cluster_sync(cl);
        stride *= 2;
        acor_pass(cl, sh, m, stride, n2, wgs, lag2, R, &c0a, &da);
        tau = da / c0prev;
    }
    if (me == 0 && threadIdx.x == 0) {
        const double scale = (double)stride * (double)(n2 - lag2);
        tau_out[d] = da * (double)(n - lag) / (scale * c0);
        mean_out[d] = mu;
        sigma_out[d] = sqrt(da / (scale * (double)n));
    }
}

// Fixed device scratch of the allocation-free acor entry point: the work copy of the
// series (dim * n doubles) followed by tau, mean and sigma (3 * dim doubles).  It is
// part of the module image, so every GPU that loads the library holds these 8 MiB
// until the process exits.  acor_kernel writes every slot it later reads, so nothing
// has to be cleared between calls; calls that overlap on the GPU share it and race.
__device__ __align__(256) double g_acor_noalloc_scratch[BAY_ACOR_NOALLOC_MAX_DOUBLES];

inline unsigned grid_for(uint64_t n, unsigned block, unsigned cap = 152u * 16u) {
    uint64_t g = (n + block - 1) / block;
    if (g < 1) g = 1;
    return (unsigned)(g < cap ? g : cap);
}

}  // namespace

namespace bay {

std::atomic<unsigned long long> g_launches{0};

unsigned long long launch_count() { return g_launches.load(); }
void count_launches(unsigned long long n) { g_launches += n; }

cudaError_t launch_ctl_apply(bay_ctl* ctl, const bay_ctl_op& op, cudaStream_t s) {
    ctl_apply<<<1, 1, 0, s>>>(ctl, op);
    g_launches++;
    return cudaGetLastError();
}

cudaError_t launch_mix_begin(bay_ctl* ctl, bay_mix_state* st, cudaStream_t s) {
    mix_begin<<<1, 32, 0, s>>>(ctl, st);
    return cudaGetLastError();
}

cudaError_t launch_mix_end(bay_ctl* ctl, bay_mix_state* st, unsigned long long W, unsigned int step,
                           double min_acc, double max_acc, cudaGraphConditionalHandle cont,
                           cudaStream_t s) {
    mix_end<<<1, 32, 0, s>>>(ctl, st, W, step, min_acc, max_acc, cont);
    return cudaGetLastError();
}

cudaError_t launch_init_uniform(float* xs, uint32_t D, uint64_t W, uint32_t seed,
                                const float* limits, cudaStream_t s) {
    init_uniform<<<grid_for((uint64_t)D * W, 256), 256, 0, s>>>(xs, D, W, seed, limits);
    g_launches++;
    return cudaGetLastError();
}

cudaError_t launch_init_normal(float* xs, uint32_t D, uint64_t W, uint32_t seed, float mean,
                               float sd, cudaStream_t s) {
    const uint64_t n = (uint64_t)D * W;
    init_normal<<<grid_for((n + 1) / 2, 256), 256, 0, s>>>(xs, n, seed, mean, sd);
    g_launches++;
    return cudaGetLastError();
}

cudaError_t launch_init_normal_members(float* xs, const bay_init_member* mem, uint32_t n,
                                       uint64_t count_max, float mean, float sd, cudaStream_t s) {
    // two pairs a thread of the largest member, up to some 32,768 CTAs over the members: with
    // equal shares of 50 CTAs the largest of 48 members held the launch (479 us against 263)
    const uint64_t want = (count_max / 2 + 511) / 512 + 1;
    for (uint32_t m0 = 0; m0 < n; m0 += 32768u) {
        const uint32_t nm = n - m0 < 32768u ? n - m0 : 32768u;
        const uint32_t most = 32768u / nm < 4u ? 4u : 32768u / nm;
        init_normal_members<<<dim3(want < most ? (uint32_t)want : most, nm), 256, 0, s>>>(xs, mem + m0,
                                                                                       mean, sd);
        g_launches++;
    }
    return cudaGetLastError();
}

cudaError_t launch_reduce_means(const bay_ctl* ctl, const float* part, float* means,
                                uint32_t means_cap, uint32_t G, uint32_t D, uint32_t nsteps,
                                double inv_W, cudaStream_t s) {
    if (nsteps == 0) return cudaSuccess;
    dim3 grid(nsteps, D);
    reduce_means<<<grid, 128, 0, s>>>(ctl, part, means, means_cap, G, D, inv_W);
    g_launches++;
    return cudaGetLastError();
}

cudaError_t launch_gemm_layout(const float* A, uint64_t ld, uint32_t rows, uint32_t F, uint32_t NP,
                               uint32_t aux_col, uint32_t aux_len, uint32_t auxs, float* lay,
                               cudaStream_t s) {
    const uint64_t n = (uint64_t)F * NP + (uint64_t)NP * auxs;
    gemm_layout<<<grid_for(n, 256), 256, 0, s>>>(A, ld, rows, F, NP, aux_col, aux_len, auxs, lay);
    g_launches++;
    return cudaGetLastError();
}

cudaError_t launch_gemm_split(const float* A, uint64_t ld, uint32_t rows, uint32_t F, uint32_t Fp,
                              uint64_t rows_pad, uint32_t aux_col, uint32_t aux_len, uint32_t auxs,
                              unsigned short* hi, unsigned short* lo, float* aux, cudaStream_t s) {
    const uint64_t n = rows_pad * Fp + rows_pad * auxs;
    gemm_split<<<grid_for(n, 256), 256, 0, s>>>(A, ld, rows, F, Fp, rows_pad, aux_col, aux_len, auxs,
                                                 hi, lo, aux);
    g_launches++;
    return cudaGetLastError();
}

cudaError_t launch_gemm_tc_image(const float* A, uint64_t ld, uint32_t rows, uint32_t F,
                                 uint32_t KC, uint32_t NP, uint32_t aux_col, uint32_t aux_len,
                                 uint32_t auxs, void* img, cudaStream_t s) {
    const uint64_t n = (uint64_t)KC * NP * 8 + (uint64_t)NP * auxs;
    gemm_tc_image<<<grid_for(n, 256), 256, 0, s>>>(A, ld, rows, F, KC, NP, aux_col, aux_len, auxs,
                                                    static_cast<unsigned char*>(img));
    g_launches++;
    return cudaGetLastError();
}

cudaError_t launch_acor(const float* series, uint32_t D, uint32_t n, uint64_t st, uint64_t sd,
                        uint32_t wgs, uint32_t lag, double* work, double* tau, double* mean,
                        double* sigma, cudaStream_t s) {
    // a CTA of the cluster for every 1,024 entries, a power of two up to 16 (8 where the
    // device takes no cluster of 16)
    cudaLaunchAttribute at[1];
    cudaLaunchConfig_t cfg{};
    cfg.blockDim = dim3(kAcorThreads);
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    uint32_t C = 1;
    while (C < kAcorCluster && (uint64_t)C * 1024u < n) C *= 2;
    if (C > 8) {
        cudaError_t e = cudaFuncSetAttribute(acor_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return e;
        at[0].val.clusterDim.x = C;
        cfg.gridDim = dim3(C);
        int fit = 0;
        e = cudaOccupancyMaxActiveClusters(&fit, acor_kernel, &cfg);
        if (e != cudaSuccess || fit < 1) {
            cudaGetLastError();
            C = 8;
        }
    }
    at[0].val.clusterDim.x = C;
    cfg.gridDim = dim3(D * C);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, acor_kernel, series, n, st, sd, wgs, lag, work, tau,
                                             mean, sigma);
    if (e != cudaSuccess) return e;
    g_launches++;
    return cudaGetLastError();
}

cudaError_t acor_noalloc_scratch(double** ptr) {
    // In host code g_acor_noalloc_scratch names a host-side stand-in, not the array: its
    // device address comes from cudaGetSymbolAddress, with the device current.
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_acor_noalloc_scratch);
    if (e != cudaSuccess) return e;
    *ptr = static_cast<double*>(p);
    return cudaSuccess;
}

cudaError_t launch_fill_bytes(void* p, uint64_t n, unsigned char v, cudaStream_t s) {
    const unsigned int w = 0x01010101u * v;
    const uint64_t n16 = n / 16;
    fill_bytes<<<grid_for(n16, 512, 152u * 8u), 512, 0, s>>>((uint4*)p, n16, w);
    g_launches++;
    return cudaGetLastError();
}

}  // namespace bay
