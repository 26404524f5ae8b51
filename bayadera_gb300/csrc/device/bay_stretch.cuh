// bay_stretch.cuh -- fused affine-invariant stretch move, compiled by NVRTC per model.
//
// One launch moves one half of the ensemble against the other (red/black update):
// Philox draw, stretch factor z ~ g(z) (Christen 2007), partner from the
// complementary half, proposal Y = S_j + z (X_k - S_j), the model's log density at Y,
// the accept step, and (in the "accu" variant) the acceptance count and the per-step
// ensemble sums that feed acor.  Reference: cuda/engines/nvidia-gtx-mcmc-stretch.cu
// stretch_move :35-99, stretch_move_accu :101-134, stretch_move_bare :136-154.
//
// Counter and key words are the reference's: key {seed_h, 0xdecafbad}, counter
// {k, step, stream, 0xbeeff00d}; stream 3333/4444 (bare) and 1111/2222 (accu) for
// halves 0/1; seed_h = seed (half 0) or seed + 1 (half 1).
//
// Layout (all forms): positions walker-major, xs[w * DIM + d] (W walkers,
// half h = walkers [h*K, h*K + K)); logfn contiguous, logfn[w].
//
// Macros supplied by the host when it compiles a model:
//   DIM            walker dimension
//   BAY_LOGFN      plain form: REAL f(uint32 data_len, uint32 params_len,
//                  const REAL* params, uint32 dim, const REAL* x)  (reference ABI)
//   BAY_TILED      1 for the data-tiled form, with
//     BAY_TILE_PREP(hyper, hyper_len, dim, x, prep)   per-walker precompute
//     BAY_TILE_TERM(row, prep) -> REAL                 one data row
//     BAY_TILE_WALKER(n_rows, hyper, hyper_len, dim, x) -> REAL   the rest
//     BAY_ROW_LEN, BAY_PREP_LEN, BAY_WPC (walkers per CTA)
//   BAY_CTA        threads per CTA
//   BAY_ACCEPT_REF 1: accept if u <= z^(D-1) exp(beta dl) in fp32 (the reference's
//                  formula); 0 (default): log u <= (D-1) log z + beta dl in fp32 with
//                  the deterministic logarithm bay_log_det (bay_accept_log).
//   BAY_STRETCH_REF 1: the stretch factor's 1/a by the compiler's fast division (the
//                  reference's build flavour, -use_fast_math); 0 (default): IEEE 1/a.
//                  Both keep the operation order the golden trajectories pin.
//   BAY_PARTNER_ELEMENT 1 (plain and tiled forms): the reference's partner offset
//                  (uint)(u0 K DIM), an element offset that straddles walkers for
//                  DIM > 1; elements past the half's end read as 0.  0 (default): the
//                  partner is walker (uint)(u0 K), clamped to the half.

#ifndef BAY_CTA
#define BAY_CTA 256
#endif
#ifndef BAY_ACCEPT_REF
#define BAY_ACCEPT_REF 0
#endif
#ifndef BAY_TILED
#define BAY_TILED 0
#endif
#ifndef BAY_STRETCH_REF
#define BAY_STRETCH_REF 0
#endif
#ifndef BAY_PARTNER_ELEMENT
#define BAY_PARTNER_ELEMENT 0
#endif
#ifndef BAY_GEMM
#define BAY_GEMM 0
#endif

// Sampler control block, resident in device memory so that captured CUDA graphs
// replay without parameter patching.
struct bay_ctl {
    unsigned int step[2];           // [0] bare move counter, [1] accu move counter
    unsigned int seed[2];           // [0] bare seed, [1] accu seed (half 1 adds 1)
    float a;
    float beta;
    unsigned int ticket[2];         // last-CTA tickets of the accu reductions
    unsigned long long accepted;    // accu: accepted proposals since the last reset
    unsigned int status;            // nonzero: a device-detected error
    unsigned int pad0[21];
    unsigned int gbar_count;        // grid barrier of the persistent form (byte 128): arrivals
    unsigned int pad1[31];
    unsigned int abort;             //   abandon flag (byte 256); both cleared before each launch
    unsigned int pad2[31];
};

struct bay_stretch_params {
    const float* params;            // data || hyperparameters
    float* xs;                      // positions, walker-major xs[w * DIM + d]
    float* logfn;                   // W log densities
    bay_ctl* ctl;
    float* part;                    // accu: per-CTA sums [step_off][half][DIM][cta]
    float* means;                   // unused by the stretch kernels (reduce_means writes it)
    unsigned long long data_len;    // floats of data in params
    unsigned int params_len;        // hyperparameters after the data
    unsigned int W, K;
    unsigned int half;
    unsigned int step_off;          // added to the device step counter
    unsigned int means_cap;         // steps the means buffer holds
    float inv_W;
    // GEMM form: matrix rows at params + gemm_base + r * gemm_ld, r < gemm_rows; the
    // sampler's copy laid out for the kernel: gemm_lay = [F][NP] feature-major, rows
    // zero-padded to NP (a multiple of 64), then [NP][aux] row-major
    unsigned long long gemm_base;
    unsigned long long gemm_rows;
    unsigned int gemm_ld;
    unsigned int gemm_np;
    const float* gemm_lay;
    // GEMM form, streaming (too many rows for shared memory): one half-step's per-walker
    // scratch and the per-row-block partial sums
    float* s_y;                     // [nk][DIM] proposals (current positions for logfn)
    float* s_b;                     // [nk][F] coefficient block
    float* s_prep;                  // [nk][BAY_PREP_LEN]
    float* s_w;                     // [nk] terms outside the row sum
    float* s_zu;                    // [nk][3] stretch factor, accept uniform, log density
    float* s_part;                  // [nsb][nk] compensated (hi, lo) partial row sums
    unsigned int s_nsb;             // row super-blocks
    unsigned int s_sbrows;          // rows per super-block (a multiple of 128)
    // GEMM form on the tensor cores: the coefficient block split into bf16 hi + lo,
    // [walker][tc_fp] each (tc_fp = F rounded up to 64; padding columns stay zero)
    unsigned short* s_bh;
    unsigned short* s_bl;
    unsigned int tc_fp;
    unsigned int gbar_extra;        // persistent form: arrivals its grid barriers wait for beyond
                                    // the grid (0; 1 makes them run out, for tests)
    // data-tiled form split into t_slices row slices per walker group (1: none): each
    // slice's CTA leaves its walkers' partial sums in t_part[k][slice] (hi, lo) and takes a
    // ticket in t_ticket[group]; the last one combines them in slice order and decides
    unsigned int t_slices;
    unsigned int beta_set;          // bare: beta of this launch below instead of the control
    float* t_part;                  // block's (an annealing step's)
    unsigned int* t_ticket;
    float beta;
    unsigned int pad_t;
};
__device__ __forceinline__ float bay_beta(const bay_stretch_params& P) {
    return P.beta_set ? P.beta : P.ctl->beta;
}

__device__ __forceinline__ float bay_stretch_z(float a, float u1) {
    // z = (a - 2 + 1/a) u1^2 + 2 (1 - 1/a) u1 + 1/a with the first product fused and
    // every other operation rounded on its own: the order the reference's golden
    // trajectories pin (the current compiler contracts the reference's spelling of the
    // expression, nvidia-gtx-mcmc-stretch.cu:71-72, differently).  1/a is IEEE by default;
    // BAY_STRETCH_REF takes the reference build's flavour, the compiler's fast division
    // (this module is compiled with -use_fast_math, as the reference's is).
#if BAY_STRETCH_REF
    const float inv_a = 1.0f / a;
#else
    const float inv_a = __fdiv_rn(1.0f, a);
#endif
    const float c1 = __fadd_rn(__fsub_rn(a, 2.0f), inv_a);
    const float c2 = __fmul_rn(2.0f, __fsub_rn(1.0f, inv_a));
    return __fadd_rn(__fmaf_rn(__fmul_rn(c1, u1), u1, __fmul_rn(c2, u1)), inv_a);
}

__device__ __forceinline__ unsigned int bay_partner(float u0, unsigned int K) {
#if BAY_PARTNER_ELEMENT
    // the reference's element offset (uint)(u0 * K * DIM), two fp32 products
    return __float2uint_rz(__fmul_rn(__fmul_rn(u0, (float)K), (float)DIM));
#else
    // Walker j = (uint)(u0 * K) of the complementary half; u0 < 1 can still round
    // u0*K up to K, so clamp (the reference would read past the half there).
    unsigned int j = __float2uint_rz(__fmul_rn(u0, (float)K));
    return j < K ? j : K - 1;
#endif
}

// Coordinate i of the partner j (bay_partner) in the complementary half S of K walkers.
__device__ __forceinline__ float bay_partner_coord(const float* S, unsigned int K, unsigned int j,
                                                   unsigned int i) {
#if BAY_PARTNER_ELEMENT
    // an element offset: past the half's last element the reference reads out of bounds
    // (or the moving half, racing with its writes); here those elements read as 0
    const unsigned long long e = (unsigned long long)j + i;
    return e < (unsigned long long)K * DIM ? S[e] : 0.0f;
#else
    return S[(size_t)j * DIM + i];
#endif
}

__device__ __forceinline__ bool bay_accept(float u2, float z, float ly, float lx, float beta) {
#if BAY_ACCEPT_REF
    const float q = isfinite(ly) ? powf(z, (float)(DIM - 1)) * expf(beta * (ly - lx)) : 0.0f;
    return u2 <= q;
#else
    return bay_accept_log(u2, z, ly, lx, beta, DIM - 1);
#endif
}

// Compensated fp32 pairs (hi, lo), hi + lo the value: sums carried without FP64 (FP64
// issue is a small fraction of FP32 on this part).  bay_cadd is symmetric in its
// arguments (TwoSum of the highs, then the lows), so an xor-butterfly of it leaves the
// same bits in every lane: the combine order is fixed and the result deterministic.
struct bay_cf {
    float hi, lo;
};
__device__ __forceinline__ bay_cf bay_cadd(bay_cf a, bay_cf b) {
    const float s = __fadd_rn(a.hi, b.hi);
    const float bb = __fsub_rn(s, a.hi);
    const float e = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bb)), __fsub_rn(b.hi, bb));
    const float lo = __fadd_rn(__fadd_rn(a.lo, b.lo), e);
    const float hi = __fadd_rn(s, lo);
    bay_cf r;
    r.hi = hi;
    r.lo = __fsub_rn(lo, __fsub_rn(hi, s));
    return r;
}
__device__ __forceinline__ bay_cf bay_cf_shfl_xor(bay_cf v, int o) {
    bay_cf r;
    r.hi = __shfl_xor_sync(0xffffffffu, v.hi, o);
    r.lo = __shfl_xor_sync(0xffffffffu, v.lo, o);
    return r;
}
// a + (s.hi + s.lo), rounded once to fp32
__device__ __forceinline__ float bay_cf_total(float a, bay_cf s) {
    bay_cf t;
    t.hi = a;
    t.lo = 0.0f;
    t = bay_cadd(t, s);
    return __fadd_rn(t.hi, t.lo);
}

// Accu epilogue: the CTA's accept count (one 64-bit atomic, integer: deterministic) and,
// when per-step means are wanted, the CTA's per-dim sums of the moved half: fp32 warp
// shuffles, per-warp sums staged in shared memory (one barrier per 64 dims), combined
// across warps with compensated fp32 in warp order, stored to part[(step_off*2 + half)][dim][cta].  The
// per-step ensemble means are reduced from these partials by a separate kernel.
// Where the group's CTA is split over a cluster (plain form, small ensembles), the warps' sums
// meet in the first CTA's shared memory: the same warps, combined in the same order.
#define BAY_SUM_CHUNK 64
__device__ __forceinline__ void bay_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ void bay_accu_epilogue(const bay_stretch_params& P, bool accepted, bool valid,
                                  const float* mine, float (*red)[BAY_SUM_CHUNK],
                                  unsigned int slot, unsigned int nslots,
                                  unsigned int ncta = 1u, unsigned int rank = 0u) {
    const int n_acc = __syncthreads_count(accepted);
    if (threadIdx.x == 0 && n_acc) atomicAdd(&P.ctl->accepted, (unsigned long long)n_acc);
    if (P.means_cap == 0) return;
    const int lane = threadIdx.x & 31, warp = (rank * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = ncta * (blockDim.x >> 5);
    float* out = P.part + ((size_t)P.step_off * 2 + P.half) * DIM * nslots + slot;
    unsigned int first = 0;                   // the first CTA's `red`
    if (ncta > 1u) {
        bay_cluster_sync();                   // every CTA of the cluster is there
        asm("mapa.shared::cluster.u32 %0, %1, 0;"
            : "=r"(first) : "r"((unsigned int)__cvta_generic_to_shared(&red[0][0])));
    }
#pragma unroll
    for (int d0 = 0; d0 < DIM; d0 += BAY_SUM_CHUNK) {
#pragma unroll
        for (int d = d0; d < DIM && d < d0 + BAY_SUM_CHUNK; ++d) {
            float v = valid ? mine[d] : 0.0f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0) {
                if (ncta > 1u)
                    asm volatile("st.shared::cluster.f32 [%0], %1;"
                                 ::"r"(first + 4u * (unsigned int)(warp * BAY_SUM_CHUNK + d - d0)), "f"(v)
                                 : "memory");
                else
                    red[warp][d - d0] = v;
            }
        }
        if (ncta > 1u) bay_cluster_sync();
        else __syncthreads();
        const int nd = (DIM - d0) < BAY_SUM_CHUNK ? (DIM - d0) : BAY_SUM_CHUNK;
        for (int d = threadIdx.x; d < nd && rank == 0u; d += blockDim.x) {
            bay_cf s;
            s.hi = 0.0f;
            s.lo = 0.0f;
            for (int w = 0; w < nwarps; ++w) {
                bay_cf y;
                y.hi = red[w][d];
                y.lo = 0.0f;
                s = bay_cadd(s, y);
            }
            out[(size_t)(d0 + d) * nslots] = __fadd_rn(s.hi, s.lo);
        }
        if (d0 + BAY_SUM_CHUNK < DIM) {       // the next chunk's sums overwrite red
            if (ncta > 1u) bay_cluster_sync();
            else __syncthreads();
        }
    }
}

#if BAY_GEMM
// ---------------------------------------------------------------- GEMM form
// log density = BAY_GEMM_WALKER(rows, hyper, hyper_len, dim, x)
//             + sum_r BAY_GEMM_TERM(eta_r, aux_r, r, x, prep),   eta = A x[COEF : COEF+F],
// A = the rows x F matrix at params + gemm_base (row stride gemm_ld; aux values of row r
// at column BAY_GEMM_AUXCOL).  A CTA owns BAY_WT walkers.  The matrix (feature-major,
// rows padded to 64) and the proposal tile are staged in shared memory once; each of
// the 256 threads accumulates a 4-walker x 4-row register tile over the F features (two
// 16-byte shared loads per 16 FMAs), applies the row term with a Kahan sum, and the 16
// row-group lanes of a walker combine as compensated fp32 pairs in a fixed xor order.
#define BAY_WT 64
#define BAY_RW 4
#define BAY_RN 4
#define BAY_NG 16
#define BAY_ROWS_PER_PASS (BAY_NG * BAY_RN)
#define BAY_DPAD (DIM | 1)
#ifndef BAY_GEMM_AUX
#define BAY_GEMM_AUX 0
#endif
#define BAY_AUXS (BAY_GEMM_AUX > 0 ? BAY_GEMM_AUX : 1)

// A row term f may come with a form for 16 rows (f_16, f_16_init and f_16_end, announced by the
// macro f_16_carry, the number of values a thread carries over its rows).  It goes with the name
// of the term that the model uses: a source may define f and use another term.
#define BAY_CAT2(a, b) a##b
#define BAY_CAT(a, b) BAY_CAT2(a, b)
#define BAY_TERM16_CARRY BAY_CAT(BAY_GEMM_TERM, _16_carry)
#if BAY_TERM16_CARRY
#define BAY_TERM16 1
#else
#define BAY_TERM16 0
#endif

// Unrolling of the feature loop, and the registers of the launches (by the CTAs an SM that they
// are to allow).  Unrolled whole a small loop takes up to 127 registers, which costs nothing while
// an SM has one CTA and is a loss with more: 40,000 walkers of 20 dims 7.8 us a bare launch and
// 12.2 accu unrolled by 20, now 6.3 and 8.3; 65,536 of 10 dims 8.0 and 9.9, now 6.3 and 8.4.  With
// four CTAs of a bare launch an SM the longer loops are scheduled better too (12,288 walkers of 77
// dims 10.8, now 9.5 us; 8,192 of 120 14.8, now 12.4).  Without a bound the accu launch of 25 to 64
// features is faster (12,290 walkers of 37 dims 5.9 us, 6.2 with three).  By 5, 8, 10, 16 and 20,
// over 20 sizes from 2 to 120 dims, 20 was the fastest above 24 features or within 1 % of it but for
// 40 dims (16: 5.6 against 6.1 us before the bound).
#define BAY_G_UNROLL (BAY_GEMM_F > 24 ? 20 : BAY_GEMM_F > 10 ? 10 : 8)
#define BAY_G_BOUNDS __launch_bounds__(256, 4)
#if BAY_GEMM_F <= 24
#define BAY_G_BOUNDS_ACCU __launch_bounds__(320, 4)
#elif BAY_GEMM_F <= 64
#define BAY_G_BOUNDS_ACCU __launch_bounds__(320)
#else
#define BAY_G_BOUNDS_ACCU __launch_bounds__(320, 3)
#endif

// barriers of the eight warps that move a tile (accu launches have two more)
__device__ __forceinline__ void bay_g_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
__device__ __forceinline__ bool bay_g_or(bool p) {
    unsigned int r;
    asm volatile("{\n .reg .pred q, o;\n setp.ne.u32 q, %1, 0;\n bar.red.or.pred o, 1, 256, q;\n"
                 " selp.u32 %0, 1, 0, o;\n}\n" : "=r"(r) : "r"((unsigned int)p) : "memory");
    return r != 0u;
}
__device__ __forceinline__ int bay_g_count(bool p) {
    int r;
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %1, 0;\n bar.red.popc.u32 %0, 1, 256, q;\n}\n"
                 : "=r"(r) : "r"((unsigned int)p) : "memory");
    return r;
}

// The statistics of a tile: per-dim compensated sums of its nv walkers' positions (rows of DIM
// floats) in walker order, dims t, t + stride, ...; out[d * gridDim.x]
__device__ __forceinline__ void bay_g_sums(const float* rows, unsigned int nv, unsigned int t,
                                           unsigned int stride, float* out) {
    for (unsigned int d = t; d < DIM; d += stride) {
        bay_cf s;
        s.hi = 0.0f;
        s.lo = 0.0f;
        for (unsigned int w0 = 0; w0 < BAY_WT; w0 += 16u) {
            float v[16];
#pragma unroll
            for (unsigned int i = 0; i < 16u; ++i)
                v[i] = w0 + i < nv ? rows[(size_t)(w0 + i) * DIM + d] : 0.0f;
#pragma unroll
            for (unsigned int i = 0; i < 16u; ++i) {
                bay_cf y;
                y.hi = v[i];
                y.lo = 0.0f;
                if (w0 + i < nv) s = bay_cadd(s, y);
            }
        }
        out[(size_t)d * gridDim.x] = __fadd_rn(s.hi, s.lo);
    }
}

template <bool ACCU, bool LOGFN_ONLY>
__device__ __forceinline__ void bay_stretch_gemm(const bay_stretch_params& P) {
    extern __shared__ __align__(128) float bay_smem[];
    const unsigned int rows = (unsigned int)P.gemm_rows;
    const unsigned int NP = P.gemm_np;
    float* As = bay_smem;                              // [F][NP]   (the sampler's layout,
    float* Aux = As + (size_t)BAY_GEMM_F * NP;         // [NP][AUXS] copied as one block)
    float* Ys = Aux + (size_t)NP * BAY_AUXS;           // [F][BAY_WT]
    float* Yw = Ys + BAY_GEMM_F * BAY_WT;              // [BAY_WT][BAY_DPAD]
    __shared__ float sZ[BAY_WT], sU2[BAY_WT], sW[BAY_WT];
    __shared__ unsigned int sJ[BAY_WT];
    __shared__ float sPrep[BAY_WT][BAY_PREP_LEN];
    __shared__ bay_cf sSum[BAY_WT];
    __shared__ float sLx[BAY_WT];
    __shared__ __align__(8) unsigned long long sBar;

    const unsigned int kind = ACCU ? 1u : 0u;
    const unsigned int tid = threadIdx.x;
    const unsigned int k0 = blockIdx.x * BAY_WT;
    const unsigned int nk = LOGFN_ONLY ? P.W : P.K;
    const float* hyper = P.params + P.data_len;
    float* X = P.xs + (LOGFN_ONLY ? 0 : (size_t)P.half * P.K * DIM);
    const float* S = P.xs + (size_t)(1u - P.half) * P.K * DIM;

    // accu: two more warps sum this tile of the other half, as the previous half-step left it
    // ((step_off, 0) for half 1, (step_off - 1, 1) for half 0; the chunk's last half-step has
    // a launch of its own), beside the eight that move the walkers.  At the end of the moving
    // half's own launch the sums were a serial chain of 64 compensated additions that
    // everything waited for: 12,290 walkers of 37 dimensions 8.3 -> 5.9 us a launch,
    // 16,384 of 50 10.7 -> 7.2.
    if (ACCU && tid >= 256u) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (P.means_cap != 0 && (P.half == 1u || P.step_off > 0u))
            bay_g_sums(S + (size_t)k0 * DIM, nk - k0 < BAY_WT ? nk - k0 : BAY_WT, tid - 256u, 64u,
                       P.part + ((size_t)(P.half == 1u ? P.step_off : P.step_off - 1u) * 2 + (1u - P.half)) *
                           DIM * gridDim.x + blockIdx.x);
        return;
    }
    // 1. one TMA bulk copy (cp.async.bulk, completion counted on an mbarrier) brings the
    //    laid-out matrix and aux values into shared memory; it overlaps the proposals.
    const unsigned int lay_bytes =
        (unsigned int)(((size_t)BAY_GEMM_F * NP + (size_t)NP * BAY_AUXS) * sizeof(float));
    const unsigned int bar = (unsigned int)__cvta_generic_to_shared(&sBar);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    bay_g_sync();
    if (tid == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                     "r"(lay_bytes) : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
            ::"r"((unsigned int)__cvta_generic_to_shared(As)), "l"(P.gemm_lay), "r"(lay_bytes),
            "r"(bar) : "memory");
    }
    // Launched with programmatic dependent launch: the matrix never changes, the rest waits
    // for the previous launch
    if (!LOGFN_ONLY) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    // 2. proposals (Philox, z, partner) for the tile, then Y in both layouts; each thread
    //    keeps all its gather loads in flight before it uses any of them
    if (!LOGFN_ONLY && tid < BAY_WT) {
        const unsigned int k = k0 + tid;
        if (k < nk) {
            const unsigned int stream = ACCU ? (P.half ? 2222u : 1111u) : (P.half ? 4444u : 3333u);
            bay_u4 c;
            c.x = k;
            c.y = P.ctl->step[kind] + P.step_off;
            c.z = stream;
            c.w = 0xbeeff00du;
            const bay_u4 r = bay_philox4x32_10(c, P.ctl->seed[kind] + P.half, 0xdecafbadu);
            const float z = bay_stretch_z(P.ctl->a, bay_u01(r.y));
            sZ[tid] = z;
            sJ[tid] = bay_partner(bay_u01(r.x), P.K);
            sU2[tid] = bay_u01(r.z);
            sLx[tid] = P.logfn[(size_t)P.half * P.K + k];
        }
    }
    bay_g_sync();
    {
        // The tile's own rows are one contiguous block of BAY_WT * DIM floats; element e is
        // (walker e / DIM, coordinate e % DIM), so a warp reads its own elements coalesced
        // and each partner row (DIM contiguous floats) in runs of consecutive coordinates.
        constexpr int NE = (BAY_WT * DIM + 255) / 256;   // elements per thread
        constexpr int CH = 16;                            // loads kept in flight per batch
        const float* Xt = X + (size_t)k0 * DIM;
        const unsigned int n_own = (nk - k0 < BAY_WT ? nk - k0 : BAY_WT) * DIM;
#pragma unroll
        for (int c0 = 0; c0 < NE; c0 += CH) {
            float xv[CH], sv[CH];
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                const unsigned int e = tid + 256u * (unsigned int)(c0 + i);
                const unsigned int w = e / DIM, d = e - w * DIM;
                const bool ev = (c0 + i < NE) && e < n_own;
                xv[i] = ev ? Xt[e] : 0.0f;
                sv[i] = (!LOGFN_ONLY && ev) ? S[(size_t)sJ[w] * DIM + d] : 0.0f;
            }
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                const unsigned int e = tid + 256u * (unsigned int)(c0 + i);
                if ((c0 + i < NE) && e < BAY_WT * DIM) {
                    const unsigned int w = e / DIM, d = e - w * DIM;
                    const float y = LOGFN_ONLY ? xv[i]
                        : (e < n_own ? __fmaf_rn(sZ[w], __fsub_rn(xv[i], sv[i]), sv[i]) : 0.0f);
                    Yw[w * BAY_DPAD + d] = y;
                }
            }
        }
    }
    bay_g_sync();
    // feature-major copy of the coefficient block for the register tiles (bank-conflict
    // free: consecutive lanes write consecutive walkers and read rows of odd stride)
    for (unsigned int e = tid; e < BAY_GEMM_F * BAY_WT; e += 256u) {
        const unsigned int f = e / BAY_WT, w = e - f * BAY_WT;
        Ys[e] = Yw[w * BAY_DPAD + BAY_GEMM_COEF + f];
    }
    // the matrix copy: bounded wait; a CTA-uniform timeout flags the sampler and exits
    {
        unsigned int done = 0;
        for (unsigned int it = 0; it < (1u << 22) && !done; ++it)
            asm volatile(
                "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                " selp.u32 %0, 1, 0, p;\n}\n"
                : "=r"(done) : "r"(bar), "r"(0u) : "memory");
        if (bay_g_or(!done)) {
            if (tid == 0) atomicOr(&P.ctl->status, 1u);
            return;
        }
    }
    // 3. per-walker precompute and the terms outside the row sum
    if (tid < BAY_WT) {
        float pr[BAY_PREP_LEN];
#pragma unroll
        for (int i = 0; i < BAY_PREP_LEN; ++i) pr[i] = 0.0f;
        float wt = 0.0f;
        if (k0 + tid < nk) {
            BAY_GEMM_PREP(hyper, P.params_len, DIM, &Yw[tid * BAY_DPAD], pr);
            wt = BAY_GEMM_WALKER(P.gemm_rows, hyper, P.params_len, DIM, &Yw[tid * BAY_DPAD]);
        }
#pragma unroll
        for (int i = 0; i < BAY_PREP_LEN; ++i) sPrep[tid][i] = pr[i];
        sW[tid] = wt;
    }
    bay_g_sync();
    // 4. eta tiles and row terms
    const unsigned int wg = tid / BAY_NG, rg = tid - wg * BAY_NG;
    const unsigned int w0 = wg * BAY_RW;
    float sum[BAY_RW], cmp[BAY_RW];
#pragma unroll
    for (int i = 0; i < BAY_RW; ++i) {
        sum[i] = 0.0f;
        cmp[i] = 0.0f;
    }
    for (unsigned int r0 = 0; r0 < NP; r0 += BAY_ROWS_PER_PASS) {
        const unsigned int n0 = r0 + rg * BAY_RN;
        float acc[BAY_RW][BAY_RN];
#pragma unroll
        for (int i = 0; i < BAY_RW; ++i)
#pragma unroll
            for (int j = 0; j < BAY_RN; ++j) acc[i][j] = 0.0f;
#pragma unroll BAY_G_UNROLL
        for (int f = 0; f < BAY_GEMM_F; ++f) {
            const float4 y = *reinterpret_cast<const float4*>(&Ys[f * BAY_WT + w0]);
            const float4 a = *reinterpret_cast<const float4*>(&As[(size_t)f * NP + n0]);
            const float yv[4] = {y.x, y.y, y.z, y.w};
            const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
            for (int i = 0; i < BAY_RW; ++i)
#pragma unroll
                for (int j = 0; j < BAY_RN; ++j) acc[i][j] = __fmaf_rn(av[j], yv[i], acc[i][j]);
        }
#pragma unroll
        for (int j = 0; j < BAY_RN; ++j) {
            const unsigned int r = n0 + j;
            if (r < rows) {
#pragma unroll
                for (int i = 0; i < BAY_RW; ++i) {
                    const float t = BAY_GEMM_TERM(acc[i][j], &Aux[(size_t)r * BAY_AUXS], (uint64_t)r,
                                                  &Yw[(w0 + i) * BAY_DPAD], sPrep[w0 + i]);
                    const float yk = __fsub_rn(t, cmp[i]);
                    const float s2 = __fadd_rn(sum[i], yk);
                    cmp[i] = __fsub_rn(__fsub_rn(s2, sum[i]), yk);
                    sum[i] = s2;
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < BAY_RW; ++i) {
        bay_cf v;
        v.hi = sum[i];
        v.lo = -cmp[i];
#pragma unroll
        for (int o = BAY_NG / 2; o > 0; o >>= 1) v = bay_cadd(v, bay_cf_shfl_xor(v, o));
        if (rg == 0) sSum[w0 + i] = v;
    }
    bay_g_sync();
    // 5. accept (one thread per walker), then the accepted walkers' rows written back
    //    cooperatively
    __shared__ unsigned char sAcc[BAY_WT];
    const unsigned int k = k0 + tid;
    const bool valid = tid < BAY_WT && k < nk;
    bool accepted = false;
    if (valid) {
        bay_cf t;
        t.hi = sW[tid];
        t.lo = 0.0f;
        t = bay_cadd(t, sSum[tid]);
        const float ly = __fadd_rn(t.hi, t.lo);
        if (LOGFN_ONLY) {
            P.logfn[k] = ly;
        } else {
            accepted = bay_accept(sU2[tid], sZ[tid], ly, sLx[tid], ACCU ? 1.0f : bay_beta(P));
            if (accepted) P.logfn[(size_t)P.half * P.K + k] = ly;
        }
    }
    if (LOGFN_ONLY) return;
    if (tid < BAY_WT) sAcc[tid] = accepted ? 1 : 0;
    const int n_acc = bay_g_count(accepted);
    {
        float* Xt = X + (size_t)k0 * DIM;
        const unsigned int n_own = (nk - k0 < BAY_WT ? nk - k0 : BAY_WT) * DIM;
        for (unsigned int e = tid; e < n_own; e += 256u) {
            const unsigned int w = e / DIM, d = e - w * DIM;
            if (sAcc[w]) Xt[e] = Yw[w * BAY_DPAD + d];
        }
    }
    if (ACCU && tid == 0 && n_acc) atomicAdd(&P.ctl->accepted, (unsigned long long)n_acc);
}

extern "C" __global__ void BAY_G_BOUNDS bay_stretch_bare(bay_stretch_params P) {
    bay_stretch_gemm<false, false>(P);
}
extern "C" __global__ void BAY_G_BOUNDS_ACCU bay_stretch_accu(bay_stretch_params P) {
    bay_stretch_gemm<true, false>(P);
}
// the statistics of the last half-step of a chunk (half P.half, step P.step_off)
extern "C" __global__ void __launch_bounds__(256) bay_gemm_stats(bay_stretch_params P) {
    const unsigned int k0 = blockIdx.x * BAY_WT;
    bay_g_sums(P.xs + ((size_t)P.half * P.K + k0) * DIM, P.K - k0 < BAY_WT ? P.K - k0 : BAY_WT, threadIdx.x,
               256u, P.part + ((size_t)P.step_off * 2 + P.half) * DIM * gridDim.x + blockIdx.x);
}
extern "C" __global__ void __launch_bounds__(256) bay_logfn_all(bay_stretch_params P) {
    bay_stretch_gemm<false, true>(P);
}

// ---------------------------------------------------------------- GEMM form, streaming
// For matrices too large for shared memory.  A half-step is three launches:
//   propose: a warp per walker -- Philox, stretch, partner, proposal row, prep and the
//            terms outside the row sum into per-walker scratch;
//   rows:    CTA (128-walker tile, row super-block): the tile's coefficient block stays in
//            shared memory (feature-major); for each 128-row sub-block the matrix is
//            streamed in 32-feature chunks; each thread owns 8 walkers x 8 rows (rows
//            rg + 16 j) of eta, applies the row term with Kahan sums, and the 16 row-group
//            lanes of a walker combine as compensated fp32 pairs -> s_part[sb][walker];
//            blockIdx.x runs over walker tiles so that the tiles sharing a row block run
//            together and the block is read from HBM once;
//   accept:  partials summed in super-block order, accept, write-back, statistics.
#define BAY_SW 128
#define BAY_SR 128
#define BAY_SF 32
#define BAY_XS (BAY_SR + 1)   // odd row stride of the staged matrix chunk (no bank conflicts)

// bf16 of a float rounded to nearest even, as its 16 bits (NaN stays a quiet NaN)
__device__ __forceinline__ unsigned short bay_bf16_rn(float x) {
    unsigned int u = __float_as_uint(x);
    if ((u & 0x7fffffffu) > 0x7f800000u) return (unsigned short)((u >> 16) | 0x40u);
    u += 0x7fffu + ((u >> 16) & 1u);
    return (unsigned short)(u >> 16);
}
__device__ __forceinline__ float bay_bf16_float(unsigned short h) {
    return __uint_as_float((unsigned int)h << 16);
}
// Two floats as packed bf16 hi + lo pairs (a in the low halves, b in the high halves), each
// rounded to nearest even by one cvt.rn.bf16x2.f32: hi = bf16(x), lo = bf16(x - hi).
__device__ __forceinline__ void bay_split_bf16x2(float a, float b, unsigned int& hi,
                                                 unsigned int& lo) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(b), "f"(a));
    const float ha = __uint_as_float(hi << 16), hb = __uint_as_float(hi & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(__fsub_rn(b, hb)), "f"(__fsub_rn(a, ha)));
}

// Propose: BAY_PW walkers per CTA, a warp per walker with its lanes over the coordinates, so
// that the walker's row, its partner's and the outputs are read and written in whole
// sectors; the proposals also stay in shared memory (odd stride), from which one thread per
// walker evaluates the model's prep and walker terms in the model's own order.  2,048 walkers
// of 257 coordinates: 5.1 us, 268 us with one thread per walker for the rows too (a sector
// per float read or written); 8 walkers per CTA are 256 CTAs there.  BAY_PW is the host's (kernel grid), 8 while the rows fit in 48 KB.
// A source that may take global rows alone (BAY_ANY_SPACE 0) gets the global copies instead.
template <int MODE>  // 0 bare, 1 accu, 2 log density of the current positions
__device__ __forceinline__ void bay_gemm_propose_impl(const bay_stretch_params& P) {
#if BAY_ANY_SPACE
    __shared__ float sY[BAY_PW][DIM | 1];
#endif
    const unsigned int kind = MODE == 1 ? 1u : 0u;
    const unsigned int nk = MODE == 2 ? P.W : P.K;
    const unsigned int k0 = blockIdx.x * BAY_PW;
    const unsigned int warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    for (unsigned int i = warp; i < BAY_PW; i += 8u) {
        const unsigned int k = k0 + i;
        if (k >= nk) break;
        float* y = P.s_y + (size_t)k * DIM;
        const float* X = P.xs + (MODE == 2 ? (size_t)0 : (size_t)P.half * P.K * DIM) + (size_t)k * DIM;
        const float* S = X;
        float z = 0.0f;
        if (MODE != 2) {
            const unsigned int stream = MODE == 1 ? (P.half ? 2222u : 1111u) : (P.half ? 4444u : 3333u);
            bay_u4 c;
            c.x = k;
            c.y = P.ctl->step[kind] + P.step_off;
            c.z = stream;
            c.w = 0xbeeff00du;
            const bay_u4 r = bay_philox4x32_10(c, P.ctl->seed[kind] + P.half, 0xdecafbadu);
            z = bay_stretch_z(P.ctl->a, bay_u01(r.y));
            const unsigned int j = bay_partner(bay_u01(r.x), P.K);
            S = P.xs + (size_t)(1u - P.half) * P.K * DIM + (size_t)j * DIM;
            if (lane == 0u) {
                P.s_zu[3 * (size_t)k] = z;
                P.s_zu[3 * (size_t)k + 1] = bay_u01(r.z);
                P.s_zu[3 * (size_t)k + 2] = P.logfn[(size_t)P.half * P.K + k];
            }
        }
        // 8 coordinates per lane per pass, their loads all in flight
        for (unsigned int d0 = lane; d0 < DIM; d0 += 256u) {
            float xv[8], sv[8];
#pragma unroll
            for (unsigned int q = 0; q < 8u; ++q) {
                const unsigned int d = d0 + 32u * q;
                xv[q] = d < DIM ? X[d] : 0.0f;
                sv[q] = MODE != 2 && d < DIM ? S[d] : 0.0f;
            }
#pragma unroll
            for (unsigned int q = 0; q < 8u; ++q) {
                const unsigned int d = d0 + 32u * q;
                if (d >= DIM) continue;
                const float v = MODE == 2 ? xv[q] : __fmaf_rn(z, __fsub_rn(xv[q], sv[q]), sv[q]);
                y[d] = v;
#if BAY_ANY_SPACE
                sY[i][d] = v;
#endif
                const unsigned int f = d - BAY_GEMM_COEF;
                if (d < BAY_GEMM_COEF || f >= BAY_GEMM_F) continue;
                if (!P.s_bh) {
                    P.s_b[(size_t)k * BAY_GEMM_F + f] = v;
                } else {
                    // the tensor-core form's operand: coefficient = hi + lo, both bf16
                    const unsigned short h = bay_bf16_rn(v);
                    P.s_bh[(size_t)k * P.tc_fp + f] = h;
                    P.s_bl[(size_t)k * P.tc_fp + f] = bay_bf16_rn(__fsub_rn(v, bay_bf16_float(h)));
                }
            }
        }
    }
    __syncthreads();
    const unsigned int k = k0 + threadIdx.x;
    if (threadIdx.x < BAY_PW && k < nk) {
#if BAY_ANY_SPACE
        const float* y = sY[threadIdx.x];
#else
        const float* y = P.s_y + (size_t)k * DIM;
#endif
        const float* hyper = P.params + P.data_len;
        float pr[BAY_PREP_LEN];
#pragma unroll
        for (int i = 0; i < BAY_PREP_LEN; ++i) pr[i] = 0.0f;
        BAY_GEMM_PREP(hyper, P.params_len, DIM, y, pr);
#pragma unroll
        for (int i = 0; i < BAY_PREP_LEN; ++i) P.s_prep[(size_t)k * BAY_PREP_LEN + i] = pr[i];
        P.s_w[k] = BAY_GEMM_WALKER(P.gemm_rows, hyper, P.params_len, DIM, y);
    }
}

template <int MODE>
__device__ __forceinline__ void bay_gemm_rows_impl(const bay_stretch_params& P) {
    extern __shared__ __align__(128) float bay_smem[];
    float* Bs = bay_smem;                              // [F][BAY_SW]
    float* Xs = Bs + (size_t)BAY_GEMM_F * BAY_SW;      // [BAY_SF][BAY_XS]
    __shared__ float sPrep[BAY_SW][BAY_PREP_LEN];
    const unsigned int nk = MODE == 2 ? P.W : P.K;
    const unsigned int tid = threadIdx.x;
    const unsigned int k0 = blockIdx.x * BAY_SW;
    const unsigned int sb = blockIdx.y;
    const unsigned int rows = (unsigned int)P.gemm_rows;
    const float* A = P.params + P.gemm_base;
    // the tile's coefficient block, feature-major (walkers past nk are zero)
    for (unsigned int e = tid; e < BAY_GEMM_F * BAY_SW; e += blockDim.x) {
        const unsigned int f = e / BAY_SW, w = e - f * BAY_SW;
        Bs[e] = (k0 + w < nk) ? P.s_b[(size_t)(k0 + w) * BAY_GEMM_F + f] : 0.0f;
    }
    for (unsigned int e = tid; e < BAY_SW * BAY_PREP_LEN; e += blockDim.x) {
        const unsigned int w = e / BAY_PREP_LEN, i = e - w * BAY_PREP_LEN;
        sPrep[w][i] = (k0 + w < nk) ? P.s_prep[(size_t)(k0 + w) * BAY_PREP_LEN + i] : 0.0f;
    }
    const unsigned int wg = tid >> 4, rg = tid & 15u;
    const unsigned int w0 = wg * 8;
    float sum[8], cmp[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        sum[i] = 0.0f;
        cmp[i] = 0.0f;
    }
    const unsigned int rb = sb * P.s_sbrows;
    const unsigned int re = rb + P.s_sbrows < rows ? rb + P.s_sbrows : rows;
    for (unsigned int r0 = rb; r0 < re; r0 += BAY_SR) {
        float acc[8][8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
        for (unsigned int f0 = 0; f0 < BAY_GEMM_F; f0 += BAY_SF) {
            __syncthreads();
            // chunk of rows r0..r0+127, features f0..f0+31: reads run along each row
            for (unsigned int e = tid; e < BAY_SR * BAY_SF; e += blockDim.x) {
                const unsigned int r = e / BAY_SF, fl = e - r * BAY_SF;
                const unsigned int f = f0 + fl;
                Xs[fl * BAY_XS + r] = (r0 + r < re && f < BAY_GEMM_F)
                    ? __ldg(A + (size_t)(r0 + r) * P.gemm_ld + f) : 0.0f;
            }
            __syncthreads();
            const unsigned int fe = BAY_GEMM_F - f0 < BAY_SF ? BAY_GEMM_F - f0 : BAY_SF;
#pragma unroll 4
            for (unsigned int fl = 0; fl < fe; ++fl) {
                const float4 b0 = *reinterpret_cast<const float4*>(&Bs[(f0 + fl) * BAY_SW + w0]);
                const float4 b1 = *reinterpret_cast<const float4*>(&Bs[(f0 + fl) * BAY_SW + w0 + 4]);
                const float bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
                float xv[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) xv[j] = Xs[fl * BAY_XS + rg + 16 * j];
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[i][j] = __fmaf_rn(bv[i], xv[j], acc[i][j]);
            }
        }
        // row terms of this sub-block
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const unsigned int r = r0 + rg + 16 * j;
            if (r < re) {
                float aux[BAY_AUXS];
#pragma unroll
                for (int c = 0; c < BAY_AUXS; ++c)
                    aux[c] = BAY_GEMM_AUX > 0 ? __ldg(A + (size_t)r * P.gemm_ld + BAY_GEMM_AUXCOL + c) : 0.0f;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const unsigned int kw = k0 + w0 + i < nk ? k0 + w0 + i : nk - 1;
                    const float t = BAY_GEMM_TERM(acc[i][j], aux, (uint64_t)r,
                                                  P.s_y + (size_t)kw * DIM, sPrep[w0 + i]);
                    const float yk = __fsub_rn(t, cmp[i]);
                    const float s2 = __fadd_rn(sum[i], yk);
                    cmp[i] = __fsub_rn(__fsub_rn(s2, sum[i]), yk);
                    sum[i] = s2;
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        bay_cf v;
        v.hi = sum[i];
        v.lo = -cmp[i];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) v = bay_cadd(v, bay_cf_shfl_xor(v, o));
        const unsigned int kw = k0 + w0 + i;
        if (rg == 0 && kw < nk) {
            P.s_part[2 * ((size_t)sb * nk + kw)] = v.hi;
            P.s_part[2 * ((size_t)sb * nk + kw) + 1] = v.lo;
        }
    }
}

// Accept: CTA (256 walkers, a slice of BAY_AD coordinates).  Every slice's CTA decides for
// its walkers (the current log density is read from the proposal's scratch, so that the
// first slice's CTA may store the new one) and then moves its coordinates, the 256 rows'
// segments in whole sectors.  2,048 walkers of 257 coordinates: 11.7 us on 40 CTAs, 86 us
// with one thread copying its walker's row on 8.
#define BAY_AD 64u
template <int MODE>
__device__ __forceinline__ void bay_gemm_accept_impl(const bay_stretch_params& P) {
    __shared__ unsigned char sAcc[256];
    const unsigned int nk = MODE == 2 ? P.W : P.K;
    const unsigned int k0 = blockIdx.x * 256u, k = k0 + threadIdx.x;
    const unsigned int d0 = blockIdx.y * BAY_AD;
    const bool valid = k < nk;
    bool accepted = false;
    if (valid) {
        bay_cf s;
        s.hi = 0.0f;
        s.lo = 0.0f;
        for (unsigned int sb = 0; sb < P.s_nsb; ++sb) {
            bay_cf p;
            p.hi = P.s_part[2 * ((size_t)sb * nk + k)];
            p.lo = P.s_part[2 * ((size_t)sb * nk + k) + 1];
            s = bay_cadd(s, p);
        }
        const float ly = bay_cf_total(P.s_w[k], s);
        if (MODE == 2) {
            P.logfn[k] = ly;
        } else {
            const float* zu = P.s_zu + 3 * (size_t)k;      // stretch factor, uniform, log density
            accepted = bay_accept(zu[1], zu[0], ly, zu[2], MODE == 1 ? 1.0f : bay_beta(P));
            if (accepted && blockIdx.y == 0u) P.logfn[(size_t)P.half * P.K + k] = ly;
        }
    }
    if (MODE == 2) return;
    sAcc[threadIdx.x] = accepted ? 1 : 0;
    const int n_acc = __syncthreads_count(accepted);
    const unsigned int nv = nk - k0 < 256u ? nk - k0 : 256u;
    const unsigned int nd = DIM - d0 < BAY_AD ? DIM - d0 : BAY_AD;
    float* Xc = P.xs + (size_t)P.half * P.K * DIM + (size_t)k0 * DIM + d0;
    const float* Yc = P.s_y + (size_t)k0 * DIM + d0;
    {
        // thread: coordinate tid % 64 of every 4th walker, 8 loads in flight
        const unsigned int d = threadIdx.x % BAY_AD;
        for (unsigned int w0 = threadIdx.x / BAY_AD; w0 < nv; w0 += 32u) {
            float v[8];
#pragma unroll
            for (unsigned int i = 0; i < 8u; ++i) {
                const unsigned int w = w0 + 4u * i;
                v[i] = w < nv && d < nd && sAcc[w] ? Yc[(size_t)w * DIM + d] : 0.0f;
            }
#pragma unroll
            for (unsigned int i = 0; i < 8u; ++i) {
                const unsigned int w = w0 + 4u * i;
                if (w < nv && d < nd && sAcc[w]) Xc[(size_t)w * DIM + d] = v[i];
            }
        }
    }
    if (MODE != 1) return;
    // accu: acceptance count and the per-dim sums of this CTA's walkers (new positions)
    if (threadIdx.x == 0 && blockIdx.y == 0u && n_acc)
        atomicAdd(&P.ctl->accepted, (unsigned long long)n_acc);
    if (P.means_cap == 0) return;
    __syncthreads();
    float* out = P.part + ((size_t)P.step_off * 2 + P.half) * DIM * gridDim.x + blockIdx.x;
    if (threadIdx.x < nd) {
        const unsigned int d = threadIdx.x;
        bay_cf s;
        s.hi = 0.0f;
        s.lo = 0.0f;
        // in walker order; unrolled so that several rows' loads are in flight
#pragma unroll 8
        for (unsigned int w = 0; w < nv; ++w) {
            bay_cf y;
            y.hi = Xc[(size_t)w * DIM + d];
            y.lo = 0.0f;
            s = bay_cadd(s, y);
        }
        out[(size_t)(d0 + d) * gridDim.x] = __fadd_rn(s.hi, s.lo);
    }
}

extern "C" __global__ void __launch_bounds__(256) bay_gemm_propose_bare(bay_stretch_params P) {
    bay_gemm_propose_impl<0>(P);
}
extern "C" __global__ void __launch_bounds__(256) bay_gemm_propose_accu(bay_stretch_params P) {
    bay_gemm_propose_impl<1>(P);
}
extern "C" __global__ void __launch_bounds__(256) bay_gemm_propose_logfn(bay_stretch_params P) {
    bay_gemm_propose_impl<2>(P);
}
extern "C" __global__ void __launch_bounds__(256) bay_gemm_rows_move(bay_stretch_params P) {
    bay_gemm_rows_impl<0>(P);
}
extern "C" __global__ void __launch_bounds__(256) bay_gemm_rows_logfn(bay_stretch_params P) {
    bay_gemm_rows_impl<2>(P);
}
extern "C" __global__ void __launch_bounds__(256) bay_gemm_accept_bare(bay_stretch_params P) {
    bay_gemm_accept_impl<0>(P);
}
extern "C" __global__ void __launch_bounds__(256) bay_gemm_accept_accu(bay_stretch_params P) {
    bay_gemm_accept_impl<1>(P);
}
extern "C" __global__ void __launch_bounds__(256) bay_gemm_accept_logfn(bay_stretch_params P) {
    bay_gemm_accept_impl<2>(P);
}

#if BAY_GEMM_TC
// ---------------------------------------------------------------- GEMM form, tensor cores
// The rows launch of the streaming form with eta on the 5th-generation tensor cores:
// eta[walker][row] = sum_f B[walker][f] A[row][f], A and B each split into bf16 hi + lo
// and three products (hi.hi + hi.lo + lo.hi) accumulated in fp32 in tensor memory; the
// dropped lo.lo product is below 2^-16 of each term.  tcgen05.mma kind::f16 with
// M = 128 walkers (TMEM lanes), N = 128 rows (TMEM columns), K = 16 per instruction,
// the rows K-major in shared memory with the 128-byte swizzle TMA writes, the walkers the
// same or in tensor memory (BAY_TC_ATM).
// CTA roles: warp 0 -- TMA producer (the CTA's walker operand once, then each 128-row
// tile in 64-feature chunks through a ring of BAY_TC_STAGES stages); warp 1 -- TMEM
// allocation and the MMA issue (one thread); warps 2 .. 17 -- epilogue, a thread per
// walker and share of a tile's rows: tcgen05.ld of its TMEM lane, the model's row terms,
// a compensated sum over the super-block's rows.  A model may give the terms of 16 rows at
// once (BAY_TERM16: their sum, and values that a thread carries over its rows, whose
// contribution is added at the end as hi + lo); rows past the last whole batch of 16 take the
// term by itself.  Two accumulator buffers in TMEM let the
// MMAs of tile t + 1 run under the epilogue of tile t.  Every wait is bounded in time; a wait
// that gives up sets the sampler's status word and the CTA's abort flag, and the CTA
// drains its own copies and MMAs, frees its TMEM and exits.
#ifndef BAY_TC_G
#define BAY_TC_G 1
#endif
#ifndef BAY_TC_STAGES
#define BAY_TC_STAGES 2
#endif
#define BAY_TC_FP ((BAY_GEMM_F + 63) / 64 * 64)
#define BAY_TC_KC (BAY_TC_FP / 64)
#define BAY_TC_TILE 16384u                      // one 128 x 64 bf16 operand chunk
// With one sub-tile and up to 256 features the walker operand lies in tensor memory (hi and
// lo of a 64-feature chunk in 32 columns each, after the two accumulator buffers; 512 columns
// in all).  From shared memory an M = N = 128 MMA reads 4 KB of each operand per 64 clocks,
// the 128 bytes a clock that shared memory delivers, and the copies of the next rows come on
// top: the tensor pipe could be busy 75 % of the time, and was (1.13 ms for 2,048 walkers x
// 524,589 rows x 256 features).  Two sub-tiles leave no columns for it (and share the rows).
#define BAY_TC_ATM (BAY_TC_G == 1 && BAY_TC_KC <= 4)
#define BAY_TC_WBYTES (BAY_TC_ATM ? 0u : (unsigned int)BAY_TC_G * BAY_TC_KC * 2u * BAY_TC_TILE)
#define BAY_TC_SBYTES (2u * BAY_TC_TILE)        // a stage: rows hi + lo chunk
#define BAY_TC_AUXF (128u * BAY_AUXS)
#define BAY_TC_NEPI 512u                        // epilogue threads (16 warps)
#define BAY_TC_THREADS 576
// Order of a 64-feature chunk's products in the accumulator.  The tensor core cuts sums off
// (toward zero), so that every product added to the large sum takes some 2^-25 of it: with a
// model that sums its rows' terms exactly enough to show it, the small products come first.
#define BAY_TC_LO_FIRST BAY_TERM16
#if BAY_TERM16
#define BAY_TC_EPI_UNROLL 2     // its arithmetic bounds the launch: logistic 2.79 -> 2.52 ms
#else
#define BAY_TC_EPI_UNROLL 1     // (tensor-bound: robust_t 0.96 ms a launch, 0.975 unrolled)
#endif
#define BAY_TC_COLS (BAY_TC_G == 2 || BAY_TC_ATM ? 512u : 256u)
#define BAY_TC_WAIT_NS 2000000000ull
// instruction descriptor: fp32 accumulator, bf16 A and B, both K-major, N = 128, M = 128
#define BAY_TC_IDESC ((1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24))

// the four TMA tensor maps (CUtensorMap, 128 bytes each), a __grid_constant__ parameter
struct __align__(64) bay_tmaps {
    unsigned long long xh[16];   // matrix rows, bf16 hi: dims {tc_fp, rows_pad}, box {64, 128}
    unsigned long long xl[16];   // matrix rows, bf16 lo
    unsigned long long bh[16];   // coefficient block, bf16 hi: dims {tc_fp, walkers_pad}
    unsigned long long bl[16];   // coefficient block, bf16 lo
};

__device__ __forceinline__ unsigned long long bay_globaltimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Wait for the completion of the phase of parity `par` of the mbarrier at shared address
// `bar`.  Gives up after BAY_TC_WAIT_NS, or as soon as another role has given up (abort
// flag set; pass abort = nullptr for a wait that must not be cut short).  Giving up on
// time sets the abort flag and the sampler's status word.
__device__ __forceinline__ bool bay_tc_wait(unsigned int bar, unsigned int par,
                                            volatile unsigned int* abort, unsigned int* status) {
    unsigned long long t0 = 0;
    for (unsigned int it = 0;; ++it) {
        unsigned int ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok) : "r"(bar), "r"(par) : "memory");
        if (ok) return true;
        if ((it & 15u) == 0u) {
            if (abort && *abort) return false;
            const unsigned long long t = bay_globaltimer();
            if (it == 0u) {
                t0 = t;
            } else if (t - t0 > BAY_TC_WAIT_NS) {
                if (abort) *abort = 1u;
                atomicOr(status, 2u);
                return false;
            }
        }
    }
}

__device__ __forceinline__ void bay_mbar_init(unsigned int bar, unsigned int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bay_expect_tx(unsigned int bar, unsigned int bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bay_tma2d(unsigned int dst, const void* map, int c0, int c1,
                                          unsigned int bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"((unsigned long long)map), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
// shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1024 B apart
__device__ __forceinline__ unsigned long long bay_sdesc(unsigned int saddr) {
    return (unsigned long long)((saddr & 0x3FFFFu) >> 4)
         | (1ull << 16)                                    // leading offset (unused here)
         | ((unsigned long long)(1024u >> 4) << 32)        // stride offset
         | (1ull << 46)                                    // tcgen05 descriptor version
         | (2ull << 61);                                   // 128-byte swizzle
}
__device__ __forceinline__ void bay_mma(unsigned int d, unsigned long long a, unsigned long long b,
                                        unsigned int acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
        ::"r"(d), "l"(a), "l"(b), "r"(BAY_TC_IDESC), "r"(acc) : "memory");
}
// the A operand in tensor memory: lane = row, two consecutive K elements per column
__device__ __forceinline__ void bay_mma_ta(unsigned int d, unsigned int a, unsigned long long b,
                                           unsigned int acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
        ::"r"(d), "r"(a), "l"(b), "r"(BAY_TC_IDESC), "r"(acc) : "memory");
}
// 128 bytes -> 32 consecutive TMEM columns of this thread's lane
__device__ __forceinline__ void bay_tmem_st32(unsigned int ta, const uint4 (&v)[8]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
        "%11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, "
        "%29, %30, %31, %32};"
        ::"r"(ta), "r"(v[0].x), "r"(v[0].y), "r"(v[0].z), "r"(v[0].w), "r"(v[1].x), "r"(v[1].y),
        "r"(v[1].z), "r"(v[1].w), "r"(v[2].x), "r"(v[2].y), "r"(v[2].z), "r"(v[2].w), "r"(v[3].x),
        "r"(v[3].y), "r"(v[3].z), "r"(v[3].w), "r"(v[4].x), "r"(v[4].y), "r"(v[4].z), "r"(v[4].w),
        "r"(v[5].x), "r"(v[5].y), "r"(v[5].z), "r"(v[5].w), "r"(v[6].x), "r"(v[6].y), "r"(v[6].z),
        "r"(v[6].w), "r"(v[7].x), "r"(v[7].y), "r"(v[7].z), "r"(v[7].w) : "memory");
}
__device__ __forceinline__ void bay_mma_commit(unsigned int bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bay_tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void bay_tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// 16 consecutive TMEM columns of this thread's lane
__device__ __forceinline__ void bay_tmem_ld16(unsigned int ta, float (&v)[16]) {
    unsigned int r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
        "%11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(ta));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

template <int MODE>  // 0: move (K walkers of the moving half), 2: log density of all W
__device__ __forceinline__ void bay_gemm_rows_tc_impl(const bay_stretch_params& P,
                                                      const bay_tmaps& T) {
    extern __shared__ __align__(1024) unsigned char bay_smem_tc[];
    const unsigned int raw = (unsigned int)__cvta_generic_to_shared(bay_smem_tc);
    const unsigned int pad = ((raw + 1023u) & ~1023u) - raw;
    unsigned char* sm = bay_smem_tc + pad;
    const unsigned int s_wop = raw + pad;                    // walker operand [G][KC][hi,lo]
    const unsigned int s_stg = s_wop + BAY_TC_WBYTES;        // row stages [S][hi,lo]
    float* saux = (float*)(sm + BAY_TC_WBYTES + BAY_TC_STAGES * BAY_TC_SBYTES);  // [2][AUXF]
    unsigned long long* bars = (unsigned long long*)(saux + 2 * BAY_TC_AUXF);
    volatile unsigned int* flags = (volatile unsigned int*)(bars + 2 * BAY_TC_STAGES + 6);
    const unsigned int bar0 = (unsigned int)__cvta_generic_to_shared(bars);
    // barriers: full[S], empty[S], tmem full[2], tmem empty[2], walker operand, drain
    const unsigned int b_full = bar0, b_empty = bar0 + 8u * BAY_TC_STAGES;
    const unsigned int b_tfull = bar0 + 16u * BAY_TC_STAGES, b_tempty = b_tfull + 16u;
    const unsigned int b_wop = b_tempty + 16u, b_drain = b_wop + 8u;
    // flags: [0] TMEM base, [1] abort, [2 + 2 set + buffer] epilogue go flags
    volatile unsigned int* abort = flags + 1;
    unsigned int* status = &P.ctl->status;

    const unsigned int warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const unsigned int nk = MODE == 2 ? P.W : P.K;
    const unsigned int k0 = blockIdx.x * (128u * BAY_TC_G);
    const unsigned int rows = (unsigned int)P.gemm_rows;
    const unsigned int rb = blockIdx.y * P.s_sbrows;
    const unsigned long long re64 = (unsigned long long)rb + P.s_sbrows;
    const unsigned int re = re64 < rows ? (unsigned int)re64 : rows;
    const unsigned int ntile = (re - rb + 127u) / 128u;

    if (threadIdx.x == 0) {
        for (unsigned int s = 0; s < BAY_TC_STAGES; ++s) {
            bay_mbar_init(b_full + 8u * s, 1u);
            bay_mbar_init(b_empty + 8u * s, 1u);
        }
        for (unsigned int b = 0; b < 2; ++b) {
            bay_mbar_init(b_tfull + 8u * b, 1u);
            bay_mbar_init(b_tempty + 8u * b, BAY_TC_NEPI / 32u);
        }
        bay_mbar_init(b_wop, BAY_TC_ATM ? BAY_TC_NEPI / 32u : 1u);
        bay_mbar_init(b_drain, 1u);
        flags[1] = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        const unsigned int dst = (unsigned int)__cvta_generic_to_shared((const void*)flags);
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(dst), "r"(BAY_TC_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    bay_tc_fence_before();
    __syncthreads();
    bay_tc_fence_after();
    const unsigned int tmem = flags[0];

    if (warp == 0) {
        if (lane == 0) {
            // ---- TMA producer
            if (!BAY_TC_ATM) bay_expect_tx(b_wop, BAY_TC_WBYTES);
            for (unsigned int g = 0; g < (BAY_TC_ATM ? 0u : BAY_TC_G); ++g)
                for (unsigned int c = 0; c < BAY_TC_KC; ++c) {
                    const unsigned int dst = s_wop + ((g * BAY_TC_KC + c) * 2u) * BAY_TC_TILE;
                    bay_tma2d(dst, T.bh, (int)(c * 64u), (int)(k0 + g * 128u), b_wop);
                    bay_tma2d(dst + BAY_TC_TILE, T.bl, (int)(c * 64u), (int)(k0 + g * 128u), b_wop);
                }
            unsigned int issued = 0;
            bool ok = true;
            for (unsigned int t = 0; t < ntile && ok; ++t) {
                for (unsigned int c = 0; c < BAY_TC_KC; ++c) {
                    const unsigned int s = issued % BAY_TC_STAGES, u = issued / BAY_TC_STAGES;
                    if (u > 0u && !bay_tc_wait(b_empty + 8u * s, (u - 1u) & 1u, abort, status)) {
                        ok = false;
                        break;
                    }
                    const unsigned int dst = s_stg + s * BAY_TC_SBYTES;
                    bay_expect_tx(b_full + 8u * s, BAY_TC_SBYTES);
                    bay_tma2d(dst, T.xh, (int)(c * 64u), (int)(rb + t * 128u), b_full + 8u * s);
                    bay_tma2d(dst + BAY_TC_TILE, T.xl, (int)(c * 64u), (int)(rb + t * 128u),
                              b_full + 8u * s);
                    ++issued;
                }
            }
            // drain: every copy issued here has landed before the CTA may exit
            bay_tc_wait(b_wop, 0u, nullptr, status);
            for (unsigned int i = issued > BAY_TC_STAGES ? issued - BAY_TC_STAGES : 0u; i < issued; ++i)
                bay_tc_wait(b_full + 8u * (i % BAY_TC_STAGES), (i / BAY_TC_STAGES) & 1u, nullptr, status);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // ---- MMA issue
            bool ok = bay_tc_wait(b_wop, 0u, abort, status);
            bay_tc_fence_after();
            unsigned int i = 0;
            for (unsigned int t = 0; t < ntile && ok; ++t) {
                const unsigned int b = t & 1u, ub = t >> 1;
                if (ub > 0u && !(ok = bay_tc_wait(b_tempty + 8u * b, (ub - 1u) & 1u, abort, status)))
                    break;
                bay_tc_fence_after();
                const unsigned int d0 = tmem + b * (128u * BAY_TC_G);
                for (unsigned int c = 0; c < BAY_TC_KC; ++c, ++i) {
                    const unsigned int s = i % BAY_TC_STAGES, u = i / BAY_TC_STAGES;
                    if (!(ok = bay_tc_wait(b_full + 8u * s, u & 1u, abort, status))) break;
                    bay_tc_fence_after();
                    const unsigned int xs = s_stg + s * BAY_TC_SBYTES;
#pragma unroll
                    for (unsigned int g = 0; g < BAY_TC_G; ++g) {
                        const unsigned int wa = s_wop + ((g * BAY_TC_KC + c) * 2u) * BAY_TC_TILE;
                        const unsigned int d = d0 + g * 128u;
                        // the three products of K step ks
                        auto product = [&](unsigned int ks, unsigned int which, unsigned int acc) {
                            const unsigned long long x =
                                bay_sdesc(xs + (which == 1u ? BAY_TC_TILE : 0u) + 32u * ks);   // hi.lo: rows' lo
#if BAY_TC_ATM
                            bay_mma_ta(d, tmem + 256u + 64u * c + (which == 2u ? 32u : 0u) + 8u * ks, x, acc);
#else
                            bay_mma(d, bay_sdesc(wa + (which == 2u ? BAY_TC_TILE : 0u) + 32u * ks), x, acc);
#endif
                        };
#if BAY_TC_LO_FIRST
#pragma unroll
                        for (unsigned int ks = 0; ks < 4u; ++ks) {
                            product(ks, 1u, (c | ks) != 0u ? 1u : 0u);
                            product(ks, 2u, 1u);
                        }
#pragma unroll
                        for (unsigned int ks = 0; ks < 4u; ++ks) product(ks, 0u, 1u);
#else
#pragma unroll
                        for (unsigned int ks = 0; ks < 4u; ++ks) {
                            product(ks, 0u, (c | ks) != 0u ? 1u : 0u);
                            product(ks, 1u, 1u);
                            product(ks, 2u, 1u);
                        }
#endif
                    }
                    bay_mma_commit(b_empty + 8u * s);  // the stage is free once these finish
                }
                if (!ok) break;
                bay_mma_commit(b_tfull + 8u * b);
            }
            // drain: every MMA issued here has finished before TMEM is released
            bay_mma_commit(b_drain);
            bay_tc_wait(b_drain, 0u, nullptr, status);
        }
    } else {
        // ---- epilogue, 16 warps in 4 groups of 4 (a group covers the 128 TMEM lanes).
        //      G = 2: group e takes walker sub-tile e / 2, rows 64 (e % 2) .. + 63 of a tile;
        //      G = 1: group e takes sub-tile 0, rows 32 e .. 32 e + 31.  A thread owns one
        //      walker (its TMEM lane): per 16-row batch it evaluates the row terms, sums them
        //      pairwise and adds the batch sum to a Kahan-compensated running sum; the
        //      groups' partial sums of a walker are combined at the end in group order.
        constexpr unsigned int GPS = 4u / BAY_TC_G;        // groups per walker sub-tile
        constexpr unsigned int NCOL = 128u / GPS;          // rows of a tile per group
        const unsigned int grp = (warp - 2u) >> 2, q = warp & 3u;
        const unsigned int g = grp / GPS;
        const unsigned int c0 = NCOL * (grp % GPS);
        const unsigned int wl = 32u * q + lane;
        const unsigned int kw = k0 + g * 128u + wl;
        const bool wv = kw < nk;
        const unsigned int kc = wv ? kw : nk - 1u;
#if BAY_TC_ATM
        // the walker operand into tensor memory: group e takes the 64-feature chunk e, a
        // thread its walker's 128 bytes of hi and of lo (rows up to the padded walker count)
        if (grp < BAY_TC_KC) {
            const unsigned int ta = tmem + ((32u * q) << 16) + 256u + 64u * grp;
#pragma unroll
            for (unsigned int h = 0; h < 2u; ++h) {
                const uint4* src = reinterpret_cast<const uint4*>(
                    (h ? P.s_bl : P.s_bh) + (size_t)kw * P.tc_fp + 64u * grp);
                uint4 v[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = src[i];
                bay_tmem_st32(ta + 32u * h, v);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        }
        bay_tc_fence_before();
        __syncwarp();
        if (lane == 0u)
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(b_wop) : "memory");
#endif
        float prep[BAY_PREP_LEN];
#pragma unroll
        for (int i = 0; i < BAY_PREP_LEN; ++i) prep[i] = P.s_prep[(size_t)kc * BAY_PREP_LEN + i];
        const float* xw = P.s_y + (size_t)kc * DIM;
        // The groups of the same rows (one per sub-tile) are a set: they stage the rows' aux
        // values and wait for a tile together, on a named barrier of their own, so that the
        // sets drift apart and one's waiting is under another's arithmetic (a scheduler has a
        // warp of every group).
        constexpr unsigned int NSET = BAY_TC_NEPI / GPS;   // threads of a set
        constexpr unsigned int AUXS = NCOL * BAY_AUXS;     // aux values of its rows of a tile
        const unsigned int set = grp % GPS, es = g * 128u + ((threadIdx.x - 64u) & 127u);
        const float* auxg = P.gemm_lay + (size_t)(rb + c0) * BAY_AUXS;   // [rows_pad][AUXS]
        constexpr unsigned int MA = (AUXS + NSET - 1u) / NSET;
        float apre[MA];
#pragma unroll
        for (unsigned int m = 0; m < MA; ++m) {
            const unsigned int j = es + m * NSET;
            apre[m] = (j < AUXS && ntile > 0u) ? __ldg(auxg + j) : 0.0f;
        }
        float sum = 0.0f, cmp = 0.0f;
#if BAY_TERM16
        float carry[BAY_TERM16_CARRY];
        BAY_CAT(BAY_GEMM_TERM, _16_init)(carry);
#endif
        bool ok = true;
        for (unsigned int t = 0; t < ntile; ++t) {
            const unsigned int b = t & 1u;
            float* sa = saux + b * BAY_TC_AUXF;
#pragma unroll
            for (unsigned int m = 0; m < MA; ++m) {
                const unsigned int j = es + m * NSET;
                if (j < AUXS) sa[c0 * BAY_AUXS + j] = apre[m];
            }
            // next tile's aux values, in flight during this tile
#pragma unroll
            for (unsigned int m = 0; m < MA; ++m) {
                const unsigned int j = es + m * NSET;
                apre[m] = (j < AUXS && t + 1u < ntile)
                    ? __ldg(auxg + (size_t)(t + 1u) * BAY_TC_AUXF + j) : 0.0f;
            }
            // one thread of the set waits for the accumulator; the decision is shared so that
            // the set leaves the loop together (the named barrier is not bounded)
            volatile unsigned int* go = flags + 2u + 2u * set + b;
            if (es == 0u) *go = bay_tc_wait(b_tfull + 8u * b, (t >> 1) & 1u, abort, status) ? 1u : 0u;
            asm volatile("bar.sync %0, %1;" ::"r"(1u + set), "r"(NSET) : "memory");
            if (!*go) {
                ok = false;
                break;
            }
            bay_tc_wait(b_tfull + 8u * b, (t >> 1) & 1u, nullptr, status);  // already complete
            bay_tc_fence_after();
            const unsigned int r0 = rb + t * 128u;
            const unsigned int nrow = re - r0 < 128u ? re - r0 : 128u;
            const unsigned int ta = tmem + ((32u * q) << 16) + b * (128u * BAY_TC_G) + g * 128u + c0;
#pragma unroll BAY_TC_EPI_UNROLL
            for (unsigned int j0 = 0; j0 < NCOL; j0 += 16u) {
                float v[16];
                bay_tmem_ld16(ta + j0, v);
                const unsigned int jb = c0 + j0;   // the batch's first row within the tile
                // the batch's aux values: 16 * AUXS consecutive floats, 16-byte aligned
                float av[16 * BAY_AUXS];
#pragma unroll
                for (unsigned int i = 0; i < 4u * BAY_AUXS; ++i) {
                    const float4 a4 = reinterpret_cast<const float4*>(sa + jb * BAY_AUXS)[i];
                    av[4 * i] = a4.x;
                    av[4 * i + 1] = a4.y;
                    av[4 * i + 2] = a4.z;
                    av[4 * i + 3] = a4.w;
                }
#if BAY_TERM16
                if (jb + 16u <= nrow) {      // the model's sum of the rows' terms, and its carry
                    v[0] = BAY_CAT(BAY_GEMM_TERM, _16)(v, av, (uint64_t)(r0 + jb), xw, prep, carry);
                } else
#endif
                {
                    if (jb + 16u <= nrow) {
#pragma unroll
                        for (unsigned int jj = 0; jj < 16u; ++jj)
                            v[jj] = BAY_GEMM_TERM(v[jj], &av[jj * BAY_AUXS],
                                                  (uint64_t)(r0 + jb + jj), xw, prep);
                    } else {
#pragma unroll
                        for (unsigned int jj = 0; jj < 16u; ++jj)
                            v[jj] = jb + jj < nrow
                                ? BAY_GEMM_TERM(v[jj], &av[jj * BAY_AUXS], (uint64_t)(r0 + jb + jj), xw,
                                                prep)
                                : 0.0f;
                    }
#pragma unroll
                    for (unsigned int w = 8u; w >= 1u; w >>= 1)
#pragma unroll
                        for (unsigned int i = 0; i < w; ++i) v[i] = __fadd_rn(v[i], v[i + w]);
                }
                const float yk = __fsub_rn(v[0], cmp);
                const float s2 = __fadd_rn(sum, yk);
                cmp = __fsub_rn(__fsub_rn(s2, sum), yk);
                sum = s2;
            }
            bay_tc_fence_before();
            __syncwarp();
            if (lane == 0u)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(b_tempty + 8u * b) : "memory");
        }
        // the groups' partial sums of each walker, combined as compensated pairs in group
        // order; stage 0 is free once the last tile's MMAs (hence its copies) are complete
        float* xchg = (float*)(sm + BAY_TC_WBYTES);        // [4 groups][128 lanes][hi, lo]
#if BAY_TERM16
        {
            bay_cf c, r;
            r.hi = sum;
            r.lo = -cmp;
            c.hi = BAY_CAT(BAY_GEMM_TERM, _16_end)(carry, &c.lo);
            r = bay_cadd(r, c);
            sum = r.hi;
            cmp = -r.lo;
        }
#endif
        if (ok) {
            xchg[2 * (grp * 128u + wl)] = sum;
            xchg[2 * (grp * 128u + wl) + 1] = -cmp;
        }
        {   // all written; a walker's groups of different sets may have left at different tiles
            unsigned int all;
            asm volatile(
                "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.and.pred q, 5, %2, p;\n"
                " selp.u32 %0, 1, 0, q;\n}\n"
                : "=r"(all) : "r"(ok ? 1u : 0u), "r"(BAY_TC_NEPI) : "memory");
            ok = all != 0u;
        }
        if (ok && set == 0u && wv) {
            bay_cf a;
            a.hi = sum;
            a.lo = -cmp;
#pragma unroll
            for (unsigned int o = 1; o < GPS; ++o) {
                bay_cf p;
                p.hi = xchg[2 * ((grp + o) * 128u + wl)];
                p.lo = xchg[2 * ((grp + o) * 128u + wl) + 1];
                a = bay_cadd(a, p);
            }
            P.s_part[2 * ((size_t)blockIdx.y * nk + kw)] = a.hi;
            P.s_part[2 * ((size_t)blockIdx.y * nk + kw) + 1] = a.lo;
        }
    }
    bay_tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        bay_tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(BAY_TC_COLS) : "memory");
    }
}

extern "C" __global__ void __launch_bounds__(BAY_TC_THREADS, 1)
bay_gemm_rows_tc_move(bay_stretch_params P, const __grid_constant__ bay_tmaps T) {
    bay_gemm_rows_tc_impl<0>(P, T);
}
extern "C" __global__ void __launch_bounds__(BAY_TC_THREADS, 1)
bay_gemm_rows_tc_logfn(bay_stretch_params P, const __grid_constant__ bay_tmaps T) {
    bay_gemm_rows_tc_impl<2>(P, T);
}

// ---------------------------------------------------------------- GEMM form, tensor cores,
// resident matrix.  For matrices of at most 256 rows that fit in shared memory with the
// walker operand (e.g. a precision matrix): one launch per half-step, a CTA per 64
// walkers (M = 128 MMAs of which lanes 0..63 are read back: small CTAs, four per SM).  The sampler keeps an image of the matrix as the MMA's B operand -- bf16 hi
// and lo, rows padded to gemm_np (a multiple of 16), K-major in 128-byte-swizzled
// 64-feature atoms -- followed by the rows' aux values; one bulk copy brings it into
// shared memory while the CTA draws its proposals.  The proposals' coefficient blocks are
// split into bf16 hi + lo and written in the same swizzled layout as the A operand; one
// thread issues the 3 x (features / 16) MMAs (N = gemm_np rows, fp32 accumulators in
// TMEM); then each walker's row terms are read back from its TMEM lane (two warps per
// lane group, half of the rows each), summed pairwise with a Kahan carry and combined,
// and the accept step and write-back follow as in the SIMT form.
#ifndef BAY_TR_W
#define BAY_TR_W 64u                                    // walkers per CTA: 64 or 128
#endif
#define BAY_TR_ATOM (BAY_TR_W * 128u)                   // BAY_TR_W walkers x 64 bf16 (one atom)
#define BAY_TR_DPAD (DIM | 1)

__device__ __forceinline__ void bay_tmem_ld8(unsigned int ta, float (&v)[8]) {
    unsigned int r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                   "=r"(r[6]), "=r"(r[7])
                 : "r"(ta));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// n8 (1..4, warp-uniform) loads of 8 TMEM columns each from ta, ta + 8, ..., then one wait:
// the loads' latencies overlap.  v[8 q + i] = column ta + 8 q + i of the thread's lane.
__device__ __forceinline__ void bay_tmem_ld32(unsigned int ta, unsigned int n8, float (&v)[32]) {
    unsigned int r[32];
#pragma unroll
    for (unsigned int q = 0; q < 4u; ++q) {
        if (q < n8)
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                         : "=r"(r[8 * q]), "=r"(r[8 * q + 1]), "=r"(r[8 * q + 2]), "=r"(r[8 * q + 3]),
                           "=r"(r[8 * q + 4]), "=r"(r[8 * q + 5]), "=r"(r[8 * q + 6]), "=r"(r[8 * q + 7])
                         : "r"(ta + 8u * q));
        else
#pragma unroll
            for (int i = 0; i < 8; ++i) r[8 * q + i] = 0u;
    }
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void bay_mma_n(unsigned int d, unsigned long long a, unsigned long long b,
                                          unsigned int idesc, unsigned int acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}

// 8 consecutive floats (dims 8u .. 8u + 7) of a walker row: float4 loads when rows are
// 16-byte aligned (DIM % 4 == 0), float2 when 8-byte aligned, else scalar; zero past DIM
// or when !ok (no access at all).  In the persistent form other CTAs rewrote the rows
// since this SM last read them: the grid barrier's acquire orders these loads after those
// writes.
__device__ __forceinline__ void bay_tr_ld8(const float* row, unsigned int u, bool ok, float (&v)[8]) {
    const unsigned int d0 = 8u * u;
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 0.0f;
    if (!ok) return;
    if (d0 + 8u <= DIM && DIM % 4u == 0u) {
        const float4 a = *(const float4*)(row + d0), b = *(const float4*)(row + d0 + 4u);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else if (d0 + 8u <= DIM && DIM % 2u == 0u) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 a = *(const float2*)(row + d0 + 2u * i);
            v[2 * i] = a.x;
            v[2 * i + 1] = a.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (d0 + i < DIM) v[i] = row[d0 + i];
    }
}

// The gather of the resident tensor-core form takes rows in items of BAY_TR_V dims.  Rows of
// at most 64 dims, even: of what one aligned load brings, 16 or 8 bytes, so that consecutive
// threads read consecutive addresses (8-dim items read every row's sectors 2 to 4 times from
// L1): 65,536 walkers of 50 and of 20 dims 7.1 -> 6.6 and 5.5 -> 5.0 us a launch.  Else 8
// dims, a whole unit of the A operand: longer rows take several rounds of loads either way
// (98 and 100 dims 13.2 -> 13.5 and 27.0 -> 27.2 us with the short items), odd ones single
// floats whose halves would go to the operand one at a time or in a pass of their own (63
// dims 7.6 -> 8.3 us).
#define BAY_TR_V (DIM > 64u || DIM % 2u ? 8u : (DIM % 4u ? 2u : 4u))
__device__ __forceinline__ void bay_tr_ld(const float* row, unsigned int u, bool ok, float (&v)[8]) {
    bay_tr_ld8(row, u, ok, v);
}
__device__ __forceinline__ void bay_tr_ld(const float* row, unsigned int u, bool ok, float (&v)[4]) {
    const float4 a = ok ? *(const float4*)(row + 4u * u) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
__device__ __forceinline__ void bay_tr_ld(const float* row, unsigned int u, bool ok, float (&v)[2]) {
    const float2 a = ok ? *(const float2*)(row + 2u * u) : make_float2(0.0f, 0.0f);
    v[0] = a.x; v[1] = a.y;
}

// the store counterpart of bay_tr_ld8 (dims past DIM are not written)
__device__ __forceinline__ void bay_tr_st8(float* row, unsigned int u, const float (&v)[8]) {
    const unsigned int d0 = 8u * u;
    if (d0 + 8u <= DIM && DIM % 4u == 0u) {
        *(float4*)(row + d0) = make_float4(v[0], v[1], v[2], v[3]);
        *(float4*)(row + d0 + 4u) = make_float4(v[4], v[5], v[6], v[7]);
    } else if (d0 + 8u <= DIM && DIM % 2u == 0u) {
#pragma unroll
        for (int i = 0; i < 4; ++i) *(float2*)(row + d0 + 2u * i) = make_float2(v[2 * i], v[2 * i + 1]);
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (d0 + i < DIM) row[d0 + i] = v[i];
    }
}

// 16-byte unit u (8 features) of walker row w in an A atom, at unit u ^ (w % 8) of its
// 128-byte row (the 128B swizzle); hi atoms first, lo atoms BAY_TC_KC atoms later
__device__ __forceinline__ void bay_tr_put_a(unsigned int s_a, unsigned int w, unsigned int u,
                                             const unsigned int (&hw)[4], const unsigned int (&lw)[4]) {
    const unsigned int off = (u >> 3) * BAY_TR_ATOM + w * 128u + (((u & 7u) ^ (w & 7u)) << 4);
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(s_a + off), "r"(hw[0]),
                 "r"(hw[1]), "r"(hw[2]), "r"(hw[3]) : "memory");
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
                 ::"r"(s_a + BAY_TC_KC * BAY_TR_ATOM + off), "r"(lw[0]), "r"(lw[1]), "r"(lw[2]),
                 "r"(lw[3]) : "memory");
}
// its halves (4 features) and quarters (2 features), the same places
__device__ __forceinline__ void bay_tr_put_a(unsigned int s_a, unsigned int w, unsigned int u,
                                             const unsigned int (&hw)[2], const unsigned int (&lw)[2]) {
    const unsigned int off = (u >> 4) * BAY_TR_ATOM + w * 128u + ((((u >> 1) & 7u) ^ (w & 7u)) << 4) +
                             8u * (u & 1u);
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(s_a + off), "r"(hw[0]), "r"(hw[1]) : "memory");
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};"
                 ::"r"(s_a + BAY_TC_KC * BAY_TR_ATOM + off), "r"(lw[0]), "r"(lw[1]) : "memory");
}
__device__ __forceinline__ void bay_tr_put_a(unsigned int s_a, unsigned int w, unsigned int u,
                                             const unsigned int (&hw)[1], const unsigned int (&lw)[1]) {
    const unsigned int off = (u >> 5) * BAY_TR_ATOM + w * 128u + ((((u >> 2) & 7u) ^ (w & 7u)) << 4) +
                             4u * (u & 3u);
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(s_a + off), "r"(hw[0]) : "memory");
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(s_a + BAY_TC_KC * BAY_TR_ATOM + off), "r"(lw[0]) : "memory");
}

// Grid barrier k (k = 1, 2, ... within a launch) of a cooperative launch (every CTA
// resident): each CTA adds 1 to the arrival count (a release reduction, no reply awaited)
// and waits until the count reaches k * nblocks; the count only grows during a launch.
// Bounded: a CTA that waits longer than BAY_TC_WAIT_NS raises ctl->abort and status bit 4;
// a raised abort ends every wait at once.  Returns false when the launch is being
// abandoned.  The count and the abort word are cleared before each launch.  `extra`
// arrivals beyond the grid (nonzero only in tests) make every barrier run out.
__device__ __forceinline__ bool bay_grid_barrier(bay_ctl* ctl, unsigned int nblocks, unsigned int k,
                                                 unsigned int extra) {
    __shared__ unsigned int s_go;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int go = 1u;
        volatile unsigned int* ab = &ctl->abort;
        if (*ab) {
            go = 0u;
        } else {
            const unsigned int target = k * nblocks + extra;
            __threadfence();                               // the CTA's writes before its arrival
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&ctl->gbar_count) : "memory");
            unsigned long long t0 = bay_globaltimer();
            for (unsigned int it = 0;; ++it) {
                unsigned int c;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(&ctl->gbar_count) : "memory");
                if (c >= target) break;
                __nanosleep(32);
                if ((it & 63u) == 63u) {
                    if (*ab) {
                        go = 0u;
                        break;
                    }
                    if (bay_globaltimer() - t0 > BAY_TC_WAIT_NS) {
                        *ab = 1u;
                        atomicOr(&ctl->status, 4u);
                        go = 0u;
                        break;
                    }
                }
            }
            __threadfence();
        }
        s_go = go;
    }
    __syncthreads();
    return s_go != 0u;
}

// Named barrier of one 256-thread tile group (ids 1..4; id 0 is the CTA's __syncthreads)
__device__ __forceinline__ void bay_gsync(unsigned int g) {
    asm volatile("bar.sync %0, 256;" ::"r"(g + 1u) : "memory");
}
__device__ __forceinline__ int bay_gsync_count(unsigned int g, bool p) {
    int n;
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n bar.red.popc.u32 %0, %1, 256, q;\n}\n"
                 : "=r"(n) : "r"(g + 1u), "r"((unsigned int)p) : "memory");
    return n;
}
// n = 256: the group's threads; 128: those that still take part
__device__ __forceinline__ bool bay_gsync_and(unsigned int g, bool p, unsigned int n) {
    unsigned int r;
    asm volatile("{\n .reg .pred q, o;\n setp.ne.u32 q, %2, 0;\n bar.red.and.pred o, %1, %3, q;\n"
                 " selp.u32 %0, 1, 0, o;\n}\n"
                 : "=r"(r) : "r"(g + 1u), "r"((unsigned int)p), "r"(n) : "memory");
    return r != 0u;
}

// Shared memory of one tile group after the A atoms: the proposals Yw [BAY_TR_W][DPAD] and
// 2 x 256 floats of reduction scratch, at least the 8 KB past the last atom that the
// M = 128 MMA reads (walker rows 64..127 of a 64-walker tile, never read back); 1 KB
// multiple.
#define BAY_TR_TAIL_RAW ((BAY_TR_W * BAY_TR_DPAD * 4u + 2048u) > (16384u - BAY_TR_ATOM) \
                         ? (BAY_TR_W * BAY_TR_DPAD * 4u + 2048u) : (16384u - BAY_TR_ATOM))
#define BAY_TR_TAIL ((BAY_TR_TAIL_RAW + 1023u) & ~1023u)
#define BAY_TR_GREG (2u * BAY_TC_KC * BAY_TR_ATOM + BAY_TR_TAIL)   // bytes per tile group

// The statistics of a tile: per-dim sums of its walkers' positions in a fixed order.
// BAY_TR_NG walker groups (256 / DIM, at most 8; one for DIM >= 128) of BAY_TR_WG
// consecutive walkers; thread (wg, d) sums its group in fp32 in walker order (pass 1, into
// scr[wg * DIM + d], or straight to out[d * ntiles] with one group), then thread d adds the
// groups' sums in group order (pass 2).  The per-step means add the tiles' sums in FP64.
#define BAY_TR_NG (DIM >= 128u ? 1u : (256u / DIM < 8u ? 256u / DIM : 8u))
#define BAY_TR_WG ((BAY_TR_W + BAY_TR_NG - 1u) / BAY_TR_NG)

// pass 1 over the rows in device memory (rows of DIM floats, nt walkers), threads 0..255
__device__ __forceinline__ void bay_tr_sums_pass1(const float* rows, unsigned int nt, unsigned int tid,
                                                  float* scr, float* out, unsigned int ntiles) {
    for (unsigned int t = tid; t < BAY_TR_NG * DIM; t += 256u) {
        const unsigned int wg = t / DIM, d = t - wg * DIM;
        float v = 0.0f;
#pragma unroll
        for (unsigned int i = 0; i < BAY_TR_WG; ++i) {
            const unsigned int w = wg * BAY_TR_WG + i;
            if (w < nt) v = __fadd_rn(v, rows[(size_t)w * DIM + d]);
        }
        if (BAY_TR_NG == 1u) out[(size_t)d * ntiles] = v;
        else scr[t] = v;
    }
}

// pass 2 (after a barrier that follows pass 1)
__device__ __forceinline__ void bay_tr_sums_pass2(unsigned int tid, const float* scr, float* out,
                                                  unsigned int ntiles) {
    if (BAY_TR_NG > 1u && tid < DIM) {
        float a = 0.0f;
#pragma unroll
        for (unsigned int wg = 0; wg < BAY_TR_NG; ++wg) a = __fadd_rn(a, scr[wg * DIM + tid]);
        out[(size_t)tid * ntiles] = a;
    }
}

// The resident tensor-core form.  A CTA holds G independent tile groups of 256 threads
// (G = 1: an ordinary CTA); each group has its own A operand, proposals, scratch, MMA
// barrier and TMEM columns, and syncs on its own named barrier; the matrix image is shared.
// PERSIST = false: one half-step (P.half, P.step_off), tile blockIdx.x (G = 1), launched
// with programmatic dependent launch.  PERSIST = true: a cooperative launch of m steps
// (both halves each, step offsets P.step_off .. + m - 1) over a grid of co-resident CTAs
// whose groups take tiles (g * gridDim.x + blockIdx.x) + k * gridDim.x * G of every half-step, with
// a grid barrier between half-steps; barriers, TMEM and the image are set up once.  Every
// tile computes what the per-launch form computes (same statistics slots), so the two
// forms give identical results.  A group whose bounded wait gives up raises ctl->abort
// and goes on to the next grid barrier, where the whole launch stops.
template <bool ACCU, bool LOGFN_ONLY, bool PERSIST, unsigned int G>
__device__ __forceinline__ void bay_stretch_tcr(const bay_stretch_params& P, unsigned int m) {
    // Shared memory: [matrix image][group 0: A hi atoms, lo atoms, Yw, red][group 1 ...].
    // The MMA runs M = 128 (an M = 64 form was measured no faster): with 64-walker tiles it
    // also reads the 8 KB after each atom's 64 rows (the next atom, or the group's Yw) as
    // walker rows 64..127, whose accumulator lanes are never read.
    extern __shared__ __align__(1024) unsigned char bay_smem_tr[];
    const unsigned int NP = P.gemm_np;                       // rows padded to 16
    const unsigned int rows = (unsigned int)P.gemm_rows;
    const unsigned int raw = (unsigned int)__cvta_generic_to_shared(bay_smem_tr);
    const unsigned int pad = ((raw + 1023u) & ~1023u) - raw;
    unsigned char* sm = bay_smem_tr + pad;
    const unsigned int img_bytes = 2u * BAY_TC_KC * NP * 128u + NP * BAY_AUXS * 4u;
    const unsigned int a_off0 = (img_bytes + 1023u) & ~1023u;
    const unsigned int s_img = raw + pad;
    const float* Aux = (const float*)(sm + 2u * BAY_TC_KC * NP * 128u);     // [NP][AUXS]
    __shared__ float sZ[G][BAY_TR_W], sU2[G][BAY_TR_W], sW[G][BAY_TR_W], sLx[G][BAY_TR_W];
    __shared__ unsigned int sJ[G][BAY_TR_W];
    __shared__ float sPrep[G][BAY_TR_W][BAY_PREP_LEN];
    __shared__ float sHalf[G][BAY_TR_W][2];
    __shared__ unsigned char sAcc[G][BAY_TR_W];
    __shared__ __align__(8) unsigned long long sBar[1 + G];
    __shared__ unsigned int sTmem, sOk[G];

    const unsigned int kind = ACCU ? 1u : 0u;
    const unsigned int g = G == 1u ? 0u : threadIdx.x >> 8;                // tile group
    const unsigned int tid = threadIdx.x & 255u, warp = tid >> 5, lane = tid & 31u;
    const unsigned int nk = LOGFN_ONLY ? P.W : P.K;
    const unsigned int ntiles = (nk + BAY_TR_W - 1u) / BAY_TR_W;
    const float* hyper = P.params + P.data_len;
    const unsigned int a_off = a_off0 + g * BAY_TR_GREG;
    const unsigned int s_a = s_img + a_off;
    float* Yw = (float*)(sm + a_off + 2u * BAY_TC_KC * BAY_TR_ATOM);         // [W][DPAD]
    float* red = Yw + BAY_TR_W * BAY_TR_DPAD;                                // [256]
    float* red2 = red + 256;                                                 // [256]
    const unsigned int bar_img = (unsigned int)__cvta_generic_to_shared(&sBar[0]);
    const unsigned int bar_mma = (unsigned int)__cvta_generic_to_shared(&sBar[1 + g]);
    unsigned int* status = &P.ctl->status;
    const unsigned int ncols = NP <= 32u ? 32u : (NP <= 64u ? 64u : (NP <= 128u ? 128u : 256u));

    // 1. barriers, TMEM (G x ncols columns), and the matrix image's bulk copy
    if (threadIdx.x == 0) {
        bay_mbar_init(bar_img, 1u);
        for (unsigned int q = 0; q < G; ++q)
            bay_mbar_init((unsigned int)__cvta_generic_to_shared(&sBar[1 + q]), 1u);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (threadIdx.x < 32u) {
        const unsigned int dst = (unsigned int)__cvta_generic_to_shared(&sTmem);
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(dst), "r"(ncols * G) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    bay_tc_fence_before();
    __syncthreads();
    bay_tc_fence_after();
    const unsigned int tmem = sTmem + g * ncols;
    // the matrix image is written once, when the sampler is created, so its copy may start
    // before this launch's dependency on the previous kernel resolves
    if (threadIdx.x == 0) {
        bay_expect_tx(bar_img, img_bytes);
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
            ::"r"(s_img), "l"(P.gemm_lay), "r"(img_bytes), "r"(bar_img) : "memory");
    }
    unsigned int mma_par = 0u;                  // phase parity of bar_mma's next completion
    const unsigned int nsteps = PERSIST ? m : 1u;
    const unsigned int h_lo = (PERSIST && !LOGFN_ONLY) ? 0u : P.half;
    const unsigned int h_hi = (PERSIST && !LOGFN_ONLY) ? 2u : P.half + 1u;
    // control words, constant during a launch: separate kernels between chunks write them,
    // and a launch after one of those starts only once it completed
    const unsigned int step0 = P.ctl->step[kind], seed0 = P.ctl->seed[kind];
    const float a_str = P.ctl->a, beta = ACCU ? 1.0f : bay_beta(P);
    // tiles g * gridDim.x + blockIdx.x, + G * gridDim.x, ...: consecutive tiles on
    // different SMs, every SM busy when the tiles outnumber the CTAs
    const unsigned int tile0 = g * gridDim.x + blockIdx.x;
    const unsigned int tstride = PERSIST ? gridDim.x * G : ntiles;
    constexpr unsigned int NU = (DIM + 7u) / 8u;               // 8-dim units of a row
    constexpr unsigned int NQ = BAY_TR_W * NU;                  // (walker, unit) items
    constexpr unsigned int IB = 2u;                             // items in flight per thread
    // the gather's items: V consecutive dims of a row
    constexpr unsigned int V = BAY_TR_V, RV = (DIM + V - 1u) / V;   // items of a row
    constexpr unsigned int NV = BAY_TR_W * RV;                       // of a tile
    constexpr unsigned int NB = (NV + 255u) / 256u;                  // of a thread
    // in flight per thread: 16 floats of each row, 32 where the shared memory leaves an SM 512
    // threads at most (80 dims 12.8 -> 12.1 us a launch)
    constexpr unsigned int FL = DIM > 64u && !PERSIST ? 32u : 16u;
    constexpr unsigned int CH = FL / V < NB ? FL / V : NB;
    // 2. proposals (Philox, z, partner) and the current log densities of a tile's walkers
    auto proposals = [&](unsigned int tile, unsigned int half, unsigned int step) {
        const unsigned int k0 = tile * BAY_TR_W;
        const unsigned int nt = nk - k0 < BAY_TR_W ? nk - k0 : BAY_TR_W;
        if (tid < nt) {
            const unsigned int k = k0 + tid;
            const unsigned int stream = ACCU ? (half ? 2222u : 1111u) : (half ? 4444u : 3333u);
            bay_u4 c;
            c.x = k;
            c.y = step;
            c.z = stream;
            c.w = 0xbeeff00du;
            const bay_u4 r = bay_philox4x32_10(c, seed0 + half, 0xdecafbadu);
            sZ[g][tid] = bay_stretch_z(a_str, bay_u01(r.y));
            sJ[g][tid] = bay_partner(bay_u01(r.x), P.K);
            sU2[g][tid] = bay_u01(r.z);
            sLx[g][tid] = P.logfn[(size_t)half * P.K + k];
        }
    };
    // the first gather pass's own rows (the tile's walkers): kept in registers, or, in the
    // persistent form (64 registers a thread at 1,024 threads), parked in Yw by the thread
    // that later reads them back
    float xpre[CH][V];
    auto own_rows = [&](const float* Xt, unsigned int nt) {
#pragma unroll
        for (unsigned int b = 0; b < CH; ++b) {
            const unsigned int q = b * 256u + tid;
            const unsigned int w = q / RV, u = q - w * RV;
            bay_tr_ld(V == 8u ? Xt + (size_t)w * DIM : Xt + V * (q - u), u, q < nt * RV, xpre[b]);
            if (PERSIST && q < NV) {
#pragma unroll
                for (unsigned int i = 0; i < V; ++i)
                    if (V * u + i < DIM) Yw[w * BAY_TR_DPAD + V * u + i] = xpre[b][i];
            }
        }
    };
#if BAY_GEMM_COEF == 0
    // the A operand's 16-byte units past the row's dims, zero for every tile (a unit with
    // some of them gets those later)
    {
        constexpr unsigned int U0 = V == 8u ? NU : DIM / 8u, U1 = BAY_TC_KC * 8u;
        constexpr unsigned int NZ = U1 > U0 ? U1 - U0 : 0u;
        const unsigned int zw[4] = {0u, 0u, 0u, 0u};
        for (unsigned int q = tid; q < BAY_TR_W * NZ; q += 256u) {
            const unsigned int w = q / (NZ ? NZ : 1u);
            bay_tr_put_a(s_a, w, U0 + (q - w * NZ), zw, zw);
        }
    }
#endif
    if (!PERSIST) {
        // One launch per half-step: this half's walkers last moved two launches back, so
        // their rows and log densities, like the draws, are final once the previous launch
        // began its work -- which it did only after waiting for its own predecessor, before
        // it let this launch start.  Load them now; only the partner rows (the half the
        // previous launch moves) wait for that launch and its memory.
        if (tile0 < ntiles) {
            const unsigned int k0 = tile0 * BAY_TR_W;
            const unsigned int nt = nk - k0 < BAY_TR_W ? nk - k0 : BAY_TR_W;
            if (!LOGFN_ONLY) proposals(tile0, P.half, step0 + P.step_off);
            own_rows(P.xs + (LOGFN_ONLY ? 0 : (size_t)P.half * P.K * DIM) + (size_t)k0 * DIM, nt);
        }
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    bool go = true;
    for (unsigned int si = 0; si < nsteps && go; ++si) {
    for (unsigned int half = h_lo; half < h_hi && go; ++half) {
    const unsigned int step_off = P.step_off + si;
    const unsigned int step = step0 + step_off;
    float* X = P.xs + (LOGFN_ONLY ? 0 : (size_t)half * P.K * DIM);
    const float* S = P.xs + (size_t)(1u - half) * P.K * DIM;
    // persistent: the group's first tile of this half-step loads its draws, own rows and
    // log densities before the grid barrier.  The tile-to-group map is fixed, so only this
    // group wrote those rows and densities (two half-steps back, ordered by its end-of-tile
    // barrier); during the half-step the barrier closes, other CTAs only read them.
    if (PERSIST && tile0 < ntiles) {
        const unsigned int nt0 = nk - tile0 * BAY_TR_W < BAY_TR_W ? nk - tile0 * BAY_TR_W : BAY_TR_W;
        if (!LOGFN_ONLY) proposals(tile0, half, step);
        own_rows(X + (size_t)tile0 * BAY_TR_W * DIM, nt0);
    }
    if (PERSIST && (si | (half - h_lo)) != 0u)
        go = bay_grid_barrier(P.ctl, gridDim.x, 2u * si + (half - h_lo), P.gbar_extra);
    if (!go) break;
    for (unsigned int tile = tile0; tile < ntiles; tile += tstride) {
    const unsigned int k0 = tile * BAY_TR_W;
    const unsigned int nt = nk - k0 < BAY_TR_W ? nk - k0 : BAY_TR_W;
    float* const Xt = X + (size_t)k0 * DIM;
    if (PERSIST && tile != tile0) {
        if (!LOGFN_ONLY) proposals(tile, half, step);
        own_rows(Xt, nt);
    }
    bay_gsync(g);
    // 3. Y of the tile (walker-major rows of odd stride): consecutive threads take
    //    consecutive items of a row (the tile's own rows are one contiguous block, a
    //    partner's row is 4 * DIM contiguous bytes), CH items' loads in flight per thread;
    //    with the coefficients at dim 0 the same thread splits its item into bf16 hi + lo
    //    and writes it to the A operand
    for (unsigned int q0 = 0; q0 < NV; q0 += CH * 256u) {
        float xv[CH][V], sv[CH][V];
#pragma unroll
        for (unsigned int b = 0; b < CH; ++b) {
            const unsigned int q = q0 + b * 256u + tid;
            const unsigned int w = q / RV, u = q - w * RV;
            const bool ok = q < nt * RV;
            if (q0 == 0u && PERSIST) {
#pragma unroll
                for (unsigned int i = 0; i < V; ++i)
                    xv[b][i] = (q < NV && V * u + i < DIM) ? Yw[w * BAY_TR_DPAD + V * u + i] : 0.0f;
            } else if (q0 == 0u) {
#pragma unroll
                for (unsigned int i = 0; i < V; ++i) xv[b][i] = xpre[b][i];
            } else {
                bay_tr_ld(V == 8u ? Xt + (size_t)w * DIM : Xt + V * (q - u), u, ok, xv[b]);
            }
            if (!LOGFN_ONLY) bay_tr_ld(S + (size_t)sJ[g][ok ? w : 0u] * DIM, u, ok, sv[b]);
        }
#pragma unroll
        for (unsigned int b = 0; b < CH; ++b) {
            const unsigned int q = q0 + b * 256u + tid;
            if (q < NV) {
                const unsigned int w = q / RV, u = q - w * RV;
                float y[V];
                const float z = LOGFN_ONLY ? 0.0f : sZ[g][w];
#pragma unroll
                for (unsigned int i = 0; i < V; ++i) {
                    y[i] = LOGFN_ONLY ? xv[b][i]
                                      : (w < nt ? __fmaf_rn(z, __fsub_rn(xv[b][i], sv[b][i]), sv[b][i]) : 0.0f);
                    if (V * u + i < DIM) Yw[w * BAY_TR_DPAD + V * u + i] = y[i];
                }
#if BAY_GEMM_COEF == 0
                if (V * u < BAY_TC_KC * 64u) {
                    unsigned int hw[V / 2u], lw[V / 2u];
#pragma unroll
                    for (unsigned int i = 0; i < V; i += 2u) {
                        const unsigned int f = V * u + i;
                        bay_split_bf16x2(f < BAY_GEMM_F ? y[i] : 0.0f,
                                         f + 1u < BAY_GEMM_F ? y[i + 1u] : 0.0f, hw[i / 2u], lw[i / 2u]);
                    }
                    bay_tr_put_a(s_a, w, u, hw, lw);
                }
#endif
            }
        }
    }
#if BAY_GEMM_COEF != 0
    // 4. the A operand from Yw (coefficients at dim BAY_GEMM_COEF): 16-byte units of hi, lo
    bay_gsync(g);
    for (unsigned int q = tid; q < BAY_TR_W * BAY_TC_KC * 8u; q += 256u) {
        const unsigned int w = q / (BAY_TC_KC * 8u), u = q - w * (BAY_TC_KC * 8u);
        unsigned int hw[4], lw[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const unsigned int f = u * 8u + 2u * i;
            const float v0 = f < BAY_GEMM_F ? Yw[w * BAY_TR_DPAD + BAY_GEMM_COEF + f] : 0.0f;
            const float v1 = f + 1u < BAY_GEMM_F ? Yw[w * BAY_TR_DPAD + BAY_GEMM_COEF + f + 1u] : 0.0f;
            bay_split_bf16x2(v0, v1, hw[i], lw[i]);
        }
        bay_tr_put_a(s_a, w, u, hw, lw);
    }
#endif
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // A visible to the MMAs
    bay_gsync(g);
    // One launch per half-step (FAST): the MMAs and all that follows are the business of the
    // epilogue's warps 0, 1, 4 and 5; warps 2, 3, 6 and 7 leave here, after the statistics of
    // the previous half-step in an accu launch -- this tile of the other half, final since
    // the previous launch completed and not written by this one: (step_off, 0) from the
    // launch of half 1, (step_off - 1, 1) from the launch of half 0 (the chunk's last one has
    // a launch of its own).  The same slots and order as bay_tr_sums_pass1 / pass2.
    // Their loads so run under the MMAs and the epilogue: 30,000 walkers of 99 dims 16.3 ->
    // 14.5 us an accu launch, 65,536 of 50 8.0 -> 7.8.
    constexpr bool FAST = !PERSIST && !LOGFN_ONLY;
    const unsigned int hand_id = 1u + G + g;        // named barriers 1..G are the groups'
    if (FAST && (warp & 2u)) {
        if (ACCU && P.means_cap != 0 && (half == 1u || step_off > 0u)) {
            float* const prev_out = P.part +
                ((size_t)(half == 1u ? step_off : step_off - 1u) * 2 + (1u - half)) * DIM * ntiles + tile;
            const unsigned int i0 = (warp >> 2) * 64u + (warp & 1u) * 32u + lane;
            const float* rows = P.xs + (size_t)(1u - half) * P.K * DIM + (size_t)k0 * DIM;
            for (unsigned int t = i0; t < BAY_TR_NG * DIM; t += 128u) {
                const unsigned int wg = t / DIM, d = t - wg * DIM;
                float v = 0.0f;
#pragma unroll
                for (unsigned int i = 0; i < BAY_TR_WG; ++i) {
                    const unsigned int w = wg * BAY_TR_WG + i;
                    if (w < nt) v = __fadd_rn(v, rows[(size_t)w * DIM + d]);
                }
                if (BAY_TR_NG == 1u) prev_out[(size_t)d * ntiles] = v;
                else red2[t] = v;
            }
            if (BAY_TR_NG > 1u) {
                asm volatile("bar.sync %0, 128;" ::"r"(1u + 2u * G + g) : "memory");
                for (unsigned int d = i0; d < DIM; d += 128u) {
                    float a = 0.0f;
#pragma unroll
                    for (unsigned int wg = 0; wg < BAY_TR_NG; ++wg) a = __fadd_rn(a, red2[wg * DIM + d]);
                    prev_out[(size_t)d * ntiles] = a;
                }
            }
        }
        continue;                                   // the tile is done (one per launch)
    }
    // 5. one thread: wait for the image, issue the MMAs, commit; the others precompute
    if (tid == 0) {
        unsigned int ok = bay_tc_wait(bar_img, 0u, nullptr, status) ? 1u : 0u;   // once done, stays
        if (ok) {
            bay_tc_fence_after();
            const unsigned int idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((NP >> 3) << 17) |
                                       ((128u >> 4) << 24);
            for (unsigned int c = 0; c < BAY_TC_KC; ++c) {
#pragma unroll
                for (unsigned int ks = 0; ks < 4u; ++ks) {
                    // past the features both sides are zeros (4,096 walkers of 98 and of 20
                    // dims 6.2 -> 6.1 and 3.16 -> 3.06 us a launch without those products)
                    if (64u * c + 16u * ks >= BAY_GEMM_F) break;
                    const unsigned int ao = c * BAY_TR_ATOM + 32u * ks;
                    const unsigned int bo = c * NP * 128u + 32u * ks;
                    const unsigned long long ah = bay_sdesc(s_a + ao);
                    const unsigned long long al = bay_sdesc(s_a + BAY_TC_KC * BAY_TR_ATOM + ao);
                    const unsigned long long bh = bay_sdesc(s_img + bo);
                    const unsigned long long bl = bay_sdesc(s_img + BAY_TC_KC * NP * 128u + bo);
                    bay_mma_n(tmem, ah, bh, idesc, (c | ks) != 0u ? 1u : 0u);
                    bay_mma_n(tmem, ah, bl, idesc, 1u);
                    bay_mma_n(tmem, al, bh, idesc, 1u);
                }
            }
        }
        bay_mma_commit(bar_mma);   // also arrives with nothing issued (a failed wait)
        sOk[g] = ok;
    }
    if (tid < BAY_TR_W) {
        float pr[BAY_PREP_LEN];
#pragma unroll
        for (int i = 0; i < BAY_PREP_LEN; ++i) pr[i] = 0.0f;
        float wt = 0.0f;
        if (tid < nt) {
            BAY_GEMM_PREP(hyper, P.params_len, DIM, &Yw[tid * BAY_TR_DPAD], pr);
            wt = BAY_GEMM_WALKER(P.gemm_rows, hyper, P.params_len, DIM, &Yw[tid * BAY_TR_DPAD]);
        }
#pragma unroll
        for (int i = 0; i < BAY_PREP_LEN; ++i) sPrep[g][tid][i] = pr[i];
        sW[g][tid] = wt;
    }
    // every thread waits for the MMAs (bounded; the commit arrives even if none were issued)
    // and observes the image copy itself before reading the aux values it brought
    const bool mma_done = bay_tc_wait(bar_mma, mma_par, nullptr, status);
    mma_par ^= 1u;
    const bool img_done = bay_tc_wait(bar_img, 0u, nullptr, status);
    // one verdict for the group's epilogue (a wait that gave up in any thread fails the tile)
    const bool ok = bay_gsync_and(g, mma_done && img_done, FAST ? 128u : 256u) && sOk[g] != 0u;
    bay_tc_fence_after();
    // 6. epilogue: warps 0, 1, 4, 5 read TMEM lanes 32 (w % 4) .. + 31 (walkers 0..63),
    //    rows [NP/2 * (w / 4), + NP/2) in 8-column loads; the two halves then combine
    if (32u * (warp & 3u) < BAY_TR_W) {
        const unsigned int wl = 32u * (warp & 3u) + lane;
        const unsigned int h = warp >> 2, half_rows = NP >> 1;
        const unsigned int c0 = h * half_rows;
        const unsigned int ta = tmem + ((32u * (warp & 3u)) << 16) + c0;
        const float* xw = &Yw[wl * BAY_TR_DPAD];
        float sum = 0.0f, cmp = 0.0f;
        // up to 32 columns per batch of loads (one wait), then per 8 columns: the row terms,
        // a pairwise sum, a Kahan step (the same order as one 8-column load at a time)
        for (unsigned int j1 = 0; j1 < half_rows; j1 += 32u) {
            const unsigned int n8 = (half_rows - j1) >= 32u ? 4u : (half_rows - j1) >> 3;
            float v32[32];
            bay_tmem_ld32(ta + j1, n8, v32);
#pragma unroll
            for (unsigned int q = 0; q < 4u; ++q) {
                if (q >= n8) break;
                float v[8];
#pragma unroll
                for (unsigned int i = 0; i < 8u; ++i) {
                    const unsigned int r = c0 + j1 + 8u * q + i;
                    v[i] = r < rows ? BAY_GEMM_TERM(v32[8u * q + i], &Aux[r * BAY_AUXS], (uint64_t)r, xw,
                                                    sPrep[g][wl])
                                    : 0.0f;
                }
#pragma unroll
                for (unsigned int s2 = 4u; s2 >= 1u; s2 >>= 1)
#pragma unroll
                    for (unsigned int i = 0; i < s2; ++i) v[i] = __fadd_rn(v[i], v[i + s2]);
                const float yk = __fsub_rn(v[0], cmp);
                const float t = __fadd_rn(sum, yk);
                cmp = __fsub_rn(__fsub_rn(t, sum), yk);
                sum = t;
            }
        }
        if (FAST) {
            if (h) {                                    // hand the second half over
                sHalf[g][wl][0] = sum;
                sHalf[g][wl][1] = -cmp;
                asm volatile("bar.arrive %0, 128;" ::"r"(hand_id) : "memory");
            } else {
                asm volatile("bar.sync %0, 128;" ::"r"(hand_id) : "memory");
                // 7. accept walker wl, write back its row and log density
                bool acc = false;
                if (wl < nt && ok) {
                    const unsigned int k = k0 + wl;
                    bay_cf t, a, b;
                    t.hi = sW[g][wl];
                    t.lo = 0.0f;
                    a.hi = sum;
                    a.lo = -cmp;
                    b.hi = sHalf[g][wl][0];
                    b.lo = sHalf[g][wl][1];
                    t = bay_cadd(t, bay_cadd(a, b));
                    const float ly = __fadd_rn(t.hi, t.lo);
                    acc = bay_accept(sU2[g][wl], sZ[g][wl], ly, sLx[g][wl], beta);
                    if (acc) {
                        P.logfn[(size_t)half * P.K + k] = ly;
                        const float* yr = &Yw[wl * BAY_TR_DPAD];
#pragma unroll 4
                        for (unsigned int u = 0; u < NU; ++u) {
                            float y[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i) y[i] = 8u * u + i < DIM ? yr[8u * u + i] : 0.0f;
                            bay_tr_st8(Xt + (size_t)wl * DIM, u, y);
                        }
                    }
                }
                if (ACCU) {
                    const unsigned int bal = __ballot_sync(0xffffffffu, acc);
                    if (lane == 0 && bal) atomicAdd(&P.ctl->accepted, (unsigned long long)__popc(bal));
                }
            }
        } else if (h) {                                 // second half of the rows
            sHalf[g][wl][0] = sum;
            sHalf[g][wl][1] = -cmp;
        } else {                                        // first half: red[wl], red[W + wl]
            red[wl] = sum;
            red[BAY_TR_W + wl] = -cmp;
        }
    }
    if (FAST) {
        if (!ok) break;
        continue;                                       // the tile is done (one per launch)
    }
    bay_tc_fence_before();
    bay_gsync(g);
    // 7. accept (one thread per walker), write-back, statistics
    bool accepted = false;
    if (tid < nt && ok) {
        const unsigned int k = k0 + tid;
        bay_cf t, a, b;
        t.hi = sW[g][tid];
        t.lo = 0.0f;
        a.hi = red[tid];
        a.lo = red[BAY_TR_W + tid];
        b.hi = sHalf[g][tid][0];
        b.lo = sHalf[g][tid][1];
        t = bay_cadd(t, bay_cadd(a, b));
        const float ly = __fadd_rn(t.hi, t.lo);
        if (LOGFN_ONLY) {
            P.logfn[k] = ly;
        } else {
            accepted = bay_accept(sU2[g][tid], sZ[g][tid], ly, sLx[g][tid], beta);
            if (accepted) P.logfn[(size_t)half * P.K + k] = ly;
        }
    }
    if (!LOGFN_ONLY) {
        if (tid < BAY_TR_W) sAcc[g][tid] = accepted ? 1 : 0;
        const int n_acc = bay_gsync_count(g, accepted);
        if (ACCU && PERSIST) {
            // the statistics need every walker's new position in Yw: the rejected walkers'
            // current rows are loaded (IB units in flight per thread), the accepted ones
            // stored
            for (unsigned int q0 = 0; q0 < NQ; q0 += IB * 256u) {
                float xv[IB][8];
#pragma unroll
                for (unsigned int b = 0; b < IB; ++b) {
                    const unsigned int q = q0 + b * 256u + tid;
                    const unsigned int w = q / NU, u = q - w * NU;
                    bay_tr_ld8(Xt + (size_t)w * DIM, u, q < NQ && w < nt && !sAcc[g][w < BAY_TR_W ? w : 0u],
                               xv[b]);
                }
#pragma unroll
                for (unsigned int b = 0; b < IB; ++b) {
                    const unsigned int q = q0 + b * 256u + tid;
                    const unsigned int w = q / NU, u = q - w * NU;
                    if (q < NQ && w < nt) {
                        float* yr = &Yw[w * BAY_TR_DPAD + 8u * u];
                        if (sAcc[g][w]) {
                            float y[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i) y[i] = 8u * u + i < DIM ? yr[i] : 0.0f;
                            bay_tr_st8(Xt + (size_t)w * DIM, u, y);
                        } else {
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                if (8u * u + i < DIM) yr[i] = xv[b][i];
                        }
                    }
                }
            }
        } else {
            // accepted walkers' rows to device memory
            for (unsigned int q = tid; q < NQ; q += 256u) {
                const unsigned int w = q / NU, u = q - w * NU;
                if (w < nt && sAcc[g][w]) {
                    const float* yr = &Yw[w * BAY_TR_DPAD + 8u * u];
                    float y[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) y[i] = 8u * u + i < DIM ? yr[i] : 0.0f;
                    bay_tr_st8(Xt + (size_t)w * DIM, u, y);
                }
            }
        }
        if (ACCU) {
            if (tid == 0 && n_acc) atomicAdd(&P.ctl->accepted, (unsigned long long)n_acc);
            if (PERSIST && P.means_cap != 0) {
                // the statistics of the tile's new positions (Yw) at the end of the tile
                bay_gsync(g);
                float* out = P.part + ((size_t)step_off * 2 + half) * DIM * ntiles + tile;
                for (unsigned int t = tid; t < BAY_TR_NG * DIM; t += 256u) {
                    const unsigned int wg = t / DIM, d = t - wg * DIM;
                    float v = 0.0f;
#pragma unroll
                    for (unsigned int i = 0; i < BAY_TR_WG; ++i) {
                        const unsigned int w = wg * BAY_TR_WG + i;
                        if (w < nt) v = __fadd_rn(v, Yw[w * BAY_TR_DPAD + d]);
                    }
                    if (BAY_TR_NG == 1u) out[(size_t)d * ntiles] = v;
                    else red[t] = v;
                }
                bay_gsync(g);
                bay_tr_sums_pass2(tid, red, out, ntiles);
            }
        }
    }
    if (PERSIST) {
        // the next tile rewrites Yw, red and the A operand, and its MMAs the accumulator
        bay_tc_fence_before();
        bay_gsync(g);
    }
    if (!ok) {
        // a bounded wait gave up: no more tiles; the persistent form raises the abort flag
        // and still meets the next grid barrier, which then stops the whole launch
        if (PERSIST && tid == 0) *(volatile unsigned int*)&P.ctl->abort = 1u;
        break;
    }
    }   // tiles
    }   // halves
    }   // steps
    // 8. release TMEM (every MMA completed before the epilogue read it); the image copy has
    //    landed (a group waited for it, or the bounded wait here)
    if (threadIdx.x == 0) bay_tc_wait(bar_img, 0u, nullptr, status);
    bay_tc_fence_before();
    __syncthreads();
    if (threadIdx.x < 32u) {
        bay_tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(sTmem),
                     "r"(ncols * G) : "memory");
    }
}

// The per-launch move kernels hold up to BAY_TR_G tile groups per CTA (1 or 2): one matrix-image
// copy and one TMEM allocation serve BAY_TR_G tiles; group g takes tile g * gridDim.x +
// blockIdx.x.  Same results for either.
#ifndef BAY_TR_G
#define BAY_TR_G 1u
#endif
extern "C" __global__ void __launch_bounds__(256 * BAY_TR_G) bay_tcr_bare(bay_stretch_params P) {
    bay_stretch_tcr<false, false, false, BAY_TR_G>(P, 1u);
}
extern "C" __global__ void __launch_bounds__(256 * BAY_TR_G) bay_tcr_accu(bay_stretch_params P) {
    bay_stretch_tcr<true, false, false, BAY_TR_G>(P, 1u);
}
extern "C" __global__ void __launch_bounds__(256) bay_tcr_logfn(bay_stretch_params P) {
    bay_stretch_tcr<false, true, false, 1u>(P, 1u);
}
// the statistics of the last half-step of a chunk (half P.half, step P.step_off): one CTA
// per tile, the same sums as the stretch launches
extern "C" __global__ void __launch_bounds__(256) bay_tcr_stats(bay_stretch_params P) {
    __shared__ float scr[256];
    const unsigned int tile = blockIdx.x, ntiles = gridDim.x, k0 = tile * BAY_TR_W;
    const unsigned int nt = P.K - k0 < BAY_TR_W ? P.K - k0 : BAY_TR_W;
    float* out = P.part + ((size_t)P.step_off * 2 + P.half) * DIM * ntiles + tile;
    bay_tr_sums_pass1(P.xs + (size_t)P.half * P.K * DIM + (size_t)k0 * DIM, nt, threadIdx.x, scr,
                      out, ntiles);
    __syncthreads();
    bay_tr_sums_pass2(threadIdx.x, scr, out, ntiles);
}
// persistent: one CTA of 4 tile groups per SM (1,024 threads, 64 registers each)
extern "C" __global__ void __launch_bounds__(1024, 1) bay_tcr_run_bare(bay_stretch_params P, unsigned int m) {
    bay_stretch_tcr<false, false, true, 4u>(P, m);
}
extern "C" __global__ void __launch_bounds__(1024, 1) bay_tcr_run_accu(bay_stretch_params P, unsigned int m) {
    bay_stretch_tcr<true, false, true, 4u>(P, m);
}
#endif  // BAY_GEMM_TC

#elif !BAY_TILED
// ---------------------------------------------------------------- plain form
// One thread per walker of the moving half, the model's LOGFN evaluated per thread
// (the reference's structure, with SoA coalesced loads and registers for Y).

// The params staged in shared memory (STAGED: a module with kernels of their own, named _s,
// launched with dynamic shared memory for them; else they stay in global memory, always so where
// the source may read them by global loads alone).  One kernel for both, with
// the density twice in it, had ptxas schedule the loads from global memory worse: 8,192 walkers
// x 65,536 rows of 65 floats 43.8 -> 62.4 ms an accu launch.  A density's loop reads them in order, all threads alike, a load
// every few arithmetic instructions of one dependent sum: from global memory, L1 hits
// included, a row of 2-D Gaussian data took 31 clocks however few warps there were, from
// shared memory 8 (8,192 walkers x 1,000 rows: 18.8 us a launch, now 5.7).
// One bulk copy, begun before the launch waits for its predecessor (the params never
// change while a sampler runs), the last floats past its 16-byte multiple by plain loads.
#if BAY_PLAIN_STAGED
#define BAY_PLAIN(name) name##_s
#else
#define BAY_PLAIN(name) name
#endif
struct bay_plain_sync {
    unsigned long long bar;
};
template <bool STAGED>
__device__ __forceinline__ void bay_stage_begin(bay_plain_sync* sy, const float* p, unsigned int n) {
    extern __shared__ __align__(16) float bay_psm[];
    if (!STAGED) return;
    const unsigned int bar = (unsigned int)__cvta_generic_to_shared(&sy->bar), bytes = (n * 4u) & ~15u;
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                     : "memory");
        if (bytes)
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                ::"r"((unsigned int)__cvta_generic_to_shared(bay_psm)), "l"(p), "r"(bytes), "r"(bar)
                : "memory");
    }
    if (bytes / 4u + threadIdx.x < n && threadIdx.x < 4u)
        bay_psm[bytes / 4u + threadIdx.x] = p[bytes / 4u + threadIdx.x];
    __syncthreads();
}
// Bounded wait (2 s) for the copy; false, with status bit 1 set, when it gave up.
template <bool STAGED>
__device__ __forceinline__ bool bay_stage_wait(bay_plain_sync* sy, unsigned int* status) {
    if (!STAGED) return true;
    const unsigned int bar = (unsigned int)__cvta_generic_to_shared(&sy->bar);
    unsigned long long t0 = 0;
    for (unsigned int it = 0;; ++it) {
        unsigned int ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n"
            " selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok) : "r"(bar) : "memory");
        if (ok) return true;
        if ((it & 15u) == 0u) {
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (it == 0u) {
                t0 = t;
            } else if (t - t0 > 2000000000ull) {
                if (status) atomicOr(status, 1u);
                return false;
            }
        }
    }
}
template <bool STAGED>
__device__ __forceinline__ float bay_density(unsigned int data_len, unsigned int params_len,
                                             const float* params, const float* x) {
    extern __shared__ __align__(16) float bay_psm[];
    if (STAGED) return BAY_LOGFN(data_len, params_len, bay_psm, DIM, x);
    return BAY_LOGFN(data_len, params_len, params, DIM, x);
}

// Launched with programmatic dependent launch where the params are staged (else a launch is
// long, and the wait's place before the density costs its loop 1 %).  A group of BAY_CTA
// walkers is a CTA, or a
// cluster of smaller ones where the ensemble has fewer groups than the device has SMs.
template <bool ACCU, bool STAGED>
__device__ __forceinline__ void bay_stretch_plain(const bay_stretch_params& P) {
    __shared__ bay_plain_sync sSync;
    bay_stage_begin<STAGED>(&sSync, P.params, (unsigned int)P.data_len + P.params_len);
    if (STAGED) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    const unsigned int kind = ACCU ? 1u : 0u;
    const unsigned int k = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = k < P.K;
    const unsigned int step = P.ctl->step[kind] + P.step_off;
    const unsigned int seed = P.ctl->seed[kind] + P.half;
    const float a = P.ctl->a;
    const float beta = ACCU ? 1.0f : bay_beta(P);
    const unsigned int stream = ACCU ? (P.half ? 2222u : 1111u) : (P.half ? 4444u : 3333u);
    float* X = P.xs + (size_t)P.half * P.K * DIM;
    const float* S = P.xs + (size_t)(1u - P.half) * P.K * DIM;
    float Y[DIM];
    bool accepted = false;
    if (valid) {
        bay_u4 c;
        c.x = k;
        c.y = step;
        c.z = stream;
        c.w = 0xbeeff00du;
        const bay_u4 r = bay_philox4x32_10(c, seed, 0xdecafbadu);
        const float u0 = bay_u01(r.x), u1 = bay_u01(r.y), u2 = bay_u01(r.z);
        const float z = bay_stretch_z(a, u1);
        const unsigned int j = bay_partner(u0, P.K);
#pragma unroll
        for (int i = 0; i < DIM; ++i) {
            const float s = bay_partner_coord(S, P.K, j, i);
            Y[i] = __fmaf_rn(z, __fsub_rn(X[(size_t)k * DIM + i], s), s);
        }
        float ly = 0.0f;
        if (STAGED) {
            const float lx = P.logfn[(size_t)P.half * P.K + k];
            if (bay_stage_wait<STAGED>(&sSync, &P.ctl->status)) {
                // else the params may be anything, lengths and offsets that it goes by too
                ly = bay_density<STAGED>((unsigned int)P.data_len, P.params_len, P.params, Y);
                accepted = bay_accept(u2, z, ly, lx, beta);
            }
        } else {
            // (the log density after the loop over the params: before it, that loop took 1,256 us
            // of a bare launch of 4,096 walkers x 60,000 rows instead of 793)
            ly = bay_density<STAGED>((unsigned int)P.data_len, P.params_len, P.params, Y);
            const float lx = P.logfn[(size_t)P.half * P.K + k];
            accepted = bay_accept(u2, z, ly, lx, beta);
        }
        if (accepted) {
#pragma unroll
            for (int i = 0; i < DIM; ++i) X[(size_t)k * DIM + i] = Y[i];
            P.logfn[(size_t)P.half * P.K + k] = ly;
        } else if (ACCU) {
#pragma unroll
            for (int i = 0; i < DIM; ++i) Y[i] = X[(size_t)k * DIM + i];
        }
    } else {
        bay_stage_wait<STAGED>(&sSync, &P.ctl->status);   // the copy lands before the CTA may end
    }
    if (ACCU) {
        __shared__ float red[BAY_CTA / 32][BAY_SUM_CHUNK];
        unsigned int ncta, rank;
        asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ncta));
        asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
        bay_accu_epilogue(P, accepted, valid, Y, red, blockIdx.x / ncta, gridDim.x / ncta, ncta, rank);
    }
}

#if BAY_PLAIN_GROUP == 1
extern "C" __global__ void __launch_bounds__(BAY_CTA) BAY_PLAIN(bay_stretch_bare)(bay_stretch_params P) {
    bay_stretch_plain<false, BAY_PLAIN_STAGED>(P);
}
extern "C" __global__ void __launch_bounds__(BAY_CTA) BAY_PLAIN(bay_stretch_accu)(bay_stretch_params P) {
    bay_stretch_plain<true, BAY_PLAIN_STAGED>(P);
}
#endif

// logfn over all W walkers (nvidia-gtx-mcmc-stretch.cu:197-206), SoA input.
template <bool STAGED>
__device__ __forceinline__ void bay_logfn_plain(const bay_stretch_params& P) {
    __shared__ bay_plain_sync sSync;
    bay_stage_begin<STAGED>(&sSync, P.params, (unsigned int)P.data_len + P.params_len);
    const unsigned int k = blockIdx.x * blockDim.x + threadIdx.x;
    const bool ok = bay_stage_wait<STAGED>(&sSync, &P.ctl->status);
    if (k >= P.W || !ok) return;
    float x[DIM];
#pragma unroll
    for (int i = 0; i < DIM; ++i) x[i] = P.xs[(size_t)k * DIM + i];
    P.logfn[k] = bay_density<STAGED>((unsigned int)P.data_len, P.params_len, P.params, x);
}
#if BAY_PLAIN_GROUP == 0
extern "C" __global__ void __launch_bounds__(BAY_CTA) BAY_PLAIN(bay_logfn_all)(bay_stretch_params P) {
    bay_logfn_plain<BAY_PLAIN_STAGED>(P);
}
#endif

// Density engines (reference cuda/engines/nvidia-gtx-distribution.cu logpdf/pdf and
// nvidia-gtx-likelihood.cu loglik/lik): the model's density at n points, x dim x n
// column-major (point i's coordinates contiguous); exp_out selects the density itself.
template <bool STAGED>
__device__ __forceinline__ void
bay_points_density(unsigned long long n, unsigned int data_len, unsigned int params_len,
                 const float* params, const float* x, float* out, unsigned int exp_out) {
    __shared__ bay_plain_sync sSync;
    bay_stage_begin<STAGED>(&sSync, params, data_len + params_len);
    const bool ok = bay_stage_wait<STAGED>(&sSync, nullptr);   // given up: NaN, not a stale value
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        float p[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) p[d] = x[i * DIM + d];
        const float v = ok ? bay_density<STAGED>(data_len, params_len, params, p) : __int_as_float(0x7fc00000);
        out[i] = exp_out ? expf(v) : v;
    }
}
#if BAY_PLAIN_GROUP == 2
extern "C" __global__ void __launch_bounds__(BAY_CTA)
BAY_PLAIN(bay_points_logfn)(unsigned long long n, unsigned int data_len, unsigned int params_len,
                            const float* params, const float* x, float* out, unsigned int exp_out) {
    bay_points_density<BAY_PLAIN_STAGED>(n, data_len, params_len, params, x, out, exp_out);
}
#endif

// Evidence (nvidia-gtx-likelihood.cu evidence_reduce): per-CTA FP64 sums of exp(density)
// over the points, each thread's points in order, then a fixed-order tree -> part[cta].
template <bool STAGED>
__device__ __forceinline__ void
bay_points_sum(unsigned long long n, unsigned int data_len, unsigned int params_len,
               const float* params, const float* x, double* part) {
    __shared__ double red[BAY_CTA];
    __shared__ bay_plain_sync sSync;
    bay_stage_begin<STAGED>(&sSync, params, data_len + params_len);
    const bool ok = bay_stage_wait<STAGED>(&sSync, nullptr);   // given up: NaN, not a stale value
    double s = ok ? 0.0 : (double)__int_as_float(0x7fc00000);
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; ok && i < n;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        float p[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) p[d] = x[i * DIM + d];
        s += (double)expf(bay_density<STAGED>(data_len, params_len, params, p));
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (unsigned int o = 512; o > 0; o >>= 1) {   // BAY_CTA: any multiple of 32 <= 1024
        if (o < BAY_CTA) {
            if (threadIdx.x < o && threadIdx.x + o < BAY_CTA) red[threadIdx.x] += red[threadIdx.x + o];
            __syncthreads();
        }
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}
#if BAY_PLAIN_GROUP == 2
extern "C" __global__ void __launch_bounds__(BAY_CTA)
BAY_PLAIN(bay_points_evidence)(unsigned long long n, unsigned int data_len, unsigned int params_len,
                               const float* params, const float* x, double* part) {
    bay_points_sum<BAY_PLAIN_STAGED>(n, data_len, params_len, params, x, part);
}
#endif

#else
// ---------------------------------------------------------------- tiled form
// A CTA owns BAY_WPC walkers (a power of two, at most 32) and BAY_CTA threads.  The data
// rows reach shared memory by TMA bulk copies (cp.async.bulk, completion counted on an
// mbarrier; the wait is bounded) in chunks of at most BAY_TILE_CHUNK floats, two chunk
// buffers in flight when the data span more than one.  Thread t works for walker
// t % BAY_WPC on row group t / BAY_WPC: walkers are fastest across lanes, so the lanes of
// one row group read the same row (a shared-memory broadcast), and each thread sums its rows
// in batches of 8 (pairwise) added with a Kahan carry.  The lanes and warps of a walker
// then combine as compensated pairs in a fixed order (deterministic for a given shape).
#ifndef BAY_WPC
#define BAY_WPC 8
#endif
#ifndef BAY_TILE_CHUNK
#define BAY_TILE_CHUNK 12288u                     // floats per staged chunk (48 KB)
#endif
#define BAY_TILE_CHUNK_ROWS ((BAY_TILE_CHUNK / BAY_ROW_LEN) & ~3u)   // 16-byte chunk starts
#define BAY_TILE_WAIT_NS 2000000000ull

__device__ __forceinline__ unsigned long long bay_tile_timer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait for phase `par` of the mbarrier at shared address `bar`: gives up after
// BAY_TILE_WAIT_NS and sets status bit 1 (the host reports the shared-memory copy).
__device__ __forceinline__ bool bay_tile_wait(unsigned int bar, unsigned int par,
                                              unsigned int* status) {
    unsigned long long t0 = 0;
    for (unsigned int it = 0;; ++it) {
        unsigned int ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok) : "r"(bar), "r"(par) : "memory");
        if (ok) return true;
        if ((it & 15u) == 0u) {
            const unsigned long long t = bay_tile_timer();
            if (it == 0u) {
                t0 = t;
            } else if (t - t0 > BAY_TILE_WAIT_NS) {
                atomicOr(status, 1u);
                return false;
            }
        }
    }
}

// Chunk c of the rows [rb, rb + n_rows) (rb a multiple of 4) -> buffer `buf` (floats): the
// 16-byte-aligned prefix by one bulk copy completing on `bar`, issued by the calling
// thread.  Returns the chunk's floats.
__device__ __forceinline__ unsigned int bay_tile_issue(const bay_stretch_params& P, unsigned long long c,
                                                       float* buf, unsigned int bar,
                                                       unsigned long long rb, unsigned long long n_rows) {
    const unsigned long long r0 = c * BAY_TILE_CHUNK_ROWS;
    const unsigned long long nr = n_rows - r0 < BAY_TILE_CHUNK_ROWS ? n_rows - r0 : BAY_TILE_CHUNK_ROWS;
    const unsigned int nf = (unsigned int)(nr * BAY_ROW_LEN);
    const unsigned int bytes = (nf * 4u) & ~15u;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
    if (bytes)
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
            ::"r"((unsigned int)__cvta_generic_to_shared(buf)), "l"(P.params + (rb + r0) * BAY_ROW_LEN),
            "r"(bytes), "r"(bar) : "memory");
    return nf;
}

// The chunk buffers' barriers and the CTA's verdict on its copies.
struct bay_tile_sync {
    unsigned long long bar[2];
    unsigned int ok;
};

// Thread 0: the chunk barriers and the first two chunks' copies.  The data never change
// while a sampler runs, so this may run before the launch waits for its predecessor.  The
// CTA's threads wait on the barriers only after a __syncthreads that follows this.
__device__ __forceinline__ void bay_tile_begin(const bay_stretch_params& P, bay_tile_sync* sy,
                                               unsigned long long rb, unsigned long long n_rows) {
    extern __shared__ __align__(128) float bay_tsm[];
    if (threadIdx.x != 0) return;
    const unsigned long long nch = (n_rows + BAY_TILE_CHUNK_ROWS - 1) / BAY_TILE_CHUNK_ROWS;
    const unsigned int bar0 = (unsigned int)__cvta_generic_to_shared(&sy->bar[0]);
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8u) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    sy->ok = 1u;
    for (unsigned long long c = 0; c < 2 && c < nch; ++c)
        bay_tile_issue(P, c, bay_tsm + (unsigned int)c * BAY_TILE_CHUNK, bar0 + 8u * (unsigned int)c,
                       rb, n_rows);
}

// Sum over all data rows of BAY_TILE_TERM(row, prep of walker w) for the CTA's walkers
// w < BAY_WPC (prep: [BAY_WPC][BAY_PREP_LEN] in shared memory) -> *out of thread w (a
// compensated pair), the copies begun by bay_tile_begin.  Every thread of the CTA calls it.  Returns
// false (and sets the status) when a bounded wait for a copy gave up; out is then
// incomplete.
// With BAY_TILE_TERM4 (the model's row term over bay_v4) and BAY_WPC a multiple of 4, a
// thread serves the four walkers 4 s .. 4 s + 3 of walker slot s = t % (BAY_WPC / 4) on row
// group t / (BAY_WPC / 4): one row load per four walkers, four times the row groups.
#if defined(BAY_TILE_TERM4) && (BAY_WPC % 4 == 0)
#define BAY_TILE_VEC 1
typedef bay_v4 bay_tval;
#define BAY_TVAL_ZERO {0.0f, 0.0f, 0.0f, 0.0f}
#define BAY_TVAL_ADD(a, b) bay_v4_add_rn(a, b)
#define BAY_TVAL_SUB(a, b) bay_v4_sub_rn(a, b)
#define BAY_TVAL_TERM(row, pv) BAY_TILE_TERM4(row, pv)
#else
#define BAY_TILE_VEC 0
typedef float bay_tval;
#define BAY_TVAL_ZERO 0.0f
#define BAY_TVAL_ADD(a, b) __fadd_rn(a, b)
#define BAY_TVAL_SUB(a, b) __fsub_rn(a, b)
#define BAY_TVAL_TERM(row, pv) BAY_TILE_TERM(row, pv)
#endif
__device__ __forceinline__ bool bay_tiled_logfn_rows(const bay_stretch_params& P,
                                                    const float (*prep)[BAY_PREP_LEN],
                                                    bay_cf (*red)[BAY_WPC], bay_cf* out,
                                                    bay_tile_sync* sy, unsigned long long rb,
                                                    unsigned long long n_rows) {
    extern __shared__ __align__(128) float bay_tsm[];
    unsigned int& sOk = sy->ok;
    constexpr unsigned int WV = BAY_TILE_VEC ? 4u : 1u;     // walkers per thread
    constexpr unsigned int WS = BAY_WPC / WV;               // walker slots
    constexpr unsigned int L = BAY_CTA / WS;                // row groups
    const unsigned int tid = threadIdx.x, w = tid % WS, l = tid / WS;
    const unsigned long long nch = (n_rows + BAY_TILE_CHUNK_ROWS - 1) / BAY_TILE_CHUNK_ROWS;
    const unsigned int bar0 = (unsigned int)__cvta_generic_to_shared(&sy->bar[0]);
#if BAY_TILE_VEC
    bay_v4 pv[BAY_PREP_LEN];
#pragma unroll
    for (int i = 0; i < BAY_PREP_LEN; ++i)
        pv[i] = {prep[4u * w][i], prep[4u * w + 1u][i], prep[4u * w + 2u][i], prep[4u * w + 3u][i]};
#else
    float pv[BAY_PREP_LEN];
#pragma unroll
    for (int i = 0; i < BAY_PREP_LEN; ++i) pv[i] = prep[w][i];
#endif
    bay_tval sum = BAY_TVAL_ZERO, cmp = BAY_TVAL_ZERO;
    for (unsigned long long c = 0; c < nch; ++c) {
        const unsigned int b = (unsigned int)(c & 1ull);
        float* R = bay_tsm + b * BAY_TILE_CHUNK;
        const unsigned long long r0 = c * BAY_TILE_CHUNK_ROWS;
        const unsigned int nr = (unsigned int)(n_rows - r0 < BAY_TILE_CHUNK_ROWS ? n_rows - r0
                                                                              : BAY_TILE_CHUNK_ROWS);
        const unsigned int nf = nr * BAY_ROW_LEN, nb = ((nf * 4u) & ~15u) / 4u;
        const bool done = bay_tile_wait(bar0 + 8u * b, (unsigned int)((c >> 1) & 1ull), &P.ctl->status);
        if (!done) sOk = 0u;
        if (nb < nf) {   // the chunk's last floats past its 16-byte-aligned prefix
            for (unsigned int e = nb + tid; e < nf; e += BAY_CTA) R[e] = P.params[(rb + r0) * BAY_ROW_LEN + e];
        }
        __syncthreads();
        if (sOk == 0u) break;
        unsigned int r = l;
        for (; r + 7u * L < nr; r += 8u * L) {
            bay_tval t[8];
#pragma unroll
            for (unsigned int i = 0; i < 8u; ++i) t[i] = BAY_TVAL_TERM(R + (r + i * L) * BAY_ROW_LEN, pv);
#pragma unroll
            for (unsigned int h = 4u; h >= 1u; h >>= 1)
#pragma unroll
                for (unsigned int i = 0; i < h; ++i) t[i] = BAY_TVAL_ADD(t[i], t[i + h]);
            const bay_tval y = BAY_TVAL_SUB(t[0], cmp);
            const bay_tval s2 = BAY_TVAL_ADD(sum, y);
            cmp = BAY_TVAL_SUB(BAY_TVAL_SUB(s2, sum), y);
            sum = s2;
        }
        for (; r < nr; r += L) {
            const bay_tval y = BAY_TVAL_SUB(BAY_TVAL_TERM(R + r * BAY_ROW_LEN, pv), cmp);
            const bay_tval s2 = BAY_TVAL_ADD(sum, y);
            cmp = BAY_TVAL_SUB(BAY_TVAL_SUB(s2, sum), y);
            sum = s2;
        }
        __syncthreads();                                // buffer b is free again
        if (tid == 0 && c + 2 < nch) bay_tile_issue(P, c + 2, R, bar0 + 8u * b, rb, n_rows);
    }
    const bool ok = sOk != 0u;
    // the lanes of a walker slot (lane bits above the slot bits) by an xor butterfly, then
    // the warps in order; walker 4 s + j of slot s at red[warp][4 s + j] (vector path)
    const unsigned int lane = tid & 31u, warp = tid >> 5;
#pragma unroll
    for (unsigned int j = 0; j < WV; ++j) {
        bay_cf v;
#if BAY_TILE_VEC
        v.hi = j == 0u ? sum.x : j == 1u ? sum.y : j == 2u ? sum.z : sum.w;
        v.lo = -(j == 0u ? cmp.x : j == 1u ? cmp.y : j == 2u ? cmp.z : cmp.w);
#else
        v.hi = sum;
        v.lo = -cmp;
#endif
#pragma unroll
        for (unsigned int o = 16u; o >= WS && o >= 1u; o >>= 1) v = bay_cadd(v, bay_cf_shfl_xor(v, o));
        if (lane < WS) red[warp][WV * lane + j] = v;
    }
    __syncthreads();
    // (a walker's total is its thread's: BAY_WPC <= 32, all in warp 0)
    if (tid < BAY_WPC) {
        bay_cf s = red[0][tid];
        for (unsigned int i = 1; i < BAY_CTA / 32u; ++i) s = bay_cadd(s, red[i][tid]);
        *out = s;
    }
    return ok;
}

template <bool ACCU>
__device__ __forceinline__ void bay_stretch_tiled(const bay_stretch_params& P) {
    const unsigned int kind = ACCU ? 1u : 0u;
    __shared__ float sY[BAY_WPC][DIM];
    __shared__ float sPrep[BAY_WPC][BAY_PREP_LEN];
    __shared__ float sW[BAY_WPC], sZ[BAY_WPC], sU2[BAY_WPC];
    __shared__ bay_cf sRed[BAY_CTA / 32][BAY_WPC];
    const unsigned int step = P.ctl->step[kind] + P.step_off;
    const unsigned int seed = P.ctl->seed[kind] + P.half;
    const float a = P.ctl->a;
    const float beta = ACCU ? 1.0f : bay_beta(P);
    const unsigned int stream = ACCU ? (P.half ? 2222u : 1111u) : (P.half ? 4444u : 3333u);
    float* X = P.xs + (size_t)P.half * P.K * DIM;
    const float* S = P.xs + (size_t)(1u - P.half) * P.K * DIM;
    const float* hyper = P.params + P.data_len;
    // walker group g and row slice sl (slice-major CTAs); slices start on 4-row boundaries
    const unsigned int NS = P.t_slices, groups = gridDim.x / NS;
    const unsigned int g = blockIdx.x % groups, sl = blockIdx.x / groups;
    const unsigned int k0 = g * BAY_WPC;
    const unsigned long long n_rows = P.data_len / BAY_ROW_LEN;
    const unsigned long long rps = NS > 1u ? (((n_rows + NS - 1u) / NS + 3ull) & ~3ull) : n_rows;
    const unsigned long long rb = (unsigned long long)sl * rps < n_rows ? (unsigned long long)sl * rps : n_rows;
    const unsigned long long rn = n_rows - rb < rps ? n_rows - rb : rps;
    __shared__ bay_tile_sync sSync;
    bay_tile_begin(P, &sSync, rb, rn);
    // Launched with programmatic dependent launch: the draws, the walker's own row and log
    // density (this half last moved two launches back, final once the previous launch began
    // its work, which it did only after waiting for its own predecessor) come before the
    // wait for the previous launch; the partner row, from the half that launch moves, after.
    const unsigned int t0 = threadIdx.x, kk = k0 + t0;
    const bool mine_ok = t0 < BAY_WPC && kk < P.K;
    float xr[DIM], z = 0.0f, u2 = 0.0f, lx = 0.0f;
    unsigned int j = 0;
    if (mine_ok) {
        bay_u4 c;
        c.x = kk;
        c.y = step;
        c.z = stream;
        c.w = 0xbeeff00du;
        const bay_u4 r = bay_philox4x32_10(c, seed, 0xdecafbadu);
        z = bay_stretch_z(a, bay_u01(r.y));
        j = bay_partner(bay_u01(r.x), P.K);
        u2 = bay_u01(r.z);
#pragma unroll
        for (int i = 0; i < DIM; ++i) xr[i] = X[(size_t)kk * DIM + i];
        lx = P.logfn[(size_t)P.half * P.K + kk];
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (threadIdx.x < BAY_WPC) {
        const unsigned int t = threadIdx.x, k = k0 + t;
        if (k < P.K) {
            float Y[DIM];
#pragma unroll
            for (int i = 0; i < DIM; ++i) {
                const float s = bay_partner_coord(S, P.K, j, i);
                Y[i] = __fmaf_rn(z, __fsub_rn(xr[i], s), s);
                sY[t][i] = Y[i];
            }
            float pr[BAY_PREP_LEN];
            BAY_TILE_PREP(hyper, P.params_len, DIM, Y, pr);
#pragma unroll
            for (int i = 0; i < BAY_PREP_LEN; ++i) sPrep[t][i] = pr[i];
            sW[t] = BAY_TILE_WALKER(n_rows, hyper, P.params_len, DIM, Y);
            sZ[t] = z;
            sU2[t] = u2;
        } else {
#pragma unroll
            for (int i = 0; i < BAY_PREP_LEN; ++i) sPrep[t][i] = 0.0f;
            sW[t] = 0.0f;
        }
    }
    __syncthreads();
    bay_cf sum;
    sum.hi = sum.lo = 0.0f;
    bool ok = bay_tiled_logfn_rows(P, sPrep, sRed, &sum, &sSync, rb, rn);
    bool accepted = false;
    const unsigned int t = threadIdx.x, k = k0 + t;
    const bool valid = t < BAY_WPC && k < P.K;
    if (NS > 1u) {
        // leave this slice's partials (NaN after a failed copy: the walker is then
        // rejected), take the group's ticket; the last slice combines them in slice order
        __shared__ unsigned int sLast;
        float2* part = reinterpret_cast<float2*>(P.t_part);
        if (valid) part[(size_t)k * NS + sl] = ok ? make_float2(sum.hi, sum.lo)
                                                 : make_float2(__int_as_float(0x7fc00000), 0.0f);
        __threadfence();
        __syncthreads();
        if (t == 0) sLast = atomicAdd(&P.t_ticket[g], 1u) == NS - 1u ? 1u : 0u;
        __syncthreads();
        if (sLast == 0u) return;
        __threadfence();
        if (t == 0) P.t_ticket[g] = 0u;             // for the next launch
        if (valid) {
            bay_cf a;
            a.hi = 0.0f;
            a.lo = 0.0f;
            for (unsigned int q = 0; q < NS; ++q) {
                const float2 v = __ldcg(&part[(size_t)k * NS + q]);
                bay_cf b;
                b.hi = v.x;
                b.lo = v.y;
                a = bay_cadd(a, b);
            }
            sum = a;
        }
        ok = true;
    }
    // the rest is the walkers' warp's: decision, write-back, and the group's statistics (the
    // warps' sums in warp order, of which the others' are zeros)
    if (t >= 32u) return;
    if (valid && ok) {
        const float ly = bay_cf_total(sW[t], sum);
        accepted = bay_accept(sU2[t], sZ[t], ly, lx, beta);
        if (accepted) {
#pragma unroll
            for (int i = 0; i < DIM; ++i) X[(size_t)k * DIM + i] = sY[t][i];
            P.logfn[(size_t)P.half * P.K + k] = ly;
        }
    }
    if (ACCU) {
        const unsigned int bal = __ballot_sync(0xffffffffu, accepted);
        if (t == 0 && bal) atomicAdd(&P.ctl->accepted, (unsigned long long)__popc(bal));
        if (P.means_cap == 0) return;
        float* out = P.part + ((size_t)P.step_off * 2 + P.half) * DIM * groups + g;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            float v = valid ? (accepted ? sY[t][d] : xr[d]) : 0.0f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            bay_cf s, w;
            s.hi = s.lo = w.lo = 0.0f;
            w.hi = v;
            s = bay_cadd(s, w);
            if (t == 0) out[(size_t)d * groups] = __fadd_rn(s.hi, s.lo);
        }
    }
}

extern "C" __global__ void __launch_bounds__(BAY_CTA) bay_stretch_bare(bay_stretch_params P) {
    bay_stretch_tiled<false>(P);
}
extern "C" __global__ void __launch_bounds__(BAY_CTA) bay_stretch_accu(bay_stretch_params P) {
    bay_stretch_tiled<true>(P);
}

// log density of all W walkers with the tiled sum (one CTA per BAY_WPC walkers).
extern "C" __global__ void __launch_bounds__(BAY_CTA) bay_logfn_all(bay_stretch_params P) {
    __shared__ float sPrep[BAY_WPC][BAY_PREP_LEN];
    __shared__ float sW[BAY_WPC];
    __shared__ bay_cf sRed[BAY_CTA / 32][BAY_WPC];
    bay_cf sum;
    sum.hi = sum.lo = 0.0f;
    const float* hyper = P.params + P.data_len;
    const unsigned long long n_rows = P.data_len / BAY_ROW_LEN;
    const unsigned int k0 = blockIdx.x * BAY_WPC;
    __shared__ bay_tile_sync sSync;
    bay_tile_begin(P, &sSync, 0ull, n_rows);
    if (threadIdx.x < BAY_WPC) {
        const unsigned int t = threadIdx.x, k = k0 + t;
        if (k < P.W) {
            float x[DIM];
#pragma unroll
            for (int i = 0; i < DIM; ++i) x[i] = P.xs[(size_t)k * DIM + i];
            float pr[BAY_PREP_LEN];
            BAY_TILE_PREP(hyper, P.params_len, DIM, x, pr);
#pragma unroll
            for (int i = 0; i < BAY_PREP_LEN; ++i) sPrep[t][i] = pr[i];
            sW[t] = BAY_TILE_WALKER(n_rows, hyper, P.params_len, DIM, x);
        } else {
#pragma unroll
            for (int i = 0; i < BAY_PREP_LEN; ++i) sPrep[t][i] = 0.0f;
            sW[t] = 0.0f;
        }
    }
    __syncthreads();
    const bool ok = bay_tiled_logfn_rows(P, sPrep, sRed, &sum, &sSync, 0ull, n_rows);
    const unsigned int t = threadIdx.x, k = k0 + t;
    if (ok && t < BAY_WPC && k < P.W) P.logfn[k] = bay_cf_total(sW[t], sum);
}
#endif
