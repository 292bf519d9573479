// pf_estimate.cu -- posterior estimate of a set of particles as a kernel-level
// entry point: FP64 partial sums of the sub-filters (one to sixteen warps each)
// into a scratch array in global memory, one row per CTA, and the last CTA to
// finish combining the rows with log-sum-exp rescaling.  The same arithmetic
// as the filter's own estimate: weights exp(key - max) in FP32 with the
// sub-filter's maximum, sums in FP64, circular means for angular variables,
// the reference's winner (first maximum key, thrust::max_element semantics,
// src/partfilt/cuda/pf_generic_soa.cu:1014-1017).
#include <cstring>
#include <mutex>
#include <string>

#include <cuda.h>

#include "pf_launch.cuh"

namespace pfdev {

constexpr int kEstMaxState = 16;
// A row of partials: [0] key maximum (0 in linear mode), [1] the first-maximum
// winner's key, [2] its particle index (-1: every key is NaN), [3] sum w,
// [4+v] sum w x_v (angles: sum w sin x_v), [4+S+a] sum w cos of the a-th angle.
constexpr int kEstStride = 4 + 2 * kEstMaxState;
constexpr int kEstThreads = 512, kEstWarps = kEstThreads / 32;

// Scratch of one call: its rows, then the ticket of the CTAs that have written
// theirs.
constexpr size_t est_scratch_doubles(int64_t rows) { return (size_t)rows * kEstStride + 1; }

// V consecutive floats (V = 4: one 16-byte load).
template <int V>
__device__ __forceinline__ void est_load(const float* __restrict__ p, float (&o)[V])
{
    if constexpr (V == 4) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(p));
        o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
    } else {
        o[0] = __ldg(p);
    }
}

// The rows part[0 .. nrow) into one pf_estimate, one CTA.  Thread r weighs row
// r, then each warp adds every 16th row, lane j its value j (a row is one
// coalesced read), in windows of 512 rows.
__device__ void est_final(const double* part, const float* __restrict__ keys, const float* __restrict__ state, int S,
                          int64_t T, int m, int nrow, uint32_t angle_mask, int log_weights,
                          pf_estimate* __restrict__ out, double (*red)[kEstStride])
{
    __shared__ double scale[kEstThreads];
    __shared__ double sum[kEstStride];
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    double gm = -INFINITY, bk = -INFINITY, bi = -1.0;
    auto offer = [&](double ok, double oi) {
        if (oi >= 0.0 && (bi < 0.0 || ok > bk || (ok == bk && oi < bi))) {
            bk = ok;
            bi = oi;
        }
    };
    for (int r = tid; r < nrow; r += kEstThreads) {
        const double* p = part + (int64_t)r * kEstStride;
        gm = fmax(gm, __ldcg(p));
        offer(__ldcg(p + 1), __ldcg(p + 2));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        gm = fmax(gm, __shfl_xor_sync(kFull, gm, o));
        const double ok = __shfl_xor_sync(kFull, bk, o);
        const double oi = __shfl_xor_sync(kFull, bi, o);
        offer(ok, oi);
    }
    if (lane == 0) {
        red[wp][0] = gm;
        red[wp][1] = bk;
        red[wp][2] = bi;
    }
    __syncthreads();
    for (int w = 0; w < kEstWarps; ++w) {
        gm = fmax(gm, red[w][0]);
        offer(red[w][1], red[w][2]);
    }
    if (!log_weights) gm = 0.0;
    const int nv = 1 + S + __popc(angle_mask & ((1u << S) - 1u));
    double a0 = 0.0, a1 = 0.0;  // values lane and lane + 32
    for (int r0 = 0; r0 < nrow; r0 += kEstThreads) {
        const int nr = min(kEstThreads, nrow - r0);
        __syncthreads();
        if (tid < nr) scale[tid] = log_weights ? exp(__ldcg(part + (int64_t)(r0 + tid) * kEstStride) - gm) : 1.0;
        __syncthreads();
        const double* p = part + (int64_t)r0 * kEstStride + 3 + lane;
        if (lane < nv) {
#pragma unroll 8
            for (int r = wp; r < nr; r += kEstWarps) a0 += scale[r] * __ldcg(p + (int64_t)r * kEstStride);
        }
        if (lane + 32 < nv)
            for (int r = wp; r < nr; r += kEstWarps) a1 += scale[r] * __ldcg(p + 32 + (int64_t)r * kEstStride);
    }
    __syncthreads();
    red[wp][lane] = a0;
    if (lane + 32 < nv) red[wp][lane + 32] = a1;
    __syncthreads();
    if (wp != 0) return;
    for (int j = lane; j < nv; j += 32) {
        double s = red[0][j];
        for (int w = 1; w < kEstWarps; ++w) s += red[w][j];
        sum[j] = s;
    }
    __syncwarp();
    const double W = sum[0];
    const int64_t best = bi >= 0.0 && (int64_t)bi < T ? (int64_t)bi : 0;
    if (lane < kEstMaxState) {
        const int v = lane;
        double mean = 0.0;
        float bv = 0.0f;
        if (v < S) {
            if ((angle_mask >> v) & 1u) {
                const int c = __popc(angle_mask & ((1u << v) - 1u));
                mean = atan2(sum[1 + v], sum[1 + S + c]);
            } else {
                mean = sum[1 + v] / W;
            }
            bv = state[(int64_t)v * T + best];
        }
        out->mean[v] = mean;
        out->best[v] = bv;
    }
    if (lane == 0) {
        out->log_norm = gm + log(W);
        out->best_key = keys[best];
        out->best_subfilter = (int32_t)(best / m);
        out->step = 0;
        out->flags = (isfinite(gm) && isfinite(W) && W > 0.0) ? 0 : 1;
    }
}

// The ticket's zero, in stream order ahead of every call: whatever happened to
// the calls before (two that overlapped on one scratch leave any count), this
// one counts its own CTAs.  Launched after all earlier work of the stream has
// completed; the estimate follows as its programmatic dependent and waits for
// it only before the ticket: 2^20 particles of 3 variables, calls back to back,
// 15.0 us without the launch, 15.8 so, 17.0 with a memset in its place; 2^18 of
// 12 variables 25.2, 24.8 and 27.0.
__global__ void k_est_clear(unsigned* ticket)
{
    allow_dependents();
    if (threadIdx.x == 0) *ticket = 0;
}

// The sub-filters' sums, TW warps each (a CTA's sixteen warps take 16 / TW
// sub-filters), combined in shared memory into one row per CTA; the last CTA
// to write its row (ticket, beside the rows) forms the estimate.  V = 4 reads four particles a
// lane and load, for rows that are 16-byte aligned.
//
// Bound: reading 4 (1 + S) bytes per particle.  The first R loads of the keys
// -- and, for states of up to 4 variables, of every state row -- are issued
// before the maximum is reduced, so a sub-filter costs one round trip to
// memory, and a lane keeps its own sums only for the variables there are.  2^20
// particles of 3 variables, 2048 sub-filters of 512: 15.3 us a call, against
// 16.4 us with the rows combined by a second kernel and 63.2 us for one 256-thread
// CTA per sub-filter with 33 sums per thread whatever S was.
template <int S, int TW, int V>
__global__ void __launch_bounds__(kEstThreads)
    k_estimate(const float* __restrict__ keys, const float* __restrict__ state, int64_t T, int m, int nsub,
               uint32_t angle_mask, int log_weights, double* part, unsigned* ticket, pf_estimate* __restrict__ out)
{
    constexpr int NW = kEstWarps;
    constexpr int R = V == 4 ? 4 : 8;            // loads of the keys held in registers
    constexpr bool PRE = S <= 4 && V == 4;       // and of the state rows
    __shared__ double red[NW][kEstStride];
    __shared__ bool s_last;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int wt = wp % TW;                      // warp within the sub-filter's team
    const int b = blockIdx.x * (NW / TW) + wp / TW;
    const bool on = b < nsub;                    // the same for a whole team
    const int64_t base = (int64_t)b * m;
    const unsigned n = (unsigned)m, i0 = on ? (unsigned)((wt * 32 + lane) * V) : n;
    constexpr unsigned step = TW * 32 * V;
    float k[R][V], x[PRE ? R : 1][S][V];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const unsigned i = i0 + r * step;
        if (i < n) {
            est_load<V>(keys + base + i, k[r]);
            if constexpr (PRE) {
#pragma unroll
                for (int v = 0; v < S; ++v) est_load<V>(state + v * T + base + i, x[r][v]);
            }
        }
    }
    // the maximum and the first particle that holds it (a NaN key never does)
    float bk = -INFINITY;
    int bi = 0x7fffffff;
    auto offer = [&](float key, int i) {
        if (key > bk || (key == bk && i < bi)) {
            bk = key;
            bi = i;
        }
    };
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const unsigned i = i0 + r * step;
        if (i < n) {
#pragma unroll
            for (int q = 0; q < V; ++q) offer(k[r][q], (int)i + q);
        }
    }
    for (unsigned i = i0 + R * step; i < n; i += step) {
        float kk[V];
        est_load<V>(keys + base + i, kk);
#pragma unroll
        for (int q = 0; q < V; ++q) offer(kk[q], (int)i + q);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ok = __shfl_xor_sync(kFull, bk, o);
        const int oi = __shfl_xor_sync(kFull, bi, o);
        offer(ok, oi);
    }
    if constexpr (TW > 1) {
        __shared__ float rk[NW];
        __shared__ int ri[NW];
        if (lane == 0) {
            rk[wp] = bk;
            ri[wp] = bi;
        }
        __syncthreads();
        for (int w = wp - wt; w < wp - wt + TW; ++w) offer(rk[w], ri[w]);
    }
    const float lmax = log_weights ? bk : 0.0f;
    double sw = 0.0, ss[S], sc[S];
#pragma unroll
    for (int v = 0; v < S; ++v) ss[v] = sc[v] = 0.0;
    auto add = [&](const float (&kk)[V], auto&& row) {
        double w[V];
#pragma unroll
        for (int q = 0; q < V; ++q) {
            w[q] = log_weights ? (double)__expf(kk[q] - lmax) : (double)kk[q];
            sw += w[q];
        }
#pragma unroll
        for (int v = 0; v < S; ++v) {
            float xv[V];
            row(v, xv);
            if ((angle_mask >> v) & 1u) {
#pragma unroll
                for (int q = 0; q < V; ++q) {
                    float sn, cs;
                    __sincosf(xv[q], &sn, &cs);
                    ss[v] = fma(w[q], (double)sn, ss[v]);
                    sc[v] = fma(w[q], (double)cs, sc[v]);
                }
            } else {
#pragma unroll
                for (int q = 0; q < V; ++q) ss[v] = fma(w[q], (double)xv[q], ss[v]);
            }
        }
    };
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const unsigned i = i0 + r * step;
        if (i < n) {
            add(k[r], [&](int v, float(&o)[V]) {
                if constexpr (PRE) {
#pragma unroll
                    for (int q = 0; q < V; ++q) o[q] = x[r][v][q];
                } else {
                    est_load<V>(state + v * T + base + i, o);
                }
            });
        }
    }
    for (unsigned i = i0 + R * step; i < n; i += step) {
        float kk[V];
        est_load<V>(keys + base + i, kk);
        add(kk, [&](int v, float(&o)[V]) { est_load<V>(state + v * T + base + i, o); });
    }
    auto tree = [&](double a) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(kFull, a, o);
        return a;
    };
    sw = tree(sw);
    if (lane == 0) {
        red[wp][0] = on ? (double)lmax : -INFINITY;
        red[wp][1] = (double)bk;
        red[wp][2] = on && bi < m ? (double)(base + bi) : -1.0;
        red[wp][3] = sw;
    }
    int a = 0;
#pragma unroll
    for (int v = 0; v < S; ++v) {
        const double s = tree(ss[v]);
        if (lane == 0) red[wp][4 + v] = s;
        if ((angle_mask >> v) & 1u) {
            const double c = tree(sc[v]);
            if (lane == 0) red[wp][4 + S + a] = c;
            ++a;
        }
    }
    __syncthreads();
    // one row: the warps' sums scaled to the CTA's maximum (a team's warps have the same one)
    double* row = part + (int64_t)blockIdx.x * kEstStride;
    const int nw = min(NW, (nsub - (int)blockIdx.x * (NW / TW)) * TW);  // warps that had a sub-filter
    double cm = red[0][0];
    for (int w = 1; w < nw; ++w) cm = fmax(cm, red[w][0]);
    __shared__ double scale[NW];
    if (threadIdx.x < nw) {
        const double l = red[threadIdx.x][0];
        scale[threadIdx.x] = log_weights && l != cm ? exp(l - cm) : 1.0;
    }
    __syncthreads();
    for (int j = 3 + threadIdx.x; j < 4 + S + a; j += blockDim.x) {
        double s = 0.0;
        for (int w = 0; w < nw; ++w) s += scale[w] * red[w][j];
        row[j] = s;
    }
    if (threadIdx.x == 0) {
        double wk = -INFINITY, wi = -1.0;
        for (int w = 0; w < nw; ++w) {
            const double ok = red[w][1], oi = red[w][2];
            if (oi >= 0.0 && (wi < 0.0 || ok > wk || (ok == wk && oi < wi))) {
                wk = ok;
                wi = oi;
            }
        }
        row[0] = cm;
        row[1] = wk;
        row[2] = wi;
    }
    wait_prerequisites();  // the ticket is cleared
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    est_final(part, keys, state, S, T, m, (int)gridDim.x, angle_mask, log_weights, out, red);
}

// Warps per sub-filter: sixteen where the CTAs of fewer would not reach every
// SM twice or a sub-filter is long, four up to 1184 sub-filters (two CTAs per
// SM), one beyond.
static int est_warps(int m, int64_t nsub)
{
    if (nsub <= 296 || m > 4096) return 16;
    return nsub <= 1184 || m > 1024 ? 4 : 1;
}
static int64_t est_rows(int m, int64_t nsub)
{
    const int per = kEstWarps / est_warps(m, nsub);
    return (nsub + per - 1) / per;
}

template <int S>
static cudaError_t launch_est(const float* keys, const float* state, int64_t T, int m, int nsub, uint32_t angle_mask,
                              int log_weights, double* scratch, pf_estimate* out, cudaStream_t st)
{
    const bool vec = ((reinterpret_cast<uintptr_t>(keys) | reinterpret_cast<uintptr_t>(state)) & 15) == 0 &&
                     m % 4 == 0 && T % 4 == 0;
    const int rows = (int)est_rows(m, nsub);
    unsigned* ticket = reinterpret_cast<unsigned*>(scratch + est_scratch_doubles(rows) - 1);
    k_est_clear<<<1, 32, 0, st>>>(ticket);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
#define PF_EST(TW, V)                                                                                        \
    return launch_maybe_dependent(true, k_estimate<S, TW, V>, rows, kEstThreads, 0, st, keys, state, T, m, nsub, \
                                  angle_mask, log_weights, scratch, ticket, out)
    switch (est_warps(m, nsub)) {
    case 16:
        if (vec) PF_EST(16, 4);
        PF_EST(16, 1);
    case 4:
        if (vec) PF_EST(4, 4);
        PF_EST(4, 1);
    default:
        if (vec) PF_EST(1, 4);
        PF_EST(1, 1);
    }
#undef PF_EST
}

// Launches the estimate on `st` with the given scratch.
static cudaError_t launch_estimate(const float* keys, const float* state, int S, int64_t T, int m,
                                   uint32_t angle_mask, int log_weights, double* scratch, pf_estimate* out,
                                   cudaStream_t st)
{
    const int nsub = (int)(T / m);
    switch (S) {
#define PF_EST_S(s) \
    case s: return launch_est<s>(keys, state, T, m, nsub, angle_mask, log_weights, scratch, out, st);
        PF_EST_S(1) PF_EST_S(2) PF_EST_S(3) PF_EST_S(4) PF_EST_S(5) PF_EST_S(6) PF_EST_S(7) PF_EST_S(8)
        PF_EST_S(9) PF_EST_S(10) PF_EST_S(11) PF_EST_S(12) PF_EST_S(13) PF_EST_S(14) PF_EST_S(15) PF_EST_S(16)
#undef PF_EST_S
    }
    return cudaErrorInvalidValue;
}

static bool estimate_shape_ok(int S, int64_t T, int m, std::string* why)
{
    if (S < 1 || S > kEstMaxState) {
        *why = "num_state must be in [1, 16]";
        return false;
    }
    if (m < 1 || T < m || T % m != 0) {
        *why = "num_particles must be a positive multiple of m";
        return false;
    }
    if (T / m > INT32_MAX) {
        *why = "too many sub-filters";
        return false;
    }
    return true;
}

}  // namespace pfdev

using namespace pfdev;

// Error recording shared with pf_api.cu (thread-local message for pf_last_error).
pf_status pfi_fail(pf_status s, const char* msg);

extern "C" pf_status pfk_estimate(const float* keys, const float* state, int32_t num_state, int64_t num_particles,
                                  int32_t m, uint32_t angle_mask, int32_t log_weights, pf_estimate* out)
{
    std::string why;
    if (!keys || !state || !out) return pfi_fail(PF_ERR_INVALID, "null argument");
    if (!estimate_shape_ok(num_state, num_particles, m, &why)) return pfi_fail(PF_ERR_INVALID, why.c_str());
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n < 1) {
        cudaGetLastError();
        return pfi_fail(PF_ERR_CUDA, "no CUDA device available (this engine has no CPU path)");
    }
    const int64_t T = num_particles;
    const int nsub = (int)(T / m);
    float *dk = nullptr, *ds = nullptr;
    double* dp = nullptr;
    pf_estimate* de = nullptr;
    cudaError_t e = cudaMalloc(&dk, (size_t)T * 4);
    if (e == cudaSuccess) e = cudaMalloc(&ds, (size_t)T * num_state * 4);
    if (e == cudaSuccess) e = cudaMalloc(&dp, est_scratch_doubles(est_rows(m, nsub)) * 8);
    if (e == cudaSuccess) e = cudaMalloc(&de, sizeof(pf_estimate));
    if (e == cudaSuccess) e = cudaMemcpy(dk, keys, (size_t)T * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(ds, state, (size_t)T * num_state * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = launch_estimate(dk, ds, num_state, T, m, angle_mask, log_weights, dp, de, 0);
    if (e == cudaSuccess) e = cudaMemcpy(out, de, sizeof(pf_estimate), cudaMemcpyDeviceToHost);
    cudaFree(dk);
    cudaFree(ds);
    cudaFree(dp);
    cudaFree(de);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return pfi_fail(PF_ERR_CUDA, cudaGetErrorString(e));
    }
    return PF_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free variant.  Some callers cannot call cudaMalloc: code running
// inside a memory pool or arena that owns every device allocation, embedded
// hosts whose allocator is locked after start-up, and work that must not
// allocate between stream captures.  pfk_estimate_noalloc computes exactly
// what pfk_estimate computes, from device pointers the caller already owns,
// with its per-sub-filter scratch in the static array below (allocated with
// the module, held by every GPU that loads the library until exit).
// ---------------------------------------------------------------------------
constexpr int kNoAllocMaxSubfilters = 4096;  // 4096 * 36 doubles = 1.18 MB per device
static __device__ __align__(256) double g_noalloc_scratch[est_scratch_doubles(kNoAllocMaxSubfilters)];

static std::mutex g_noalloc_mu;
// Device address of g_noalloc_scratch per device ordinal, valid for the CUDA
// context whose process-unique id is stored beside it: cudaDeviceReset (or a
// caller switching to another context on the same ordinal) loads the module
// afresh, possibly at another address, and the new context has a new id, so
// the next call looks the address up again instead of using a stale one.
static double* g_noalloc_ptr[256];
static unsigned long long g_noalloc_ctx[256];

// The current context's process-unique id (cuCtxGetId; ids are never reused
// within a process), through the runtime's driver entry points so the library
// needs no link against libcuda.  0 when no context is current.
static unsigned long long current_context_id()
{
    using GetCurrent = CUresult (*)(CUcontext*);
    using GetId = CUresult (*)(CUcontext, unsigned long long*);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    if (!get_current || !get_id) {
        void* a = nullptr;
        void* b = nullptr;
        cudaDriverEntryPointQueryResult qa, qb;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &a, cudaEnableDefault, &qa) != cudaSuccess ||
            cudaGetDriverEntryPoint("cuCtxGetId", &b, cudaEnableDefault, &qb) != cudaSuccess ||
            qa != cudaDriverEntryPointSuccess || qb != cudaDriverEntryPointSuccess || !a || !b) {
            cudaGetLastError();
            return 0;
        }
        get_current = reinterpret_cast<GetCurrent>(a);
        get_id = reinterpret_cast<GetId>(b);
    }
    CUcontext c = nullptr;
    unsigned long long id = 0;
    if (get_current(&c) != CUDA_SUCCESS || !c || get_id(c, &id) != CUDA_SUCCESS) return 0;
    return id;
}

extern "C" pf_status pfk_estimate_noalloc(const float* d_keys, const float* d_state, int32_t num_state,
                                          int64_t num_particles, int32_t m, uint32_t angle_mask,
                                          int32_t log_weights, pf_estimate* d_out, void* stream)
{
    std::string why;
    if (!d_keys || !d_state || !d_out) return pfi_fail(PF_ERR_INVALID, "null argument");
    if (!estimate_shape_ok(num_state, num_particles, m, &why)) return pfi_fail(PF_ERR_INVALID, why.c_str());
    if (num_particles / m > kNoAllocMaxSubfilters)
        return pfi_fail(PF_ERR_INVALID, "pfk_estimate_noalloc: more than 4096 sub-filters (num_particles / m) "
                                        "exceed its static scratch; use pfk_estimate");
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 256) {
        cudaGetLastError();
        return pfi_fail(PF_ERR_CUDA, "no current CUDA device");
    }
    double* scratch = nullptr;
    {
        // Once per device (and again after the device's context was replaced),
        // with that device current: the host-side name of the array is only a
        // stand-in, so ask the runtime for its device address.
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        unsigned long long ctx = current_context_id();
        if (!g_noalloc_ptr[dev] || !ctx || ctx != g_noalloc_ctx[dev]) {
            void* p = nullptr;
            e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
            if (e != cudaSuccess || !p) {
                cudaGetLastError();
                return pfi_fail(PF_ERR_CUDA, "cudaGetSymbolAddress of the static scratch failed");
            }
            g_noalloc_ptr[dev] = static_cast<double*>(p);
            g_noalloc_ctx[dev] = current_context_id();  // the lookup made the context current if none was
        }
        scratch = g_noalloc_ptr[dev];
    }
    e = launch_estimate(d_keys, d_state, num_state, num_particles, m, angle_mask, log_weights, scratch, d_out,
                        static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) {
        cudaGetLastError();
        return pfi_fail(PF_ERR_CUDA, cudaGetErrorString(e));
    }
    return PF_OK;
}
