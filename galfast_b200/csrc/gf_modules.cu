/*
 * gf_modules.cu -- sm_100a kernels of the postprocessing modules on the
 * catalog path.  Each restates the reference kernel named beside it with the
 * portable math of gf_math.h; expressions keep the reference's types and
 * evaluation order (the library is compiled with -fmad=false).
 *
 *   clipper_kernel     os_clipper::process (src/skygen/os_skygen.cpp:999-1044), analytic footprints
 *   fixedfeh_kernel    os_fixedFeH_kernel (src/modules/fixedFeH_gpu.cu.h:34-50)
 *   stream_rows_kernel, and thread_rows_kernel for many chunks, with
 *     BondOps          os_Bond2010_kernel (src/modules/Bond2010_gpu.cu.h:81-218)
 *     FehOps           os_FeH_kernel (src/modules/FeH_gpu.cu.h:43-87)
 *     GaussFehOps      os_GaussianFeH_kernel (src/modules/GaussianFeH_gpu.cu.h:42-73)
 *     MultOps          os_unresolvedMultiples_kernel (src/modules/unresolvedMultiples_gpu.cu.h:36-123)
 *   photometry_kernel  os_photometry_kernel (src/modules/photometry_gpu.cu.h:87-174)
 *   photoerr_kernel    os_photometricErrors::process (photometricErrors_host.cpp:112-131)
 *   vel2pm_kernel      os_vel2pm_kernel (src/modules/vel2pm_gpu.cu.h:253-301)
 *   gal2other_kernel   os_gal2other_kernel (src/modules/gal2other_gpu.cu.h:62-96)
 */
#include "gf_launch.h"
#include "gf_math.h"
#include "gf_rng.h"
#include "gf_footprint.h"

namespace gfk {

static const double D2R = 0.01745329251994329576923691;

static int grid_for(int64_t n, int threads)
{
    int64_t b = (n + threads - 1) / threads;
    int64_t cap = (int64_t)sm_count() * 32;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (int)b;
}

/* ---------------- sampler check: Poisson deviates of one stream ---------------- */
/* rng_t::poisson (cuda_rng.h:344-376) applied to mu[0..n) one after another on a
 * single stream: the device form of the sampler, including the gamma_int /
 * binomial reduction for mu > 10 that catalog bins rarely reach. */
__global__ void poisson_stream_kernel(uint32_t *st, const float *mu, int32_t n, uint32_t *out)
{
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    gfr::Mwc r;
    r.a = st[0]; r.c = st[1]; r.x = st[2]; r.used = 0;
    for (int32_t i = 0; i < n; i++) out[i] = r.poisson(mu[i]);
    st[0] = r.a; st[1] = r.c; st[2] = r.x;
}

cudaError_t launch_poisson_stream(uint32_t *st, const float *mu, int32_t n, uint32_t *out, cudaStream_t s)
{
    poisson_stream_kernel<<<1, 32, 0, s>>>(st, mu, n, out);
    count_launches(1);
    return cudaGetLastError();
}

/* ---------------- clipper ---------------- */
__device__ __forceinline__ void clip_row(const gf_footprint &foot, gf_table &t, int64_t row)
{
    const int64_t P = t.capacity;
    if (t.hidden[row]) return;
    bool in = true;
        if (foot.kind == GF_FOOT_LAMBERT_RECT) {
            float x = t.projXY[row], y = t.projXY[P + row];
            in = t.projIdx[row] == foot.proj && x >= foot.a && x < foot.b && y >= foot.c && y < foot.d;
        } else if (foot.kind == GF_FOOT_CAP) {
            double l = t.lb[row] * D2R, b = t.lb[P + row] * D2R;
            double l0 = foot.a * D2R, b0 = foot.b * D2R;
            double cosd = gfm::sin_d(b) * gfm::sin_d(b0) + gfm::cos_d(b) * gfm::cos_d(b0) * gfm::cos_d(l - l0);
            in = cosd >= gfm::cos_d(foot.c * D2R);
        } else if (foot.kind == GF_FOOT_LATCUT) {
            in = fabs(t.lb[P + row]) > foot.a;
        } else if (foot.kind == GF_FOOT_LB_RECT) {
            const double l = t.lb[row], b = t.lb[P + row];
            in = b >= foot.c && b < foot.d && ((foot.a <= foot.b) ? (l >= foot.a && l < foot.b) : (l >= foot.a || l < foot.b));
        } else if (foot.kind == GF_FOOT_REGIONS) {
            in = gff::regions_inside(foot, t.lb[row], t.lb[P + row]);
        }
        if (!in) t.hidden[row] = 1;
}

__global__ void clipper_kernel(gf_footprint foot, gf_table t, int64_t begin, int64_t end)
{
    for (int64_t row = begin + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; row < end; row += (int64_t)gridDim.x * blockDim.x)
        clip_row(foot, t, row);
}

/* each row clipped by its own request's footprint */
__global__ void clipper_multi_kernel(const gf_footprint *foot_by_job, MultiRows R, gf_table t, int64_t begin, int64_t end)
{
    for (int64_t row = begin + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; row < end; row += (int64_t)gridDim.x * blockDim.x) {
        const gf_footprint &f = foot_by_job[R.slot_job[R.row_slot[row]]];
        if (f.kind != GF_FOOT_ALL) clip_row(f, t, row);
    }
}

cudaError_t launch_clipper_multi(const gf_footprint *foot_by_job, MultiRows R, gf_table t, int64_t begin, int64_t end,
                                 cudaStream_t s)
{
    if (end <= begin) return cudaSuccess;
    clipper_multi_kernel<<<grid_for(end - begin, 256), 256, 0, s>>>(foot_by_job, R, t, begin, end);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_clipper(const gf_footprint &foot, gf_table t, int64_t begin, int64_t end, cudaStream_t s)
{
    if (end <= begin || foot.kind == GF_FOOT_ALL) return cudaSuccess;
    clipper_kernel<<<grid_for(end - begin, 256), 256, 0, s>>>(foot, t, begin, end);
    count_launches(1);
    return cudaGetLastError();
}

/* ---------------- fixedFeH ---------------- */
__global__ void fixedfeh_kernel(gf_fixedfeh_config c, gf_table t, int64_t begin, int64_t end)
{
    for (int64_t row = begin + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; row < end; row += (int64_t)gridDim.x * blockDim.x) {
        if (t.hidden[row]) continue;
        int cmp = t.comp[row];
        if (!((c.comp_mask >> cmp) & 1u)) continue;
        t.FeH[row] = c.FeH;
    }
}

cudaError_t launch_fixedfeh(const gf_fixedfeh_config &c, gf_table t, int64_t begin, int64_t end, cudaStream_t s)
{
    if (end <= begin) return cudaSuccess;
    fixedfeh_kernel<<<grid_for(end - begin, 256), 256, 0, s>>>(c, t, begin, end);
    count_launches(1);
    return cudaGetLastError();
}

/* ---------------- rows that draw from a stream, 256 to a stream ---------------- */
/* The reference gives each stream 256 consecutive rows, one thread walking them: the
 * uniforms a row takes depend on the rejections of the rows before it.  What depends on
 * the order is only where each row's uniforms begin; so one warp takes a stream and
 *   1  generates a run of W = 32 R uniforms, R to a lane: the MWC is a Lehmer generator,
 *      and lane l starts at the state times a^(l R);
 *   2  marks the positions where a Gaussian's pair is accepted and finds for every
 *      position where a Gaussian (next), and a row's NG Gaussians (fh), begun there end;
 *   3  walks the rows through fh, one shared-memory read a row;
 *   4  forms the rows' values, 32 rows at a time, reading and writing whole lines.
 * A row that the run ends in begins the next run.  Measured (Bond2010): 20001 rows 0.73 ms as one thread
 * a stream, 0.06 ms now (latency of one chunk); 4.0e6 rows 0.94 -> 0.39 ms (instruction issue: 56 % of slots,
 * 16e3 warp instructions a chunk, half of them the rows' functions).  Many chunks take a thread each instead
 * (thread_rows).
 */
#define GF_PAIR_TRIES 4096              /* pairs of a row's Gaussians (one in 4.7 is rejected): no stream that steps comes near */
#define GF_RUN_LANE 26                  /* uniforms of a lane in a run (even): three runs serve 256 rows of three Gaussians */
#define GF_RUN_PITCH 33
#define GF_RUN_END 0xffffu

/* Position p of a run of 32 R uniforms (lane p / R holds it, as its (p mod R)-th) is kept at
 * (p mod R) 33 + p / R: a lane's run is a column, and the run's end (p = 32 R) has an index of its own.
 * The tables hold such indexes, so following them takes no arithmetic. */
struct RowStream {
    float u[GF_RUN_PITCH * GF_RUN_LANE];
    uint16_t next[GF_RUN_PITCH * GF_RUN_LANE];      /* end of the Gaussian that begins here */
    uint16_t fh[GF_RUN_PITCH * GF_RUN_LANE];        /* end of the NG Gaussians that begin here (from the next position when every row leads with a uniform) */
    uint16_t start[256];
    uint16_t list[256];                 /* the rows that draw: row | kind << 8 */
};

template <int R>
__device__ __forceinline__ int run_forward(int q) { return q < (R - 1) * GF_RUN_PITCH ? q + GF_RUN_PITCH : q - (R - 1) * GF_RUN_PITCH + 1; }
template <int R>
__device__ __forceinline__ int run_back(int q) { return q >= GF_RUN_PITCH ? q - GF_RUN_PITCH : q + (R - 1) * GF_RUN_PITCH - 1; }

__device__ __forceinline__ float row_step(uint64_t &v, uint32_t a)
{
    const uint64_t t = (uint64_t)a * (uint32_t)v + (v >> 32);
    v = t;
    return GF_MWC_SCALE * (float)(uint32_t)t;
}

/* a chunk's stream: its multiplier, and the powers that jump it */
struct RowJump {
    const uint64_t *lo, *hi;            /* the context's tables of stream th, or null (another multiplier was set) */
    uint32_t a;
    bool ok;                            /* the multiplier is within the bounds of mwc_fold3 */
};

__device__ __forceinline__ RowJump row_jump(const StreamPowers &pw, const uint32_t *rng, int64_t th)
{
    RowJump j;
    j.a = rng[th];
    const bool same = j.a == pw.mult[th];
    j.lo = same ? pw.jt.lo + (size_t)th * 32 : nullptr;
    j.hi = same ? pw.jt.hi + (size_t)th * GF_JUMP_HI : nullptr;
    j.ok = j.a >= 16u && j.a <= 0xfffffff0u;
    return j;
}

/* the state of the lane's part of a run, lane R steps after v; false when v is not a residue of the Lehmer
 * generator modulo p = a 2^32 - 1 (0 < v < p).  mwc_mulmod_scaled(x, y) = x y a^3 mod p, so s(n) = a^(n-3)
 * jumps n steps and s(n + m) = mulmod(s(n), s(m)); s(1) = a^-2 = 2^64 mod p. */
template <int R>
__device__ __forceinline__ bool stream_runs(const RowJump &j, uint64_t v, int lane, uint64_t &w)
{
    const uint64_t p = ((uint64_t)j.a << 32) - 1;
    if (!j.ok || v == 0 || v >= p) return false;
    const int n = lane * R;
    w = v;
    if (j.hi) {
        w = gfr::mwc_mulmod_scaled(__ldg(j.hi + (n >> 5)), w, j.a, p);
        w = gfr::mwc_mulmod_scaled(__ldg(j.lo + (n & 31)), w, j.a, p);
    } else {
        uint64_t m = (0ull - p) % p;
        for (int k = n; k; k >>= 1) {
            if (k & 1) w = gfr::mwc_mulmod_scaled(m, w, j.a, p);
            m = gfr::mwc_mulmod_scaled(m, m, j.a, p);
        }
    }
    return true;
}

/* the stream's state at index q of the run (the run's end included), given each lane's start w0 */
template <int R>
__device__ __forceinline__ uint64_t stream_state_at(uint32_t a, uint64_t w0, int q, int lane)
{
    int steps = q / GF_RUN_PITCH, src = q - steps * GF_RUN_PITCH;
    if (src == 32) { src = 31; steps = R; }
    uint64_t w = w0;
    for (int s = 0; s < steps; s++) (void)row_step(w, a);
    const uint32_t lo = __shfl_sync(0xffffffffu, (uint32_t)w, src), hi = __shfl_sync(0xffffffffu, (uint32_t)(w >> 32), src);
    return ((uint64_t)hi << 32) | lo;
}

/* the polar Box-Muller test of a pair of uniforms (gaussian, cuda_rng.h:165-182) */
__device__ __forceinline__ float pair_r2(float u0, float u1, float &y)
{
    const float x = -1.f + 2.f * u0;
    y = -1.f + 2.f * u1;
    return x * x + y * y;
}
__device__ __forceinline__ bool pair_accepted(float r2) { return !(r2 > 1.0f || r2 == 0.f || r2 == 4.f); }

/* One run of 32 R uniforms: the places of the rows from r0 on that it holds (S.start, S.next, S.u).  lead:
 * every row's kind, or -1 when they differ.  Returns the row after the last one, with v the state there; r0
 * when none fits or v cannot be jumped. */
template <int NG, int R>
__device__ __forceinline__ int rows_of_run(const RowJump &j, uint64_t &v, int r0, int na, int lead, RowStream &S, int lane)
{
    constexpr unsigned full = 0xffffffffu;
    uint64_t w0;
    if (!stream_runs<R>(j, v, lane, w0)) return r0;
    /* the uniforms, and the accepted pairs that begin in the lane's part */
    uint32_t acc = 0;
    {
        uint64_t w = w0;
        float y, prev = row_step(w, j.a);
        const float first = prev;
        S.u[lane] = prev;
#pragma unroll 5
        for (int s = 1; s < R; s++) {
            const float u = row_step(w, j.a);
            S.u[s * GF_RUN_PITCH + lane] = u;
            if (pair_accepted(pair_r2(prev, u, y))) acc |= 1u << (s - 1);
            prev = u;
        }
        const float after = __shfl_down_sync(full, first, 1);
        if (lane < 31 && pair_accepted(pair_r2(prev, after, y))) acc |= 1u << (R - 1);
    }
    /* the end of the first accepted pair of each parity in the lanes after this one (R is even) */
    uint32_t later[2];
#pragma unroll
    for (int par = 0; par < 2; par++) {
        const uint32_t mine = acc & (0x55555555u << par);
        const int at = run_forward<R>(run_forward<R>((__ffs(mine) - 1) * GF_RUN_PITCH + lane));
        const unsigned has = __ballot_sync(full, mine != 0) & (0xfffffffeu << lane);
        const int there = __shfl_sync(full, at, has ? __ffs(has) - 1 : lane);
        later[par] = has ? (uint32_t)there : GF_RUN_END;
    }
    uint32_t even = later[0], odd = later[1];
    int at = (R - 1) * GF_RUN_PITCH + lane;           /* the odd position of a pair of positions */
#pragma unroll 2
    for (int s = R - 2; s >= 0; s -= 2, at -= 2 * GF_RUN_PITCH) {
        if ((acc >> s) & 2u) odd = (uint32_t)run_forward<R>(run_forward<R>(at));
        if ((acc >> s) & 1u) even = (uint32_t)run_forward<R>(at);
        S.next[at] = (uint16_t)odd;
        S.next[at - GF_RUN_PITCH] = (uint16_t)even;
    }
    __syncwarp();
    /* the indexes of whole rows; the run's end is at column 32 and ends every chain */
    if (NG > 1 || lead == 1) {
#pragma unroll 2
        for (int s = 0; s < R; s++) {
            int q = s * GF_RUN_PITCH + lane;
            if (lead == 1) q = run_forward<R>(q);
#pragma unroll
            for (int g = 0; g < NG; g++) q = (q < R * GF_RUN_PITCH && q != 32) ? S.next[q] : (int)GF_RUN_END;
            S.fh[s * GF_RUN_PITCH + lane] = (uint16_t)q;
        }
        __syncwarp();
    }
    /* where each row begins */
    const uint16_t *fh = (NG > 1 || lead == 1) ? S.fh : S.next;
    int q = 0, r = r0;
    if (lead >= 0) {
        while (r < na && q != 32) {
            const int e = fh[q];
            if (e == (int)GF_RUN_END) break;
            if (lane == 0) S.start[r] = (uint16_t)q;
            q = e;
            r++;
        }
    } else {
        while (r < na && q != 32) {
            const int b = (S.list[r] >> 8) ? run_forward<R>(q) : q;
            const int e = b != 32 ? fh[b] : (int)GF_RUN_END;
            if (e == (int)GF_RUN_END) break;
            if (lane == 0) S.start[r] = (uint16_t)q;
            q = e;
            r++;
        }
    }
    if (r > r0) v = stream_state_at<R>(j.a, w0, q, lane);
    return r;
}

/* the rows [begin + 256 th, ...) of one chunk with stream th, on one warp */
template <class Ops>
__device__ __forceinline__ void chunk_rows(const Ops &ops, const StreamPowers &pw, uint32_t *rng, int32_t NS,
                                           gf_table &t, int64_t begin, int64_t end, int64_t th, RowStream &S)
{
    constexpr int NG = Ops::NG, R = GF_RUN_LANE;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t rb = begin + 256 * th;
    const int nrow = (int)(end - rb < 256 ? end - rb : 256);
    int na = 0, leads = 0;
    for (int q = 0; q < nrow; q += 32) {
        const int i = q + lane;
        const int kind = i < nrow ? ops.kind(t, rb + i) : -1;
        const unsigned m = __ballot_sync(full, kind >= 0);
        if (kind >= 0) S.list[na + __popc(m & ((1u << lane) - 1u))] = (uint16_t)(i | (kind << 8));
        na += __popc(m);
        leads += __popc(__ballot_sync(full, kind == 1));
    }
    __syncwarp();
    if (na == 0) return;
    const int lead = leads == na ? 1 : leads == 0 ? 0 : -1;
    const RowJump j = row_jump(pw, rng, th);
    uint64_t v = ((uint64_t)rng[NS + th] << 32) | rng[2 * NS + th];
    int r0 = 0;
    while (r0 < na) {
        int r = rows_of_run<NG, R>(j, v, r0, na, lead, S, lane);
        if (r == r0) {
            /* a state outside the Lehmer range, or a row longer than a run: its uniforms one after
             * another, the accepted ones laid out as the first of a run */
            const int kind = S.list[r0] >> 8;
            int q = 0, tries = 0;
            __syncwarp();                                  /* (the run's tables have been read) */
            if (kind) {
                S.u[0] = row_step(v, j.a);
                q = GF_RUN_PITCH;
            }
            for (int g = 0; g < NG; g++, q += 2 * GF_RUN_PITCH) {
                float u0, u1, y;
                bool accepted;
                do {
                    u0 = row_step(v, j.a);
                    u1 = row_step(v, j.a);
                    accepted = pair_accepted(pair_r2(u0, u1, y));
                } while (!accepted && ++tries < GF_PAIR_TRIES);
                if (!accepted) {
                    /* a state that repeats itself (v = 0, a 2^32 - 1, or any of a multiplier 0): the rows left keep
                     * what they hold, and the caller learns of it at its next synchronisation */
                    if (lane == 0) *(volatile unsigned long long *)pw.stuck = 1ull;
                    return;
                }
                S.u[q] = u0;
                S.u[q + GF_RUN_PITCH] = u1;
                S.next[q] = (uint16_t)(q + 2 * GF_RUN_PITCH);
            }
            S.start[r0] = 0;
            r = r0 + 1;
        }
        __syncwarp();
        for (int i = r0 + lane; i < r; i += 32) {
            const int entry = S.list[i], kind = entry >> 8;
            int b = S.start[i];
            float pu = 0.f;
            if (kind) {
                pu = S.u[b];
                b = run_forward<R>(b);
            }
            float ys[NG], ss[NG];
#pragma unroll
            for (int g = 0; g < NG; g++) {
                b = S.next[b];
                const int b1 = run_back<R>(b);
                const float r2 = pair_r2(S.u[run_back<R>(b1)], S.u[b1], ys[g]);
                ss[g] = sqrtf(-2.0f * gfm::logf_(r2) / r2);
            }
            ops.apply(t, rb + (entry & 0xff), kind, pu, ys, ss);
        }
        r0 = r;
        __syncwarp();
    }
    if (lane == 0) {
        rng[NS + th] = (uint32_t)(v >> 32);
        rng[2 * NS + th] = (uint32_t)v;
    }
}

#define GF_ROW_WARPS 4

template <class Ops>
__global__ void __launch_bounds__(32 * GF_ROW_WARPS, 6) stream_rows_kernel(const Ops ops, const StreamPowers pw, uint32_t *rng, int32_t NS, gf_table t,
                                                                        int64_t begin, int64_t end, int64_t nchunks)
{
    __shared__ RowStream S[GF_ROW_WARPS];
    const int64_t th = (int64_t)blockIdx.x * GF_ROW_WARPS + (threadIdx.x >> 5);
    if (th >= nchunks) return;
    chunk_rows(ops, pw, rng, NS, t, begin, end, th, S[threadIdx.x >> 5]);
}

/* the last slot whose first chunk is at or before c */
__device__ __forceinline__ int slot_of_chunk(const int64_t *slot_chunk_begin, int nslots, int64_t c)
{
    int lo = 0, hi = nslots - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (slot_chunk_begin[mid] <= c) lo = mid; else hi = mid - 1;
    }
    return lo;
}

/* the 256-row chunks of every request of a pass, each drawing from its request's streams */
template <class Ops>
__global__ void __launch_bounds__(32 * GF_ROW_WARPS, 6) stream_rows_multi_kernel(const Ops ops, const StreamPowers pw, uint32_t *rng_all, int32_t NS,
                                                                              MultiRows R, const int64_t *slot_chunk_begin,
                                                                              int32_t nslots, int64_t nchunks,
                                                                              const int64_t *slot_rows, gf_table t)
{
    __shared__ RowStream S[GF_ROW_WARPS];
    const int64_t c = (int64_t)blockIdx.x * GF_ROW_WARPS + (threadIdx.x >> 5);
    if (c >= nchunks) return;
    const int slot = slot_of_chunk(slot_chunk_begin, nslots, c);
    const int64_t b = R.slot_row_begin[slot];
    chunk_rows(ops, pw, rng_all + (size_t)R.slot_job[slot] * 3 * NS, NS, t, b, b + slot_rows[slot], c - slot_chunk_begin[slot],
               S[threadIdx.x >> 5]);
}

/* The rows of a chunk on one thread, one row after another: the better arrangement once there are enough
 * chunks to fill the chip with threads, since it makes no tables (a warp's 16e3 instructions a chunk are 500
 * for a thread's share).  Threads against warps, one component: Bond2010 10e6 rows 1.03 and 0.93 ms, 12e6
 * 1.08 and 1.11, 16.7e6 1.25 and 1.53; FeH 10e6 0.43 and 0.44, 16.7e6 0.53 and 0.71; GaussianFeH of two components
 * 12e6 0.62 and 0.62, 16.7e6 0.65 and 0.83; multiples 8e6 0.46 and 0.47, 16.7e6 0.69 and 0.94.  So 11.5e6 rows are the
 * line, for the multiples, whose walk reads every row's fraction, 8e6 (THREADS_FROM, in chunks).
 * CTAs are of one warp, so that a call's spread evenly, and at most GF_THREAD_CTAS to an SM: each thread holds a
 * line of every column that it walks, 1 KB of them, and with 16 warps an SM (78 MB) they stay in L2.  Bond2010
 * over the passes of 2048 requests (5.3e8 rows, the largest 2.4e8): 8 warps 52.8 ms, 12 40.5, 16 37.0, 24 58.1, as
 * many as fit 62; a warp a chunk 47.3. */
template <class Ops>
__device__ __forceinline__ void thread_rows(const Ops &ops, const StreamPowers &pw, uint32_t *rng, int32_t NS, gf_table &t,
                                            int64_t begin, int64_t end, int64_t th)
{
    const uint32_t a = rng[th];
    uint64_t v = ((uint64_t)rng[NS + th] << 32) | rng[2 * NS + th];
    const int64_t rb = begin + 256 * th, re = rb + 256 < end ? rb + 256 : end;
    for (int64_t row = rb; row < re; row++) {
        const int kind = ops.kind(t, row);
        if (kind < 0) continue;
        const float pu = kind ? row_step(v, a) : 0.f;
        float ys[Ops::NG], ss[Ops::NG];
        int tries = 0;
#pragma unroll
        for (int g = 0; g < Ops::NG; g++) {
            float r2;
            bool accepted;
            do {
                const float u0 = row_step(v, a), u1 = row_step(v, a);
                r2 = pair_r2(u0, u1, ys[g]);
                accepted = pair_accepted(r2);
            } while (!accepted && ++tries < GF_PAIR_TRIES);
            if (!accepted) {
                *(volatile unsigned long long *)pw.stuck = 1ull;
                return;
            }
            ss[g] = sqrtf(-2.0f * gfm::logf_(r2) / r2);
        }
        ops.apply(t, row, kind, pu, ys, ss);
    }
    rng[NS + th] = (uint32_t)(v >> 32);
    rng[2 * NS + th] = (uint32_t)v;
}

template <class Ops>
__global__ void __launch_bounds__(32) thread_rows_kernel(const Ops ops, const StreamPowers pw, uint32_t *rng, int32_t NS, gf_table t,
                                                          int64_t begin, int64_t end, int64_t nchunks)
{
    for (int64_t th = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; th < nchunks; th += (int64_t)gridDim.x * blockDim.x)
        thread_rows(ops, pw, rng, NS, t, begin, end, th);
}

template <class Ops>
__global__ void __launch_bounds__(32) thread_rows_multi_kernel(const Ops ops, const StreamPowers pw, uint32_t *rng_all, int32_t NS,
                                                                MultiRows R, const int64_t *slot_chunk_begin, int32_t nslots,
                                                                int64_t nchunks, const int64_t *slot_rows, gf_table t)
{
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < nchunks; c += (int64_t)gridDim.x * blockDim.x) {
        const int slot = slot_of_chunk(slot_chunk_begin, nslots, c);
        const int64_t b = R.slot_row_begin[slot];
        thread_rows(ops, pw, rng_all + (size_t)R.slot_job[slot] * 3 * NS, NS, t, b, b + slot_rows[slot], c - slot_chunk_begin[slot]);
    }
}

#define GF_THREAD_CTAS 16
inline unsigned thread_ctas(int64_t nchunks) { return (unsigned)std::min<int64_t>((nchunks + 31) / 32, (int64_t)sm_count() * GF_THREAD_CTAS); }

template <class Ops>
cudaError_t launch_stream_rows(const Ops &ops, const StreamPowers &pw, uint32_t *rng, int32_t NS, gf_table t, int64_t begin, int64_t end,
                               int64_t nchunks, cudaStream_t s)
{
    if (nchunks >= Ops::THREADS_FROM)
        thread_rows_kernel<Ops><<<thread_ctas(nchunks), 32, 0, s>>>(ops, pw, rng, NS, t, begin, end, nchunks);
    else
        stream_rows_kernel<Ops><<<(unsigned)((nchunks + GF_ROW_WARPS - 1) / GF_ROW_WARPS), 32 * GF_ROW_WARPS, 0, s>>>(
        ops, pw, rng, NS, t, begin, end, nchunks);
    count_launches(1);
    return cudaGetLastError();
}

template <class Ops>
cudaError_t launch_stream_rows_multi(const Ops &ops, const StreamPowers &pw, uint32_t *rng_all, int32_t NS, MultiRows R, const int64_t *slot_chunk_begin,
                                     int32_t nslots, int64_t nchunks, const int64_t *slot_rows, gf_table t, cudaStream_t s)
{
    if (nchunks >= Ops::THREADS_FROM)
        thread_rows_multi_kernel<Ops><<<thread_ctas(nchunks), 32, 0, s>>>(ops, pw, rng_all, NS, R, slot_chunk_begin, nslots,
                                                                                       nchunks, slot_rows, t);
    else
        stream_rows_multi_kernel<Ops><<<(unsigned)((nchunks + GF_ROW_WARPS - 1) / GF_ROW_WARPS), 32 * GF_ROW_WARPS, 0, s>>>(
        ops, pw, rng_all, NS, R, slot_chunk_begin, nslots, nchunks, slot_rows, t);
    count_launches(1);
    return cudaGetLastError();
}

/* ---------------- Bond2010 kinematics ---------------- */
__device__ __forceinline__ float modfun(float Rsquared, float Z, const float *val)
{
    /* a + b|Z|^c + d R^e, Bond2010_gpu.cu.h:106-110 */
    return val[0] + val[1] * gfm::powf_(fabsf(Z), val[2]) + val[3] * gfm::powf_(Rsquared, (float)(0.5 * (double)val[4]));
}

__device__ __forceinline__ void trivar_gauss(float y[3], const float sg[6], const float z[3])
{
    /* Cholesky draw, Bond2010_gpu.cu.h:81-103 */
    float s11 = sg[0], s12 = sg[1], s13 = sg[2], s22 = sg[3], s23 = sg[4], s33 = sg[5];
    float b10 = s12;      float b11 = s22 * s22;
    float b20 = s13;      float b21 = s23;      float b22 = s33 * s33;
    float a00 = s11; float oneDivA00 = 1.0f / a00;
    float a10 = b10 * oneDivA00;
    float a11 = sqrtf(b11 - a10 * a10);
    float a20 = b20 * oneDivA00;
    float a21 = (b21 - a20 * a10) / a11;
    float a22 = sqrtf(b22 - a20 * a20 - a21 * a21);
    y[0] += a00 * z[0];
    y[1] += a10 * z[0] + a11 * z[1];
    y[2] += a20 * z[0] + a21 * z[1] + a22 * z[2];
}

__device__ __forceinline__ void draw_moments(float v[3], float R2, float Z, const gf_vmoments &mo, bool disk, const float z[3])
{
    for (int i = 0; i < 3; i++) v[i] = modfun(R2, Z, mo.m[i]);
    if (disk && v[1] > 0.f) v[1] = 0.f;
    float sg[6];
    for (int i = 0; i < 6; i++) sg[i] = modfun(R2, Z, mo.ss[i]);
    trivar_gauss(v, sg, z);
}

/* os_Bond2010_kernel's row (Bond2010_gpu.cu.h:140-215): disk stars draw the disk
 * component's uniform, then three Gaussians; halo stars three Gaussians */
struct BondOps {
    gf_bond2010_config par;
    static constexpr int NG = 3;
    static constexpr int64_t THREADS_FROM = 45000;

    __device__ __forceinline__ int kind(const gf_table &t, int64_t row) const
    {
        if (t.hidden[row]) return -1;
        const int cmp = t.comp[row];
        if (((par.comp_thin | par.comp_thick) >> cmp) & 1u) return 1;
        return ((par.comp_halo >> cmp) & 1u) ? 0 : -1;
    }
    __device__ __forceinline__ void apply(gf_table &t, int64_t row, int kind, float pu, const float *y, const float *s) const
    {
        const int64_t P = t.capacity;
        float vx = t.XYZ[row] + par.T[0], vy = t.XYZ[P + row] + par.T[1], vz = t.XYZ[2 * P + row] + par.T[2];
        float wx = par.M[0] * vx + par.M[1] * vy + par.M[2] * vz;
        float wy = par.M[3] * vx + par.M[4] * vy + par.M[5] * vz;
        float wz = par.M[6] * vx + par.M[7] * vy + par.M[8] * vz;
        const float R2 = (float)(1e-6 * (double)(wx * wx + wy * wy));
        const float Z = (float)(1e-3 * (double)wz);
        const float z[3] = {y[0] * s[0], y[1] * s[1], y[2] * s[2]};
        float v[3];
        if (kind == 1) {
            draw_moments(v, R2, Z, pu < par.fk ? par.disk_1 : par.disk_2, true, z);
        } else {
            draw_moments(v, R2, Z, par.halo, false, z);
            float invR = 1.f / sqrtf(R2 + Z * Z);
            float cosa = sqrtf(R2) * invR;
            float sina = Z * invR;
            float vR = cosa * v[0] - sina * v[1];
            float vZ = sina * v[0] + cosa * v[1];
            v[0] = vR;
            v[1] = v[2];
            v[2] = vZ;
        }
        t.vcyl[row] = v[0];
        t.vcyl[P + row] = v[1];
        t.vcyl[2 * P + row] = v[2];
    }
};

cudaError_t launch_bond2010_multi(const gf_bond2010_config &c, const StreamPowers &pw, uint32_t *rng_all, int32_t NS, MultiRows R,
                                  const int64_t *slot_chunk_begin, int32_t nslots, int64_t nchunks,
                                  const int64_t *slot_rows, gf_table t, cudaStream_t s)
{
    if (nchunks <= 0) return cudaSuccess;
    BondOps o;
    o.par = c;
    return launch_stream_rows_multi(o, pw, rng_all, NS, R, slot_chunk_begin, nslots, nchunks, slot_rows, t, s);
}

cudaError_t launch_bond2010(const gf_bond2010_config &c, const StreamPowers &pw, uint32_t *rng, int32_t NS, gf_table t, int64_t begin, int64_t end,
                            cudaStream_t s)
{
    if (end <= begin) return cudaSuccess;
    int64_t n = end - begin;
    int64_t nchunks = n / 256 + (n % 256 ? 1 : 0);
    if (nchunks > NS) return cudaErrorInvalidValue;
    BondOps o;
    o.par = c;
    return launch_stream_rows(o, pw, rng, NS, t, begin, end, nchunks, s);
}

/* ---------------- FeH (Ivezic et al. 2008) and GaussianFeH ---------------- */

/* os_FeH_kernel's row (FeH_gpu.cu.h:43-87): disk stars draw the Gaussian's number, then it; halo stars one Gaussian */
struct FehOps {
    gf_feh_config par;
    static constexpr int NG = 1;
    static constexpr int64_t THREADS_FROM = 45000;

    __device__ __forceinline__ int kind(const gf_table &t, int64_t row) const
    {
        if (t.hidden[row]) return -1;
        const int cmp = t.comp[row];
        if (((par.comp_thin | par.comp_thick) >> cmp) & 1u) return 1;
        return ((par.comp_halo >> cmp) & 1u) ? 0 : -1;
    }
    __device__ __forceinline__ void apply(gf_table &t, int64_t row, int kind, float pu, const float *y, const float *s) const
    {
        const int64_t P = t.capacity;
        if (kind == 1) {
            /* the Gaussian to draw from */
            const float p = pu * (par.A[0] + par.A[1]);
            const int i = p < par.A[0] ? 0 : 1;
            /* the star's place in the disk */
            const float vx = t.XYZ[row] + par.T[0], vy = t.XYZ[P + row] + par.T[1], vz = t.XYZ[2 * P + row] + par.T[2];
            const float wz = par.M[6] * vx + par.M[7] * vy + par.M[8] * vz;
            /* Bond et al. A2; exp in single precision through the portable expf */
            const float muD = par.muInf + par.DeltaMu * gfm::expf_(-fabsf(wz) / par.Hmu);
            const float aZ = muD - 0.067f;
            t.FeH[row] = par.sigma[i] * y[0] * s[0] + aZ + par.offs[i];
        } else {
            t.FeH[row] = par.offs[2] + par.sigma[2] * y[0] * s[0];
        }
    }
};

/* os_GaussianFeH_kernel's row (GaussianFeH_gpu.cu.h:42-73): the component's uniform when there
 * are several, then one Gaussian */
struct GaussFehOps {
    gf_gaussfeh_config par;
    static constexpr int NG = 1;
    static constexpr int64_t THREADS_FROM = 45000;

    __device__ __forceinline__ int kind(const gf_table &t, int64_t row) const
    {
        if (t.hidden[row] || !((par.comp_mask >> t.comp[row]) & 1u)) return -1;
        return par.ncomp != 1 ? 1 : 0;
    }
    __device__ __forceinline__ void apply(gf_table &t, int64_t row, int kind, float u, const float *y, const float *s) const
    {
        int at = 0;
        if (kind == 1)
            while (par.pcum[at] < u) ++at;
        t.FeH[row] = par.mean[at] + par.sigma[at] * y[0] * s[0];
        t.FeH_comp[row] = at;
    }
};

cudaError_t launch_feh(const gf_feh_config *fp, const gf_gaussfeh_config *gp, const StreamPowers &pw, uint32_t *rng, int32_t NS, gf_table t,
                       int64_t begin, int64_t end, cudaStream_t s)
{
    if (end <= begin) return cudaSuccess;
    const int64_t n = end - begin, nchunks = n / 256 + (n % 256 ? 1 : 0);
    if (nchunks > NS) return cudaErrorInvalidValue;
    if (fp) {
        FehOps o;
        o.par = *fp;
        return launch_stream_rows(o, pw, rng, NS, t, begin, end, nchunks, s);
    }
    GaussFehOps o;
    o.par = *gp;
    return launch_stream_rows(o, pw, rng, NS, t, begin, end, nchunks, s);
}

cudaError_t launch_feh_multi(const gf_feh_config *fp, const gf_gaussfeh_config *gp, const StreamPowers &pw, uint32_t *rng_all, int32_t NS,
                             MultiRows R, const int64_t *slot_chunk_begin, int32_t nslots, int64_t nchunks,
                             const int64_t *slot_rows, gf_table t, cudaStream_t s)
{
    if (nchunks <= 0) return cudaSuccess;
    if (fp) {
        FehOps o;
        o.par = *fp;
        return launch_stream_rows_multi(o, pw, rng_all, NS, R, slot_chunk_begin, nslots, nchunks, slot_rows, t, s);
    }
    GaussFehOps o;
    o.par = *gp;
    return launch_stream_rows_multi(o, pw, rng_all, NS, R, slot_chunk_begin, nslots, nchunks, slot_rows, t, s);
}

/* ---------------- unresolved multiple systems ---------------- */

/* nearest-texel lookup of a 1-D table (cux.h:786-792, 849-855) */
__device__ __forceinline__ float mult_tex(const float *tab, int n, float x0, float inv_dx, float x)
{
    float xi = (x - x0) * inv_dx + 0.5f;
    if (xi < 0.f) xi = 0.f;
    else if (xi >= (float)n) xi = (float)n - 1;
    return tab[(uint32_t)xi];
}

/* os_unresolvedMultiples_kernel's row (unresolvedMultiples_gpu.cu.h:46-123) with two system
 * components: a uniform against the binary fraction and, for a companion drawn from the
 * luminosity function, a second one */
struct MultOps {
    gf_multiples_config c;
    static constexpr int64_t THREADS_FROM = 31000;

    __device__ __forceinline__ bool active(const gf_table &t, int64_t row) const
    {
        return !t.hidden[row] && ((c.comp_mask >> t.comp[row]) & 1u);
    }
    __device__ __forceinline__ float fraction(const gf_table &t, int64_t row) const
    {
        return mult_tex(c.secprob, c.nsec, c.sec_x0, c.sec_inv_dx, t.absmag[row]);
    }
    __device__ __forceinline__ void single(gf_table &t, int64_t row) const
    {
        t.absmagSys[row] = t.absmag[row];
        t.absmagSys[t.capacity + row] = 99.999f;
        t.absmagSysNcomp[row] = 1;
    }
    /* companion: whether one was drawn; u: its uniform (not used by equal-mass pairs) */
    __device__ __forceinline__ void apply(gf_table &t, int64_t row, bool companion, float u) const
    {
        const int64_t P = t.capacity;
        const float M1 = t.absmag[row];
        t.absmagSys[row] = M1;
        float Ltot = gfm::exp10f_(-0.4f * M1);
        int ncomps = 1;
        float M2 = 99.999f;
        if (companion) {
            if (c.algo == GF_MULT_EQUAL_MASS) {
                M2 = M1;
            } else {
                const float pprim = mult_tex(c.cumlf, c.ncum, c.cum_x0, c.cum_inv_dx, M1);
                /* fainter than the primary: u rescaled into [pprim, 1] in double, as written */
                if (c.algo == GF_MULT_LF_M2_GT_M1) u = (float)((double)pprim + (double)u * (1. - (double)pprim));
                M2 = mult_tex(c.invcumlf, c.ninv, c.inv_x0, c.inv_inv_dx, u);
                if (c.algo == GF_MULT_LF_M2_GT_M1 && M2 < M1) M2 = M1;
            }
            Ltot += gfm::exp10f_(-0.4f * M2);
            ncomps++;
        }
        t.absmagSys[P + row] = M2;
        /* -2.5 is a double: the product is formed in double and stored as float */
        t.absmag[row] = (float)(-2.5 * (double)gfm::log10f_(Ltot));
        t.absmagSysNcomp[row] = ncomps;
    }
};

/* rows [begin + 256 th, ...) with stream th on one warp: at most two uniforms a row, so one run of 512 serves
 * the chunk; the walk over the rows only counts them, the magnitudes are formed by all lanes */
__device__ __forceinline__ void chunk_rows(const MultOps &ops, const StreamPowers &pw, uint32_t *rng,
                                           int32_t NS, gf_table &t, int64_t begin, int64_t end, int64_t th, RowStream &S)
{
    const int lane = threadIdx.x & 31;
    const int64_t rb = begin + 256 * th;
    const int nrow = (int)(end - rb < 256 ? end - rb : 256);
    float *psec = (float *)S.next;                     /* binary fraction of each active row */
    int na = 0;
    for (int q = 0; q < nrow; q += 32) {
        const int i = q + lane;
        const bool in = i < nrow, on = in && ops.active(t, rb + i);
        const unsigned m = __ballot_sync(0xffffffffu, on);
        if (on) {
            const int k = na + __popc(m & ((1u << lane) - 1u));
            S.list[k] = (uint16_t)i;
            psec[k] = ops.fraction(t, rb + i);
        } else if (in) {
            ops.single(t, rb + i);
        }
        na += __popc(m);
    }
    if (na == 0) return;
    const bool two = ops.c.algo != GF_MULT_EQUAL_MASS;
    const RowJump j = row_jump(pw, rng, th);
    uint64_t v = ((uint64_t)rng[NS + th] << 32) | rng[2 * NS + th];
    constexpr int R = 16;
    uint64_t w0;
    const bool run = stream_runs<R>(j, v, lane, w0);
    if (run) {
        uint64_t w = w0;
#pragma unroll 4
        for (int s = 0; s < R; s++) S.u[s * GF_RUN_PITCH + lane] = row_step(w, j.a);
    }
    __syncwarp();
    int q = 0;
    for (int r = 0; r < na; r++) {
        /* (a state outside the Lehmer range: its uniforms one after another, from every lane's copy of v) */
        const float u = run ? S.u[q] : row_step(v, j.a);
        const bool companion = !(u > psec[r]);
        const float u2 = run || !(companion && two) ? 0.f : row_step(v, j.a);
        if (lane == 0) {
            S.start[r] = (uint16_t)(q | (companion ? 0x8000 : 0));
            if (!run) S.u[256 + r] = u2;
        }
        q = run_forward<R>(q);
        if (companion && two) q = run_forward<R>(q);
        if (!run) q = r + 1;
    }
    __syncwarp();
    for (int r = lane; r < na; r += 32) {
        const int st = S.start[r];
        const bool companion = (st & 0x8000) != 0;
        float u2 = 0.f;
        if (companion && two) u2 = run ? S.u[run_forward<R>(st & 0x7fff)] : S.u[256 + r];
        ops.apply(t, rb + S.list[r], companion, u2);
    }
    const uint64_t ve = run ? stream_state_at<R>(j.a, w0, q, lane) : v;
    if (lane == 0) {
        rng[NS + th] = (uint32_t)(ve >> 32);
        rng[2 * NS + th] = (uint32_t)ve;
    }
}

__device__ __forceinline__ void thread_rows(const MultOps &ops, const StreamPowers &, uint32_t *rng, int32_t NS, gf_table &t,
                                            int64_t begin, int64_t end, int64_t th)
{
    const bool two = ops.c.algo != GF_MULT_EQUAL_MASS;
    const uint32_t a = rng[th];
    uint64_t v = ((uint64_t)rng[NS + th] << 32) | rng[2 * NS + th];
    const int64_t rb = begin + 256 * th, re = rb + 256 < end ? rb + 256 : end;
    for (int64_t row = rb; row < re; row++) {
        if (!ops.active(t, row)) {
            ops.single(t, row);
            continue;
        }
        const bool companion = !(row_step(v, a) > ops.fraction(t, row));
        ops.apply(t, row, companion, companion && two ? row_step(v, a) : 0.f);
    }
    rng[NS + th] = (uint32_t)(v >> 32);
    rng[2 * NS + th] = (uint32_t)v;
}

cudaError_t launch_multiples(const gf_multiples_config &c, const StreamPowers &pw, uint32_t *rng, int32_t NS, gf_table t, int64_t begin, int64_t end,
                             cudaStream_t s)
{
    if (end <= begin) return cudaSuccess;
    const int64_t n = end - begin, nchunks = n / 256 + (n % 256 ? 1 : 0);
    if (nchunks > NS) return cudaErrorInvalidValue;
    MultOps o;
    o.c = c;
    return launch_stream_rows(o, pw, rng, NS, t, begin, end, nchunks, s);
}

cudaError_t launch_multiples_multi(const gf_multiples_config &c, const StreamPowers &pw, uint32_t *rng_all, int32_t NS, MultiRows R,
                                   const int64_t *slot_chunk_begin, int32_t nslots, int64_t nchunks, const int64_t *slot_rows,
                                   gf_table t, cudaStream_t s)
{
    if (nchunks <= 0) return cudaSuccess;
    MultOps o;
    o.c = c;
    return launch_stream_rows_multi(o, pw, rng_all, NS, R, slot_chunk_begin, nslots, nchunks, slot_rows, t, s);
}

/* ---------------- photometry ---------------- */
__device__ __forceinline__ uint32_t brev(uint32_t a) { return __brev(a); }

__global__ void __launch_bounds__(256) photometry_kernel(PhotTables lt, gf_table t, int64_t begin, int64_t end)
{
    const int64_t P = t.capacity;
    const int ncolors = lt.nbands - 1;
    const bool sys = t.systems && t.absmagSys;
    const float *Mr = sys ? t.absmagSys : t.absmag;
    const int nabsmag = sys ? 2 : 1;
    for (int64_t row = begin + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; row < end; row += (int64_t)gridDim.x * blockDim.x) {
        if (t.hidden[row]) continue;
        int cmp = t.comp[row];
        if (!((lt.comp_mask >> cmp) & 1u)) continue;
        float fFeH = t.FeH[row];
        uint32_t flag = 0;
        float c[GF_MAX_BANDS];
        /* the system's components (absmagSys when unresolved multiples ran, else the
         * single absmag): their luminosities are summed band by band */
        for (int syscomp = 0; syscomp < nabsmag; syscomp++) {
            const float fMr = Mr[(size_t)syscomp * P + row];
            if (fMr >= 99.999f) break;
            float xi = (fFeH - lt.tcFeH[0]) * lt.tcFeH[1] + 0.5f;
            float yi = (fMr - lt.tcMr[0]) * lt.tcMr[1] + 0.5f;
            if (xi < 0.f) xi = 0.f; else if (xi >= (float)lt.nFeH) xi = (float)lt.nFeH - 1;
            if (yi < 0.f) yi = 0.f; else if (yi >= (float)lt.nMr) yi = (float)lt.nMr - 1;
            uint32_t i = (uint32_t)xi, j = (uint32_t)yi;
            for (int ic = 0; ic < ncolors; ic++) {
                size_t off = ((size_t)ic * lt.nMr + j) * lt.nFeH + i;
                c[ic] = lt.colors[off];
                flag |= ((uint32_t)(lt.eflags[off] != 0)) << ic;
            }
            for (int b = 0; b <= ncolors; b++) {
                float M = fMr;
                if (b < lt.bidx) { for (int q = b; q != lt.bidx; q++) M += c[q]; }
                if (b > lt.bidx) { for (int q = lt.bidx; q != b; q++) M -= c[q]; }
                float L = gfm::exp10f_(-0.4f * M);
                if (syscomp) L += t.mags[b * P + row];
                t.mags[b * P + row] = L;
            }
        }
        bool fl = false;
        for (int q = lt.bidx - 1; q >= 0; q--) {
            fl = fl || (flag & (1u << q));
            flag |= ((uint32_t)fl) << q;
        }
        fl = false;
        for (int q = lt.bidx; q < ncolors; q++) {
            fl = fl || (flag & (1u << q));
            flag |= ((uint32_t)fl) << q << 1;
        }
        flag &= ~(1u << lt.bidx);
        flag = brev(flag);
        flag >>= (8 * sizeof(flag) - ncolors - 1);
        t.photoflags[row] = (int32_t)flag;
        float dm = t.DM[row];
        float Am0 = t.Am[row];
        for (int b = 0; b <= ncolors; b++) {
            float Msys = -2.5f * gfm::log10f_(t.mags[b * P + row]);
            float msys = dm + Msys;
            float Am = Am0 * lt.reddening[b];
            t.mags[b * P + row] = msys + Am;
        }
    }
}

cudaError_t launch_photometry(const PhotTables &c, gf_table t, int64_t begin, int64_t end, cudaStream_t s)
{
    if (end <= begin) return cudaSuccess;
    photometry_kernel<<<grid_for(end - begin, 256), 256, 0, s>>>(c, t, begin, end);
    count_launches(1);
    return cudaGetLastError();
}

/* ---------------- photometric errors ---------------- */
/* Philox4x32-10 (Salmon, Moraes, Dror, Shaw 2011) */
__device__ __forceinline__ void philox(uint32_t ctr[4], uint32_t k0, uint32_t k1)
{
#pragma unroll
    for (int r = 0; r < 10; r++) {
        uint32_t hi0 = __umulhi(0xD2511F53u, ctr[0]), lo0 = 0xD2511F53u * ctr[0];
        uint32_t hi1 = __umulhi(0xCD9E8D57u, ctr[2]), lo1 = 0xCD9E8D57u * ctr[2];
        uint32_t n0 = hi1 ^ ctr[1] ^ k0;
        uint32_t n2 = hi0 ^ ctr[3] ^ k1;
        ctr[0] = n0; ctr[1] = lo1; ctr[2] = n2; ctr[3] = lo0;
        k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
    }
}

__device__ __forceinline__ double error_normal(uint64_t seed, uint64_t row, uint32_t band)
{
    uint32_t ctr[4] = {(uint32_t)row, (uint32_t)(row >> 32), band, 0x67616c66u};
    philox(ctr, (uint32_t)seed, (uint32_t)(seed >> 32));
    uint64_t a = ((uint64_t)ctr[0] << 21) ^ (ctr[1] >> 11);
    uint64_t b = ((uint64_t)ctr[2] << 21) ^ (ctr[3] >> 11);
    double u1 = ((double)(a & ((1ull << 53) - 1)) + 1.0) * 0x1p-53;
    double u2 = (double)(b & ((1ull << 53) - 1)) * 0x1p-53;
    double r = sqrt(-2.0 * gfm::log_d(u1));
    return r * gfm::cos_d(6.283185307179586 * u2);
}

/* gsl_interp_linear at x: the bisection's bracket (the last knot <= x, within
 * [0, n-2]), found from the guide cell when the knots are strictly increasing --
 * the same bracket, since the guide never starts past it -- and by bisection
 * otherwise (NaN takes the bisection's answer, n - 2). */
__device__ __forceinline__ double linear_eval(const double *xa, const double *ya, int n, double x, const int32_t *guide,
                                              int nguide, double gx0, double ginv)
{
    int ilo = 0;
    if (guide && x == x) {
        ilo = guide[perr_cell(x, gx0, ginv, nguide)];
        while (ilo < n - 2 && xa[ilo + 1] <= x) ilo++;
    } else {
        int ihi = n - 1;
        while (ihi > ilo + 1) {
            int i = (ihi + ilo) / 2;
            if (xa[i] > x) ihi = i; else ilo = i;
        }
    }
    double x_lo = xa[ilo], x_hi = xa[ilo + 1];
    double y_lo = ya[ilo], y_hi = ya[ilo + 1];
    double dx = x_hi - x_lo;
    if (dx > 0.0) return y_lo + (x - x_lo) / dx * (y_hi - y_lo);
    return 0.0;
}

/* guide cell g of a band: its last knot (at most nknots - 2) whose own cell is before g, or 0 */
__global__ void perr_guide_kernel(PerrTables c, int32_t *guide)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= c.nbands * c.nguide) return;
    const int b = k / c.nguide, g = k - b * c.nguide;
    const double *xa = c.mag + (size_t)b * c.nknots;
    int lo = 0, hi = c.nknots - 1;          /* knots before lo: cell < g; from hi on: not (or out of range) */
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (perr_cell(xa[mid], c.gx0[b], c.ginv[b], c.nguide) < g) lo = mid + 1; else hi = mid;
    }
    guide[k] = lo > 0 ? lo - 1 : 0;
}

cudaError_t launch_perr_guide(const PerrTables &c, int32_t *guide, cudaStream_t s)
{
    const int n = c.nbands * c.nguide;
    perr_guide_kernel<<<(n + 255) / 256, 256, 0, s>>>(c, guide);
    count_launches(1);
    return cudaGetLastError();
}

/* observed magnitudes of one row; catalog_row numbers the row within its request's catalog */
__device__ __forceinline__ void photoerr_row(const PerrTables &c, uint64_t seed, int64_t catalog_row, gf_table &t, int64_t row)
{
    const int64_t P = t.capacity;
    if (t.hidden[row]) return;
    for (int b = 0; b < c.nbands; b++) {
        float mag = t.mags[b * P + row];
        float sigma = (float)linear_eval(c.mag + (size_t)b * c.nknots, c.sigma + (size_t)b * c.nknots, c.nknots, mag,
                                         c.guide ? c.guide + (size_t)b * c.nguide : nullptr, c.nguide, c.gx0[b], c.ginv[b]);
        double z = error_normal(seed, (uint64_t)catalog_row, (uint32_t)b);
        t.obsmags[b * P + row] = mag + (float)((double)sigma * z);
    }
}

__global__ void __launch_bounds__(256) photoerr_kernel(PerrTables c, int64_t row_offset, gf_table t, int64_t begin, int64_t end)
{
    for (int64_t row = begin + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; row < end; row += (int64_t)gridDim.x * blockDim.x)
        photoerr_row(c, c.seed, row_offset + row, t, row);
}

__global__ void __launch_bounds__(256) photoerr_multi_kernel(PerrTables c, const uint64_t *seed_by_job,
                                                              const int64_t *catalog_offset_by_job, MultiRows R, gf_table t,
                                                              int64_t begin, int64_t end)
{
    for (int64_t row = begin + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; row < end; row += (int64_t)gridDim.x * blockDim.x) {
        const int sl = R.row_slot[row];
        const int job = R.slot_job[sl];
        photoerr_row(c, seed_by_job[job], catalog_offset_by_job[job] + (row - R.slot_row_begin[sl]), t, row);
    }
}

cudaError_t launch_photoerrors_multi(const PerrTables &c, const uint64_t *seed_by_job, const int64_t *catalog_offset_by_job,
                                     MultiRows R, gf_table t, int64_t begin, int64_t end, cudaStream_t s)
{
    if (end <= begin) return cudaSuccess;
    photoerr_multi_kernel<<<grid_for(end - begin, 256), 256, 0, s>>>(c, seed_by_job, catalog_offset_by_job, R, t, begin, end);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_photoerrors(const PerrTables &c, int64_t row_offset, gf_table t, int64_t begin, int64_t end, cudaStream_t s)
{
    if (end <= begin) return cudaSuccess;
    photoerr_kernel<<<grid_for(end - begin, 256), 256, 0, s>>>(c, row_offset, t, begin, end);
    count_launches(1);
    return cudaGetLastError();
}

/* ---------------- vel2pm ---------------- */
__device__ __forceinline__ void vel_xyz2lbr(float &vl, float &vb, float &vr, const float vx, const float vy, const float vz,
                                            const float l, const float b)
{
    float cl = gfm::cosf_(l), sl = gfm::sinf_(l), cb = gfm::cosf_(b), sb = gfm::sinf_(b);
    float tmp;
    vl = -vx * sl + vy * cl;
    tmp = vx * cl + vy * sl;
    vr = cb * tmp + vz * sb;
    vb = -sb * tmp + vz * cb;
}

__device__ __forceinline__ void transform_pm(float &vlout, float &vbout, float l, float b, float vl, float vb,
                                             const double ce, const double se, const double l0)
{
    double cb = gfm::cos_d((double)b);
    double sb = gfm::sin_d((double)b);
    double cl = gfm::cos_d((double)l - l0);
    double sl = gfm::sin_d((double)l - l0);
    double tmp1 = cb * se - ce * sb * sl;
    double tmp2 = ce * sb - cb * se * sl;
    double tmp4 = cb * cl;
    double tmp3 = sb * se + cb * ce * sl;
    if (fabs(tmp3) > 0.9999999) {
        vlout = vbout = 999.99f;
    } else {
        double denom1 = 1. / (tmp4 * tmp4 + tmp2 * tmp2);
        double cd = sqrt(1. - tmp3 * tmp3);
        vl = (float)((double)vl / cb);
        vlout = (float)((-ce * cl * (double)vb + cb * tmp1 * (double)vl) * denom1);
        vbout = (float)((tmp1 * (double)vb + cb * ce * cl * (double)vl) / cd);
        vlout = (float)((double)vlout * cd);
    }
}

__global__ void __launch_bounds__(256) vel2pm_kernel(gf_vel2pm_config par, gf_table t, int64_t begin, int64_t end)
{
    const int64_t P = t.capacity;
    const double ce = 0.88998740217659689, se = 0.45598511375586859, l0 = D2R * 32.932;
    for (int64_t row = begin + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; row < end; row += (int64_t)gridDim.x * blockDim.x) {
        if (t.hidden[row]) continue;
        float l = 0.017453292519943295769f * (float)t.lb[row];
        float b = 0.017453292519943295769f * (float)t.lb[P + row];
        float X = par.Rg - t.XYZ[row];
        float Y = -t.XYZ[P + row];
        float Z = t.XYZ[2 * P + row];
        float vx = t.vcyl[row], vy = t.vcyl[P + row], vz = t.vcyl[2 * P + row];
        /* vel_cyl2xyz */
        float rho = sqrtf(X * X + Y * Y);
        float cphi = X / rho;
        float sphi = Y / rho;
        float px = -sphi * vy + cphi * vx;
        float py = cphi * vy + sphi * vx;
        float pz = vz;
        px -= par.u0;
        py -= par.v0 + par.vLSR;
        pz -= par.w0;
        float ix = -px, iy = -py, iz = pz;
        vel_xyz2lbr(px, py, pz, ix, iy, iz, l, b);
        float D = sqrtf((8000.f - X) * (8000.f - X) + Y * Y + Z * Z);
        px = (float)((double)px / (4.74 * (double)D * 1e-3));
        py = (float)((double)py / (4.74 * (double)D * 1e-3));
        if (par.coordsys == 1) {
            float ivl = px, ivb = py;
            transform_pm(px, py, l, b, ivl, ivb, ce, se, l0);
        } else if (par.coordsys != 0) {
            px = py = pz = -9.99f;
        }
        t.pm[row] = px;
        t.pm[P + row] = py;
        t.pm[2 * P + row] = pz;
    }
}

cudaError_t launch_vel2pm(const gf_vel2pm_config &c, gf_table t, int64_t begin, int64_t end, cudaStream_t s)
{
    if (end <= begin) return cudaSuccess;
    vel2pm_kernel<<<grid_for(end - begin, 256), 256, 0, s>>>(c, t, begin, end);
    count_launches(1);
    return cudaGetLastError();
}

/* ---------------- gal2other ---------------- */
__global__ void __launch_bounds__(256) gal2other_kernel(int32_t coordsys, gf_table t, int64_t begin, int64_t end)
{
    const int64_t P = t.capacity;
    const double angp = D2R * 192.859508333, l0 = D2R * 32.932;
    const double ce = 0.88998740217659689, se = 0.45598511375586859;
    const double pi2 = 2 * 3.14159265358979323846264338;
    for (int64_t row = begin + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; row < end; row += (int64_t)gridDim.x * blockDim.x) {
        if (t.hidden[row]) continue;
        double lx = t.lb[row] * D2R, ly = t.lb[P + row] * D2R;
        double rx, ry;
        if (coordsys == 1) {
            const double cb = gfm::cos_d(ly), sb = gfm::sin_d(ly);
            const double cl = gfm::cos_d(lx - l0), sl = gfm::sin_d(lx - l0);
            rx = gfm::atan2_d(cb * cl, sb * ce - cb * se * sl) + angp;
            ry = gfm::asin_d(cb * ce * sl + sb * se);
            while (rx < 0.) rx += pi2;
            while (rx >= pi2) rx -= pi2;
        } else {
            rx = ry = -9999.;
        }
        t.radec[row] = rx / D2R;
        t.radec[P + row] = ry / D2R;
    }
}

cudaError_t launch_gal2other(int32_t coordsys, gf_table t, int64_t begin, int64_t end, cudaStream_t s)
{
    if (end <= begin) return cudaSuccess;
    gal2other_kernel<<<grid_for(end - begin, 256), 256, 0, s>>>(coordsys, t, begin, end);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace gfk
