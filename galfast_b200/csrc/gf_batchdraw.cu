/*
 * gf_batchdraw.cu -- the Poisson draw pass of many requests (the batched form).
 *
 * The bins, uniforms and star draws are exactly those of the reference's
 * draw pass (skygenGPU<T>::kernel with draw = 1, skygen.cu.h:469-618, and
 * draw_stars, :366-457): stream t of a request crawls blocks t, t + N, t + 2N, ...
 * of 10 consecutive bins (N streams), takes one uniform per uncut bin, and a
 * bin with stars consumes the Poisson sampler's uniforms and 2 or 4 per star.
 * The arrangement is this library's, for requests whose nm * nM is a multiple
 * of 10 (so every pixel's blocks start at local indices 0, 10, 20, ...):
 *
 *   block words     the model density at each slot distance of the request's anchor plan
 *                   along the pixel's direction (the anchor quantity that depends on the
 *                   pixel), and from them one 32-bit word per block of 10 bins and row of
 *                   up to 4 neighbouring pixels with the same cut: how many bins are live
 *                   (not cut), and a threshold that no uniform of an empty block's bins
 *                   reaches in any of the row's pixels.
 *   draw            one warp per up to 32 consecutive streams, one lane per stream.  Stream t
 *                   takes blocks t, t + N, t + 2N, ... of the request: a step loads the
 *                   word of the lane's next block, steps the MWC over the live bins and
 *                   compares the largest uniform with the threshold.  A lane whose block
 *                   may hold stars parks; when enough lanes are parked they find their
 *                   first candidate bin together, test it exactly, run the reference's
 *                   Poisson sampler and the star uniforms, record the bin (an event: its k
 *                   and the stream state at its first star) and go on with the bins after it.
 *                   (A single request's generator walks the same words with a warp a stream:
 *                   stream_draw_kernel, gf_skygen.cu.)
 *   expand          (thread per event) the star records of each event, regenerated
 *                   from its stream state, at offsets from a scan over k.
 *
 * The streams' final states are written back for the modules that continue them (Bond2010).
 */
#include "gf_crawl.cuh"
#include "gf_launch.h"
#include "gf_rng.h"
#include <cub/cub.cuh>

namespace gfk {

namespace {

#define BD_FULL 0xffffffffu
#define GF_EVBUF 64                /* events staged in shared memory per warp (a pass over the parked lanes adds at most 32) */
#define GF_BINS 0x3ffu             /* the bins of a block as bits */

/* one MWC step; returns the new x (the uniform is 2^-32 x) */
__device__ __forceinline__ uint32_t bd_mwc_x(uint64_t &v, uint32_t a)
{
    const uint64_t t = (uint64_t)a * (uint32_t)v + (v >> 32);
    v = t;
    return (uint32_t)t;
}

/* exp(-mu) >= 1 - mu: bins that surely draw no star, without exp */
__device__ __forceinline__ bool bd_surely_empty(float u, float mu)
{
    return u <= (1.0f - mu) - 3.0e-7f;
}

/* the sampler's exact test (mu > 10 takes the branch that never compares with exp(-mu)) */
__device__ __forceinline__ bool bd_has_stars(float u, float mu)
{
    return mu > 10.f || gfr::exceeds_exp_neg(u, mu);
}

template <class T>
__device__ __forceinline__ const T *plan_at(const unsigned char *plan, int off)
{
    return (const T *)(plan + off);
}

/* Per request of a chunk and block of its grid: the block's first bin (i | j << 16), its
 * binfo word, its block-start slot | the slot of its first diagonal start << 16, and a bound
 * C of LF(M) D^3 norm over its 10 bins (negative values count as 0; NaN where the
 * bound does not hold: a negative density factor or normalisation).  A bin's expected count
 * (((LF ms) norm) D^3) K, four rounded products of non-negative factors, is at most
 * (1 + 2^-24)^4 its exact value, and C ms K with ms the largest density of the block's
 * slots is at least (1 - 2^-24)^6 (1 + 1e-6) times that: the factor 1 + 1e-6 covers all ten. */
__global__ void __launch_bounds__(256) block_records_kernel(BlockLfParams P)
{
    for (long long f = blockIdx.x * (long long)blockDim.x + threadIdx.x; f < P.total; f += (long long)gridDim.x * blockDim.x) {
        int lo = 0, hi = P.njobs;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (P.blk_off[mid] <= f) lo = mid; else hi = mid;
        }
        const int job = P.job_list[lo];
        const int b = (int)(f - P.blk_off[lo]);
        const SkyModel &m = P.jobs[job].m;
        const unsigned char *plan = P.plans[job];
        const IntegPlanHdr *h = (const IntegPlanHdr *)plan;
        const float *slotD = plan_at<float>(plan, h->off_slot);
        const uint16_t *dslot = plan_at<uint16_t>(plan, h->off_dslot);
        const uint32_t bij = plan_at<uint32_t>(plan, h->off_blk)[b];
        int i = (int)(bij & 0xffffu), j = (int)(bij >> 16);
        const uint32_t bi = plan_at<uint32_t>(plan, h->off_binfo)[b];
        const uint32_t wm = (bi >> 16) & GF_BINS;
        const uint32_t s0 = plan_at<uint16_t>(plan, h->off_bslot)[b];
        const uint32_t s1 = wm ? dslot[i + j + 1] : 0u;
        float D = slotD[s0];
        float mx = gfc::lf_sample(m, m.lf, m.M1 - (float)j * m.dM);
        for (int s = 1; s < GF_BLOCK; s++) {
            if (gfc::step_in_pixel(i, j, m.nm, m.nM)) D = fmaxf(D, slotD[dslot[i + j]]);
            mx = fmaxf(mx, gfc::lf_sample(m, m.lf, m.M1 - (float)j * m.dM));
        }
        float C = fmaxf(mx, 0.f) * m.norm;
        C *= D * D * D;
        C *= 1.0f + 1.0e-6f;
        if (!(m.f >= 0.f && m.norm >= 0.f)) C = __int_as_float(0x7fffffff);
        P.brec[job][b] = make_uint4(bij, bi, s0 | (s1 << 16), __float_as_uint(C));
        /* a request's threads also sample its LF(M) at every absolute-magnitude row */
        for (int q = b; q < m.nM; q += h->nblocks) P.lfm[job][q] = gfc::lf_sample(m, m.lf, m.M1 - (float)q * m.dM);
    }
}

/* The live bins of a block: im below the pixel's cut row, and the anchor's distance inside [dmin, dmax).
 * At most one diagonal start (bin p): bins before it continue the first diagonal (im = i0 + s), bins from it
 * on the next one from im = max(0, d + 1 - (nM - 1)); each run's live bins are a prefix of it. */
__device__ __forceinline__ uint32_t block_live(const uint4 &br, int icut, int nM)
{
    const int i0 = (int)(br.x & 0xffffu), j0 = (int)(br.x >> 16);
    if ((int)(br.y & 0xffffu) < icut) return GF_BINS;                       /* the block's largest im */
    const uint32_t wm = (br.y >> 16) & GF_BINS;
    if (!(wm & (wm - 1u))) {
        const int p = wm ? __ffs(wm) - 1 : GF_BLOCK;
        const int iB = max(0, i0 + j0 + 1 - (nM - 1));
        uint32_t live = (1u << min(p, max(0, icut - i0))) - 1u;
        if (wm) live |= ((1u << min(GF_BLOCK - p, max(0, icut - iB))) - 1u) << p;
        return live;
    }
    /* several diagonal starts (short diagonals at the grid's corners) */
    int ii = i0, dd = i0 + j0;
    uint32_t live = ii < icut ? 1u : 0u;
    for (int s = 1; s < GF_BLOCK; s++) {
        if ((wm >> s) & 1u) {
            dd++;
            ii = max(0, dd - (nM - 1));
        } else {
            ii++;
        }
        live |= ii < icut ? (1u << s) : 0u;
    }
    return live;
}

/* the bins of a block whose anchor lies in [dmin, dmax) */
__device__ __noinline__ uint32_t block_inside(const uint4 &br, const float *slotD, const uint16_t *dslot, float dmin, float dmax)
{
    const uint32_t wm = (br.y >> 16) & GF_BINS;
    int d = (int)(br.x & 0xffffu) + (int)(br.x >> 16);
    float D = slotD[br.z & 0xffffu];
    uint32_t in = 0;
    for (int s = 0; s < GF_BLOCK; s++) {
        if ((wm >> s) & 1u) D = slotD[dslot[++d]];
        in |= (dmin > D || dmax <= D) ? 0u : 1u << s;
    }
    return in;
}

/* A CTA takes up to P.tile rows of one request: the slot densities of their pixels (a warp a
 * row) into the request's tables, for the exact tests of candidate bins, and each slot's largest
 * in the row into shared memory; then every block's word, a thread's block for all the tile's
 * rows (the block record is decoded once).  Pixels of a row are neighbours: their densities
 * differ by a few percent, and so do the thresholds' candidates from each pixel's own. */
template <int MODEL>
__global__ void __launch_bounds__(256) block_words_kernel(BlockWordParams P)
{
    extern __shared__ __align__(16) float s_ms[];      /* [tile][nslots] */
    __shared__ SkyModel m;
    __shared__ int s_icut[GF_WORD_TILE];
    __shared__ float s_K[GF_WORD_TILE];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int loaded = -1;
    for (int unit = blockIdx.x; unit < P.total_tiles; unit += gridDim.x) {
        int lo = 0, hi = P.njobs;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (P.tile_off[mid] <= unit) lo = mid; else hi = mid;
        }
        const int job = P.job_list[lo];
        const CrawlJob &J = P.jobs[job];
        const DrawJob &V = P.view[job];
        const int q0 = (unit - P.tile_off[lo]) * P.tile;             /* within the segment's rows */
        const int nr = min(V.nrows - q0, P.tile);
        __syncthreads();
        if (job != loaded) {
            for (int w = tid; w < (int)(sizeof(SkyModel) / 4); w += blockDim.x) ((uint32_t *)&m)[w] = ((const uint32_t *)&J.m)[w];
            loaded = job;
            __syncthreads();
        }
        const int nslots = V.nslots;
        for (int q = warp; q < nr; q += 8) {
            const int row = V.row0 + q0 + q;
            const int pa = max(V.rowpx[row], V.px0), pb = min(V.rowpx[row + 1], V.px0 + V.npx);
            float K = 0.f;
            for (int p = pa; p < pb; p++) {
                const gf_pencil_beam pix = J.g.pixels[p];
                K = fmaxf(K, pix.dA * GF_POGSON * m.dm * m.dM);
                if (lane == 0) V.roff[p - V.px0] = (uint32_t)(q0 + q) * (uint32_t)V.Bp;
                float *ms_row = V.ms + (size_t)(p - V.px0) * nslots;
                for (int s = lane; s < nslots; s += 32) {
                    const float D = V.slotD[s];
                    const float px = D * pix.cl * pix.cb;
                    const float py = D * pix.sl * pix.cb;
                    const float pz = D * pix.sb;
                    const float ms = gfc::model_rho<MODEL>(m, px, py, pz);
                    if (V.ms) ms_row[s] = ms;
                    s_ms[q * nslots + s] = p == pa ? ms : fmaxf(s_ms[q * nslots + s], ms);
                }
            }
            if (lane == 0) {
                s_icut[q] = (int)(V.prow[pa].y & 0xffffu);
                s_K[q] = K;
            }
        }
        __syncthreads();
        const bool dlim = m.dmin != 0.f || m.dmax != 0.f;
        uint32_t *words = V.words + (size_t)q0 * V.Bp;
        for (int lb = tid; lb < V.Bp; lb += blockDim.x) {
            const uint4 br = __ldg(V.brec + lb);
            const uint32_t wm = (br.y >> 16) & GF_BINS;
            const bool several = (wm & (wm - 1u)) != 0;
            const int s0 = (int)(br.z & 0xffffu), s1 = wm ? (int)(br.z >> 16) : s0;
            const float C = __uint_as_float(br.w);
            const uint32_t in = dlim ? block_inside(br, V.slotD, V.dslot, m.dmin, m.dmax) : GF_BINS;
            int icut = -1;
            uint32_t n = 0;
            for (int q = 0; q < nr; q++) {
                if (s_icut[q] != icut) {
                    icut = s_icut[q];
                    n = __popc(block_live(br, icut, m.nM) & in);
                }
                const float *ms = s_ms + q * nslots;
                float msmax = fmaxf(ms[s0], ms[s1]);
                if (several) {
                    int d = (int)(br.x & 0xffffu) + (int)(br.x >> 16) + 1;
                    for (uint32_t mm = wm & (wm - 1u); mm; mm &= mm - 1u) msmax = fmaxf(msmax, ms[V.dslot[++d]]);
                }
                const float mub = C * msmax * s_K[q];
                /* u <= 1 - mub - 3e-7 proves a bin empty; x <= X implies it (uniform_threshold_lower), and the
                 * word keeps X rounded down to 16s: a bin is a candidate when x >= that (conversion of a
                 * negative or NaN threshold gives 0: every bin is one; so it is without a bound, C NaN) */
                const uint32_t X = __float2uint_rz(((1.0f - mub) - 3.0e-7f) * 4294967296.0f * 0.99999976f);
                words[(size_t)q * V.Bp + lb] = n ? (X & ~GF_NLIVE) | n : GF_DEAD_WORD;
            }
        }
    }
}

/* A candidate bin on the lane (stream) that found it: whether its stars k > 0, from the first
 * uniform u (drawn from state wb; w the state after it).  The reference's Poisson sampler: the
 * product of uniforms against exp(-mu), bracketed as in Mwc::poisson_small, or for large means its
 * gamma and binomial stages from wb.  w becomes the state after the sampler. */
__device__ __forceinline__ int draw_count(uint32_t a, uint64_t wb, float u, float mu, uint64_t &w)
{
    if (mu >= GF_FASTEXP_MIN_MU && mu <= 10.f) {
        const float ea = __expf(-mu);
        const float lo = ea * (1.0f - GF_FASTEXP_MARGIN), hi = ea * (1.0f + GF_FASTEXP_MARGIN);
        float prod = u;
        int k = 0;
        for (;;) {
            if (prod <= lo) break;
            if (!(prod > hi) && !(prod > gfm::expf_(-mu))) break;
            k++;
            prod *= GF_MWC_SCALE * (float)bd_mwc_x(w, a);
        }
        return k;
    }
    if (!bd_has_stars(u, mu)) return 0;
    gfr::Mwc r;
    r.a = a;
    r.set_v(wb);
    r.used = 0;
    const int k = (int)r.poisson(mu);
    w = r.v();
    return k;
}

/* the state after the uniforms of k stars (draw_stars: x, y, and M, m unless x^2 + y^2 > 2) */
__device__ __forceinline__ uint64_t skip_stars(uint32_t a, uint64_t w, int k, bool edge, const gf_pencil_beam *pix)
{
    if (!edge) {
        /* no point of the pixel lies beyond x^2 + y^2 = 2 */
        for (int n = 0; n < 4 * k; n++) (void)bd_mwc_x(w, a);
        return w;
    }
    const float X = pix->X, Y = pix->Y, dx = pix->dx;
    for (int n = 0; n < k; n++) {
        const float u0 = GF_MWC_SCALE * (float)bd_mwc_x(w, a);
        const float u1 = GF_MWC_SCALE * (float)bd_mwc_x(w, a);
        float xx = X, yy = Y;
        xx += dx * (u0 - 0.5f);
        yy += dx * (u1 - 0.5f);
        if (!(xx * xx + yy * yy > 2.f)) {
            (void)bd_mwc_x(w, a);
            (void)bd_mwc_x(w, a);
        }
    }
    return w;
}

/* write the warp's staged events to the global list (all lanes) */
__device__ __forceinline__ void flush_events(const BatchDrawParams &P, EventRecord *evb, int *nev, int lane)
{
    __syncwarp();
    const int n = *nev;
    if (n == 0) return;
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(P.ev_count, (unsigned long long)n);
    base = __shfl_sync(BD_FULL, base, 0);
    for (int q = lane; q < n; q += 32)
        if (base + q < (unsigned long long)P.ev_capacity) P.ev[base + q] = evb[q];
    __syncwarp();
    if (lane == 0) *nev = 0;
    __syncwarp();
}

/* One warp per item of up to 32 consecutive streams of a request, one lane per stream.  A step of a lane
 * is one block: its word (loaded three steps ahead), at most 10 MWC steps, one comparison.
 * Almost every block is empty, and the few lanes that find a candidate bin would hold up
 * the others if the warp served each at once; so they park and are served together, when
 * their waiting has cost about what a service does (whatever the rate of candidates, that is
 * within twice the best choice).  The lanes drift apart by the steps they waited; their words
 * come from a table small enough for the caches.
 * Bound by the integer pipes: a step takes about 160 scheduler cycles (104 of them the walk), a
 * service about 430.  Measured, three models: 256 beams of 0.5-5 deg (5.1e9 blocks, 6.2e7 stars)
 * 34 ms, against 64 ms when each warp bounded its blocks itself and walked those with candidates
 * again at once; 64 beams 27 -> 10 ms.  With 64 registers (4 CTAs an SM) 38 ms at 256 beams; one vote
 * per step or two instead of four, or three times the patience: 35 to 41 ms. */
__global__ void __launch_bounds__(256, 3) batch_draw_kernel(BatchDrawParams P)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    EventRecord *evb = (EventRecord *)(smem + (size_t)wib * (sizeof(EventRecord) * GF_EVBUF + 16));
    int *nev = (int *)(evb + GF_EVBUF);
    if (lane == 0) *nev = 0;
    __syncwarp();

    /* The first items, streams of the largest requests, go round the SMs, and round the warps of an SM's
     * CTAs, so that no scheduler gets more of the longest chains than another; then the warps that finish
     * take the rest in order.  Taken in order from the start, the 240 warps of a call's largest request
     * sat on a few SMs (one busy for 57 % of the time, all of them for 8 %): 16.2 -> 13.7 ms at twelve
     * requests, 11.0 -> 10.0 ms at 64 beams, 256 beams the same. */
    const int wpc = blockDim.x >> 5, rank = (wib + blockIdx.x / P.sms) % wpc;
    for (int it = rank * gridDim.x + blockIdx.x; it < P.nitems;) {
        const uint32_t wi = P.items[it];
        const int job = (int)(wi >> 16), t = (int)(wi & 0xffffu) + lane;
        const DrawJob &V = P.view[job];
        const uint32_t Bp = (uint32_t)V.Bp;
        const bool stream_ok = t < V.N && lane < V.lanes;
        const int NS = V.rng_nstreams;
        uint32_t *rng = V.rng;
        const uint32_t a = stream_ok ? rng[t] : 0u;
        uint64_t w = stream_ok ? (((uint64_t)rng[NS + t] << 32) | rng[2 * NS + t]) : 0ull;
        const uint32_t *words = V.words, *roff = V.roff;
        const uint32_t npx = (uint32_t)V.npx, QN = (uint32_t)V.QN, RN = (uint32_t)V.RN;
        uint32_t x = (uint32_t)w, c = (uint32_t)(w >> 32);
        /* the block whose word is loaded next: pixel, block in the pixel, the words of the pixel's row.
         * The stream's first block of the segment (block r of stream t is the request's t + r N -th): */
        uint32_t lb = (uint32_t)(t >= V.first ? t - V.first : t - V.first + V.N);
        uint32_t px = (__umulhi(lb, V.fB.mul) + lb) >> V.fB.shift;
        lb -= px * Bp;
        if (!stream_ok) px = npx;
        uint32_t ro = px < npx ? __ldg(roff + px) : 0u;
        auto next_word = [&]() {
            const uint32_t word = px < npx ? __ldg(words + (ro + lb)) : GF_END_WORD;
            px += QN;
            lb += RN;
            if (lb >= Bp) { lb -= Bp; px++; }
            ro = px < npx ? __ldg(roff + px) : 0u;
            return word;
        };
        uint32_t c0 = next_word(), c1 = next_word(), c2 = next_word();
        int skip = 0;                  /* live bins of the current block that are done */
        bool parked = false;
        int idle = 0;                  /* rounds of four steps that parked lanes have waited */
        for (;;) {
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const bool act = !parked && c0 != GF_END_WORD;
                uint32_t x1 = x, cc = c;
                const uint32_t mx = gfc::walk_bins(x1, cc, a, act ? c0 & GF_NLIVE : (uint32_t)GF_BLOCK);
                if (act) {
                    if (mx >= (c0 & ~GF_NLIVE)) {
                        parked = true;
                    } else {
                        x = x1;
                        c = cc;
                        skip = 0;
                        c0 = c1;
                        c1 = c2;
                        c2 = next_word();
                    }
                }
            }
            const unsigned waiting = __ballot_sync(BD_FULL, parked), left = __ballot_sync(BD_FULL, c0 != GF_END_WORD);
            if (left == 0) break;
            /* serve the parked lanes when they have waited, together, as long as a service holds up the lanes left */
            idle += __popc(waiting);
            if (waiting == 0 || (2 * idle < __popc(left) && waiting != left)) continue;
            idle = 0;
            if (parked) {
                parked = false;
                /* the block, three steps behind the next word's */
                uint32_t pixel = px - 3 * QN;
                int lbc = (int)lb - 3 * (int)RN;
                while (lbc < 0) { lbc += (int)Bp; pixel--; }
                const uint4 br = __ldg(V.brec + lbc);
                const uint2 cut = __ldg(V.prow + V.px0 + pixel);
                const gf_pencil_beam *pix = V.pixels + V.px0 + pixel;
                const float dA = __ldg(&pix->dA);
                /* its first candidate bin, the states before and after it */
                uint32_t n = c0 & GF_NLIVE, k = 0, xk = 0;
                const uint32_t T = c0 & ~GF_NLIVE;
                w = ((uint64_t)c << 32) | x;
                uint64_t wb = w;
                for (; k < n; k++) {
                    wb = w;
                    xk = bd_mwc_x(w, a);
                    if (xk >= T) break;
                }
                const float K = dA * GF_POGSON * V.dm * V.dM;
                uint32_t live = block_live(br, (int)(cut.y & 0xffffu), V.nM);
                if (V.dlim) live &= block_inside(br, V.slotD, V.dslot, V.dmin, V.dmax);
                for (int q = skip + (int)k; q > 0; q--) live &= live - 1u;
                const int s = __ffs(live) - 1;
                /* the bin's position follows from the block's diagonal starts, as step_in_pixel walks it */
                const int i0 = (int)(br.x & 0xffffu), j0 = (int)(br.x >> 16);
                const uint32_t starts = (br.y >> 16) & ((2u << s) - 2u);         /* diagonal starts in bins 1..s */
                const int d = i0 + j0 + __popc(starts);
                int i = i0 + s, slot = (int)(br.z & 0xffffu);
                if (starts) {
                    i = max(0, d - (V.nM - 1)) + s - (31 - __clz(starts));
                    slot = d == i0 + j0 + 1 ? (int)(br.z >> 16) : (int)__ldg(V.dslot + d);
                }
                const int j = d - i;
                const float D = __ldg(V.slotD + slot);
                float mu = __ldg(V.lfm + j) * V.ms[(size_t)pixel * V.nslots + slot];
                mu *= V.norm;
                mu *= D * D * D;
                mu *= K;
                const float u = GF_MWC_SCALE * (float)xk;
                if (k < n && !bd_surely_empty(u, mu)) {
                    if (!(mu < 3.0e38f) && bd_has_stars(u, mu)) {
                        /* an infinite expected count would never leave the sampler's gamma loop: the stream ends
                         * here, its block's later bins too (px no longer tells which block a word is of) */
                        atomicOr(P.err, 1ull);
                        n = k + 1;
                        c1 = c2 = GF_END_WORD;
                        px = npx;
                    } else {
                        const int stars = draw_count(a, wb, u, mu, w);
                        if (stars > 0) {
                            EventRecord e;
                            e.stream = (job << 16) | t;
                            e.ilb = V.px0 + (int)pixel;
                            e.im = (int16_t)i;
                            e.iM = (int16_t)j;
                            e.k = stars;
                            e.v_star = w;
                            evb[atomicAdd(nev, 1)] = e;
                            w = skip_stars(a, w, stars, (cut.y & 0x10000u) != 0, pix);
                        }
                    }
                }
                x = (uint32_t)w;
                c = (uint32_t)(w >> 32);
                /* the bins after it remain */
                skip += (int)k + 1;
                if (k + 1 < n) {
                    c0 = T | (n - k - 1);
                } else {
                    skip = 0;
                    c0 = c1;
                    c1 = c2;
                    c2 = next_word();
                }
            }
            __syncwarp();
            if (*nev >= GF_EVBUF / 2) flush_events(P, evb, nev, lane);
        }
        if (stream_ok) {
            rng[NS + t] = c;
            rng[2 * NS + t] = x;
        }
        if (lane == 0) it = (int)(gridDim.x * wpc + atomicAdd(P.next_item, 1u));
        it = __shfl_sync(BD_FULL, it, 0);
    }
    flush_events(P, evb, nev, lane);
}

__global__ void event_k_kernel(const EventRecord *ev, int64_t n, int64_t *k64)
{
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
        k64[e] = ev[e].k;
}

/* the star records of each event (draw_stars' uniforms, skygen.cu.h:366-457) */
__global__ void __launch_bounds__(256) expand_kernel(const EventRecord *ev, int64_t n, const int64_t *off, const int64_t *k64,
                                                     const CrawlJob *jobs, StarRecord *rec, int64_t cap, int64_t *total)
{
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
        const EventRecord E = ev[e];
        const int job = E.stream >> 16, t = E.stream & 0xffff;
        const CrawlJob &J = jobs[job];
        const gf_pencil_beam pix = J.g.pixels[E.ilb];
        gfr::Mwc r;
        r.a = J.rng[t];
        r.set_v(E.v_star);
        r.used = 0;
        const int64_t o = off[e];
        for (int q = 0; q < E.k; q++) {
            StarRecord s;
            s.stream = E.stream;
            s.ilb = E.ilb + J.pix_base;
            s.im = E.im;
            s.iM = E.iM;
            s.seq = q;
            s.u[0] = r.uniform();
            s.u[1] = r.uniform();
            float xx = pix.X, yy = pix.Y;
            xx += pix.dx * (s.u[0] - 0.5f);
            yy += pix.dx * (s.u[1] - 0.5f);
            if (xx * xx + yy * yy > 2.f) {
                s.u[2] = s.u[3] = 0.f;
            } else {
                s.u[2] = r.uniform();
                s.u[3] = r.uniform();
            }
            if (o + q < cap) rec[o + q] = s;
        }
        if (e == n - 1) *total = o + k64[e];
    }
}

}  // namespace

cudaError_t launch_block_records(const BlockLfParams &P, cudaStream_t s)
{
    if (P.total <= 0) return cudaSuccess;
    const int blocks = (int)std::min<long long>((P.total + 255) / 256, (long long)sm_count() * 16);
    block_records_kernel<<<blocks, 256, 0, s>>>(P);
    count_launches(1);
    return cudaGetLastError();
}

int block_word_tile(int64_t rows, int max_slots)
{
    /* as many rows as 96 KB of densities hold, but four tiles an SM while there are fewer rows than that */
    const int64_t fit = (96 * 1024) / (4 * (int64_t)std::max(max_slots, 1));
    const int64_t want = std::min<int64_t>(std::min<int64_t>(fit, GF_WORD_TILE), rows / (4 * (int64_t)sm_count()));
    return (int)std::max<int64_t>(want, 1);
}

template <int MODEL>
static cudaError_t launch_block_words_t(const BlockWordParams &P, int max_slots, cudaStream_t s)
{
    const size_t smem = 4 * (size_t)P.tile * max_slots;
    cudaError_t e = cudaFuncSetAttribute(block_words_kernel<MODEL>, cudaFuncAttributeMaxDynamicSharedMemorySize, GF_WORD_SMEM);
    int per_sm = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, block_words_kernel<MODEL>, 256, smem);
    if (e != cudaSuccess) return e;
    const int blocks = (int)std::min<long long>(P.total_tiles, (long long)sm_count() * std::max(per_sm, 1));
    block_words_kernel<MODEL><<<blocks, 256, smem, s>>>(P);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_block_words(const BlockWordParams &P, int model_type, int max_slots, cudaStream_t s)
{
    if (P.total_tiles <= 0) return cudaSuccess;
    if (P.tile < 1 || P.tile > GF_WORD_TILE || !block_words_fit(P.tile, max_slots)) return cudaErrorInvalidValue;
    return model_type == GF_MODEL_EXP_DISK ? launch_block_words_t<GF_MODEL_EXP_DISK>(P, max_slots, s)
                                           : launch_block_words_t<GF_MODEL_POWER_LAW_ELLIPSOID>(P, max_slots, s);
}

cudaError_t launch_batch_draw(const BatchDrawParams &P, int warps_per_cta, cudaStream_t s)
{
    if (P.nitems <= 0) return cudaSuccess;
    if (warps_per_cta < 1 || warps_per_cta > 8) warps_per_cta = 4;
    const size_t smem = (size_t)warps_per_cta * (sizeof(EventRecord) * GF_EVBUF + 16);
    cudaError_t e = cudaMemsetAsync(P.next_item, 0, sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
    const int threads = 32 * warps_per_cta;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_draw_kernel, threads, smem);
    if (e != cudaSuccess) return e;
    const long long want = ((long long)P.nitems + warps_per_cta - 1) / warps_per_cta;
    const int blocks = (int)std::min<long long>(want, (long long)sm_count() * std::max(per_sm, 1));
    BatchDrawParams Q = P;
    Q.sms = sm_count();
    batch_draw_kernel<<<blocks, threads, smem, s>>>(Q);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t expand_temp_bytes(int64_t nev, size_t *bytes)
{
    *bytes = 0;
    if (nev <= 0) return cudaSuccess;
    return cub::DeviceScan::ExclusiveSum(nullptr, *bytes, (const int64_t *)nullptr, (int64_t *)nullptr, (int)nev);
}

cudaError_t launch_expand_events(const EventRecord *ev, int64_t nev, const CrawlJob *jobs, int64_t *k64, int64_t *off64,
                                 void *temp, size_t temp_bytes, StarRecord *rec, int64_t rec_capacity, int64_t *total,
                                 cudaStream_t s)
{
    cudaError_t e = cudaMemsetAsync(total, 0, sizeof(int64_t), s);
    if (e != cudaSuccess || nev <= 0) return e;
    const int blocks = (int)std::min<long long>((nev + 255) / 256, (long long)sm_count() * 16);
    event_k_kernel<<<blocks, 256, 0, s>>>(ev, nev, k64);
    size_t tb = temp_bytes;
    e = cub::DeviceScan::ExclusiveSum(temp, tb, k64, off64, (int)nev, s);
    if (e != cudaSuccess) return e;
    expand_kernel<<<blocks, 256, 0, s>>>(ev, nev, off64, k64, jobs, rec, rec_capacity, total);
    count_launches(3);
    return cudaGetLastError();
}

}  // namespace gfk
