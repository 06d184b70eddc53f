/*
 * gf_integrate.cu -- the expected-count (integrate) pass of many requests,
 * pixel by pixel.
 *
 * The reference integrates with the same crawl as the draw pass: stream t
 * takes blocks of 10 consecutive bins, and evaluates the model at an anchor
 * bin at every block start and every diagonal start (skygen.cu.h:469-611);
 * each later bin of the block reuses its anchor.  When nm * nM is a multiple
 * of 10 the blocks of every pixel start at the local indices k = 0, 10, 20 ...,
 * so the anchors of a pixel are the same positions in every pixel and in
 * every stream decomposition.  This pass computes every bin's expected count
 * with the reference's anchor and float expression, without the streams:
 *
 *   plan    (per magnitude grid) the anchor positions of each diagonal and the
 *           anchor's distance D[im][iM].  Along a diagonal the distance
 *           modulus is the same number rounded in a few different ways, so
 *           the anchors of a diagonal take only 1-4 distinct D; the plan lists
 *           the distinct values (the slots) and maps every anchor to its slot.
 *   pixels  (two pixels a lane, 64 pixels of a request to a warp) the warp walks
 *           the plan's diagonals and anchors together: on a diagonal each lane
 *           forms the model density at the diagonal's slot distances along its own
 *           pixels' directions (the only anchor quantity that depends on D and the
 *           pixel), then every bin's mu = (((LF(M) * ms) * norm) * D^3) * K, bins
 *           with m + Am > m1 cut.  Per pixel the counts and covered counts are
 *           summed in FP64.
 *   totals  (32 CTAs per request, then their sums) the pixel sums in a fixed order.
 *
 * Every bin's mu is bit-identical to the crawl's; the totals differ from a
 * per-stream summation only by the order of the FP64 additions.
 */
#include "gf_crawl.cuh"
#include "gf_launch.h"

namespace gfk {

namespace {

/* first local index of diagonal d (cells before it) and its length, for an x-by-y grid */
__device__ __forceinline__ long long diag_start(int d, int x, int y)
{
    const long long l = x < y ? x : y, m = x < y ? y : x, n = x + y - 1 - (long long)d;
    if (d < l) return (long long)d * (d + 1) / 2;
    if (d < m) return l * (l + 1) / 2 + ((long long)d - l) * l;
    return (long long)x * y - n * (n + 1) / 2;
}

__device__ __forceinline__ int diag_len(int d, int x, int y)
{
    const int l = x < y ? x : y;
    int n = d + 1;
    n = n < l ? n : l;
    const int r = x + y - 1 - d;
    return n < r ? n : r;
}

/* first anchor after position 0 on a diagonal that starts at local index k0 */
__device__ __forceinline__ int first_block_start(long long k0)
{
    const int r = (int)(k0 % GF_BLOCK);
    return r == 0 ? GF_BLOCK : GF_BLOCK - r;
}

#define GF_PLAN_REMEMBER 8          /* distinct distances remembered per diagonal */

/* distinct anchor distances of diagonal d, in order of first appearance; calls
 * emit(anchor ordinal, slot ordinal on the diagonal, D, local index, i, j) for every anchor */
template <class F>
__device__ __forceinline__ int diag_anchors(const float *Dtab, int nM_tab, int d, int x, int y, F emit)
{
    const long long k0 = diag_start(d, x, y);
    const int len = diag_len(d, x, y);
    const int i0 = d - (y - 1) > 0 ? d - (y - 1) : 0;
    uint32_t seen[GF_PLAN_REMEMBER];
    int nseen = 0, nslot = 0, q = 0;
    for (int t = 0; t < len; t = (t == 0 ? first_block_start(k0) : t + GF_BLOCK), q++) {
        const int i = i0 + t, j = d - i;
        const float D = Dtab[(size_t)i * nM_tab + j];
        const uint32_t b = __float_as_uint(D);
        int s = -1;
        for (int r = 0; r < nseen; r++)
            if (seen[r] == b) s = r;
        if (s < 0) {
            s = nslot++;
            if (nseen < GF_PLAN_REMEMBER) seen[nseen++] = b;
        }
        emit(q, s, D, k0 + t, i, j);
    }
    return nslot;
}

/* block-wide exclusive scan of two counters (blockDim.x = 1024) */
__device__ __forceinline__ void scan2(int &a, int &b, int *sa, int *sb, int &tot_a, int &tot_b)
{
    const int t = threadIdx.x;
    sa[t] = a;
    sb[t] = b;
    __syncthreads();
    for (int o = 1; o < blockDim.x; o <<= 1) {
        int va = 0, vb = 0;
        if (t >= o) { va = sa[t - o]; vb = sb[t - o]; }
        __syncthreads();
        sa[t] += va;
        sb[t] += vb;
        __syncthreads();
    }
    tot_a = sa[blockDim.x - 1];
    tot_b = sb[blockDim.x - 1];
    a = sa[t] - a;
    b = sb[t] - b;
    __syncthreads();
}

/* byte layout of a plan (the header's offsets) */
__host__ __device__ inline void plan_layout(int nm, int nM, int max_anchors, int max_slots, IntegPlanHdr &h)
{
    const long long nd = (long long)nm + nM - 1, nb = (long long)nm * nM / GF_BLOCK;
    long long off = (sizeof(IntegPlanHdr) + 15) & ~15ll;
    off += (8 * nd + 15) & ~15ll;
    h.off_slot = (int32_t)off;
    off += (4 * (long long)max_slots + 15) & ~15ll;
    h.off_anc = (int32_t)off;
    off += (2 * (long long)max_anchors + 15) & ~15ll;
    h.off_blk = (int32_t)off;
    off += (4 * nb + 15) & ~15ll;
    h.off_bslot = (int32_t)off;
    off += (2 * nb + 15) & ~15ll;
    h.off_dslot = (int32_t)off;
    off += (2 * nd + 15) & ~15ll;
    h.off_binfo = (int32_t)off;
    off += (4 * nb + 15) & ~15ll;
    h.nd = (int32_t)nd;
    h.nblocks = (int32_t)nb;
    h.max_anchors = max_anchors;
    h.max_slots = max_slots;
    h.bytes = (int32_t)off;
    h.nanchors = 0;
    h.nslots = 0;
    h.ok = 0;
    h.pad[0] = h.pad[1] = 0;
}

__global__ void __launch_bounds__(1024) plan_kernel(const IntegPlanDesc *desc)
{
    __shared__ int sa[1024], sb[1024];
    const IntegPlanDesc P = desc[blockIdx.x];
    const int x = P.nm, y = P.nM, nd = x + y - 1;
    unsigned char *plan = P.plan;
    IntegPlanHdr h;
    plan_layout(x, y, P.max_anchors, P.max_slots, h);
    int2 *diag = (int2 *)(plan + ((sizeof(IntegPlanHdr) + 15) & ~15));
    float *slotD = (float *)(plan + h.off_slot);
    uint16_t *anc = (uint16_t *)(plan + h.off_anc);
    uint32_t *blk = (uint32_t *)(plan + h.off_blk);
    uint16_t *bslot = (uint16_t *)(plan + h.off_bslot);
    uint16_t *dslot = (uint16_t *)(plan + h.off_dslot);
    int base_a = 0, base_s = 0;
    bool overflow = false;
    for (int c0 = 0; c0 < nd; c0 += blockDim.x) {
        const int d = c0 + threadIdx.x;
        int na = 0, ns = 0;
        if (d < nd) ns = diag_anchors(P.Dtab, P.nM_tab, d, x, y, [&](int q, int, float, long long, int, int) { na = q + 1; });
        int ea = na, es = ns, ta = 0, ts = 0;
        scan2(ea, es, sa, sb, ta, ts);
        const int abase = base_a + ea, sbase = base_s + es;
        if (d < nd) {
            diag[d] = make_int2(abase, first_block_start(diag_start(d, x, y)));
            if (abase + na <= P.max_anchors && sbase + ns <= P.max_slots && sbase + ns <= 65536)
                diag_anchors(P.Dtab, P.nM_tab, d, x, y, [&](int q, int s, float D, long long k, int i, int j) {
                    const int slot = sbase + s;
                    anc[abase + q] = (uint16_t)slot;
                    slotD[slot] = D;
                    if (q == 0) dslot[d] = (uint16_t)slot;
                    if (k % GF_BLOCK == 0) {
                        blk[k / GF_BLOCK] = (uint32_t)i | ((uint32_t)j << 16);
                        bslot[k / GF_BLOCK] = (uint16_t)slot;
                    }
                });
            else
                overflow = true;
        }
        base_a += ta;
        base_s += ts;
    }
    overflow = __syncthreads_or(overflow);
    /* per block: its largest m row and its diagonal starts, from the block-start bins above */
    if (!overflow) {
        uint32_t *binfo = (uint32_t *)(plan + h.off_binfo);
        for (int b = threadIdx.x; b < h.nblocks; b += blockDim.x) {
            const uint32_t bij = blk[b];
            int i = (int)(bij & 0xffffu), j = (int)(bij >> 16);
            int imax = i;
            uint32_t wm = 0;
            for (int s = 1; s < GF_BLOCK; s++) {
                if (gfc::step_in_pixel(i, j, x, y)) wm |= 1u << s;
                imax = i > imax ? i : imax;
            }
            binfo[b] = (uint32_t)imax | (wm << 16);
        }
    }
    if (threadIdx.x == 0) {
        h.nanchors = base_a;
        h.nslots = base_s;
        h.ok = overflow ? 0 : 1;
        *(IntegPlanHdr *)plan = h;
    }
}

#define GF_IG_WARPS 4               /* warps of a CTA, all on one request */
#define GF_IG_SLOTS 8               /* slots of a diagonal kept per lane (a plan has 1-4; further ones are formed anew) */

/* a float's bits as a double: exact for positive normal floats.  One wide multiply-add places the
 * mantissa and adds the difference of the exponent biases; the conversion instruction runs at an
 * eighth of the rate of an addition, so a run's bins take the two ways in turn. */
__device__ __forceinline__ double widen_positive(float v)
{
    return __longlong_as_double((long long)((uint64_t)__float_as_uint(v) * (1ull << 29) + (0x380ull << 52)));
}

/* the products of two pixels at once (each rounded to nearest, as FMUL) */
__device__ __forceinline__ float2 mul2(float2 a, float2 b)
{
    float2 r;
    asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmul.rn.f32x2 c, a, b;\n\tmov.b64 {%0, %1}, c;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}

/* scalar additions: the compiler contracts packed products and packed sums even though both ask for rounding */
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y)); }

__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }

/* sums of a lane's two pixels: counts, covered counts */
struct PixelSums {
    double cx = 0.0, cy = 0.0, vx = 0.0, vy = 0.0;
};

/* what the lanes of a warp share while they walk a request's diagonals */
struct DiagonalWalk {
    const int2 *diag;
    const uint16_t *anc, *dslot;
    const float *slotD;
    int nslots, d0, d1;
    int icmin, icmax;              /* the lanes' cut rows lie between */
    const float2 *lf;              /* LF rows reversed (entry k is LF(nM - 1 - k)), each twice; a second copy from entry 1 on, pitch apart */
    int pitch;
    float lfmin, lfmax;
};

/* the directions of a lane's two pixels */
struct PixelPair {
    float2 cl, cb, sl, sb;
};

/* model density of both pixels at distance D (anchor_x's expressions: px = D cl cb ..., then the model's frame) */
template <int MODEL>
__device__ __forceinline__ float2 pair_density(const SkyModel &m, const PixelPair &P, float D)
{
    const float2 D2 = both(D);
    const float2 vx = add2(mul2(mul2(D2, P.cl), P.cb), both(m.T[0]));
    const float2 vy = add2(mul2(mul2(D2, P.sl), P.cb), both(m.T[1]));
    const float2 vz = add2(mul2(D2, P.sb), both(m.T[2]));
    const float2 wx = add2(add2(mul2(both(m.M[0]), vx), mul2(both(m.M[1]), vy)), mul2(both(m.M[2]), vz));
    const float2 wy = add2(add2(mul2(both(m.M[3]), vx), mul2(both(m.M[4]), vy)), mul2(both(m.M[5]), vz));
    const float2 wz = add2(add2(mul2(both(m.M[6]), vx), mul2(both(m.M[7]), vy)), mul2(both(m.M[8]), vz));
    return make_float2(gfc::model_rho_frame<MODEL>(m, wx.x, wy.x, wz.x), gfc::model_rho_frame<MODEL>(m, wx.y, wy.y, wz.y));
}

/* One pair of bins of both pixels (entries lp->xy and lp->zw): products, then the sums; odd: the second bin counts too */
template <bool COV>
__device__ __forceinline__ void add_bins(const float4 *lp, float2 ms, float2 D3, float2 K, float2 cf, bool odd, bool turn, PixelSums &sum)
{
    const float4 l = *lp;
    float2 p = mul2({l.x, l.y}, ms), q = mul2({l.z, l.w}, ms);
    p = mul2(p, D3);
    q = mul2(q, D3);
    p = mul2(p, K);
    q = mul2(q, K);
    sum.cx += (double)p.x;
    sum.cy += widen_positive(p.y);
    if (odd) {
        sum.cx += widen_positive(q.x);
        sum.cy += turn ? (double)q.y : widen_positive(q.y);
    }
    if (COV) {
        p = mul2(p, cf);
        q = mul2(q, cf);
        sum.vx += (double)p.x;
        sum.vy += widen_positive(p.y);
        if (odd) {
            sum.vx += widen_positive(q.x);
            sum.vy += turn ? (double)q.y : widen_positive(q.y);
        }
    }
}

/* The diagonals [d0, d1) of the lanes' pixels; K, cf, icut: of each lane's two pixels. */
template <int MODEL, bool COV>
__device__ __forceinline__ void walk_diagonals(const SkyModel &m, const DiagonalWalk &W, const PixelPair &pix, int2 icut, float2 K,
                                               float2 cf, float2 (*s_ms)[32], int lane, PixelSums &sum)
{
    const int x = m.nm, y = m.nM, nd = x + y - 1;
    const float norm = m.norm;
    const bool dlim = m.dmin != 0.f || m.dmax != 0.f;
    for (int d = W.d0; d < W.d1; d++) {
        const int i0 = d - (y - 1) > 0 ? d - (y - 1) : 0;
        const int len = (d < x - 1 ? d : x - 1) - i0 + 1;
        const int tmax = min(len, W.icmax - i0);
        if (tmax <= 0) continue;
        const int tmin = min(len, W.icmin - i0);
        const int2 dg = __ldg(W.diag + d);
        const int s0 = __ldg(W.dslot + d), ns = (d + 1 < nd ? (int)__ldg(W.dslot + d + 1) : W.nslots) - s0;
        /* The densities, and for which slots every product of the diagonal is a positive normal float in all
         * lanes' pixels (then the widening by bits is exact). */
        unsigned plain = 0;
        for (int k = 0; k < ns && k < GF_IG_SLOTS; k++) {
            const float D = __ldg(W.slotD + s0 + k);
            const float2 ms = pair_density<MODEL>(m, pix, D);
            s_ms[k][lane] = ms;
            const float f3 = D * D * D;
            const float fx = ms.x * f3 * K.x * (COV ? cf.x : 1.0f), fy = ms.y * f3 * K.y * (COV ? cf.y : 1.0f);
            /* (each factor for itself: a minimum of two drops the one that is no number; with a row that is not
             * positive, bounds of negative products would pass) */
            const bool in = W.lfmin > 0.0f && W.lfmin * fx > 1.0e-30f && W.lfmin * fy > 1.0e-30f && W.lfmax * fx < 1.0e30f && W.lfmax * fy < 1.0e30f;
            if (__all_sync(0xffffffffu, in)) plain |= 1u << k;
        }
        if (norm != 1.0f) plain = 0;
        const int st = (y - 1) - (d - i0);             /* the entry of the diagonal's first bin */
        const uint16_t *ap = W.anc + dg.x;
        int t = 0, seg_end = min(dg.y, tmax), slot = __ldg(ap);
        for (;;) {
            const int rel = slot - s0, n = seg_end - t;
            const float D = __ldg(W.slotD + slot);
            if (seg_end < tmax) slot = __ldg(++ap);
            if (!(dlim && (m.dmin > D || m.dmax <= D))) {
                const float2 ms = rel < GF_IG_SLOTS ? s_ms[rel][lane] : pair_density<MODEL>(m, pix, D);
                const float2 D3 = both(D * D * D);
                if (rel < GF_IG_SLOTS && ((plain >> rel) & 1u) && seg_end <= tmin) {
                    const int at = st + t;
                    const float4 *lp = (const float4 *)(W.lf + (at & 1) * W.pitch + (at & ~1));
                    if (n == GF_BLOCK) {
#pragma unroll
                        for (int u = 0; u < GF_BLOCK / 2; u++) add_bins<COV>(lp + u, ms, D3, K, cf, true, u & 1, sum);
                    } else {
#pragma unroll 1
                        for (int u = 0; u < n; u += 2) add_bins<COV>(lp++, ms, D3, K, cf, u + 1 < n, false, sum);
                    }
                } else {
                    for (int q = t; q < seg_end; q++) {
                        float2 mu = mul2(W.lf[st + q], ms);
                        mu = mul2(mu, both(norm));
                        mu = mul2(mu, D3);
                        mu = mul2(mu, K);
                        if (i0 + q < icut.x) {
                            sum.cx += (double)mu.x;
                            if (COV) sum.vx += (double)(mu.x * cf.x);
                        }
                        if (i0 + q < icut.y) {
                            sum.cy += (double)mu.y;
                            if (COV) sum.vy += (double)(mu.y * cf.y);
                        }
                    }
                }
            }
            t = seg_end;
            if (t >= tmax) break;
            seg_end = min(t + GF_BLOCK, tmax);
        }
    }
}

/* A warp takes a group of 64 pixels of one request (in P.order: the fully covered ones first, so that
 * only the groups with partly covered pixels form the covered products) and one of P.splits parts of
 * their diagonals; a CTA's warps share the request's model and LF table.  The plan's control flow, its
 * loads and the LF reads are the same for all lanes; per bin and pixel there remain the float products
 * (two pixels to an instruction), a conversion and an FP64 addition.  Bound by instruction issue: 10 warp
 * instructions per bin of 32 pixels, 58 % of the slots used (4.3e9 bins: 1.35e9 instructions; with a warp a
 * pixel and a lane a diagonal 2.57e9, at 22 of 32 lanes, the conversions alone half the time).  Three models:
 * 256 beams 35.3 -> 29.6 ms (27.0 with the exponentials rounded from a table), 8 beams 1.43 -> 0.62 ms.
 * The runs of two pixels to an instruction need every LF row of the model positive and a normalisation of 1
 * (the widening by bits holds for positive normal products only): one zero row anywhere, or a norm that was
 * set, sends all bins through the general loop.  19600 pixels, three models: 1.59 ms, and 1.91 with zero rows or a
 * norm (11.5 by streams); 64 beams 7.3 ms, and 9.6 with zero rows (9.5 before this kernel). */
template <int MODEL>
__global__ void __launch_bounds__(32 * GF_IG_WARPS) integrate_pixels_kernel(IntegPixParams P)
{
    extern __shared__ __align__(16) float2 s_lf[];
    __shared__ SkyModel m;
    __shared__ float2 s_ms[GF_IG_WARPS][GF_IG_SLOTS][32];
    __shared__ float s_ext[2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int loaded = -1;
    for (int cta = blockIdx.x; cta < P.total_ctas; cta += gridDim.x) {
        int job = 0, hi = P.njobs;
        while (hi - job > 1) {
            const int mid = (job + hi) >> 1;
            if (P.cta_off[mid] <= cta) job = mid; else hi = mid;
        }
        const CrawlJob &J = P.jobs[job];
        if (job != loaded) {
            __syncthreads();
            for (int w = threadIdx.x; w < (int)(sizeof(SkyModel) / 4); w += blockDim.x) ((uint32_t *)&m)[w] = ((const uint32_t *)&J.m)[w];
            __syncthreads();
            for (int k = threadIdx.x; k < P.pitch; k += blockDim.x) {
                const float v = k < m.nM ? gfc::lf_sample(m, m.lf, m.M1 - (float)(m.nM - 1 - k) * m.dM) : 0.f;
                s_lf[k] = make_float2(v, v);
                if (k > 0) s_lf[P.pitch + k - 1] = make_float2(v, v);
            }
            __syncthreads();
            if (warp == 0) {
                float lo = s_lf[0].x, up = lo;
                bool number = true;
                for (int k = lane; k < m.nM; k += 32) {
                    lo = fminf(lo, s_lf[k].x);
                    up = fmaxf(up, s_lf[k].x);
                    number = number && s_lf[k].x == s_lf[k].x;
                }
                if (!__all_sync(0xffffffffu, number)) lo = -1.0f;         /* no slot is plain */
                for (int o = 16; o > 0; o >>= 1) {
                    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
                    up = fmaxf(up, __shfl_xor_sync(0xffffffffu, up, o));
                }
                if (lane == 0) { s_ext[0] = lo; s_ext[1] = up; }
            }
            __syncthreads();
            loaded = job;
        }
        const unsigned char *plan = P.plans[job];
        const IntegPlanHdr *h = (const IntegPlanHdr *)plan;
        const int npix = J.g.npixels, unit = (cta - P.cta_off[job]) * GF_IG_WARPS + warp;
        const int g = unit / P.splits, sp = unit - g * P.splits;
        if (g * 64 >= npix || !h->ok) continue;
        const int qa = g * 64 + lane, qb = qa + 32, base = P.pix_off[job];
        const uint32_t ia = P.order[base + min(qa, npix - 1)], ib = P.order[base + min(qb, npix - 1)];
        const gf_pencil_beam pa = J.g.pixels[ia], pb = J.g.pixels[ib];
        const float2 K = {pa.dA * GF_POGSON * m.dm * m.dM, pb.dA * GF_POGSON * m.dm * m.dM};
        const float2 cf = {pa.coveredFraction, pb.coveredFraction};
        const PixelPair pix = {{pa.cl, pb.cl}, {pa.cb, pb.cb}, {pa.sl, pb.sl}, {pa.sb, pb.sb}};
        const int2 icut = make_int2((int)(P.prow[base + ia].y & 0xffffu), (int)(P.prow[base + ib].y & 0xffffu));
        /* the diagonals whose first bin lies in the part's share of the bins */
        const int x = m.nm, y = m.nM, nd = x + y - 1;
        auto diagonal_at = [&](long long bin) {
            int lo = 0, up = nd;
            while (lo < up) {
                const int mid = (lo + up) >> 1;
                if (diag_start(mid, x, y) < bin) lo = mid + 1; else up = mid;
            }
            return lo;
        };
        const long long bins = (long long)x * y;
        DiagonalWalk W;
        W.d0 = sp == 0 ? 0 : diagonal_at(bins * sp / P.splits);
        W.d1 = sp + 1 == P.splits ? nd : diagonal_at(bins * (sp + 1) / P.splits);
        W.icmin = __reduce_min_sync(0xffffffffu, min(icut.x, icut.y));
        W.icmax = __reduce_max_sync(0xffffffffu, max(icut.x, icut.y));
        W.diag = (const int2 *)(plan + ((sizeof(IntegPlanHdr) + 15) & ~15));
        W.slotD = (const float *)(plan + h->off_slot);
        W.anc = (const uint16_t *)(plan + h->off_anc);
        W.dslot = (const uint16_t *)(plan + h->off_dslot);
        W.nslots = h->nslots;
        W.lf = s_lf;
        W.pitch = P.pitch;
        W.lfmin = s_ext[0];
        W.lfmax = s_ext[1];
        PixelSums sum;
        if (__all_sync(0xffffffffu, cf.x == 1.0f && cf.y == 1.0f)) {
            /* fully covered pixels: mu * cf == mu, so the covered sum is the sum */
            walk_diagonals<MODEL, false>(m, W, pix, icut, K, cf, s_ms[warp], lane, sum);
            sum.vx = sum.cx;
            sum.vy = sum.cy;
        } else {
            walk_diagonals<MODEL, true>(m, W, pix, icut, K, cf, s_ms[warp], lane, sum);
        }
        double2 *out = P.pix_sum + (size_t)sp * P.total_pix + base;
        if (qa < npix) out[ia] = make_double2(sum.cx, sum.vx);
        if (qb < npix) out[ib] = make_double2(sum.cy, sum.vy);
    }
}

/* GF_TOTAL_PARTS CTAs a request sum its pixels, one more launch their sums: a single large request
 * (20k pixels in 32 parts: 10 MB) is latency-bound with one CTA. */
#define GF_TOTAL_PARTS 32

__global__ void __launch_bounds__(256) job_totals_kernel(const double2 *pix_sum, const int32_t *pix_off, int splits, int total_pix,
                                                          const unsigned char *const *plans, double2 *part)
{
    __shared__ double sc[256], sv[256];
    const int j = blockIdx.y;
    double c = 0.0, v = 0.0;
    if (plans[j])
        for (int sp = 0; sp < splits; sp++)
            for (int p = pix_off[j] + blockIdx.x * blockDim.x + threadIdx.x; p < pix_off[j + 1]; p += GF_TOTAL_PARTS * blockDim.x) {
                const double2 s = pix_sum[(size_t)sp * total_pix + p];
                c += s.x;
                v += s.y;
            }
    sc[threadIdx.x] = c;
    sv[threadIdx.x] = v;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            sc[threadIdx.x] += sc[threadIdx.x + o];
            sv[threadIdx.x] += sv[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) part[(size_t)j * GF_TOTAL_PARTS + blockIdx.x] = make_double2(sc[0], sv[0]);
}

__global__ void __launch_bounds__(256) sum_totals_kernel(const double2 *part, int njobs, double2 *tot)
{
    const int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (j >= njobs) return;
    double2 s = part[(size_t)j * GF_TOTAL_PARTS + lane];
    for (int o = 16; o > 0; o >>= 1) {
        s.x += __shfl_down_sync(0xffffffffu, s.x, o);
        s.y += __shfl_down_sync(0xffffffffu, s.y, o);
    }
    if (lane == 0) tot[j] = s;
}

__global__ void __launch_bounds__(256) pixel_counts_kernel(const double2 *pix_sum, int splits, int npix, double *out)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npix) return;
    double v = 0.0;
    for (int sp = 0; sp < splits; sp++) v += pix_sum[(size_t)sp * npix + p].y;
    out[p] = v;
}

}  // namespace

size_t integ_plan_bytes(int nm, int nM, int *max_anchors, int *max_slots)
{
    const long long nd = (long long)nm + nM - 1;
    const long long na = (long long)nm * nM / GF_BLOCK + nd;
    *max_anchors = (int)std::min<long long>(na, 1ll << 30);
    *max_slots = (int)std::min<long long>(na, 65536);
    IntegPlanHdr h;
    plan_layout(nm, nM, *max_anchors, *max_slots, h);
    return (size_t)h.bytes;
}

cudaError_t launch_integ_plans(const IntegPlanDesc *desc_dev, int nplans, cudaStream_t s)
{
    if (nplans <= 0) return cudaSuccess;
    plan_kernel<<<nplans, 1024, 0, s>>>(desc_dev);
    count_launches(1);
    return cudaGetLastError();
}

int integ_splits(int64_t groups)
{
    /* parts of the diagonals: about 128 warps an SM (several rounds of them, so that a large request does not end last) */
    const int64_t want = (int64_t)sm_count() * 128;
    return (int)std::max<int64_t>(1, std::min<int64_t>(32, want / std::max<int64_t>(groups, 1)));
}

int64_t integ_ctas(int64_t npix, int splits) { return ((npix + 63) / 64 * splits + GF_IG_WARPS - 1) / GF_IG_WARPS; }

size_t integ_smem(int nM_max, int32_t *pitch)
{
    *pitch = (int32_t)((nM_max + 15) & ~3);
    return 16 * (size_t)*pitch;
}

template <int MODEL>
static cudaError_t launch_integrate_pixels_t(const IntegPixParams &P, cudaStream_t s)
{
    const size_t smem = 16 * (size_t)P.pitch;
    cudaError_t e = cudaFuncSetAttribute(integrate_pixels_kernel<MODEL>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    int per_sm = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, integrate_pixels_kernel<MODEL>, 32 * GF_IG_WARPS, smem);
    if (e != cudaSuccess) return e;
    const int blocks = (int)std::min<long long>(P.total_ctas, (long long)sm_count() * std::max(per_sm, 1));
    integrate_pixels_kernel<MODEL><<<blocks, 32 * GF_IG_WARPS, smem, s>>>(P);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_integrate_pixels(const IntegPixParams &P, int model_type, double2 *tot, cudaStream_t s)
{
    if (P.total_ctas <= 0) return cudaSuccess;
    if (16 * (size_t)P.pitch > 200 * 1024 || P.splits < 1) return cudaErrorInvalidValue;
    cudaError_t e = model_type == GF_MODEL_EXP_DISK ? launch_integrate_pixels_t<GF_MODEL_EXP_DISK>(P, s)
                                                    : launch_integrate_pixels_t<GF_MODEL_POWER_LAW_ELLIPSOID>(P, s);
    if (e != cudaSuccess) return e;
    double2 *part = tot + P.njobs;
    job_totals_kernel<<<dim3(GF_TOTAL_PARTS, P.njobs), 256, 0, s>>>(P.pix_sum, P.pix_off, P.splits, P.total_pix, P.plans, part);
    sum_totals_kernel<<<(P.njobs + 7) / 8, 256, 0, s>>>(part, P.njobs, tot);
    count_launches(2);
    return cudaGetLastError();
}

size_t integ_totals(int njobs) { return (size_t)njobs * (1 + GF_TOTAL_PARTS); }

cudaError_t launch_pixel_counts(const IntegPixParams &P, double *out, cudaStream_t s)
{
    pixel_counts_kernel<<<(P.total_pix + 255) / 256, 256, 0, s>>>(P.pix_sum, P.splits, P.total_pix, out);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace gfk
