// gkm_core.cu -- packing, self-kernels, the ballot/popc pair join, the l-mer
// table, ISM's mutant self-kernels and the dense FP64 epilogues.
//
// Mismatch counts are accumulated as integers: per-lane 16-bit fields of a
// uint64 (four mismatch levels per word, gkm_shl64 drops levels past the
// word), flushed into uint64 totals before a field can overflow.  The FP64
// weighting sum_m h(m) n_m happens once per (row, column).
#include <cuda_runtime.h>
#include <stdint.h>

#include <cooperative_groups.h>

#include <type_traits>

#include "gkm_common.cuh"

namespace {

constexpr int SELF_THREADS = 256;
constexpr int SMEM_WINDOWS = 12288;  // rows staged in shared memory up to this

// staged-window capacity of a launch over rows of W window slots: the
// shared memory is sized to the rows, not to the limit, so short rows leave
// room for more blocks per SM
static int staged_windows(int64_t W) { return (int)(W < 1 ? 1 : W < SMEM_WINDOWS ? W : SMEM_WINDOWS); }

// ---------------------------------------------------------------------------
// Packing (kernels/packed.py:130-187)
// ---------------------------------------------------------------------------

constexpr int PACK_THREADS = 256, PACK_WINDOWS = 4 * PACK_THREADS;

// Rows of at least this many windows take blocks of their own (pack_rows), shorter ones
// a thread per window: calls over 4M bases in rows of 20 / 100 / 200 / 300 / 1,000 take
// 38 / 49 / 51 / 50 / 51 us so, and 290 / 80 / 55 / 46 / 35 with a block a row.
constexpr int PACK_ROW = 256;

__global__ void pack_kernel(const uint8_t *__restrict__ codes, const int64_t *__restrict__ lengths,
                            int64_t B, int64_t L, int l, uint32_t *__restrict__ fwd,
                            uint32_t *__restrict__ rc, int32_t *__restrict__ counts)
{
    int64_t W = L - l + 1;
    int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= B * W) return;
    int64_t b = idx / W, i = idx - b * W;
    int64_t n = W;
    if (lengths) {
        n = lengths[b] - l + 1;
        n = n < 0 ? 0 : (n > W ? W : n);
    }
    if (i == 0 && counts) counts[b] = (int32_t)n;
    uint32_t w = GKM_PAD;
    if (i < n) {
        const uint8_t *c = codes + b * L + i;
        w = 0;
        for (int k = 0; k < l; k++) w |= ((uint32_t)(c[k] & 3u)) << (2 * k);
    }
    fwd[idx] = w;
    if (rc) rc[b * W + (W - 1 - i)] = w == GKM_PAD ? GKM_PAD : gkm_rc_word(w, l);
}

// PACK_WINDOWS windows of a row per block: its bases go to shared memory as two bits
// each, a window is then two words funnel-shifted.  Bound by the stores.  Measured
// 8,192 rows of 2,000 bases (50 .. 2,000 used): pack_kernel 86 us, this 40 us.
__global__ void __launch_bounds__(PACK_THREADS) pack_rows(
    const uint8_t *__restrict__ codes, const int64_t *__restrict__ lengths, int64_t L, int l, int64_t chunks,
    uint32_t *__restrict__ fwd, uint32_t *__restrict__ rc, int32_t *__restrict__ counts)
{
    __shared__ uint32_t bases[PACK_WINDOWS / 16 + 2];  // 16 a word, and those past the last window
    const int64_t W = L - l + 1, b = blockIdx.x / chunks, c0 = (blockIdx.x - b * chunks) * PACK_WINDOWS;
    int64_t n = W;
    if (lengths) {
        n = lengths[b] - l + 1;
        n = n < 0 ? 0 : (n > W ? W : n);
    }
    if (c0 == 0 && threadIdx.x == 0 && counts) counts[b] = (int32_t)n;
    if (c0 < n) {
        const uint8_t *c = codes + b * L;
        const int64_t end = n + l - 1;
        for (int k = threadIdx.x; k < PACK_WINDOWS / 4 + 8; k += PACK_THREADS) {
            const int64_t p = c0 + 4 * k;
            uint32_t v = 0;
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (p + j < end) v |= (c[p + j] & 3u) << (2 * j);
            ((uint8_t *)bases)[k] = (uint8_t)v;
        }
        __syncthreads();
    }
    const uint32_t mask = (1u << (2 * l)) - 1u;
#pragma unroll
    for (int k = 0; k < PACK_WINDOWS / PACK_THREADS; k++) {
        const int at = k * PACK_THREADS + threadIdx.x;
        const int64_t i = c0 + at;
        if (i >= W) break;
        const uint32_t w = i < n ? __funnelshift_r(bases[at >> 4], bases[(at >> 4) + 1], 2 * (at & 15)) & mask : GKM_PAD;
        fwd[b * W + i] = w;
        if (rc) rc[b * W + (W - 1 - i)] = w == GKM_PAD ? GKM_PAD : gkm_rc_word(w, l);
    }
}

// ---------------------------------------------------------------------------
// Pair counting
// ---------------------------------------------------------------------------

template <int NW>
struct Packed {
    uint64_t w[NW];
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int k = 0; k < NW; k++) w[k] = 0;
    }
    // add a (<= 16 bits) to level m's field; levels past 4*NW drop out
    __device__ __forceinline__ void add(uint32_t m, uint64_t a)
    {
#pragma unroll
        for (int k = 0; k < NW; k++) w[k] += gkm_shl64(a, 16u * (m - 4u * k));
    }
    // tot[m] += scale * field m
    __device__ __forceinline__ void flush(uint64_t *tot, uint64_t scale)
    {
#pragma unroll
        for (int k = 0; k < NW; k++) {
#pragma unroll
            for (int f = 0; f < 4; f++) tot[4 * k + f] += scale * ((w[k] >> (16 * f)) & 0xFFFFu);
            w[k] = 0;
        }
    }
};

// Row staged for the self-kernel: f[k] its forward windows, r[k] = rc(f[k]).
struct RowView {
    const uint32_t *f;   // forward windows (smem or global)
    const uint32_t *r;   // rc(f[k]) at k (smem), or the RC row read reversed
    int64_t W;           // row stride of the global RC row (reverse read)
    bool reversed;       // r is the global RC row: rc(f[k]) = r[W - 1 - k]
    __device__ __forceinline__ uint32_t rcf(int k) const { return reversed ? r[W - 1 - k] : r[k]; }
};

// Per-thread partial pair counts of one row against itself: forward x forward
// and forward x RC, each unordered pair once (j > i doubled, j == i once),
// kernels/direct.py:109-137.
template <int NW>
__device__ void self_pairs(const RowView rv, int n, bool has_rc, const uint8_t *wd, bool weighted,
                           uint64_t *tot)
{
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    Packed<NW> acc;
    acc.zero();
    for (int i = warp; i < n; i += nw) {
        uint32_t fi = rv.f[i];
        uint64_t wi = weighted ? gkm_wt(wd, n, i) : 1;
        int it = 0;
        for (int j = i + 1 + lane; j < n; j += 32) {
            uint64_t wj = weighted ? gkm_wt(wd, n, j) : 1;
            acc.add((uint32_t)gkm_mism(fi, rv.f[j]), wj);
            if (has_rc) acc.add((uint32_t)gkm_mism(fi, rv.rcf(j)), wj);
            if (++it == 128) {  // 2 * 255 * 128 < 2^16
                acc.flush(tot, 2 * wi);
                it = 0;
            }
        }
        acc.flush(tot, 2 * wi);
        if (lane == 0) {
            tot[0] += wi * wi;  // m(f_i, f_i) = 0
            if (has_rc) {
                int m = gkm_mism(fi, rv.rcf(i));
                if (m < 4 * NW) tot[m] += wi * wi;
            }
        }
    }
}

// Block reduction of per-thread level totals; result in sums[] (smem, all threads).
template <int NL>
__device__ void block_reduce_levels(uint64_t *tot, uint64_t *red, uint64_t *sums)
{
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int m = 0; m < NL; m++) {
        uint64_t v = tot[m];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(GKM_FULL, v, o);
        if (lane == 0) red[warp * NL + m] = v;
    }
    __syncthreads();
    if (threadIdx.x < NL) {
        uint64_t s = 0;
        for (int w = 0; w < nw; w++) s += red[w * NL + threadIdx.x];
        sums[threadIdx.x] = s;
    }
    __syncthreads();
}

// Mismatches of 32 neighbouring window pairs at once, bit-sliced: bit p of plane
// k is bit k of the mismatches of the windows at p, given e (bit p: the bases at p
// differ) and the word after it.  The L shifted copies of e are summed by carry-
// save adders (a full adder is two logic operations).  L = 0: run-time length l.
struct Planes {
    uint32_t v[4];
};

template <int L>
__device__ __forceinline__ Planes mismatch_planes(uint32_t e, uint32_t en, int l)
{
    Planes r;
    if constexpr (L == 0) {
        r.v[0] = r.v[1] = r.v[2] = r.v[3] = 0;
        for (int k = 0; k < l; k++) {
            uint32_t c = __funnelshift_r(e, en, k);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint32_t x = r.v[j] & c;
                r.v[j] ^= c;
                c = x;
            }
        }
    } else {
        uint32_t a[4][L];
        int n[4] = {L, 0, 0, 0};
#pragma unroll
        for (int k = 0; k < L; k++) a[0][k] = k ? __funnelshift_r(e, en, k) : e;
#pragma unroll
        for (int j = 0; j < 4; j++) {
#pragma unroll
            for (int k = 0; k < L; k++) {  // at most L adders a plane
                if (n[j] >= 3) {
                    const uint32_t x = a[j][n[j] - 1], y = a[j][n[j] - 2], z = a[j][n[j] - 3];
                    if (j < 3) a[j + 1][n[j + 1]++] = (x & y) | (x & z) | (y & z);
                    n[j] -= 2;
                    a[j][n[j] - 1] = x ^ y ^ z;
                } else if (n[j] == 2) {
                    const uint32_t x = a[j][1], y = a[j][0];
                    if (j < 3) a[j + 1][n[j + 1]++] = x & y;
                    n[j] = 1;
                    a[j][0] = x ^ y;
                }
            }
            r.v[j] = n[j] ? a[j][0] : 0u;
        }
    }
    return r;
}

// bits of `valid` whose pair has m mismatches
__device__ __forceinline__ uint32_t level_mask(const Planes &p, int m, uint32_t valid)
{
    return valid & (m & 1 ? p.v[0] : ~p.v[0]) & (m & 2 ? p.v[1] : ~p.v[1]) & (m & 4 ? p.v[2] : ~p.v[2]) &
           (m & 8 ? p.v[3] : ~p.v[3]);
}

// A row's bases as bit planes: x (forward) and y (reverse complement), two words
// per 32 bases each, zero past the row.  Returns whether the packed windows are
// not those of one sequence (all threads).
__device__ __forceinline__ bool stage_planes(const uint32_t *frow, int n, int l, uint32_t *pl, int pw)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5, nb = n + l - 1;
    const uint32_t low = (1u << (2 * (l - 1))) - 1u;
    bool bad = false;
    auto base = [&](int p) -> uint32_t {
        return p < n ? frow[p] & 3u : (frow[n - 1] >> (2 * (p - n + 1))) & 3u;
    };
    for (int k = warp; k < pw; k += nw) {
        const int p = k * 32 + lane;
        const uint32_t x = n > 0 && p < nb ? base(p) : 0u, y = n > 0 && p < nb ? 3u - base(nb - 1 - p) : 0u;
        if (p + 1 < n) bad |= (frow[p + 1] & low) != (frow[p] >> 2);
        const uint32_t x0 = __ballot_sync(GKM_FULL, x & 1u), x1 = __ballot_sync(GKM_FULL, x & 2u);
        const uint32_t y0 = __ballot_sync(GKM_FULL, y & 1u), y1 = __ballot_sync(GKM_FULL, y & 2u);
        if (lane == 0) {
            pl[k] = x0;
            pl[pw + k] = x1;
            pl[2 * pw + k] = y0;
            pl[3 * pw + k] = y1;
        }
    }
    return __syncthreads_or(bad);
}

constexpr int SELF_PLANES = 200 * 1024;  // the most shared memory for a row's planes

// bit plane words of a row of W windows: the bases and three words past them
__host__ __device__ inline int plane_words(int64_t W, int l) { return (int)((W + l - 1 + 31) / 32) + 3; }

// What both forms do with a row's level sums (tot of every thread).
template <int NL>
__device__ __forceinline__ void self_finish(const gkm_spec spec, uint64_t *tot, uint64_t *red, uint64_t *sums, double *dred, int64_t b,
                            int n, const uint32_t *frow, double *diag, uint64_t *profile, const double *table, double bias,
                            int normalize, double *scores, double *raw_out)
{
    block_reduce_levels<NL>(tot, red, sums);
    double k = 0.0;
#pragma unroll
    for (int m = 0; m < NL; m++)
        if (m <= spec.dmax) k += spec.h[m] * (double)sums[m];
    if (threadIdx.x == 0) {
        if (diag) diag[b] = k;
        if (profile)
            for (int m = 0; m <= spec.l; m++)
                profile[b * (spec.l + 1) + m] = (m < NL && m <= spec.dmax) ? sums[m] : 0;
    }
    if (table) {
        double t = 0.0;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            double a = spec.weighted ? (double)gkm_wt(spec.wd, n, i) : 1.0;
            t += a * table[frow[i]];
        }
        t = gkm_block_sum(t, dred);
        if (threadIdx.x == 0) {
            if (raw_out) raw_out[b] = t;
            double s = normalize ? t / sqrt(fmax(k, 1e-10)) : t;
            scores[b] = s + bias;
        }
    }
}

// Self-kernel of one row per block, optionally fused with the l-mer table sum
// (svm.py:559-582: score = sum_i wt_i table[x_i] / sqrt(K(x, x)) + b).
//
// A pair of windows (i, i + s) compares the same positions as its neighbour on
// the diagonal, shifted by one: along a diagonal the mismatches are a sliding sum
// of the bits "bases p and p + s differ", which 32 pairs at a time take ~50
// operations (a pair alone took 11 and a quarter-rate population count).  Forward x
// RC pairs are the diagonals of the sequence against its reverse complement, each
// symmetric about its middle: half of it is summed.  Bound by the integer pipe;
// measured fused with the table sum (t=2): 8,192 rows of 50 .. 2,000 bp 4,516 us
// pair by pair -> 633 us, 512 rows of 1,000 bp 544 -> 71 us.  Rows whose windows do not
// overlap (not one sequence's) or whose planes do not fit shared memory are still taken
// pair by pair.
template <int L, int NL, bool WT>
__global__ void __launch_bounds__(SELF_THREADS) self_kernel(
    gkm_spec spec, const uint32_t *__restrict__ fwd, const uint32_t *__restrict__ rc,
    const int32_t *__restrict__ counts, int64_t W, double *__restrict__ diag,
    uint64_t *__restrict__ profile, const double *__restrict__ table, double bias, int normalize,
    double *__restrict__ scores, double *__restrict__ raw_out, int pw)
{
    extern __shared__ uint32_t pl[];  // x0, x1, y0, y1, pw words each
    __shared__ uint64_t red[(SELF_THREADS / 32) * NL];
    __shared__ uint64_t sums[NL];
    __shared__ double dred[32];
    int64_t b = blockIdx.x;
    const int n = counts[b], l = L ? L : spec.l;
    const bool has_rc = spec.include_rc && rc != nullptr;
    const uint32_t *frow = fwd + b * W;
    const uint8_t *wd = spec.wd;
    uint64_t tot[NL];
#pragma unroll
    for (int m = 0; m < NL; m++) tot[m] = 0;
    if (pw == 0 || stage_planes(frow, n, l, pl, pw)) {
        RowView rv;
        rv.f = frow;
        rv.r = has_rc ? rc + b * W : nullptr;
        rv.W = W;
        rv.reversed = true;
        self_pairs<NL / 4>(rv, n, has_rc, wd, WT, tot);
    } else {
        uint32_t cnt[NL], mid[NL];
#pragma unroll
        for (int m = 0; m < NL; m++) cnt[m] = mid[m] = 0;
        // diagonal s of x against x (0), x against y (1) and y against x (2)
        for (int t = threadIdx.x; t < (has_rc ? 3 * n : n); t += SELF_THREADS) {
            const int mode = t >= 2 * n ? 2 : t >= n ? 1 : 0, s = t - mode * n, len = n - s;
            if (s == 0 && mode != 1) continue;  // mode 0: a window with itself, below; mode 2: mode 1's
            const int H = mode ? (len + 1) >> 1 : len;
            const bool odd = mode && (len & 1);  // the last of the half is its own mirror image
            const uint32_t *P = pl + (mode == 2 ? 2 * pw : 0), *Q = pl + (mode == 1 ? 2 * pw : 0) + (s >> 5);
            uint32_t q0 = Q[0], q1 = Q[pw];
            auto differ = [&](int w) -> uint32_t {  // words in turn
                const uint32_t n0 = Q[w + 1], n1 = Q[pw + w + 1];
                const uint32_t e = (P[w] ^ __funnelshift_r(q0, n0, s)) | (P[pw + w] ^ __funnelshift_r(q1, n1, s));
                q0 = n0;
                q1 = n1;
                return e;
            };
            uint32_t e = differ(0);
            const int nw = (H + 31) >> 5;
            for (int w = 0; w < nw; w++) {
                const uint32_t en = differ(w + 1);
                const Planes pn = mismatch_planes<L>(e, en, l);
                const bool last = w == nw - 1;
                const uint32_t valid = last && (H & 31) ? (1u << (H & 31)) - 1u : GKM_FULL;
                e = en;
                uint32_t near = valid;
                if (NL == 4) near &= ~pn.v[2] & ~pn.v[3];
                if (WT) {
#pragma unroll
                    for (int m = 0; m < NL; m++) {
                        if (m > spec.dmax) break;
                        for (uint32_t h = level_mask(pn, m, near); h; h &= h - 1) {
                            const int i = w * 32 + __ffs(h) - 1;
                            // windows i and i + s; an RC window has its forward window's weight
                            const int j = mode ? n - 1 - (i + s) : i + s, i2 = mode == 2 ? n - 1 - i : i,
                                      j2 = mode == 2 ? i + s : j;
                            tot[m] += (odd && i == H - 1 ? 1ull : 2ull) * gkm_wt(wd, n, i2) * gkm_wt(wd, n, j2);
                        }
                    }
                } else {
#pragma unroll
                    for (int m = 0; m < NL; m++) {
                        const uint32_t h = level_mask(pn, m, near);
                        cnt[m] += __popc(h);
                        if (last && odd) mid[m] += (h >> ((H - 1) & 31)) & 1u;
                    }
                }
            }
        }
        if (WT) {
            for (int i = threadIdx.x; i < n; i += SELF_THREADS) {
                const uint64_t w = gkm_wt(wd, n, i);
                tot[0] += w * w;
            }
        } else {
#pragma unroll
            for (int m = 0; m < NL; m++) tot[m] = 2ull * cnt[m] - mid[m];
            if (threadIdx.x == 0) tot[0] += n;
        }
    }
    self_finish<NL>(spec, tot, red, sums, dred, b, n, frow, diag, profile, table, bias, normalize, scores, raw_out);
}

// The same pair by pair, for weighted kernels whose pairs mostly count (pairs_pay): there
// the diagonals above take every counted pair one by one, with 64-bit sums, and this does
// so with less work a pair.
template <int NW>
__global__ void __launch_bounds__(SELF_THREADS) self_pairs_kernel(
    gkm_spec spec, const uint32_t *__restrict__ fwd, const uint32_t *__restrict__ rc,
    const int32_t *__restrict__ counts, int64_t W, double *__restrict__ diag,
    uint64_t *__restrict__ profile, const double *__restrict__ table, double bias, int normalize,
    double *__restrict__ scores, double *__restrict__ raw_out, int sw)
{
    constexpr int NL = 4 * NW;
    extern __shared__ uint32_t sm[];  // the row's forward and RC windows, sw words each
    __shared__ uint64_t red[(SELF_THREADS / 32) * NL];
    __shared__ uint64_t sums[NL];
    __shared__ double dred[32];
    const int64_t b = blockIdx.x;
    const int n = counts[b];
    const bool has_rc = spec.include_rc && rc != nullptr;
    const uint32_t *frow = fwd + b * W, *rrow = has_rc ? rc + b * W : nullptr;
    RowView rv = {frow, rrow, W, true};
    if (n <= sw) {
        for (int k = threadIdx.x; k < n; k += SELF_THREADS) {
            sm[k] = frow[k];
            if (has_rc) sm[sw + k] = rrow[W - 1 - k];
        }
        rv.f = sm;
        rv.r = sm + sw;
        rv.reversed = false;
    }
    __syncthreads();
    uint64_t tot[NL];
#pragma unroll
    for (int m = 0; m < NL; m++) tot[m] = 0;
    self_pairs<NW>(rv, n, has_rc, spec.wd, spec.weighted, tot);
    self_finish<NL>(spec, tot, red, sums, dred, b, n, frow, diag, profile, table, bias, normalize, scores, raw_out);
}

// ---------------------------------------------------------------------------
// Pair join by warp ballot/popc: K_raw[b, s] over every window pair
// ---------------------------------------------------------------------------

constexpr int JOIN_WARPS = 8;
constexpr int JOIN_WINDOWS = 56000;  // the longest query row (in shared memory)

template <int NW>
__global__ void __launch_bounds__(JOIN_WARPS * 32) join_kernel(
    gkm_spec spec, const uint32_t *__restrict__ bx, const int32_t *__restrict__ cx, int64_t Wx,
    const uint32_t *__restrict__ by, const uint32_t *__restrict__ ry, const int32_t *__restrict__ cy,
    int64_t S, int64_t Wy, double *__restrict__ raw, uint64_t *__restrict__ profile)
{
    constexpr int NL = 4 * NW;
    extern __shared__ uint32_t xs[];  // query row windows
    int64_t b = blockIdx.x;
    int nx = cx[b];
    for (int i = threadIdx.x; i < nx; i += blockDim.x) xs[i] = bx[b * Wx + i];
    __syncthreads();
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t s = (int64_t)blockIdx.y * JOIN_WARPS + warp;
    if (s >= S) return;
    int ny = cy[s];
    bool has_rc = spec.include_rc && ry != nullptr;
    int nt = has_rc ? 2 * ny : ny;
    const int dmax = spec.dmax;
    uint64_t tot[NL];
#pragma unroll
    for (int m = 0; m < NL; m++) tot[m] = 0;
    for (int c0 = 0; c0 < nt; c0 += 32) {
        int t = c0 + lane;
        uint32_t y = GKM_PAD;
        uint64_t wy = 1;
        if (t < nt) {
            if (t < ny) {
                y = by[s * Wy + t];
                if (spec.weighted) wy = gkm_wt(spec.wd, ny, t);
            } else {  // RC window of forward window ny - 1 - (t - ny)
                int f = ny - 1 - (t - ny);
                y = ry[s * Wy + (Wy - 1 - f)];
                if (spec.weighted) wy = gkm_wt(spec.wd, ny, f);
            }
        }
        Packed<NW> acc;
        acc.zero();
        int hits = 0;
        for (int i = 0; i < nx; i++) {
            int m = y == GKM_PAD ? 99 : gkm_mism(xs[i], y);
            if (__ballot_sync(GKM_FULL, m <= dmax)) {
                if (spec.weighted) {
                    if (m <= dmax) acc.add((uint32_t)m, gkm_wt(spec.wd, nx, i));
                    if (++hits == 256) {  // 255 * 256 < 2^16
                        acc.flush(tot, wy);
                        hits = 0;
                    }
                } else {
#pragma unroll
                    for (int lev = 0; lev < NL; lev++)
                        if (lev <= dmax) tot[lev] += __popc(__ballot_sync(GKM_FULL, m == lev));
                }
            }
        }
        if (spec.weighted) acc.flush(tot, wy);
    }
    if (spec.weighted) {
#pragma unroll
        for (int m = 0; m < NL; m++)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) tot[m] += __shfl_xor_sync(GKM_FULL, tot[m], o);
    }
    if (lane == 0) {
        double k = 0.0;
#pragma unroll
        for (int m = 0; m < NL; m++)
            if (m <= dmax) k += spec.h[m] * (double)tot[m];
        if (raw) raw[b * S + s] = k;
        if (profile)
            for (int m = 0; m <= spec.l; m++)
                profile[(b * S + s) * (spec.l + 1) + m] = (m < NL && m <= dmax) ? tot[m] : 0;
    }
}

// ---------------------------------------------------------------------------
// l-mer table (lmer_table.py:58-98): table[u] = sum_t h(level_t) V[u ^ mask_t]
// ---------------------------------------------------------------------------

__global__ void lmer_table_kernel(gkm_spec spec, const double *__restrict__ V,
                                  const uint32_t *__restrict__ masks, int n_masks,
                                  double *__restrict__ table, int64_t n_lmers)
{
    __shared__ double hs[16];
    if (threadIdx.x < 16) hs[threadIdx.x] = threadIdx.x <= spec.l ? spec.h[threadIdx.x] : 0.0;
    __syncthreads();
    int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= n_lmers) return;
    double acc = 0.0;
    for (int t = 0; t < n_masks; t++) {
        uint32_t mk = __ldg(masks + t);
        double v = __ldg(V + ((uint32_t)u ^ (mk & 0x00FFFFFFu)));
        acc += hs[mk >> 24] * v;
    }
    table[u] = acc;
}

// ---------------------------------------------------------------------------
// ISM: mutant self-kernels and table deltas (ism.py:118-144, 254-320;
// kernels/direct.py:160-201)
// ---------------------------------------------------------------------------

constexpr int MUT_THREADS = 128;

// Per (position p, row b): for each substituted base v the change in pair
// counts of the row's self-kernel, from the pairs touching the windows A that
// cover p.  Pairs (i in A, j not in A) stand for both orders (x2); pairs inside
// A are counted once per order.  The reference base gives new == old, so its
// change is exactly 0.
template <int NW>
__global__ void __launch_bounds__(MUT_THREADS) mutant_kernel(
    gkm_spec spec, const uint32_t *__restrict__ fwd, const int32_t *__restrict__ counts, int64_t B,
    int64_t W, int64_t L, const double *__restrict__ diag, double *__restrict__ mut_diag,
    const double *__restrict__ table, const double *__restrict__ ref_raw, int normalize,
    double *__restrict__ ism_out, int sw)
{
    constexpr int NL = 4 * NW;
    // the pair counts with base v at p, v = 0..3; the reference base's are
    // the row's own (its substitution changes nothing), so they serve as "old"
    constexpr int NA = 4;
    extern __shared__ uint32_t sm[];
    __shared__ uint64_t red[(MUT_THREADS / 32) * NA * NL];
    __shared__ uint64_t sums[NA * NL];
    int64_t p = blockIdx.x, b = blockIdx.y;
    int n = counts[b];
    int l = spec.l;
    int a_s = (int)(p - l + 1 > 0 ? p - l + 1 : 0);
    int a_e = (int)(p + 1 < n ? p + 1 : n);
    double d0 = diag ? diag[b] : 0.0;
    if (a_s >= a_e) {  // p past the row's windows: nothing changes
        if (threadIdx.x < 4) {
            if (mut_diag) mut_diag[(threadIdx.x * L + p) * B + b] = d0;
            if (ism_out) ism_out[(b * 4 + threadIdx.x) * L + p] = 0.0;
        }
        return;
    }
    bool has_rc = spec.include_rc != 0;
    const uint32_t *frow = fwd + b * W;
    uint32_t *f = sm;  // [n] forward, [n] rc(f)
    bool in_smem = n <= sw;
    if (in_smem) {
        for (int k = threadIdx.x; k < n; k += blockDim.x) {
            uint32_t w = frow[k];
            f[k] = w;
            f[sw + k] = gkm_rc_word(w, l);
        }
        __syncthreads();
    }
    const uint32_t *F = in_smem ? f : frow;
    const int na = a_e - a_s;
    const int xp = (int)((F[a_s] >> (2 * (p - a_s))) & 3u);  // the row's base at p
    const uint8_t *wd = spec.wd;
    const bool wt = spec.weighted != 0;
    uint64_t tot[NA][NL];
#pragma unroll
    for (int a = 0; a < NA; a++)
#pragma unroll
        for (int m = 0; m < NL; m++) tot[a][m] = 0;
    if (diag || mut_diag) {
        for (int j = threadIdx.x; j < n; j += blockDim.x) {
            uint32_t fj = F[j];
            uint32_t rj = in_smem ? f[sw + j] : gkm_rc_word(fj, l);
            bool jin = j >= a_s && j < a_e;
            uint64_t wj = wt ? gkm_wt(wd, n, j) : 1;
            Packed<NW> acc[NA];
#pragma unroll
            for (int a = 0; a < NA; a++) acc[a].zero();
            for (int ii = 0; ii < na; ii++) {
                int i = a_s + ii;
                uint32_t fi = F[i];
                uint64_t wi = wt ? gkm_wt(wd, n, i) : 1;
                uint32_t sh = 2u * (uint32_t)(p - i);
                if (!jin) {
                    // only window i changes: its mismatches with j away from
                    // offset k = p - i, plus one where j's base at k is not v
                    const uint32_t keep = ~(1u << sh);
                    uint32_t x = fi ^ fj;
                    const uint32_t mf = (uint32_t)__popc((x | (x >> 1)) & 0x55555555u & keep);
                    const uint32_t bf = (fj >> sh) & 3u;
                    x = fi ^ rj;
                    const uint32_t mr = (uint32_t)__popc((x | (x >> 1)) & 0x55555555u & keep);
                    const uint32_t br = (rj >> sh) & 3u;
#pragma unroll
                    for (int v = 0; v < 4; v++) {
                        acc[v].add(mf + (bf != (uint32_t)v), wi);
                        if (has_rc) acc[v].add(mr + (br != (uint32_t)v), wi);
                    }
                    continue;
                }
                uint32_t cleared = fi & ~(3u << sh);
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    uint32_t fn = cleared | ((uint32_t)v << sh);
                    // both windows change
                    const uint32_t shj = 2u * (uint32_t)(p - j);
                    const uint32_t gj = (fj & ~(3u << shj)) | ((uint32_t)v << shj);
                    const uint32_t grj = gkm_rc_word(gj, l);
                    acc[v].add((uint32_t)gkm_mism(fn, gj), wi);
                    if (has_rc) acc[v].add((uint32_t)gkm_mism(fn, grj), wi);
                }
            }
            uint64_t scale = (jin ? 1 : 2) * wj;  // 2 * 11 * 255 < 2^16
#pragma unroll
            for (int a = 0; a < NA; a++) acc[a].flush(tot[a], scale);
        }
        // block reduction of the NA * NL totals
        int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
        for (int a = 0; a < NA; a++)
#pragma unroll
            for (int m = 0; m < NL; m++) {
                uint64_t v = tot[a][m];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(GKM_FULL, v, o);
                if (lane == 0) red[(warp * NA + a) * NL + m] = v;
            }
        __syncthreads();
        for (int k = threadIdx.x; k < NA * NL; k += blockDim.x) {
            uint64_t s = 0;
            for (int w = 0; w < nw; w++) s += red[w * NA * NL + k];
            sums[k] = s;
        }
        __syncthreads();
    }
    if (threadIdx.x < 4) {
        int v = threadIdx.x;
        double md = d0;
        if (diag || mut_diag) {
            double delta = 0.0;
            for (int m = 0; m < NL && m <= spec.dmax; m++) {
                int64_t dn = (int64_t)(sums[v * NL + m] - sums[xp * NL + m]);
                delta += spec.h[m] * (double)dn;
            }
            md = d0 + delta;
            if (mut_diag) mut_diag[((int64_t)v * L + p) * B + b] = md;
        }
        if (ism_out) {
            double r = ref_raw[b];
            double dt = 0.0;
            for (int i = a_s; i < a_e; i++) {
                uint32_t fi = F[i];
                uint32_t sh = 2u * (uint32_t)(p - i);
                uint32_t fn = (fi & ~(3u << sh)) | ((uint32_t)v << sh);
                double a = wt ? (double)gkm_wt(wd, n, i) : 1.0;
                dt += a * (table[fn] - table[fi]);
            }
            double kn = r + dt;
            double out;
            if (normalize)
                out = kn / sqrt(fmax(md, 1e-10)) - r / sqrt(fmax(d0, 1e-10));
            else
                out = kn - r;
            ism_out[(b * 4 + v) * L + p] = out;
        }
    }
}

// The same for kernels of at most four levels, by bit-sliced diagonals: a block
// takes MT_WINDOWS - l + 1 positions of a row and the windows that cover them.  Only
// pairs within dmax + 1 mismatches can count after a substitution (~1 % of them), so
// those are found 32 pairs at a time as in self_kernel -- every diagonal of the
// tile's windows against the row and against its reverse complement -- queued per
// warp and taken one per lane: the pair's l positions add to the counts of (position,
// base, level).  Pairs whose second window covers the position, too, are the l x l
// ones about it and are tested directly.  Bound by the integer pipe (52 %) and by how few
// warps there are (27 %).  Measured (t=2,
// 128 x 300 bp): mutant_kernel, every pair at every position, 685 us; this 76 us.
// mutant_kernel stays for d >= 4, for rows whose planes outgrow shared memory and where
// it is the faster form (tiles_pay).
constexpr int MT_THREADS = 256;
constexpr int MT_WINDOWS = 128;
constexpr int MT_PLANES = 128 * 1024;  // the most shared memory for a row's planes

// words of one plane: pw zeros, the row's pw, and what the last windows' partners
// read past them (a tile's words and two more)
__host__ __device__ inline int mutant_plane(int pw) { return 2 * pw + MT_WINDOWS / 32 + 4; }

template <int L, bool WT>
__global__ void __launch_bounds__(MT_THREADS) mutant_tiles(
    gkm_spec spec, const uint32_t *__restrict__ fwd, const int32_t *__restrict__ counts, int64_t B,
    int64_t W, int64_t len, const double *__restrict__ diag, double *__restrict__ mut_diag,
    const double *__restrict__ table, const double *__restrict__ ref_raw, int normalize,
    double *__restrict__ ism_out, int pw)
{
    typedef typename std::conditional<WT, unsigned long long, uint32_t>::type Acc;
    // x0, x1, y0, y1: pw words of zeros, then the row's (and zeros past it)
    extern __shared__ uint32_t pl[];
    const int ps = mutant_plane(pw);
    __shared__ Acc acc[MT_WINDOWS][4][4];  // position, base, level
    __shared__ uint32_t queue[MT_THREADS / 32][64];
    const int l = L ? L : spec.l, P = MT_WINDOWS - l + 1, D = spec.dmax;
    const int64_t b = blockIdx.y;
    const int n = counts[b], p0 = (int)(blockIdx.x * P), np = (int)min((int64_t)P, len - p0);
    const int i0 = max(0, p0 - l + 1), i1 = min(n, p0 + np);  // the windows that cover the tile's positions
    const double d0 = diag ? diag[b] : 0.0;
    if (i0 >= i1) {  // past the row's windows: nothing changes
        for (int t = threadIdx.x; t < 4 * np; t += MT_THREADS) {
            const int v = t / np, p = p0 + t - v * np;
            if (mut_diag) mut_diag[((int64_t)v * len + p) * B + b] = d0;
            if (ism_out) ism_out[(b * 4 + v) * len + p] = 0.0;
        }
        return;
    }
    const uint32_t *F = fwd + b * W;
    const bool has_rc = spec.include_rc != 0;
    const uint8_t *wd = spec.wd;
    for (int t = threadIdx.x; t < MT_WINDOWS * 16; t += MT_THREADS) (&acc[0][0][0])[t] = 0;
    if (diag || mut_diag) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        for (int t = threadIdx.x; t < 4 * pw; t += MT_THREADS) pl[(t / pw) * ps + t % pw] = 0;
        {
            const int nb = n + l - 1;
            auto base = [&](int p) -> uint32_t { return p < n ? F[p] & 3u : (F[n - 1] >> (2 * (p - n + 1))) & 3u; };
            for (int k = warp; k < ps - pw; k += MT_THREADS / 32) {
                const int p = k * 32 + lane;
                const uint32_t x = p < nb ? base(p) : 0u, y = p < nb ? 3u - base(nb - 1 - p) : 0u;
                const uint32_t x0 = __ballot_sync(GKM_FULL, x & 1u), x1 = __ballot_sync(GKM_FULL, x & 2u);
                const uint32_t y0 = __ballot_sync(GKM_FULL, y & 1u), y1 = __ballot_sync(GKM_FULL, y & 2u);
                if (lane == 0) {
                    pl[pw + k] = x0;
                    pl[ps + pw + k] = x1;
                    pl[2 * ps + pw + k] = y0;
                    pl[3 * ps + pw + k] = y1;
                }
            }
        }
        __syncthreads();
        int nq = 0;  // queued pairs of this warp: window - i0 | RC << 8 | other window << 9
        auto take = [&](int c) {
            __syncwarp();
            if (lane < c) {
                const uint32_t e = queue[warp][lane];
                const int i = i0 + (int)(e & 0xFFu), j = (int)(e >> 9);
                const uint32_t fi = F[i], g = (e >> 8) & 1u ? gkm_rc_word(F[j], l) : F[j];
                const uint32_t x = fi ^ g, differ = (x | (x >> 1)) & 0x55555555u;
                const int m = __popc(differ);
                const Acc w = WT ? (Acc)2 * gkm_wt(wd, n, i) * gkm_wt(wd, n, j) : (Acc)2;
                for (int k = 0; k < l; k++) {
                    const int p = i + k - p0, me = m - (int)((differ >> (2 * k)) & 1u);
                    // me: mismatches away from p; a position j covers, too, is left to the pairs below
                    if (me > D || p < 0 || p >= np || (unsigned)(i + k - j) < (unsigned)l) continue;
                    const uint32_t same = (g >> (2 * k)) & 3u;
                    atomicAdd(&acc[p][same][me], w);
                    if (me < D)
#pragma unroll
                        for (uint32_t v = 0; v < 4; v++)
                            if (v != same) atomicAdd(&acc[p][v][me + 1], w);
                }
            }
            __syncwarp();
            if (c == 32 && lane < nq - 32) queue[warp][lane] = queue[warp][32 + lane];
            __syncwarp();
            nq -= c;
        };
        // diagonals: shift s of the row (strand 0) and of its reverse complement (1)
        const int nd = 2 * n - 1, nt = has_rc ? 2 * nd : nd, nwd = (i1 - i0 + 31) >> 5;
        for (int t0 = 0; t0 < nt; t0 += MT_THREADS) {
            const int t = t0 + threadIdx.x, st = t >= nd, s = t - st * nd - (n - 1);
            // windows whose partner is one of the row's
            const int lo = max(i0, -s), hi = min(i1, n - s);
            const bool live = t < nt && (st || s != 0) && lo < hi;
            // bit of the first window's partner, after the zeros: within n - 1 before
            // and MT_WINDOWS after the row's bits
            const int at = live ? pw * 32 + i0 + s : pw * 32;
            const uint32_t *X = pl + pw + (i0 >> 5), *Q = pl + (live && st ? 2 * ps : 0) + (at >> 5);
            auto differ = [&](int w) -> uint32_t {
                const uint32_t x0 = __funnelshift_r(X[w], X[w + 1], i0), x1 = __funnelshift_r(X[ps + w], X[ps + w + 1], i0);
                const uint32_t q0 = __funnelshift_r(Q[w], Q[w + 1], at), q1 = __funnelshift_r(Q[ps + w], Q[ps + w + 1], at);
                return (x0 ^ q0) | (x1 ^ q1);
            };
            uint32_t e = differ(0);
            for (int w = 0; w < nwd; w++) {
                const uint32_t en = differ(w + 1);
                const Planes pn = mismatch_planes<L>(e, en, l);
                e = en;
                const int a0 = max(lo - i0 - 32 * w, 0), a1 = min(hi - i0 - 32 * w, 32);
                uint32_t h = live && a1 > a0 ? (a1 < 32 ? (1u << a1) - 1u : GKM_FULL) & ~((1u << a0) - 1u) : 0u;
                // at most D + 1 <= 4 mismatches
                uint32_t near = ~pn.v[3] & (~pn.v[2] | (~pn.v[0] & ~pn.v[1]));  // <= 4
                if (D < 3) near &= ~pn.v[2] & (D == 2 ? GKM_FULL : D == 1 ? ~(pn.v[0] & pn.v[1]) : ~pn.v[1]);
                h &= near;
                while (__any_sync(GKM_FULL, h != 0)) {
                    const uint32_t who = __ballot_sync(GKM_FULL, h != 0);
                    if (h) {
                        const int i = 32 * w + __ffs(h) - 1, q = i0 + i + s, j = st ? n - 1 - q : q;
                        queue[warp][nq + __popc(who & ((1u << lane) - 1u))] = (uint32_t)i | (uint32_t)st << 8 | (uint32_t)j << 9;
                        h &= h - 1;
                    }
                    nq += __popc(who);
                    if (nq >= 32) take(32);
                }
            }
        }
        if (nq) take(nq);
        __syncthreads();
        // both windows cover the position: windows a_s .. a_e - 1, unordered pairs
        // twice (a window with itself has no mismatch whatever the base)
        for (int t = threadIdx.x; t < 4 * np; t += MT_THREADS) {
            const int v = t & 3, p = p0 + (t >> 2), as = max(0, p - l + 1), ae = min(n, p + 1);
            for (int i = as; i < ae; i++) {
                const uint32_t sh = 2u * (uint32_t)(p - i), fi = (F[i] & ~(3u << sh)) | (uint32_t)v << sh;
                const uint32_t wi = WT ? gkm_wt(wd, n, i) : 1u;
                for (int j = i; j < ae; j++) {
                    const uint32_t shj = 2u * (uint32_t)(p - j), fj = (F[j] & ~(3u << shj)) | (uint32_t)v << shj;
                    const Acc w = (Acc)(i == j ? 1u : 2u) * wi * (WT ? gkm_wt(wd, n, j) : 1u);
                    const int mf = gkm_mism(fi, fj);
                    if (mf <= D) acc[p - p0][v][mf] += w;
                    if (has_rc) {
                        const int mr = gkm_mism(fi, gkm_rc_word(fj, l));
                        if (mr <= D) acc[p - p0][v][mr] += w;
                    }
                }
            }
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < 4 * np; t += MT_THREADS) {
        const int v = t / np, q = t - v * np, p = p0 + q;
        const int as = max(0, p - l + 1), ae = min(n, p + 1);
        const bool none = as >= ae;
        const int xp = none ? v : (int)((F[as] >> (2 * (p - as))) & 3u);  // the row's base at p
        double md = d0;
        if (diag || mut_diag) {
            double delta = 0.0;
            for (int m = 0; m < 4 && m <= D; m++)
                delta += spec.h[m] * (double)((int64_t)acc[q][v][m] - (int64_t)acc[q][xp][m]);
            md = d0 + delta;
            if (mut_diag) mut_diag[((int64_t)v * len + p) * B + b] = md;
        }
        if (ism_out) {
            double out = 0.0;
            if (!none) {
                const double r = ref_raw[b];
                double dt = 0.0;
                if (v != xp)
                    for (int i = as; i < ae; i++) {
                        const uint32_t fi = F[i], sh = 2u * (uint32_t)(p - i);
                        const uint32_t fn = (fi & ~(3u << sh)) | ((uint32_t)v << sh);
                        const double a = WT ? (double)gkm_wt(wd, n, i) : 1.0;
                        dt += a * (table[fn] - table[fi]);
                    }
                const double kn = r + dt;
                out = normalize ? kn / sqrt(fmax(md, 1e-10)) - r / sqrt(fmax(d0, 1e-10)) : kn - r;
            }
            ism_out[(b * 4 + v) * len + p] = out;
        }
    }
}

// ---------------------------------------------------------------------------
// Dense FP64 epilogues over materialised [rows, S] blocks
// ---------------------------------------------------------------------------

__global__ void raw_score_kernel(const double *__restrict__ raw, int64_t S, const double *__restrict__ dx,
                                 const double *__restrict__ ds, const double *__restrict__ coef,
                                 double gamma, int rbf, double bias, double *__restrict__ out)
{
    __shared__ double red[32];
    int64_t b = blockIdx.x;
    double acc = 0.0;
    for (int64_t s = threadIdx.x; s < S; s += blockDim.x) {
        double k = raw[b * S + s];
        if (dx) k /= fmax(sqrt(dx[b] * ds[s]), 1e-10);
        if (rbf) k = exp(gamma * (k - 1.0));
        acc += coef[s] * k;
    }
    acc = gkm_block_sum(acc, red);
    if (threadIdx.x == 0) out[b] = acc + bias;
}

// A cluster of blocks per row (a row a block left most SMs idle: 96 rows x 72,000 SVs
// 353 us, this 103 us); their sums meet in the first block's shared memory and are
// added in rank order.
constexpr int IMPACT_BLOCKS = 8;

__global__ void __cluster_dims__(IMPACT_BLOCKS, 1, 1) __launch_bounds__(256) impact_kernel(
    const double *__restrict__ raw, int64_t n, int64_t S, const double *__restrict__ dr, const double *__restrict__ ds,
    const double *__restrict__ coef, double gamma, int rbf, double *__restrict__ out)
{
    __shared__ double red[32], sums[IMPACT_BLOCKS];
    auto cluster = cooperative_groups::this_cluster();
    const unsigned rank = cluster.block_rank();
    cluster.sync();  // every block of the cluster runs before one writes to another
    const int64_t b = blockIdx.x / IMPACT_BLOCKS;
    double fl = rbf ? exp(-gamma) : 0.0;
    double acc = 0.0;
    for (int64_t s = rank * blockDim.x + threadIdx.x; s < S; s += IMPACT_BLOCKS * blockDim.x) {
        double k = raw[b * S + s];
        double dk = raw[(n + b) * S + s] - k;
        if (dr) {
            double z = fmax(sqrt(dr[b] * ds[s]), 1e-10);
            k /= z;
            dk /= z;
        }
        if (rbf) {
            if (k <= 0) continue;
            dk *= (exp(gamma * (k - 1.0)) - fl) / k;
        }
        acc += coef[s] * dk;
    }
    acc = gkm_block_sum(acc, red);
    if (threadIdx.x == 0) cluster.map_shared_rank(sums, 0)[rank] = acc;
    cluster.sync();
    if (rank == 0 && threadIdx.x == 0) {
        double t = 0.0;
        for (int k = 0; k < IMPACT_BLOCKS; k++) t += sums[k];
        out[b] = t;
    }
}

__global__ void gram_finish_kernel(const double *__restrict__ raw, int64_t N, int64_t M,
                                   const double *__restrict__ dx, const double *__restrict__ dy,
                                   double gamma, int rbf, int symmetric, double *__restrict__ out)
{
    int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= N * M) return;
    int64_t r = idx / M, c = idx - r * M;
    int64_t rr = r, cc = c;
    if (symmetric && c < r) {  // mirror the upper triangle exactly
        rr = c;
        cc = r;
    }
    double k = raw[rr * M + cc];
    if (dx) k /= fmax(sqrt(dx[rr] * dy[cc]), 1e-10);
    if (rbf) k = exp(gamma * (k - 1.0));
    out[idx] = k;
}

int nw_for(int dmax)
{
    return dmax < 4 ? 1 : (dmax < 8 ? 2 : 4);
}

int check_spec(const gkm_spec *spec)
{
    if (!spec) return gkm_fail(GKM_ERR_INVALID, "spec is null");
    if (spec->l < 1 || spec->l > GKM_MAX_L) return gkm_fail(GKM_ERR_INVALID, "l must be in 1..15, got %d", spec->l);
    if (spec->dmax < 0 || spec->dmax > spec->l) return gkm_fail(GKM_ERR_INVALID, "dmax %d out of range", spec->dmax);
    if (spec->weighted && (!spec->wd || spec->wd_len < 1)) return gkm_fail(GKM_ERR_INVALID, "weighted spec without weights");
    return GKM_OK;
}

}  // namespace

// ---------------------------------------------------------------------------
// Entry points (C ABI)
// ---------------------------------------------------------------------------

extern "C" int gkm_pack(const gkm_spec *spec, const uint8_t *codes, const int64_t *lengths, int64_t B,
                        int64_t L, uint32_t *fwd, uint32_t *rc, int32_t *counts, gkm_stream_t stream)
{
    GKM_TRY(check_spec(spec));
    if (L < spec->l) return gkm_fail(GKM_ERR_INVALID, "Sequence length %lld is shorter than window length %d", (long long)L, spec->l);
    if (!codes || !fwd) return gkm_fail(GKM_ERR_INVALID, "null codes or output");
    int64_t W = L - spec->l + 1;
    int64_t n = B * W;
    if (n == 0) return GKM_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const int64_t chunks = (W + PACK_WINDOWS - 1) / PACK_WINDOWS;
    if (W >= PACK_ROW && B * chunks <= 0x7FFFFFFFLL) {
        GKM_PREFER_SHARED(pack_rows);
        pack_rows<<<(unsigned)(B * chunks), PACK_THREADS, 0, st>>>(codes, lengths, L, spec->l, chunks, fwd, rc, counts);
    } else {
        GKM_PREFER_SHARED(pack_kernel);
        pack_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(codes, lengths, B, L, spec->l, fwd, rc, counts);
    }
    GKM_CHECK_LAUNCH("pack");
    return GKM_OK;
}

// The share of window pairs of uniform bases within d mismatches.
static double pair_share(int l, int d)
{
    double c = 1.0, n = 0.0, p = 1.0;
    for (int m = 0; m <= d && m <= l; m++) {
        n += c;
        c = c * 3.0 * (l - m) / (m + 1);
    }
    for (int k = 0; k < l; k++) p *= 0.25;
    return n * p;
}

// Whether a weighted self-kernel costs less pair by pair: past this share of pairs that
// count (d past 7 makes a pair dearer, 16 levels), and a larger one for many short rows,
// whose warps the pair loop leaves half empty.  Measured on B200, by diagonals and pair by
// pair: 32 rows of 2,000 bp, l = 8, d = 7 (90 % of the pairs) 3,494 and 1,086 us; l = 9, d =
// 5 (17 %) 1,409 and 1,084; l = 9, d = 4 (5 %) 831 and 1,088; l = 15, d = 14 (99 %) 5,083
// and 2,434; 512 rows of 150 bp, l = 12, d = 9 (61 %) 66 and 128.  Of 1,552 shapes (l = 3 ..
// 15, every d) diagonals for all are slower by more than a tenth in 290, by up to 3.2
// times, by this rule 9, by up to 1.25.
static bool pairs_pay(const gkm_spec *spec, int64_t B, int64_t W)
{
    if (!spec->weighted) return false;
    double share = spec->dmax < 4 ? 0.16 : spec->dmax < 8 ? 0.14 : 0.45;
    if (B > 2 * gkm_sm_count() && W < 512) share *= 750.0 / (double)W;
    return pair_share(spec->l, spec->dmax) > share;
}

static int self_launch(const gkm_spec *spec, const uint32_t *fwd, const uint32_t *rc, const int32_t *counts,
                       int64_t B, int64_t W, double *diag, uint64_t *profile, const double *table, double bias,
                       int normalize, double *scores, double *raw, cudaStream_t st)
{
    if (B == 0) return GKM_OK;
    int pw = plane_words(W, spec->l);
    size_t smem = (size_t)4 * pw * sizeof(uint32_t);
    if (smem > SELF_PLANES) smem = pw = 0;
    if (pairs_pay(spec, B, W)) {
        const int sw = staged_windows(W), nw = nw_for(spec->dmax);
        const size_t staged = (size_t)2 * sw * sizeof(uint32_t);
#define GKM_SELF_PAIRS(NW)                                                                                \
    do {                                                                                                  \
        GKM_ALLOW_SHARED(self_pairs_kernel<NW>, 2 * SMEM_WINDOWS * sizeof(uint32_t));                     \
        GKM_PREFER_SHARED(self_pairs_kernel<NW>);                                                         \
        self_pairs_kernel<NW><<<(unsigned)B, SELF_THREADS, staged, st>>>(                                 \
            *spec, fwd, rc, counts, W, diag, profile, table, bias, normalize, scores, raw, sw);           \
    } while (0)
        if (nw == 1) GKM_SELF_PAIRS(1);
        else if (nw == 2) GKM_SELF_PAIRS(2);
        else GKM_SELF_PAIRS(4);
#undef GKM_SELF_PAIRS
        GKM_CHECK_LAUNCH("self_pairs_kernel");
        return GKM_OK;
    }
#define GKM_SELF_AS(L, NL, WT)                                                                                \
    do {                                                                                                      \
        GKM_ALLOW_SHARED((self_kernel<L, NL, WT>), SELF_PLANES);                                              \
        GKM_PREFER_SHARED((self_kernel<L, NL, WT>));                                                          \
        self_kernel<L, NL, WT><<<(unsigned)B, SELF_THREADS, smem, st>>>(                                      \
            *spec, fwd, rc, counts, W, diag, profile, table, bias, normalize, scores, raw, pw);               \
    } while (0)
#define GKM_SELF(L)                                                       \
    do {                                                                  \
        if (spec->dmax < 4 && spec->weighted) GKM_SELF_AS(L, 4, true);    \
        else if (spec->dmax < 4) GKM_SELF_AS(L, 4, false);                \
        else if (spec->weighted) GKM_SELF_AS(L, 16, true);                \
        else GKM_SELF_AS(L, 16, false);                                   \
    } while (0)
    // l = 10 and 11 compiled in (32 rows of 2,000 bp, d = 3: 89 and 79 us), other lengths at
    // run time (l = 9: 151, l = 12: 165)
    if (spec->l == 11) GKM_SELF(11);
    else if (spec->l == 10) GKM_SELF(10);
    else GKM_SELF(0);
#undef GKM_SELF
#undef GKM_SELF_AS
    GKM_CHECK_LAUNCH("self_kernel");
    return GKM_OK;
}

extern "C" int gkm_self_kernel(const gkm_spec *spec, const uint32_t *fwd, const uint32_t *rc,
                               const int32_t *counts, int64_t B, int64_t W, double *diag,
                               uint64_t *profile, gkm_stream_t stream)
{
    GKM_TRY(check_spec(spec));
    if (!fwd || !counts) return gkm_fail(GKM_ERR_INVALID, "null windows or counts");
    return self_launch(spec, fwd, rc, counts, B, W, diag, profile, nullptr, 0.0, 0, nullptr, nullptr,
                       (cudaStream_t)stream);
}

extern "C" int gkm_table_score(const gkm_spec *spec, const double *table, const uint32_t *fwd,
                               const uint32_t *rc, const int32_t *counts, int64_t B, int64_t W, double bias,
                               int32_t normalize, double *scores, double *raw, double *diag,
                               gkm_stream_t stream)
{
    GKM_TRY(check_spec(spec));
    if (!table || !scores) return gkm_fail(GKM_ERR_INVALID, "null table or scores");
    return self_launch(spec, fwd, rc, counts, B, W, diag, nullptr, table, bias, normalize, scores, raw,
                       (cudaStream_t)stream);
}

extern "C" int gkm_join_pairwise(const gkm_spec *spec, const uint32_t *bx, const int32_t *cx, int64_t B,
                                 int64_t Wx, const uint32_t *by, const uint32_t *ry, const int32_t *cy,
                                 int64_t S, int64_t Wy, double *raw, uint64_t *profile, gkm_stream_t stream)
{
    GKM_TRY(check_spec(spec));
    if (B == 0 || S == 0) return GKM_OK;
    if (Wx > JOIN_WINDOWS) return gkm_fail(GKM_ERR_UNSUPPORTED, "query rows longer than 56,000 windows");
    size_t smem = (size_t)Wx * sizeof(uint32_t);
    dim3 grid((unsigned)B, (unsigned)((S + JOIN_WARPS - 1) / JOIN_WARPS));
    if (grid.y > 65535) return gkm_fail(GKM_ERR_UNSUPPORTED, "too many columns for one join launch");
    cudaStream_t st = (cudaStream_t)stream;
    int nw = nw_for(spec->dmax);
#define GKM_JOIN(NW)                                                                                   \
    do {                                                                                               \
        GKM_ALLOW_SHARED(join_kernel<NW>, JOIN_WINDOWS * sizeof(uint32_t));                            \
        join_kernel<NW><<<grid, JOIN_WARPS * 32, smem, st>>>(*spec, bx, cx, Wx, by, ry, cy, S, Wy, raw, \
                                                             profile);                                 \
    } while (0)
    if (nw == 1) GKM_JOIN(1);
    else if (nw == 2) GKM_JOIN(2);
    else GKM_JOIN(4);
#undef GKM_JOIN
    GKM_CHECK_LAUNCH("join");
    return GKM_OK;
}

extern "C" int gkm_lmer_table(const gkm_spec *spec, const double *V, const uint32_t *masks, int32_t n_masks,
                              double *table, gkm_stream_t stream)
{
    GKM_TRY(check_spec(spec));
    if (spec->l > 12) return gkm_fail(GKM_ERR_UNSUPPORTED, "l-mer tables need l <= 12");
    int64_t n = (int64_t)1 << (2 * spec->l);
    lmer_table_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(*spec, V, masks, n_masks,
                                                                                   table, n);
    GKM_CHECK_LAUNCH("lmer_table");
    return GKM_OK;
}

// DeltaSVM weights read off the l-mer table (svm.py:667-704): out[idx], idx in
// DeltaSVM order (first base most significant), = table[idx with its digits
// reversed] times the lone window's weight, divided by sqrt(K(u, u)) of the
// l-mer alone when qnorm (h(0), plus h(m(u, rc u)) with RC, times the weight
// squared).
__global__ void deltasvm_table_kernel(gkm_spec sp, const double *__restrict__ table, double wt, int qnorm,
                                      double *__restrict__ out, int64_t n)
{
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n) return;
    const int l = sp.l;
    const uint32_t u = (uint32_t)idx;
    uint32_t packed = 0;
    for (int p = 0; p < l; p++) packed |= ((u >> (2 * (l - 1 - p))) & 3u) << (2 * p);
    double w = table[packed] * wt;
    if (qnorm) {
        double self_k = sp.h[0];
        if (sp.include_rc) self_k = self_k + sp.h[gkm_mism(packed, gkm_rc_word(packed, l))];
        self_k = self_k * (wt * wt);
        w = w / sqrt(fmax(self_k, 1e-10));
    }
    out[idx] = w;
}

extern "C" int gkm_deltasvm_table(const gkm_spec *spec, const double *table, double window_weight,
                                  int32_t query_norm, double *out, gkm_stream_t stream)
{
    GKM_TRY(check_spec(spec));
    if (!table || !out) return gkm_fail(GKM_ERR_INVALID, "null table or out");
    if (spec->l > 12) return gkm_fail(GKM_ERR_UNSUPPORTED, "l-mer tables need l <= 12");
    int64_t n = (int64_t)1 << (2 * spec->l);
    deltasvm_table_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(*spec, table, window_weight,
                                                                                        query_norm, out, n);
    GKM_CHECK_LAUNCH("deltasvm_table");
    return GKM_OK;
}

// Whether mutant_tiles costs less than mutant_kernel for B rows of W windows.  Microseconds
// measured on B200 (l = 3 .. 12, d = 0 .. 3, 1 and 32 rows of 20 .. 2,000 bp): a block of
// mutant_tiles runs every diagonal of its row and each pair within dmax + 1 mismatches one
// lane per l positions (weighted: 64-bit adds), however few blocks there are; mutant_kernel
// has a block per position and looks at every window there.  A lone 300 bp row, l = 11, d =
// 3: 38 against 15 us, 32 of them 46 against 178; short l-mers, where every pair is near:
// 32 rows of 300 bp at l = 6, d = 3 296 against 119 us, weighted 940.
static bool tiles_pay(const gkm_spec *spec, int64_t B, int64_t W, int64_t L)
{
    const int l = spec->l, P = MT_WINDOWS - l + 1;
    const double near = pair_share(l, spec->dmax + 1), w = (double)W;
    const double block = 20.0 + w * (0.016 + near * (spec->weighted ? 1.75 * (spec->dmax + 1) : 0.33 * l));
    const double fill = (double)((L + P - 1) / P * B) / gkm_sm_count() / 2.1;
    const double all = 12.0 + (double)B * (double)L * w * (10.0 + 4.0 * l) * 1e-6;
    return block * (fill > 1.0 ? fill : 1.0) < all;
}

// Whether mutant_tiles takes a launch: four levels, rows whose bit planes fit shared
// memory, and work enough.
static size_t tile_planes(const gkm_spec *spec, int64_t W, int *pw)
{
    *pw = plane_words(W, spec->l) + 1;
    return (size_t)4 * mutant_plane(*pw) * sizeof(uint32_t);
}
static bool tiles_apply(const gkm_spec *spec, int64_t B, int64_t W, int64_t L)
{
    int pw;
    return spec->dmax < 4 && tile_planes(spec, W, &pw) <= MT_PLANES && tiles_pay(spec, B, W, L);
}

extern "C" int gkm_self_form(const gkm_spec *spec, int64_t B, int64_t W)
{
    return spec && check_spec(spec) == GKM_OK && pairs_pay(spec, B, W) ? 1 : 0;
}

extern "C" int gkm_mutant_form(const gkm_spec *spec, int64_t B, int64_t W, int64_t L)
{
    return spec && check_spec(spec) == GKM_OK && tiles_apply(spec, B, W, L) ? 1 : 0;
}

static int mutant_launch(const gkm_spec *spec, const uint32_t *fwd, const int32_t *counts, int64_t B,
                         int64_t W, int64_t L, const double *diag, double *mut_diag, const double *table,
                         const double *ref_raw, int normalize, double *out, cudaStream_t st)
{
    if (B == 0 || L == 0) return GKM_OK;
    if (B > 65535) return gkm_fail(GKM_ERR_UNSUPPORTED, "more than 65,535 rows per ISM launch");
    if (tiles_apply(spec, B, W, L)) {
        int pw;
        const size_t planes = tile_planes(spec, W, &pw);
        const int P = MT_WINDOWS - spec->l + 1;
        const dim3 grid((unsigned)((L + P - 1) / P), (unsigned)B);
#define GKM_MUT_AS(LT, WT)                                                                                     \
    do {                                                                                                       \
        GKM_ALLOW_SHARED((mutant_tiles<LT, WT>), MT_PLANES);                                                   \
        GKM_PREFER_SHARED((mutant_tiles<LT, WT>));                                                             \
        mutant_tiles<LT, WT><<<grid, MT_THREADS, planes, st>>>(*spec, fwd, counts, B, W, L, diag, mut_diag,    \
                                                               table, ref_raw, normalize, out, pw);            \
    } while (0)
        if (spec->l == 11 && spec->weighted) GKM_MUT_AS(11, true);
        else if (spec->l == 11) GKM_MUT_AS(11, false);
        else if (spec->l == 10 && spec->weighted) GKM_MUT_AS(10, true);
        else if (spec->l == 10) GKM_MUT_AS(10, false);
        else if (spec->weighted) GKM_MUT_AS(0, true);
        else GKM_MUT_AS(0, false);
#undef GKM_MUT_AS
        GKM_CHECK_LAUNCH("mutant_tiles");
        return GKM_OK;
    }
    const int sw = staged_windows(W);
    size_t smem = (size_t)2 * sw * sizeof(uint32_t);
    dim3 grid((unsigned)L, (unsigned)B);
    int nw = nw_for(spec->dmax);
#define GKM_MUT(NW)                                                                                      \
    do {                                                                                                 \
        GKM_ALLOW_SHARED(mutant_kernel<NW>, 2 * SMEM_WINDOWS * sizeof(uint32_t));                        \
        GKM_PREFER_SHARED(mutant_kernel<NW>);                                                            \
        mutant_kernel<NW><<<grid, MUT_THREADS, smem, st>>>(*spec, fwd, counts, B, W, L, diag, mut_diag,  \
                                                           table, ref_raw, normalize, out, sw);          \
    } while (0)
    if (nw == 1) GKM_MUT(1);
    else if (nw == 2) GKM_MUT(2);
    else GKM_MUT(4);
#undef GKM_MUT
    GKM_CHECK_LAUNCH("mutant");
    return GKM_OK;
}

extern "C" int gkm_mutant_diag(const gkm_spec *spec, const uint32_t *fwd, const int32_t *counts, int64_t B,
                               int64_t W, int64_t L, const double *diag, double *mut_diag, gkm_stream_t stream)
{
    GKM_TRY(check_spec(spec));
    if (!diag || !mut_diag) return gkm_fail(GKM_ERR_INVALID, "null diag or mut_diag");
    return mutant_launch(spec, fwd, counts, B, W, L, diag, mut_diag, nullptr, nullptr, 0, nullptr,
                         (cudaStream_t)stream);
}

extern "C" int gkm_ism_table(const gkm_spec *spec, const double *table, const uint32_t *fwd,
                             const int32_t *counts, int64_t B, int64_t W, int64_t L, const double *ref_raw,
                             const double *diag, double *mut_diag, int32_t normalize, double *out,
                             gkm_stream_t stream)
{
    GKM_TRY(check_spec(spec));
    if (!table || !ref_raw || !out) return gkm_fail(GKM_ERR_INVALID, "null table, ref_raw or out");
    if (normalize && !diag) return gkm_fail(GKM_ERR_INVALID, "normalize needs diag");
    return mutant_launch(spec, fwd, counts, B, W, L, normalize ? diag : nullptr, mut_diag, table, ref_raw,
                         normalize, out, (cudaStream_t)stream);
}

extern "C" int gkm_raw_score(const double *raw, int64_t B, int64_t S, const double *dx, const double *ds,
                             const double *coef, double gamma, int32_t rbf, double bias, double *scores,
                             gkm_stream_t stream)
{
    if (B == 0) return GKM_OK;
    GKM_PREFER_SHARED(raw_score_kernel);
    raw_score_kernel<<<(unsigned)B, 256, 0, (cudaStream_t)stream>>>(raw, S, dx, ds, coef, gamma, rbf, bias, scores);
    GKM_CHECK_LAUNCH("raw_score");
    return GKM_OK;
}

extern "C" int gkm_impact(const double *raw, int64_t n, int64_t S, const double *dr, const double *ds,
                          const double *coef, double gamma, int32_t rbf, double *out, gkm_stream_t stream)
{
    if (n == 0) return GKM_OK;
    GKM_PREFER_SHARED(impact_kernel);
    impact_kernel<<<(unsigned)(n * IMPACT_BLOCKS), 256, 0, (cudaStream_t)stream>>>(raw, n, S, dr, ds, coef, gamma, rbf, out);
    GKM_CHECK_LAUNCH("impact");
    return GKM_OK;
}

extern "C" int gkm_gram_finish(const double *raw, int64_t N, int64_t M, const double *dx, const double *dy,
                               double gamma, int32_t rbf, int32_t symmetric, double *out, gkm_stream_t stream)
{
    int64_t n = N * M;
    if (n == 0) return GKM_OK;
    if (symmetric && N != M) return gkm_fail(GKM_ERR_INVALID, "symmetric Gram must be square");
    gram_finish_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(raw, N, M, dx, dy, gamma, rbf,
                                                                                     symmetric, out);
    GKM_CHECK_LAUNCH("gram_finish");
    return GKM_OK;
}
