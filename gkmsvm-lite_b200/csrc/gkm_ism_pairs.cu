// gkm_ism_pairs.cu -- ISM deltas of every substitution for kernels without an l-mer
// table (RBF), from one pass over the window pairs of a row and an SV.
//
// A substitution at p changes only pairs of a window (i, strand) of the row that
// covers p and a window u of the SV, and for them
//     h changes from h(t) to h(t + 1) or back,
// t the mismatches outside p, by whether u has the old or the new base there.  With
// G[p][a][t] the pairs covering p whose u has base a there and t mismatches
// elsewhere (products of the window weights for weighted kernels),
//     K(mutant v) - K(x) = sum_t (h(t) - h(t + 1)) (G[p][v][t] - G[p][x_p][t]),
// and only pairs within dmax + 1 mismatches count.  A pair adds to G at the places
// where it mismatches (a != x_p, at most dmax + 1 adds); the pairs that match there
// follow from C[i][m], the pairs of row window i with m mismatches:
//     G[p][x_p][t] = sum over i covering p of C[i][t] - sum over a != x_p of G[p][a][t - 1].
//
//   1. pair_lists: per l-mer (rows folded as in the count tables) the row's windows
//      within dmax + 1 mismatches, 16 bits each;
//   2. pair_gather: per SV the lists of its windows, G and C in shared memory, then
//      the SV's term of every mutant's score added in registers;
//   3. pair_finish: the blocks' sums, minus the reference's.
//
// The walk (gkm_index_mutants) queries the index with l windows for each of three
// mutants per position and writes K of every (mutant, SV); this visits a pair once for
// all of them.
#include <cuda_runtime.h>
#include <stdint.h>

#include "gkm_common.cuh"

namespace {

constexpr int PL_ROWS = 1024;  // table rows per list tile: five positions
constexpr int PL_THREADS = 256;
constexpr int PL_BALL = 781;   // masks of five positions within four mismatches
constexpr int PG_POS = 2;      // positions of a gather thread

struct Ball {
    uint16_t v[PL_BALL];
};

constexpr Ball make_ball()
{
    Ball b{};
    int k = 0;
    for (int m = 0; m <= 4; m++)
        for (int x = 0; x < PL_ROWS; x++) {
            int n = 0;
            for (int j = 0; j < 5; j++) n += ((x >> (2 * j)) & 3) != 0;
            if (n == m) b.v[k++] = (uint16_t)x;
        }
    return b;
}

__constant__ Ball c_ball = make_ball();  // masks of the suffix by mismatches

struct PairArgs {
    const uint32_t *fwd;     // [B, W]
    const int32_t *counts;
    int64_t B, W, L, b;      // this call's row
    gkm_rows sh;
    const uint8_t *wd;       // weighted: window weights by distance from the centre
    uint32_t *off;           // [tiles + 1][PL_ROWS + 1] list bounds; the last tile stays empty
    uint16_t *ents;          // window i | strand << 15
    uint32_t *cursor;
    int tiles;
    const uint32_t *ids;     // gather lists of the SVs (see gkm_count_table.cu)
    const uint8_t *wts;
    const uint32_t *goff;
    const uint32_t *perm;
    int64_t S;
    double dh[4];            // h(t) - h(t + 1)
    const double *ref;       // [B, S] K(x, s)
    const double *inv_dx;    // [B]
    const double *inv_dmut;  // [4, L, B]
    const double *inv_ds;
    const double *coef;
    double gamma;
    int rbf;
    double *partial;         // [blocks, 3 L + 1]
    double *out;             // [B, 4, L]
};

__global__ void __launch_bounds__(PL_THREADS) pair_lists(PairArgs a)
{
    __shared__ __align__(16) uint32_t cnt[PL_ROWS];
    __shared__ uint16_t ball[PL_BALL];
    __shared__ uint32_t warp_sum[PL_THREADS / 32], base_s;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t tile = blockIdx.x;
    const gkm_rows sh = a.sh;
    const int n = a.counts[a.b], words = n > 0 ? n * sh.strands : 0;
    ((uint4 *)cnt)[threadIdx.x] = make_uint4(0, 0, 0, 0);
    for (int k = threadIdx.x; k < PL_BALL; k += PL_THREADS) ball[k] = c_ball.v[k];
    __syncthreads();
    for (int pass = 0; pass < 2; pass++) {
        auto hit = [&](uint32_t r, uint32_t e) {
            const uint32_t at = atomicAdd(&cnt[r], 1u);
            if (pass) a.ents[at] = (uint16_t)e;
        };
        for (int k0 = warp * 32; k0 < words; k0 += PL_THREADS) {
            const int k = k0 + lane, st = k >= n, i = st ? k - n : k;
            int budget = -1;
            uint32_t c = 0;
            if (k < words) {
                uint32_t v = __ldg(a.fwd + a.b * a.W + i);
                if (st) v = gkm_rc_word(v, sh.l);
                c = v;
                if (sh.fold) {  // the middle base goes on top
                    const uint32_t low = (1u << (2 * sh.mid)) - 1u;
                    c = (v & low) | ((v >> 2) & ~low & ((1u << (2 * (sh.l - 1))) - 1u)) |
                        (((v >> (2 * sh.mid)) & 3u) << (2 * (sh.l - 1)));
                }
                budget = sh.D + 1 - gkm_mism(c >> 10, tile);
            }
            const uint32_t suffix = c & (PL_ROWS - 1), e = (uint32_t)i | (uint32_t)st << 15;
            if (budget == 0) hit(suffix, e);
            for (uint32_t rest = __ballot_sync(GKM_FULL, budget > 0); rest; rest &= rest - 1) {
                const int j = __ffs(rest) - 1, bj = __shfl_sync(GKM_FULL, budget, j);
                const uint32_t sj = __shfl_sync(GKM_FULL, suffix, j), ej = __shfl_sync(GKM_FULL, e, j);
                const int masks = bj == 1 ? 16 : bj == 2 ? 106 : bj == 3 ? 376 : 781;
                for (int m = lane; m < masks; m += 32) hit(sj ^ ball[m], ej);
            }
        }
        __syncthreads();
        if (pass) break;
        // the rows' places: an exclusive scan, and the tile's share of the entries
        const uint4 c4 = ((const uint4 *)cnt)[threadIdx.x];
        const uint32_t own = c4.x + c4.y + c4.z + c4.w;
        uint32_t x = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(GKM_FULL, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_sum[warp] = x;
        __syncthreads();
        uint32_t before = 0, total = 0;
        for (int w = 0; w < PL_THREADS / 32; w++) {
            if (w < warp) before += warp_sum[w];
            total += warp_sum[w];
        }
        if (threadIdx.x == 0) base_s = atomicAdd(a.cursor, total);
        __syncthreads();
        x = base_s + before + x - own;
        const uint4 first = make_uint4(x, x + c4.x, x + c4.x + c4.y, x + own - c4.w);
        ((uint4 *)cnt)[threadIdx.x] = first;
        uint32_t *o = a.off + (size_t)tile * (PL_ROWS + 1) + 4 * threadIdx.x;
        o[0] = first.x, o[1] = first.y, o[2] = first.z, o[3] = first.w;
        if (threadIdx.x == PL_THREADS - 1) o[4] = x + own;
        __syncthreads();
    }
}

// Shared-memory add where m is not zero (predicated rather than branched around).
__device__ __forceinline__ void pair_add(uint32_t m, uint32_t addr, uint32_t v)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p red.shared.add.u32 [%1], %2;\n\t}" ::"r"(m), "r"(addr),
                 "r"(v)
                 : "memory");
}

// A two's complement word as a double: placed in the mantissa of 2^52 with its sign bit
// flipped, exactly.
__device__ __forceinline__ double pair_double(uint32_t x)
{
    return __hiloint2double(0x43300000, (int)(x ^ 0x80000000u)) - 4503601774854144.0;  // 2^52 + 2^31
}

// Shared memory of a gather block: G (16 planes of a multiple of 32 positions: most
// pairs have the same t, so that a position's counters side by side would leave 8 of
// the 32 banks to them), C twice (cleared while the other is in use), both strands'
// words, weights.
__host__ __device__ __forceinline__ int64_t pg_plane(int64_t L) { return (L + 31) & ~(int64_t)31; }
inline size_t pg_bytes(int64_t L) { return (size_t)(64 * pg_plane(L) + (2 * 16 + 8 + 1) * L); }

// One block per SV at a time; thread t has positions t and t + T of every SV, their
// normalisers and sums in registers.  Bound by instruction issue (181M pairs at 500 bp
// against 72,000 SVs of 350 bp).  Measured there: the walk and its reduction 7.1 ms,
// lists, gather and sums 2.2 ms (with a position's 16 counters side by side 2.4).
template <int T, bool WT>
__global__ void __launch_bounds__(T, 1024 / T) pair_gather(PairArgs a)
{
    extern __shared__ __align__(16) uint8_t pg_smem[];
    constexpr int WARPS = T / 32;
    __shared__ uint2 slot_s[WARPS][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const gkm_rows sh = a.sh;
    const int l = sh.l, n = a.counts[a.b], P = n > 0 ? n + l - 1 : 0;
    const uint32_t plane = (uint32_t)pg_plane(a.L);
    uint32_t *G = (uint32_t *)pg_smem;    // [base][t][plane]
    uint4 *C = (uint4 *)(G + 16 * plane);  // [2][n]: four m
    uint32_t *word = (uint32_t *)(C + 2 * a.L);  // [2][n]
    uint8_t *wx = (uint8_t *)(word + 2 * a.L);
    for (int k = threadIdx.x; k < 4 * (int)plane + 2 * n; k += T) ((uint4 *)G)[k] = make_uint4(0, 0, 0, 0);  // (and C)
    for (int i = threadIdx.x; i < n; i += T) {
        const uint32_t v = a.fwd[a.b * a.W + i];
        word[i] = v;
        word[n + i] = gkm_rc_word(v, l);
        if (WT) wx[i] = (uint8_t)gkm_wt(a.wd, n, i);
    }
    __syncthreads();
    double z[PG_POS][3], sum[PG_POS][3], ref_sum = 0.0;
    int xp[PG_POS];
#pragma unroll
    for (int q = 0; q < PG_POS; q++) {
        const int p = threadIdx.x + q * T;
        xp[q] = 0;
        if (p < P) xp[q] = p < n ? word[p] & 3u : (word[n - 1] >> (2 * (p - n + 1))) & 3u;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            sum[q][k] = 0.0;
            z[q][k] = p < P ? a.inv_dmut[((int64_t)(k + (k >= xp[q])) * a.L + p) * a.B + a.b] : 0.0;
        }
    }
    const double zx = a.inv_dx[a.b];
    const uint32_t gbase = (uint32_t)__cvta_generic_to_shared(G);
    uint2 *slot = slot_s[warp];
    int par = 0;
    for (int64_t g = blockIdx.x; g < a.S && P > 0; g += gridDim.x, par ^= 1) {
        const uint32_t p0 = a.goff[g], wins = a.goff[g + 1] - p0;
        uint32_t *Cw = (uint32_t *)(C + par * n);
        const uint32_t per = (wins + WARPS - 1) / WARPS, mine = min(wins, (warp + 1) * per);
        for (uint32_t c = warp * per; c < mine; c += 32) {
            uint32_t beg = 0, upto = 0, u = 0, ws = 1;
            if (c + lane < mine) {
                const uint32_t r = __ldg(a.ids + p0 + c + lane);
                const uint32_t *o = a.off + (size_t)(r / PL_ROWS) * (PL_ROWS + 1) + r % PL_ROWS;
                beg = __ldg(o);
                upto = __ldg(o + 1) - beg;
                u = sh.lmer(r);
                if (WT) ws = __ldg(a.wts + p0 + c + lane);
            }
            const uint32_t len = upto;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(GKM_FULL, upto, o);
                if (lane >= o) upto += y;
            }
            const uint32_t all = __shfl_sync(GKM_FULL, upto, 31), start = upto - len;
            // the windows with pairs, side by side: pair h of the chunk is entry .x + h
            // (in 32 bits: .x may lie below zero)
            const uint32_t some = __ballot_sync(GKM_FULL, len != 0);
            if (len) slot[__popc(some & ((1u << lane) - 1u))] = make_uint2(beg - start, u | ws << 24);
            __syncwarp();
            // Pairs h0 + lane: their window is the last one that starts at or before
            // them, found by counting starts.
            uint32_t begun = 0;
            uint2 win;
            auto fetch = [&](uint32_t h0) -> uint32_t {
                const uint32_t at = start - h0, starts = __reduce_or_sync(GKM_FULL, len && at < 32 ? 1u << at : 0u);
                win = slot[(begun + __popc(starts & (0xFFFFFFFFu >> (31 - lane))) - 1u) & 31u];
                begun += __popc(starts);
                return h0 + lane < all ? (uint32_t)__ldg(a.ents + (win.x + (h0 + lane))) : 0u;
            };
            uint32_t e = fetch(0);
            for (uint32_t h0 = 0; h0 < all; h0 += 32) {
                const uint32_t now = e, uu = win.y & 0xFFFFFFu, i = now & 0x7FFFu, st = now >> 15;
                const bool in = h0 + lane < all;
                const uint32_t w = WT ? (win.y >> 24) * wx[i] : 1u;
                e = fetch(h0 + 32);  // in flight meanwhile
                const uint32_t x = uu ^ word[i + (st ? n : 0)];
                uint32_t m = in ? (x | (x >> 1)) & 0x55555555u : 0u;
                const uint32_t nm = __popc(m);
                if (in && (int)nm <= sh.D) atomicAdd(Cw + 4 * i + nm, w);
                // strand 1 reads the row backwards, complemented
                const uint32_t to = gbase + 4 * (i + (st ? l - 1 : 0) + plane * (nm - 1)), step = st ? -2 : 2, ub = st ? ~uu : uu;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const uint32_t bit = 31 - __clz(m);
                    pair_add(m, to + step * bit + 16 * plane * ((ub >> (bit & 31u)) & 3u), w);
                    m &= ~(1u << (bit & 31u));
                }
            }
            __syncwarp();
        }
        __syncthreads();
        const int64_t s = a.perm[g];
        const double ref = a.ref[a.b * a.S + s], ds = a.inv_ds[s], co = a.coef[s];
#pragma unroll
        for (int q = 0; q < PG_POS; q++) {
            const int p = threadIdx.x + q * T;
            if (p >= P) break;
            // pairs covering p by mismatches
            uint32_t t[4] = {0, 0, 0, 0};
            for (int i = max(0, p - l + 1), e = min(n - 1, p); i <= e; i++) {
                const uint4 v = C[par * n + i];
                t[0] += v.x, t[1] += v.y, t[2] += v.z, t[3] += v.w;
            }
            uint32_t own[3][4];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                uint32_t *at = G + 4 * plane * (k + (k >= xp[q])) + p;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    own[k][j] = at[j * plane];
                    at[j * plane] = 0;
                    if (j < 3) t[j + 1] -= own[k][j];
                }
            }
#pragma unroll
            for (int k = 0; k < 3; k++) {
                double d = ref;
#pragma unroll
                for (int j = 0; j < 4; j++) d += a.dh[j] * pair_double(own[k][j] - t[j]);
                const double kn = d * z[q][k] * ds;
                sum[q][k] += co * (a.rbf ? exp(a.gamma * (kn - 1.0)) : kn);
            }
        }
        if (threadIdx.x == T - 1) {  // the reference's score, by the same arithmetic
            const double kn = ref * zx * ds;
            ref_sum += co * (a.rbf ? exp(a.gamma * (kn - 1.0)) : kn);
        }
        for (int i = threadIdx.x; i < n; i += T) C[(par ^ 1) * n + i] = make_uint4(0, 0, 0, 0);
        __syncthreads();
    }
    double *part = a.partial + (int64_t)blockIdx.x * (3 * a.L + 1);
#pragma unroll
    for (int q = 0; q < PG_POS; q++)
        if ((int)threadIdx.x + q * T < P)
#pragma unroll
            for (int k = 0; k < 3; k++) part[k * a.L + threadIdx.x + q * T] = sum[q][k];
    if (threadIdx.x == T - 1) part[3 * a.L] = ref_sum;
}

// Sums column c of the blocks' parts in the order of 32 slices (thread y: one slice).
__device__ __forceinline__ double pair_slice(const double *__restrict__ part, int blocks, int64_t stride, int64_t c, int y)
{
    double t = 0.0;
    for (int k = y; k < blocks; k += 32) t += part[k * stride + c];
    return t;
}

// 32 positions x 32 slices a block: the three mutants' scores minus the reference's.
__global__ void __launch_bounds__(1024) pair_finish(PairArgs a, int blocks)
{
    __shared__ double red[4][32][33];
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const int64_t p = (int64_t)blockIdx.x * 32 + x, stride = 3 * a.L + 1;
    const int l = a.sh.l, n = a.counts[a.b], P = n > 0 ? n + l - 1 : 0;
    for (int k = 0; k < 3; k++) red[k][y][x] = p < P ? pair_slice(a.partial, blocks, stride, k * a.L + p, y) : 0.0;
    if (x == 0 && P > 0) red[3][y][0] = pair_slice(a.partial, blocks, stride, 3 * a.L, y);
    __syncthreads();
    if (y >= 4 || p >= a.L) return;
    double *out = a.out + a.b * 4 * a.L + p;
    const uint32_t *w = a.fwd + a.b * a.W;
    const int xp = p >= P ? -1 : (int)(p < n ? w[p] & 3u : (w[n - 1] >> (2 * (p - n + 1))) & 3u);
    if (p >= P || y == 3) {
        out[(p >= P ? y : xp) * a.L] = 0.0;
        return;
    }
    double t = 0.0, r = 0.0;
    for (int k = 0; k < 32; k++) t += red[y][k][x], r += red[3][k][0];
    out[(y + (y >= xp)) * a.L] = t - r;
}

}  // namespace

static int64_t pair_up(int64_t n) { return (n + 255) & ~(int64_t)255; }

struct PairPlan {
    int threads, blocks;
    int64_t tiles, off, ents, partial, bytes;
    size_t smem;
};

static bool pair_plan(const gkm_index *ix, int64_t W, int64_t L, PairPlan &p)
{
    // the count tables' gather lists (and their limits); a thread has two positions and
    // an SV's G and C fit shared memory; every window lies within the L positions
    if (!ix->ct_ids || W < 1 || L > 2048 || W > L - ix->spec.l + 1) return false;
    p.threads = L <= 512 ? 256 : L <= 1024 ? 512 : 1024;
    p.smem = pg_bytes(L);
    if ((int64_t)p.smem > gkm_smem_limit()) return false;
    p.blocks = gkm_sm_count() * (1024 / p.threads);
    p.tiles = gkm_row_count(ix) / PL_ROWS;
    const gkm_rows sh = gkm_rows_of(ix);
    int64_t ball = 0, c = 1;  // l-mers within dmax + 1 mismatches
    for (int m = 0; m <= sh.D + 1; m++) {
        ball += c;
        c = c * 3 * (sh.l - m) / (m + 1);
    }
    const int64_t cap = W * ball * (sh.strands == 2 && !sh.fold ? 2 : 1);
    if (cap > 0x7FFFFFFFLL) return false;
    p.off = pair_up(4 * (p.tiles + 1) * (PL_ROWS + 1));
    p.ents = pair_up(2 * cap);
    p.partial = pair_up(8 * (int64_t)p.blocks * (3 * L + 1));
    p.bytes = 256 + p.off + p.ents + p.partial;
    return true;
}

extern "C" int gkm_ism_pairs_workspace(const gkm_index_t *ix, int64_t W, int64_t L, int64_t *bytes)
{
    if (!ix || !bytes) return gkm_fail(GKM_ERR_INVALID, "null argument");
    PairPlan p;
    *bytes = pair_plan(ix, W, L, p) ? p.bytes : 0;
    return GKM_OK;
}

extern "C" int gkm_ism_pairs(const gkm_index_t *ix, const uint32_t *fwd, const int32_t *counts, int64_t B, int64_t W,
                             int64_t L, const double *ref_raw, const double *inv_dx, const double *inv_dmut,
                             const double *inv_ds, const double *coef, double gamma, int32_t rbf, double *out,
                             void *workspace, int64_t workspace_bytes, gkm_stream_t stream)
{
    if (!ix || !fwd || !counts || !ref_raw || !inv_dx || !inv_dmut || !inv_ds || !coef || !out)
        return gkm_fail(GKM_ERR_INVALID, "null argument");
    if (B < 0 || L < 0 || W < 0) return gkm_fail(GKM_ERR_INVALID, "negative size");
    if (B == 0 || L == 0) return GKM_OK;
    PairPlan p;
    if (!pair_plan(ix, W, L, p)) return gkm_fail(GKM_ERR_UNSUPPORTED, "this index or row length has no pair lists");
    if (!workspace || ((uintptr_t)workspace & 255) || workspace_bytes < p.bytes)
        return gkm_fail(GKM_ERR_CAPACITY, "ISM pair lists need a 256-byte aligned workspace of %lld bytes", (long long)p.bytes);
    cudaStream_t st = (cudaStream_t)stream;
    const bool wt = ix->spec.weighted != 0;
    PairArgs a = {};
    a.fwd = fwd;
    a.counts = counts;
    a.B = B;
    a.W = W;
    a.L = L;
    a.sh = gkm_rows_of(ix);
    a.wd = ix->spec.wd;
    uint8_t *w = (uint8_t *)workspace;
    a.cursor = (uint32_t *)w;
    a.off = (uint32_t *)(w + 256);
    a.ents = (uint16_t *)(w + 256 + p.off);
    a.partial = (double *)(w + 256 + p.off + p.ents);
    a.tiles = (int)p.tiles;
    a.ids = ix->ct_ids;
    a.wts = ix->ct_wts;
    a.goff = ix->ct_off;
    a.perm = ix->ct_perm;
    a.S = ix->S;
    for (int t = 0; t < 4; t++) {
        const double h0 = t <= a.sh.D ? ix->spec.h[t] : 0.0, h1 = t + 1 <= a.sh.D ? ix->spec.h[t + 1] : 0.0;
        a.dh[t] = h0 - h1;
    }
    a.ref = ref_raw;
    a.inv_dx = inv_dx;
    a.inv_dmut = inv_dmut;
    a.inv_ds = inv_ds;
    a.coef = coef;
    a.gamma = gamma;
    a.rbf = rbf;
    a.out = out;
    cudaError_t e = cudaMemsetAsync(a.off + p.tiles * (PL_ROWS + 1), 0, 4 * (PL_ROWS + 1), st);
    if (e != cudaSuccess) return gkm_cuda_status(e, "ISM pair lists");
    // a limit on the thread's persistent grids holds here, too
    int blocks = gkm_query_blocks() * (1024 / p.threads);
    if (blocks > p.blocks) blocks = p.blocks;
    if (blocks > ix->S) blocks = (int)ix->S;
    auto gather = p.threads == 256 ? (wt ? pair_gather<256, true> : pair_gather<256, false>)
                  : p.threads == 512 ? (wt ? pair_gather<512, true> : pair_gather<512, false>)
                                     : (wt ? pair_gather<1024, true> : pair_gather<1024, false>);
    GKM_ALLOW_SHARED(gather, pg_bytes(2 * p.threads));
    for (a.b = 0; a.b < B; a.b++) {
        e = cudaMemsetAsync(a.cursor, 0, 4, st);
        if (e != cudaSuccess) return gkm_cuda_status(e, "ISM pair lists");
        pair_lists<<<(unsigned)p.tiles, PL_THREADS, 0, st>>>(a);
        GKM_CHECK_LAUNCH("pair_lists");
        gather<<<(unsigned)blocks, (unsigned)p.threads, p.smem, st>>>(a);
        GKM_CHECK_LAUNCH("pair_gather");
        pair_finish<<<(unsigned)((L + 31) / 32), 1024, 0, st>>>(a, blocks);
        GKM_CHECK_LAUNCH("pair_finish");
    }
    return GKM_OK;
}
