// gkm_count_table.cu -- index queries through count tables: K_raw(x, s) of a
// group of query rows x against every SV s, without visiting the (window,
// neighbour, entry) hits one by one.
//
// With X_m(v) the number of windows of x (forward and reverse complement; for
// weighted kernels the sum of their weights) exactly m mismatches from l-mer v,
//     K_raw(x, s) = sum_m h(m) sum over the forward windows w of s  X_m(w),
// because a window of s and its reverse complement see the two strands of x the
// same way.  So per group of rows:
//   1. count_tiles writes X_0 .. X_dmax of every l-mer for every row of the
//      group into a table, one row of RB bytes per l-mer, the group's query
//      rows side by side (odd l: a window and its reverse complement share the
//      row of the one whose middle base is A or C, so 4^l / 2 rows);
//   2. gather_kernel sums, per SV, the table rows of its windows: coalesced
//      RB-byte reads added in registers, no atomics.
// The neighbourhood of a query window is visited once (not once per SV tile),
// and a table row read serves every query of the group: at 72,000 SVs and 300 bp
// rows an index walk visits 16.7M entries per query by shared-memory atomics,
// the gather reads 24.5M / 32 rows of 64 bytes.  Measured against the walk (with
// its query self-kernels): 1,000 x 300 bp, t=3: 43.5 -> 9.2 ms; 2,048 rows of 50 ..
// 2,000 bp: 135 -> 20.9 ms; 512 of them, weighted t=5: 77.8 -> 9.6 ms; one 300 bp
// row: 1.3 -> 0.2 ms.
//
// Entries are exact.  Unweighted entries take 16 bits (5, 4, 4 and 3 for levels
// dmax, dmax - 1, ...: t = dmax - m indexes the fields), weighted ones four bytes,
// one per level.  They are counted in shared memory in fields of those widths
// (weighted: 9 / 8 / 8 / 7 bits).  A weighted count past its byte is clipped and
// the excess added to the (SV, query) counts of that l-mer's SVs through the
// index's buckets (spill_excess: C and its dirty bits, read back by the gather).
// A tile whose shared fields overflowed (its decoded fields do not sum to the
// adds made) is counted again with 32-bit counters, one level of one query each,
// and clipped alike.
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>

#include <type_traits>

#include "gkm_common.cuh"

namespace {

constexpr int CT_ROWS = 4096;     // table rows per tile: six of the l-mer's positions
constexpr int CT_THREADS = 1024;
constexpr int CT_WARPS = CT_THREADS / 32;
constexpr int CT_SLOTS = 8;       // counter words per table row a block holds (128 KB)
constexpr int CT_LIST = 512;      // entries of a tile a block queues for a second look
constexpr int CT_RECS = 12288;    // window records of a pass a block keeps in shared memory
constexpr int64_t CT_EXC = 4096;   // clipped counts a group queues, per query (weighted)
// unweighted counter halves (and entries): fields of 5 / 4 / 4 / 3 bits for t = 0
// .. 3, placed so that two byte dot products sum all of them
constexpr uint32_t CT_F0 = 0, CT_F1 = 8, CT_F2 = 12, CT_F3 = 5;
constexpr int CT_R2 = 6, CT_R3 = 26;  // rounds of 32 lanes over the 154 / 694 neighbour masks of budgets 2 / 3
constexpr int CT_BALL = 376;      // masks of up to five positions within three mismatches
constexpr int G_THREADS = 128;
constexpr int G_BLOCKS = 4, G_BLOCKS_W = 6;   // gather blocks per SM, unweighted / weighted

// Shared-memory position of the table row with suffix s (12 bits): a linear
// bijection, its own inverse, chosen so that the masks of a budget spread evenly
// over the 32 banks: lane b takes the masks of bank class b, so a warp's adds
// around any one window hit 32 different banks.
__host__ __device__ __forceinline__ uint32_t ct_phys(uint32_t s)
{
    const uint32_t h = s >> 5;
    return s ^ ((h ^ (h << 2) ^ (h >> 3)) & 31u);
}

struct CtShape {
    int l, D, fold, strands, mid;
    // l-mer -> table row.  fold: the middle position keeps one bit (A / C),
    // moved to the top; the other positions stay in order.
    __host__ __device__ __forceinline__ uint32_t row(uint32_t u) const
    {
        if (!fold) return u;
        const uint32_t low = (1u << (2 * mid)) - 1u;
        return (u & low) | ((u >> 2) & ~low & ((1u << (2 * (l - 1))) - 1u)) | (((u >> (2 * mid)) & 1u) << (2 * (l - 1)));
    }
    __host__ __device__ __forceinline__ uint32_t lmer(uint32_t r) const
    {
        if (!fold) return r;
        const uint32_t low = (1u << (2 * mid)) - 1u, top = (1u << (2 * (l - 1))) - 1u;
        return (r & low) | (((r & top) & ~low) << 2) | ((r >> (2 * (l - 1))) << (2 * mid));
    }
};

struct CtArgs {
    const uint32_t *bx;
    const int32_t *cx;
    int64_t W;
    const int32_t *order;
    int64_t r0;  // first row of the group (position in order)
    int nq;      // rows of the group
    int qg;      // queries a table row holds
    int rb;      // bytes of a table row
    int items, passes;  // (tile, pass of queries) items of the group, passes per tile
    CtShape sh;
    const uint32_t *lists;  // neighbour masks of the six suffix positions by bank class
    const uint32_t *ball;   // masks of the other positions by mismatches
    int nball[4];           // how many of each
    // windows of the call's rows by the bases outside the suffix (ct_buckets):
    // records [pass][rec_cap], bucket offsets [pass][n_pre + 1]
    uint32_t *recs;
    uint32_t *roff;
    int64_t rec_cap;
    int n_pre;
    int pass0;  // pass of the group's first row
    int words, rec_smem;  // count_tiles' counter words per row and staged records
    uint8_t *T;
    unsigned long long *exc;  // [cap_exc] clipped counts of the group: row | q << 22 | excess << 32
    unsigned int *nexc;       // how many (past cap_exc: added at once)
    unsigned int cap_exc;
    unsigned long long *C;   // [S, qg, 2]: excess counts, levels (t0 | t1 << 32, t2 | t3 << 32)
    uint32_t *dirty;         // bit s * qg + q: C holds an excess
    unsigned long long *self;  // [B, 4] by t: the rows' self-kernel counts
    const uint8_t *wd;
    // index buckets
    const uint32_t *off;
    const uint32_t *ent;
    const uint16_t *ent16;
    int64_t n_lmers;
    int tiles;
    int tile_svs;
    // gather
    const uint32_t *ids;   // table rows of each SV's windows, padded to a multiple of 8 with the zero row
    const uint8_t *wts;    // their window weights (weighted)
    const uint32_t *goff;  // [S + 1] in gather order
    const uint32_t *perm;  // gather order: SVs by falling window count
    int64_t S;
    double h[4];           // by t
    int normalize;
    const double *inv_dx;  // [B] by row, or null: from self
    double *diag;          // [B] by row (nullable)
    const double *inv_ds;
    const double *coef;
    double gamma;
    int rbf;
    double *partial;       // [gridDim.x, qg] of this group
    double *raw;           // [B, S] (RAW)
    int64_t diag_offset;   // >= 0: only columns >= diag_offset + row
};

__device__ __forceinline__ int64_t ct_row_of(const CtArgs &a, int q)
{
    return a.order ? (int64_t)a.order[a.r0 + q] : a.r0 + q;
}

// ---------------------------------------------------------------------------
// 1. count tables
// ---------------------------------------------------------------------------

// Adds the excess counts ex (by t) of l-mer v and query q to the counts of the
// SVs holding v, lanes lane, lane + nl, ... of its buckets.  Without folding the
// rows of v and rc(v) hold the same counts and both strands of an SV are in the
// buckets, so v <= rc(v) stands for both; a palindrome's bucket holds every
// window twice in a row.
template <bool WT>
__device__ void ct_excess(const CtArgs &a, uint32_t v, int q, const uint64_t *ex, int lane, int nl)
{
    bool pal = false;
    if (!a.sh.fold && a.sh.strands == 2) {
        const uint32_t r = gkm_rc_word(v, a.sh.l);
        if (r < v) return;
        pal = r == v;
    }
    for (int t = 0; t < a.tiles; t++) {
        const uint32_t *o = a.off + (int64_t)t * a.n_lmers + v;
        const uint32_t b = o[0], e = o[1];
        for (uint32_t k = b + lane; k < e; k += nl) {
            if (pal && ((k - b) & 1u)) continue;
            const uint32_t en = a.ent16 ? (uint32_t)a.ent16[k] | (1u << 24) : a.ent[k];
            const int64_t s = (int64_t)t * a.tile_svs + (en & 0x00FFFFFFu);
            const uint64_t w = WT ? en >> 24 : 1;
            const int64_t at = s * a.qg + q;
            const unsigned long long c0 = w * ex[0] | (w * ex[1]) << 32, c1 = w * ex[2] | (w * ex[3]) << 32;
            if (c0) atomicAdd(a.C + 2 * at, c0);
            if (c1) atomicAdd(a.C + 2 * at + 1, c1);
            atomicOr(a.dirty + (at >> 5), 1u << (at & 31));
        }
    }
}

// plain add to shared memory (byte address), no value returned
__device__ __forceinline__ void ct_add(uint32_t addr, uint32_t v)
{
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

template <bool WT>
__host__ __device__ __forceinline__ uint32_t ct_shift(uint32_t t)
{
    return WT ? (t ? 8u * t + 1u : 0u) : t == 0 ? CT_F0 : t == 1 ? CT_F1 : t == 2 ? CT_F2 : CT_F3;
}

// Counter index (plane of the query, position of the suffix), half and weight of
// a window: how ct_buckets hands it to count_tiles.
//   bits 0..14 counter index, 15 upper half, 16.. weight
template <bool WT>
__device__ __forceinline__ uint32_t ct_record(const CtShape &sh, uint32_t v, int q, uint32_t w, uint32_t *pre)
{
    uint32_t c = v;  // the l-mer without its middle base, which goes on top (fold)
    if (sh.fold) {
        const uint32_t low = (1u << (2 * sh.mid)) - 1u;
        c = (v & low) | ((v >> 2) & ~low & ((1u << (2 * (sh.l - 1))) - 1u)) | (((v >> (2 * sh.mid)) & 3u) << (2 * (sh.l - 1)));
    }
    *pre = c >> 12;
    const uint32_t plane = WT ? (uint32_t)q : (uint32_t)q >> 1;
    return plane * CT_ROWS + ct_phys(c & 0xFFFu) | (WT ? 0u : (uint32_t)(q & 1) << 15) | w << 16;
}

// One block per pass of queries: their windows (both strands) sorted by the
// bases outside the six suffix positions (counting sort in shared memory), so
// that a tile visits the buckets within D mismatches of it and tests nothing.
template <bool WT>
__global__ void __launch_bounds__(CT_THREADS) ct_buckets(CtArgs a, int64_t B)
{
    constexpr int PASS = WT ? CT_SLOTS : 2 * CT_SLOTS;
    __shared__ uint32_t hist[1024], wtot[32];
    const int64_t pass = a.pass0 + blockIdx.x;
    const int64_t q0 = pass * PASS;
    const int nq = (int)min((int64_t)PASS, B - q0);
    uint32_t *recs = a.recs + (int64_t)blockIdx.x * a.rec_cap, *roff = a.roff + (int64_t)blockIdx.x * (a.n_pre + 1);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    hist[threadIdx.x] = 0;
    __syncthreads();
    for (int phase = 0; phase < 2; phase++) {
        for (int q = warp; q < nq * 4; q += CT_WARPS) {  // four warps a row
            const int64_t r = a.order ? (int64_t)a.order[q0 + (q >> 2)] : q0 + (q >> 2);
            const int n = a.cx[r];
            for (int i = (q & 3) * 32 + lane; i < n; i += 128) {
                uint32_t v = __ldg(a.bx + r * a.W + i);
                const uint32_t w = WT ? gkm_wt(a.wd, n, i) : 1u;
                for (int st = 0; st < a.sh.strands; st++) {
                    if (st) v = gkm_rc_word(v, a.sh.l);
                    uint32_t pre;
                    const uint32_t rec = ct_record<WT>(a.sh, v, q >> 2, w, &pre);
                    const uint32_t at = atomicAdd(&hist[pre], 1u);
                    if (phase) recs[at] = rec;
                }
            }
        }
        __syncthreads();
        if (phase) break;
        // exclusive scan: the buckets' first records
        const uint32_t c = hist[threadIdx.x];
        uint32_t x = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(GKM_FULL, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wtot[warp] = x;
        __syncthreads();
        if (warp == 0) {
            uint32_t t = wtot[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(GKM_FULL, t, o);
                if (lane >= o) t += y;
            }
            wtot[lane] = t;
        }
        __syncthreads();
        x = x - c + (warp ? wtot[warp - 1] : 0u);
        hist[threadIdx.x] = x;
        if ((int)threadIdx.x < a.n_pre) roff[threadIdx.x] = x;
        if ((int)threadIdx.x == a.n_pre - 1) roff[a.n_pre] = x + c;
        __syncthreads();
    }
}

// Items of (tile, pass of queries): a tile is the l-mers that agree outside the
// six suffix positions.  Windows whose other positions differ from the tile's at
// dp <= D places reach the suffixes within budget D - dp of their own: one row
// (budget 0), 19, 154 or 694.  Warps take buckets of windows of one budget:
// budgets 0 and 1 a window per lane, budgets 2 and 3 a window per warp with a
// lane on each bank (no two of its adds conflict).
//
// Shared counters: unweighted, one word per two queries (fields: CT_F0 ..);
// weighted, one word per query with 9 / 8 / 8 / 7 bits (entry: a byte each).
template <bool WT>
__global__ void __launch_bounds__(CT_THREADS, 1) count_tiles(CtArgs a)
{
    constexpr int PASS = WT ? CT_SLOTS : 2 * CT_SLOTS;
    extern __shared__ __align__(16) uint8_t ct_smem[];
    __shared__ uint2 l3[CT_R3 * 32];
    __shared__ uint32_t off_s[1025];
    __shared__ uint16_t ball_s[CT_BALL];
    // by tile parity: the entries that need a second look, and the fields' sum and
    // the adds made
    __shared__ uint16_t list_at[2][CT_LIST];
    __shared__ uint32_t list_w[2][CT_LIST];
    __shared__ int nlist[2];
    __shared__ unsigned long long chk[2][2];
    // counters [words][CT_ROWS], aligned to a word's plane so that a neighbour's
    // address is an exclusive or
    const uint32_t raw0 = (uint32_t)__cvta_generic_to_shared(ct_smem), cbase = (raw0 + 16383u) & ~16383u;
    uint32_t *cnt = (uint32_t *)(ct_smem + (cbase - raw0));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const CtShape sh = a.sh;
    const int D = sh.D;
    // a mask: byte offset and increment (0: none in this round)
    auto entry = [&](uint32_t e) -> uint2 {
        return (e >> 31) ? make_uint2((uint32_t)lane * 4u, 0u)
                         : make_uint2((e & 0xFFFu) * 4u, 1u << ct_shift<WT>((e >> 12) & 3u));
    };
    uint2 e2[CT_R2];
#pragma unroll
    for (int k = 0; k < CT_R2; k++) e2[k] = entry(a.lists[k * 32 + lane]);
    for (int k = threadIdx.x; k < CT_R3 * 32; k += CT_THREADS) l3[k] = entry(a.lists[CT_R2 * 32 + k]);
    const int pass = blockIdx.x % a.passes;  // grid: a multiple of passes
    const uint32_t *recs = a.recs + (int64_t)pass * a.rec_cap;
    uint32_t *recs_s = cnt + a.words * CT_ROWS;
    const uint32_t n_rec = a.roff[(int64_t)pass * (a.n_pre + 1) + a.n_pre];
    const bool staged = n_rec <= (uint32_t)a.rec_smem;
    if (staged)
        for (uint32_t k = threadIdx.x; k < n_rec; k += CT_THREADS) recs_s[k] = recs[k];
    auto load_rec = [&](uint32_t k) -> uint32_t { return staged ? recs_s[k] : __ldg(recs + k); };
    for (int k = threadIdx.x; k <= a.n_pre; k += CT_THREADS) off_s[k] = a.roff[(int64_t)pass * (a.n_pre + 1) + k];
    for (int k = threadIdx.x; k < CT_BALL; k += CT_THREADS) ball_s[k] = (uint16_t)a.ball[k];
    const int q0 = pass * PASS;
    const int nqp = min(PASS, a.nq - q0);
    const int words = WT ? nqp : (nqp + 1) >> 1;
    // tasks: buckets of budget 3 (in 8 parts), 2 (in 4 parts), 1, 0; nb[b] of them,
    // their masks from ball_s[sb[b]]
    const int nb3 = D >= 3 ? a.nball[D - 3] : 0, nb2 = D >= 2 ? a.nball[D - 2] : 0, nb1 = D >= 1 ? a.nball[D - 1] : 0,
              nb0 = a.nball[D];
    const int t3 = 8 * nb3, t2 = t3 + 4 * nb2, t1 = t2 + nb1, ntask = t1 + nb0;
    // the level-0 field (t = D) of a counter word; slow words have a window of the
    // query itself there, or (weighted) a count past its entry byte
    const uint32_t f0 = WT ? (D == 3 ? 0xFE000000u : D == 2 ? 0x01FE0000u : D == 1 ? 0x0001FE00u : 0x000001FFu)
                           : D == 3 ? 0x00E000E0u : D == 2 ? 0xF000F000u : D == 1 ? 0x0F000F00u : 0x001F001Fu;
    const uint32_t slow_mask = f0 | (WT ? 0x100u : 0u);

    // fields of a counter word (half)
    auto fields = [](uint32_t v, uint32_t (&c)[4]) {
        if (WT)
            c[0] = v & 0x1FFu, c[1] = (v >> 9) & 0xFFu, c[2] = (v >> 17) & 0xFFu, c[3] = v >> 25;
        else
            c[0] = v & 31u, c[1] = (v >> CT_F1) & 15u, c[2] = (v >> CT_F2) & 15u, c[3] = (v >> CT_F3) & 7u;
    };
    // a count's entry, and what the entry's fields do not hold
    auto clip = [](const uint32_t (&c)[4], uint32_t (&x)[4]) -> uint32_t {
        const uint32_t k0 = min(c[0], WT ? 255u : 31u), k1 = min(c[1], WT ? 255u : 15u), k2 = min(c[2], WT ? 255u : 15u),
                       k3 = min(c[3], WT ? 255u : 7u);
        x[0] = c[0] - k0, x[1] = c[1] - k1, x[2] = c[2] - k2, x[3] = c[3] - k3;
        return WT ? k0 | k1 << 8 | k2 << 16 | k3 << 24 : k0 | k1 << CT_F1 | k2 << CT_F2 | k3 << CT_F3;
    };
    // A count c (by t) of query q: its row's part of the query's self-kernel, sum
    // over its windows u of X_t(u) = sum over rows of X(level 0) X_t.
    auto self_part = [&](const uint32_t (&c)[4], int q) {
        const uint32_t n0 = D == 3 ? c[3] : D == 2 ? c[2] : D == 1 ? c[1] : c[0];
        if (n0)
#pragma unroll
            for (int t = 0; t < 4; t++)
                if (c[t]) atomicAdd(a.self + (a.r0 + q0 + q) * 4 + t, (unsigned long long)n0 * c[t]);
    };
    // A second look at counter word w, `at` = j * CT_ROWS + position of a tile, one
    // query per lane (unweighted: two neighbouring lanes share the word): the
    // query's self-kernel part and, weighted, a clipped count's entry and excess,
    // which goes to the group's list (full: to the SVs at once).  All lanes call it.
    auto look = [&](uint32_t tl, bool in, uint32_t at, uint32_t w) {
        const uint32_t j = at / CT_ROWS, q = WT ? j : 2 * j + (lane & 1);
        const uint32_t v = !in ? 0u : WT ? w : (w >> (16 * (lane & 1))) & 0xFFFFu;
        uint32_t c[4];
        fields(v, c);
        if (v & slow_mask) self_part(c, q);
        if constexpr (WT) {
            const bool over = (v & 0x100u) != 0;
            const uint32_t overs = __ballot_sync(GKM_FULL, over);
            if (!overs) return;
            uint32_t base = 0, x[4];
            if (lane == 0) base = atomicAdd(a.nexc, (unsigned)__popc(overs));
            const uint32_t pos = __shfl_sync(GKM_FULL, base, 0) + __popc(overs & ((1u << lane) - 1u));
            if (!over) return;
            const uint32_t row = tl * CT_ROWS + ct_phys(at & (CT_ROWS - 1));
            ((uint32_t *)(a.T + (size_t)row * a.rb))[q0 + q] = clip(c, x);
            if (pos < a.cap_exc) {
                a.exc[pos] = row | (unsigned long long)(q0 + q) << 22 | (unsigned long long)x[0] << 32;
            } else {
                const uint64_t ex[4] = {x[0], 0, 0, 0};
                ct_excess<WT>(a, sh.lmer(row), q0 + (int)q, ex, 0, 1);
            }
        }
    };
    // the words a tile queued, spread over the warps
    auto look_queued = [&](uint32_t tl, int par) {
        const int n = nlist[par];
        for (int k0 = 0; k0 < n; k0 += WT ? CT_THREADS : CT_THREADS / 2) {
            const int k = k0 + warp + CT_WARPS * (WT ? lane : lane >> 1);
            const bool in = k < n;
            if (!__any_sync(GKM_FULL, in)) continue;
            look(tl, in, in ? list_at[par][k] : 0u, in ? list_w[par][k] : 0u);
        }
    };

    if (n_rec == 0) return;  // rows of length 0 pad a batch: the gather reads nothing of them
    const int tiles = a.items / a.passes;
    int par = 0, queued = -1;  // the tile whose queued entries wait for their second look
    for (int tile = blockIdx.x / a.passes; tile < tiles; tile += gridDim.x / a.passes, par ^= 1) {
    if (threadIdx.x == 0) {
        nlist[par] = 0;
        chk[par][0] = chk[par][1] = 0;
    }
    for (int k = threadIdx.x; k < words * CT_ROWS / 4; k += CT_THREADS) ((uint4 *)cnt)[k] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    if (queued >= 0) look_queued(queued, par ^ 1);

    // counts the windows of queries qa .. qb - 1 (safe: the recount of two
    // queries with 32-bit counters, plane (q - qa) * 4 + t; else all)
    auto count_buckets = [&](auto SAFE, int qa, int qb) -> unsigned long long {
        constexpr bool safe = decltype(SAFE)::value;
        unsigned long long adds = 0;
        // counter address, increment of one window of weight 1 (0: not counted)
        auto where = [&](uint32_t rec, uint32_t &sa, uint32_t &inc) {
            const uint32_t at = rec & 0x7FFFu;
            if (safe) {
                const int q = WT ? at / CT_ROWS : 2 * (at / CT_ROWS) + ((rec >> 15) & 1u);
                const bool in = q >= qa && q < qb;
                sa = cbase + ((in ? (q - qa) * 4 * CT_ROWS + (at & (CT_ROWS - 1)) : 0u) << 2);
                inc = in ? rec >> 16 : 0u;
            } else {
                sa = cbase + (at << 2);
                inc = WT ? rec >> 16 : 1u << ((rec >> 11) & 16u);
            }
        };
        // add at the neighbour with byte offset x, field increment f = 1 << ct_shift(t)
        auto add = [&](uint32_t sa, uint32_t x, uint32_t f, uint32_t inc) {
            if (safe) {
                const uint32_t t = f == 1u ? 0u : f == 1u << ct_shift<WT>(1) ? 1u : f == 1u << ct_shift<WT>(2) ? 2u : 3u;
                if (f && inc) ct_add((sa ^ x) + t * (4 * CT_ROWS), inc);
            } else {
                ct_add(sa ^ x, f * inc);
            }
        };
        // lane j: the warp's j-th task (at most 14), its bucket's records
        uint32_t my_beg = 0, my_end = 0, my_kind = 0;
        {
            const int task = warp + CT_WARPS * lane;
            if (task < ntask) {
                int k;
                if (task < t3) {
                    my_kind = 3u | (task & 7) << 2;
                    k = task >> 3;
                } else if (task < t2) {
                    my_kind = 2u | ((task - t3) & 3) << 2;
                    k = nb3 + ((task - t3) >> 2);
                } else {
                    my_kind = task < t1 ? 1u : 0u;
                    k = nb3 + nb2 + task - t2;
                }
                const uint32_t pre = (uint32_t)tile ^ ball_s[k];
                my_beg = off_s[pre];
                my_end = off_s[pre + 1];
            }
        }
        uint32_t c = __shfl_sync(GKM_FULL, my_beg, 0), end = __shfl_sync(GKM_FULL, my_end, 0);
        uint32_t rec = c + lane < end ? load_rec(c + lane) : 0u;
        const int mine = (ntask - warp + CT_WARPS - 1) / CT_WARPS;
        for (int j0 = 0; j0 < mine; j0++) {
            const uint32_t kind = __shfl_sync(GKM_FULL, my_kind, j0);
            const int b = kind & 3, part = kind >> 2;
            // the next task's records, in flight while this one is counted
            const int jn = j0 + 1 < mine ? j0 + 1 : j0;
            const uint32_t nc = __shfl_sync(GKM_FULL, my_beg, jn), nend = __shfl_sync(GKM_FULL, my_end, jn);
            const uint32_t nrec = nc + lane < nend ? load_rec(nc + lane) : 0u;
            while (c < end) {
                const int n = min(32u, end - c);
                uint32_t sa, inc;
                where(rec, sa, inc);
                const uint32_t w = rec >> 16;
                if (b <= 1) {
                    if (lane < n) {
                        if (b == 0) {
                            add(sa, 0u, 1u, inc);
                            adds += w;
                        } else {
                            add(sa, 0u, 1u << ct_shift<WT>(1), inc);
#pragma unroll
                            for (int pos = 0; pos < 6; pos++)
#pragma unroll
                                for (uint32_t d = 1; d < 4; d++) add(sa, ct_phys(d << (2 * pos)) << 2, 1u, inc);
                            adds += 19u * w;
                        }
                    }
                } else if (b == 2) {
                    if (part == 0 && lane < n) adds += 154u * w;
                    for (int j = part; j < n; j += 4) {
                        const uint32_t ss = __shfl_sync(GKM_FULL, sa, j), si = __shfl_sync(GKM_FULL, inc, j);
#pragma unroll
                        for (int k = 0; k < CT_R2; k++) add(ss, e2[k].x, e2[k].y, si);
                    }
                } else {
                    if (part == 0 && lane < n) adds += 694u * w;
                    for (int j = part; j < n; j += 8) {
                        const uint32_t ss = __shfl_sync(GKM_FULL, sa, j), si = __shfl_sync(GKM_FULL, inc, j);
#pragma unroll 2
                        for (int k = 0; k < CT_R3; k++) {
                            const uint2 e = l3[k * 32 + lane];
                            add(ss, e.x, e.y, si);
                        }
                    }
                }
                c += 32;
                if (c < end) rec = c + lane < end ? load_rec(c + lane) : 0u;
            }
            c = nc, end = nend, rec = nrec;
        }
        return adds;
    };

    unsigned long long adds = count_buckets(std::false_type{}, 0, nqp);
    __syncthreads();
    // The tile's entries (row by row; a thread takes four neighbouring counters
    // of every word), the words that need more queued, and the fields' sum: it
    // equals the adds made unless some field carried into the next.
    uint8_t *T = a.T + (size_t)tile * CT_ROWS * a.rb + q0 * (WT ? 4 : 2);
    {
        uint32_t fa = 0, fb = 0;
#pragma unroll
        for (int i = 0; i < CT_ROWS / CT_THREADS; i++) {
            const uint32_t p = i * CT_THREADS + threadIdx.x;
            uint32_t o[CT_SLOTS], slow = 0;
#pragma unroll
            for (int j = 0; j < CT_SLOTS; j++) {
                const uint32_t w = j < words ? cnt[j * CT_ROWS + p] : 0u;
                if (WT) {
                    fa = __dp4a(w >> 9, 0x00010101u, fa) + (w & 0x1FFu);
                    o[j] = (w & 0xFFu) | ((w >> 1) & 0xFFFFFF00u);
                } else {
                    // t = 0 and 1 are the bytes' low fields; t = 3 and 2 the high
                    // ones, 32 and 16 times too large
                    fa = __dp4a(w & 0x0F1F0F1Fu, 0x01010101u, fa);
                    fb = __dp4a(w & 0xF0E0F0E0u, 0x02010201u, fb);
                    o[j] = w;
                }
                slow |= (uint32_t)((w & slow_mask) != 0) << j;
            }
            uint4 *out = (uint4 *)(T + (size_t)ct_phys(p) * a.rb);
            out[0] = make_uint4(o[0], o[1], o[2], o[3]);
            out[1] = make_uint4(o[4], o[5], o[6], o[7]);
            for (; slow; slow &= slow - 1) {
                const int j = __ffs(slow) - 1, n = atomicAdd(&nlist[par], 1);
                if (n < CT_LIST) {
                    list_at[par][n] = (uint16_t)(j * CT_ROWS + p);
                    list_w[par][n] = cnt[j * CT_ROWS + p];
                }
            }
        }
        unsigned long long sum = fa + (fb >> 5);
#pragma unroll
        for (int o2 = 16; o2; o2 >>= 1) {
            sum += __shfl_xor_sync(GKM_FULL, sum, o2);
            adds += __shfl_xor_sync(GKM_FULL, adds, o2);
        }
        if (lane == 0) {
            atomicAdd(&chk[par][0], sum);
            atomicAdd(&chk[par][1], adds);
        }
    }
    __syncthreads();

    queued = -1;
    if (chk[par][0] == chk[par][1]) {
        if (nlist[par] <= CT_LIST) {
            queued = tile;
        } else {  // every word
            for (int k0 = 0; k0 < words * CT_ROWS; k0 += WT ? CT_THREADS : CT_THREADS / 2) {
                const int k = k0 + (WT ? threadIdx.x : threadIdx.x >> 1);
                look(tile, true, k, cnt[k]);
            }
            __syncthreads();
        }
    } else {
        // a field overflowed: 32-bit counters, two queries x four levels at a time
        for (int qa = 0; qa < nqp; qa += 2) {
            const int nb = min(2, nqp - qa);
            __syncthreads();
            for (int k = threadIdx.x; k < 4 * nb * CT_ROWS; k += CT_THREADS) cnt[k] = 0;
            __syncthreads();
            count_buckets(std::true_type{}, qa, qa + nb);
            __syncthreads();
            for (int p = threadIdx.x; p < CT_ROWS; p += CT_THREADS) {
                const uint32_t suf = ct_phys(p);
                for (int q = 0; q < nb; q++) {
                    const uint32_t *cq = cnt + q * 4 * CT_ROWS + p;
                    const uint32_t c[4] = {cq[0], cq[CT_ROWS], cq[2 * CT_ROWS], cq[3 * CT_ROWS]};
                    self_part(c, qa + q);
                    uint32_t x[4];
                    const uint32_t v = clip(c, x);
                    if (WT)
                        ((uint32_t *)(T + (size_t)suf * a.rb))[qa + q] = v;
                    else
                        ((uint16_t *)(T + (size_t)suf * a.rb))[qa + q] = (uint16_t)v;
                    const uint64_t ex[4] = {x[0], x[1], x[2], x[3]};
                    if (x[0] | x[1] | x[2] | x[3]) ct_excess<WT>(a, sh.lmer(tile * CT_ROWS + suf), q0 + qa + q, ex, 0, 1);
                }
            }
        }
        __syncthreads();
    }
    }
    if (queued >= 0) look_queued(queued, par ^ 1);
}

// The queued excess counts of a group (weighted: level t = 0), eight lanes each.
__global__ void spill_excess(CtArgs a)
{
    const unsigned n = min(*a.nexc, a.cap_exc);
    for (unsigned k = (blockIdx.x * blockDim.x + threadIdx.x) >> 3; k < n; k += (gridDim.x * blockDim.x) >> 3) {
        const unsigned long long e = a.exc[k];
        const uint64_t ex[4] = {e >> 32, 0, 0, 0};
        ct_excess<true>(a, a.sh.lmer((uint32_t)e & 0x3FFFFFu), (int)((e >> 22) & 0x3FFu), ex, threadIdx.x & 7, 8);
    }
}

// ---------------------------------------------------------------------------
// 2. gather
// ---------------------------------------------------------------------------

__device__ __forceinline__ void ct_fa(uint32_t &s, uint32_t &c, uint32_t a, uint32_t b)
{
    const uint32_t x = s;
    s = x ^ a ^ b;
    c = (x & a) | (x & b) | (a & b);
}

// acc[t] (two 16-bit sums, a query each) += the fields of entry word x times 2^p
__device__ __forceinline__ void ct_unpack(uint32_t *acc, uint32_t x, int p)
{
    acc[0] += (x & 0x001F001Fu) << p;
    acc[1] += ((x >> CT_F1) & 0x000F000Fu) << p;
    acc[2] += ((x >> CT_F2) & 0x000F000Fu) << p;
    acc[3] += ((x >> CT_F3) & 0x00070007u) << p;
}

// Epilogue of four queries j0 .. of SV s: their counts n[q][t], the excess counts
// where `dirty` has their bits (read and cleared), then the SV's terms added to
// part[q] or K_raw written.
template <bool RAW>
__device__ __forceinline__ void ct_finish(const CtArgs &a, int64_t s, int j0, const uint32_t (&n)[4][4], uint32_t dirty,
                                          const double *inv_dx, double z, double c, double (&part)[4])
{
    ulonglong2 ex[4];
    if (dirty) {
        ulonglong2 *g = (ulonglong2 *)a.C + s * a.qg + j0;
#pragma unroll
        for (int q = 0; q < 4; q++) ex[q] = (dirty >> q) & 1u ? g[q] : make_ulonglong2(0, 0);
#pragma unroll
        for (int q = 0; q < 4; q++)
            if ((dirty >> q) & 1u) g[q] = make_ulonglong2(0, 0);
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        if (j0 + q >= a.nq) break;
        uint64_t v[4] = {n[q][0], n[q][1], n[q][2], n[q][3]};
        if (dirty) {
            v[0] += (uint32_t)ex[q].x;
            v[1] += ex[q].x >> 32;
            v[2] += (uint32_t)ex[q].y;
            v[3] += ex[q].y >> 32;
        }
        double k = 0.0;  // level 0 first
#pragma unroll
        for (int t = 3; t >= 0; t--) k += a.h[t] * (double)(int64_t)v[t];
        if (RAW) {
            const int64_t row = ct_row_of(a, j0 + q);
            if (a.diag_offset < 0 || s >= a.diag_offset + row) a.raw[row * a.S + s] = k;
        } else {
            const double kn = k * inv_dx[j0 + q] * z;
            part[q] = c * (a.rbf ? exp(a.gamma * (kn - 1.0)) : kn);
        }
    }
}

// RB-byte rows, 16 bytes per lane, RB / 16 lanes per SV; persistent blocks take
// SVs round robin in gather order (long SVs first).  Bound by L2 and HBM latency
// times bandwidth: every lane keeps two stages of eight row pieces in flight in
// its own slots of shared memory (asynchronous copies; nothing is shared between
// lanes, so no barriers) while it adds a third.
template <int RB, bool WT, bool RAW>
__global__ void __launch_bounds__(G_THREADS, WT ? G_BLOCKS_W : G_BLOCKS) gather_kernel(CtArgs a)
{
    constexpr int NQ = WT ? 4 : 8;  // queries a lane owns
    constexpr int LPG = RB / 16, GPB = G_THREADS / LPG, QG = LPG * NQ;
    __shared__ uint4 rows_s[4 * G_THREADS];
    __shared__ double inv_dx[QG];
    __shared__ uint32_t empty_s[QG];  // a query without windows (its columns may hold another group's counts)
    __shared__ double part_s[G_THREADS / 32][QG];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = threadIdx.x % LPG, j0 = sub * NQ;
    bool some = false;
    for (int j = threadIdx.x; j < QG; j += G_THREADS) {
        inv_dx[j] = 0.0;
        empty_s[j] = 1;
        if (j < a.nq) {
            const int64_t row = ct_row_of(a, j);
            empty_s[j] = a.cx[row] <= 0;
            some |= a.cx[row] > 0;
            double k = 0.0;
            // both strands of every l-mer counted (no folding): each pair twice
            const int twice = !a.sh.fold && a.sh.strands == 2;
            for (int t = 3; t >= 0; t--) k += a.h[t] * (double)(a.self[(a.r0 + j) * 4 + t] >> twice);
            if (a.diag && blockIdx.x == 0) a.diag[row] = k;
            inv_dx[j] = a.inv_dx ? a.inv_dx[row] : a.normalize ? 1.0 / sqrt(fmax(k, 1e-20)) : 1.0;
        }
    }
    for (int j = threadIdx.x; j < G_THREADS / 32 * QG; j += G_THREADS) (&part_s[0][0])[j] = 0.0;
    some = __syncthreads_or(some);
    const uint8_t *base = a.T + sub * 16;
    const int64_t rounds = (a.S + (int64_t)gridDim.x * GPB - 1) / ((int64_t)gridDim.x * GPB);
    for (int64_t it = 0; it < rounds; it++) {
        const int64_t g = (it * gridDim.x + blockIdx.x) * GPB + threadIdx.x / LPG;
        const bool live = g < a.S;
        const int64_t s = live ? a.perm[g] : 0;
        const uint32_t p0 = live ? a.goff[g] : 0;
        uint32_t nst = live ? (a.goff[g + 1] - p0) >> 3 : 0;
        if (!some || (RAW && a.diag_offset >= 0 && s < a.diag_offset + a.r0)) nst = 0;  // nothing there, or wholly below the diagonal
        uint32_t id[8];
        // stage k: its row pieces into slot `at`, and the next stage's row numbers
        auto load_ids = [&](uint32_t k) {
            if (k >= nst) return;
            const uint4 i0 = __ldg((const uint4 *)(a.ids + p0) + 2 * k), i1 = __ldg((const uint4 *)(a.ids + p0) + 2 * k + 1);
            id[0] = i0.x, id[1] = i0.y, id[2] = i0.z, id[3] = i0.w;
            id[4] = i1.x, id[5] = i1.y, id[6] = i1.z, id[7] = i1.w;
        };
        load_ids(0);
        uint32_t acc[16];  // WT: [query][t]; else [word][t], two 16-bit sums each
#pragma unroll
        for (int k = 0; k < 16; k++) acc[k] = 0;
        // 16 bits per query: carry-save adders over the 32-bit words sum rows with
        // ~2 logic operations per row and word whatever the fields; every 32 rows the
        // carries of weight 32 are added field by field into 16-bit sums (31 x 2,048
        // rows < 2^16).  (p8, p16: carries waiting for the second of a pair)
        uint32_t ones[4] = {}, twos[4] = {}, fours[4] = {}, eights[4] = {}, s16[4] = {}, p8[4] = {}, p16[4] = {};
        for (uint32_t k = 0; k < nst; k++) {
            uint4 r[8];
#pragma unroll
            for (int j = 0; j < 8; j++) r[j] = __ldg((const uint4 *)(base + (size_t)id[j] * RB));
            uint2 wt = make_uint2(0, 0);
            if (WT) wt = __ldg((const uint2 *)(a.wts + p0) + k);
            load_ids(k + 1);
            if constexpr (!WT) {
                uint32_t f[2][4];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint4 r0 = r[4 * h], r1 = r[4 * h + 1], r2 = r[4 * h + 2], r3 = r[4 * h + 3];
                    const uint32_t x0[4] = {r0.x, r0.y, r0.z, r0.w}, x1[4] = {r1.x, r1.y, r1.z, r1.w},
                                   x2[4] = {r2.x, r2.y, r2.z, r2.w}, x3[4] = {r3.x, r3.y, r3.z, r3.w};
#pragma unroll
                    for (int w = 0; w < 4; w++) {
                        uint32_t t0, t1;
                        ct_fa(ones[w], t0, x0[w], x1[w]);
                        ct_fa(ones[w], t1, x2[w], x3[w]);
                        ct_fa(twos[w], f[h][w], t0, t1);
                    }
                }
#pragma unroll
                for (int w = 0; w < 4; w++) {
                    uint32_t e;
                    ct_fa(fours[w], e, f[0][w], f[1][w]);
                    if ((k & 1) == 0) {
                        p8[w] = e;
                        continue;
                    }
                    uint32_t c;
                    ct_fa(eights[w], c, p8[w], e);
                    p8[w] = 0;
                    if ((k & 2) == 0) {
                        p16[w] = c;
                    } else {
                        uint32_t x;
                        ct_fa(s16[w], x, p16[w], c);
                        p16[w] = 0;
                        ct_unpack(acc + 4 * w, x, 0);
                    }
                }
            } else {
                // four bytes per query: the level bytes of four rows side by side
                // (byte permutes), multiplied by the rows' window weights and
                // summed by dp4a into 32 bits
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint32_t ww = h ? wt.y : wt.x;
                    const uint4 r0 = r[4 * h], r1 = r[4 * h + 1], r2 = r[4 * h + 2], r3 = r[4 * h + 3];
                    const uint32_t w0[4] = {r0.x, r0.y, r0.z, r0.w}, w1[4] = {r1.x, r1.y, r1.z, r1.w},
                                   w2[4] = {r2.x, r2.y, r2.z, r2.w}, w3[4] = {r3.x, r3.y, r3.z, r3.w};
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const uint32_t x0 = __byte_perm(w0[q], w1[q], 0x5140), x1 = __byte_perm(w0[q], w1[q], 0x7362);
                        const uint32_t y0 = __byte_perm(w2[q], w3[q], 0x5140), y1 = __byte_perm(w2[q], w3[q], 0x7362);
                        acc[4 * q] = __dp4a(__byte_perm(x0, y0, 0x5410), ww, acc[4 * q]);
                        acc[4 * q + 1] = __dp4a(__byte_perm(x0, y0, 0x7632), ww, acc[4 * q + 1]);
                        acc[4 * q + 2] = __dp4a(__byte_perm(x1, y1, 0x5410), ww, acc[4 * q + 2]);
                        acc[4 * q + 3] = __dp4a(__byte_perm(x1, y1, 0x7632), ww, acc[4 * q + 3]);
                    }
                }
            }
        }
        if constexpr (!WT) {
#pragma unroll
            for (int w = 0; w < 4; w++) {
                // the waiting carries, then the planes below 32
                uint32_t x = eights[w] & p8[w], y;
                eights[w] ^= p8[w];
                ct_fa(s16[w], y, p16[w], x);
                ct_unpack(acc + 4 * w, y, 0);
#pragma unroll
                for (int k = 0; k < 4; k++) acc[4 * w + k] <<= 5;
                ct_unpack(acc + 4 * w, ones[w], 0);
                ct_unpack(acc + 4 * w, twos[w], 1);
                ct_unpack(acc + 4 * w, fours[w], 2);
                ct_unpack(acc + 4 * w, eights[w], 3);
                ct_unpack(acc + 4 * w, s16[w], 4);
            }
        }
        // epilogue, four queries at a time (the sums wait in the lane's slots, so
        // that the loop above has the registers).  Weighted: two lanes share a byte
        // of dirty bits.
        const int64_t dat = s * a.qg + j0;
        uint8_t *db = (uint8_t *)a.dirty + (dat >> 3);
        const uint32_t dirty = live ? (*db >> (dat & 7)) & ((1u << NQ) - 1u) : 0u;
        const double z = RAW || !live ? 0.0 : a.inv_ds[s], coef = RAW || !live ? 0.0 : a.coef[s];
        __syncwarp();
        if (dirty) *db = 0;
        uint4 *sums = rows_s + threadIdx.x;
#pragma unroll
        for (int k = 0; k < 4; k++) sums[k * G_THREADS] = make_uint4(acc[4 * k], acc[4 * k + 1], acc[4 * k + 2], acc[4 * k + 3]);
#pragma unroll 1
        for (int w = 0; w < NQ / 4; w++) {
            uint32_t n[4][4];
#pragma unroll
            for (int k = 0; k < (WT ? 4 : 2); k++) {
                const uint4 v = sums[((WT ? 0 : 2 * w) + k) * G_THREADS];
                if (WT) {
                    n[k][0] = v.x, n[k][1] = v.y, n[k][2] = v.z, n[k][3] = v.w;
                } else {  // a word: two queries
                    n[2 * k][0] = v.x & 0xFFFFu, n[2 * k][1] = v.y & 0xFFFFu, n[2 * k][2] = v.z & 0xFFFFu, n[2 * k][3] = v.w & 0xFFFFu;
                    n[2 * k + 1][0] = v.x >> 16, n[2 * k + 1][1] = v.y >> 16, n[2 * k + 1][2] = v.z >> 16, n[2 * k + 1][3] = v.w >> 16;
                }
            }
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (empty_s[j0 + 4 * w + q]) n[q][0] = n[q][1] = n[q][2] = n[q][3] = 0;
            double part[4] = {0.0, 0.0, 0.0, 0.0};
            if (live) ct_finish<RAW>(a, s, j0 + 4 * w, n, (dirty >> (4 * w)) & 15u, inv_dx, z, coef, part);
            if (!RAW) {
                // the warp's SVs, in a fixed order
#pragma unroll
                for (int q = 0; q < 4; q++) {
#pragma unroll
                    for (int o = LPG; o < 32; o <<= 1) part[q] += __shfl_xor_sync(GKM_FULL, part[q], o);
                    if (lane < LPG) part_s[warp][j0 + 4 * w + q] += part[q];
                }
            }
        }
    }
    if (RAW) return;
    __syncthreads();
    for (int j = threadIdx.x; j < QG; j += G_THREADS) {
        double t = 0.0;
        for (int k = 0; k < G_THREADS / 32; k++) t += part_s[k][j];
        a.partial[(int64_t)blockIdx.x * QG + j] = t;
    }
}

// scores of every group: the blocks' partial sums in a fixed order, 32 slices
__global__ void ct_scores(const double *__restrict__ partial, int nblk, int qg, const int32_t *__restrict__ order,
                          int64_t B, double bias, double *__restrict__ scores)
{
    __shared__ double red[32][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = qg < 32 ? qg : 32;
    const int parts = qg / per;
    const int64_t grp = blockIdx.x / parts;
    const int j = (int)(blockIdx.x % parts) * per + lane;
    double t = 0.0;
    if (lane < per)
        for (int k = warp; k < nblk; k += 32) t += partial[(grp * nblk + k) * qg + j];
    red[warp][lane] = t;
    __syncthreads();
    if (warp == 0 && lane < per) {
        t = 0.0;
        for (int k = 0; k < 32; k++) t += red[k][lane];
        const int64_t r = grp * qg + j;
        if (r < B) scores[order ? (int64_t)order[r] : r] = t + bias;
    }
}

// ---------------------------------------------------------------------------
// gather lists (built with the index)
// ---------------------------------------------------------------------------

__global__ void ct_perm_keys(const int32_t *__restrict__ counts, int64_t S, uint32_t *__restrict__ keys,
                             uint32_t *__restrict__ vals)
{
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= S) return;
    keys[s] = 0xFFFFu - (uint32_t)min(counts[s], 0xFFFF);
    vals[s] = (uint32_t)s;
}

__global__ void ct_padded(const int32_t *__restrict__ counts, const uint32_t *__restrict__ perm, int64_t S,
                          uint32_t *__restrict__ out)
{
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g <= S) out[g] = g < S ? ((uint32_t)counts[perm[g]] + 7u) & ~7u : 0u;
}

// One SV per block: its windows' table rows in rising order (neighbouring SVs
// then sweep the table together, which keeps the rows they share in L2), padded
// with the zero row.
__global__ void ct_rows(CtShape sh, const uint32_t *__restrict__ fwd, const int32_t *__restrict__ counts, int64_t W,
                        const uint32_t *__restrict__ perm, const uint32_t *__restrict__ goff, uint32_t zero_row,
                        const uint8_t *__restrict__ wd, uint32_t *__restrict__ ids, uint8_t *__restrict__ wts)
{
    extern __shared__ uint32_t key[];
    const int64_t g = blockIdx.x, s = perm[g];
    const int n = counts[s];
    int m = 1;
    while (m < n) m <<= 1;
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        uint32_t k = 0xFFFFFFFFu;
        if (i < n) {
            uint32_t u = fwd[s * W + i];
            if (sh.fold && ((u >> (2 * sh.mid + 1)) & 1u)) u = gkm_rc_word(u, sh.l);
            k = sh.row(u) << 8 | (wd ? gkm_wt(wd, n, i) : 0u);
        }
        key[i] = k;
    }
    for (int k = 2; k <= m; k <<= 1)
        for (int j = k >> 1; j; j >>= 1) {
            __syncthreads();
            for (int i = threadIdx.x; i < m; i += blockDim.x) {
                const int o = i ^ j;
                if (o > i) {
                    const uint32_t x = key[i], y = key[o];
                    if ((x > y) == ((i & k) == 0)) {
                        key[i] = y;
                        key[o] = x;
                    }
                }
            }
        }
    __syncthreads();
    const uint32_t b = goff[g], e = goff[g + 1];
    for (uint32_t i = threadIdx.x; i < e - b; i += blockDim.x) {
        const bool in = (int)i < n;
        ids[b + i] = in ? key[i] >> 8 : zero_row;
        if (wts) wts[b + i] = in ? (uint8_t)(key[i] & 0xFFu) : 0;
    }
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

static CtShape ct_shape(const gkm_index *ix)
{
    CtShape sh;
    sh.l = ix->spec.l;
    sh.D = ix->spec.dmax;
    sh.strands = ix->strands;
    sh.fold = ix->strands == 2 && (sh.l & 1);
    sh.mid = sh.l / 2;
    return sh;
}

static int64_t ct_table_rows(const gkm_index *ix)
{
    const CtShape sh = ct_shape(ix);
    return sh.fold ? (int64_t)1 << (2 * sh.l - 1) : (int64_t)1 << (2 * sh.l);
}

// Neighbour masks of the six suffix positions with 0 .. b mismatches for b = 2,
// 3, arranged so that lane k of every round holds a mask of bank class k:
// position | t << 12, or bit 31.
static void ct_lists(uint32_t *out)
{
    const int rounds[4] = {0, 0, CT_R2, CT_R3};
    uint32_t *p = out;
    for (int b = 2; b <= 3; b++) {
        int used[32] = {0};
        for (int k = 0; k < rounds[b] * 32; k++) p[k] = 0x80000000u;
        for (uint32_t x = 0; x < CT_ROWS; x++) {
            const int m = __builtin_popcount((x | (x >> 1)) & 0x555u), cls = ct_phys(x) & 31;
            if (m <= b) p[32 * used[cls]++ + cls] = ct_phys(x) | (uint32_t)(b - m) << 12;
        }
        p += rounds[b] * 32;
    }
}

// Masks of n positions (l - 6 of them) with m mismatches; returns how many.
static int ct_ball(int n, int m, uint32_t *out)
{
    int k = 0;
    for (uint32_t x = 0; x < (1u << (2 * n)); x++)
        if (__builtin_popcount((x | (x >> 1)) & 0x55555555u) == m) {
            if (out) out[k] = x;
            k++;
        }
    return k;
}

int gkm_ct_build(gkm_index *ix, const uint32_t *fwd, const int32_t *counts, cudaStream_t st)
{
    ix->ct_ids = nullptr;
    const CtShape sh = ct_shape(ix);
    // 16-bit gather sums (31 x windows) and the in-block sort bound the SV rows;
    // weighted entries are bytes: three windows of the largest weight fit
    if (sh.l < 8 || sh.l > 11 || sh.D < 0 || sh.D > 3 || ix->W > 2048 || ix->S < 64 || ix->wmax > 85) return GKM_OK;
    const int64_t S = ix->S;
    uint32_t *k0 = nullptr, *k1 = nullptr, *v1 = nullptr;
    int s = GKM_OK;
    uint32_t total = 0;
    do {
        if (cudaMalloc(&ix->ct_perm, sizeof(uint32_t) * S) != cudaSuccess ||
            cudaMalloc(&ix->ct_off, sizeof(uint32_t) * (S + 1)) != cudaSuccess ||
            cudaMalloc(&ix->ct_lists, sizeof(uint32_t) * (32 * (CT_R2 + CT_R3) + CT_BALL)) != cudaSuccess ||
            cudaMallocAsync(&k0, sizeof(uint32_t) * (S + 1), st) != cudaSuccess ||
            cudaMallocAsync(&k1, sizeof(uint32_t) * (S + 1), st) != cudaSuccess ||
            cudaMallocAsync(&v1, sizeof(uint32_t) * (S + 1), st) != cudaSuccess) {
            s = gkm_fail(GKM_ERR_OOM, "gather lists");
            break;
        }
        uint32_t lists[32 * (CT_R2 + CT_R3) + CT_BALL] = {};
        ct_lists(lists);
        for (int m = 0, k = 32 * (CT_R2 + CT_R3); m <= sh.D; m++) k += ct_ball(sh.l - 6, m, lists + k);
        if (cudaMemcpyAsync(ix->ct_lists, lists, sizeof(lists), cudaMemcpyHostToDevice, st) != cudaSuccess) {
            s = gkm_cuda_status(cudaGetLastError(), "mask lists");
            break;
        }
        const unsigned nb = (unsigned)((S + 256) / 256);
        ct_perm_keys<<<nb, 256, 0, st>>>(counts, S, k0, ix->ct_perm);
        uint32_t *keys = k0, *vals = ix->ct_perm, *kt = k1, *vt = v1;
        if ((s = gkm_radix_sort(keys, vals, kt, vt, S, 16, st)) != GKM_OK) break;
        if (vals != ix->ct_perm) cudaMemcpyAsync(ix->ct_perm, vals, sizeof(uint32_t) * S, cudaMemcpyDeviceToDevice, st);
        ct_padded<<<nb, 256, 0, st>>>(counts, ix->ct_perm, S, k0);
        if ((s = gkm_scan_exclusive(k0, ix->ct_off, S + 1, st)) != GKM_OK) break;
        if (cudaMemcpyAsync(&total, ix->ct_off + S, sizeof(uint32_t), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess) {
            s = gkm_cuda_status(cudaGetLastError(), "gather lists");
            break;
        }
        ix->ct_entries = total;
        if (cudaMalloc(&ix->ct_ids, sizeof(uint32_t) * ((size_t)total + 8)) != cudaSuccess ||
            (ix->spec.weighted && cudaMalloc(&ix->ct_wts, (size_t)total + 8) != cudaSuccess)) {
            s = gkm_fail(GKM_ERR_OOM, "gather lists");
            break;
        }
        int m = 1;
        while (m < ix->W) m <<= 1;
        ct_rows<<<(unsigned)S, m >= 512 ? 256 : m >= 64 ? m / 2 : 32, sizeof(uint32_t) * m, st>>>(
            sh, fwd, counts, ix->W, ix->ct_perm, ix->ct_off, (uint32_t)ct_table_rows(ix),
            ix->spec.weighted ? ix->spec.wd : nullptr, ix->ct_ids, ix->ct_wts);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) s = gkm_cuda_status(e, "gather lists");
        ix->bytes += (int64_t)sizeof(uint32_t) * (2 * S + total) + (ix->ct_wts ? total : 0);
    } while (0);
    cudaFreeAsync(k0, st);
    cudaFreeAsync(k1, st);
    cudaFreeAsync(v1, st);
    return s;
}

void gkm_ct_free(gkm_index *ix)
{
    cudaFree(ix->ct_ids);
    cudaFree(ix->ct_wts);
    cudaFree(ix->ct_off);
    cudaFree(ix->ct_perm);
    cudaFree(ix->ct_lists);
}

// The row width of a call: 32 bytes for batches that fit a few groups of them,
// else 128.
struct CtPlan {
    int rb, qg, blocks;
    int64_t groups, rows, table, c, dirty, self, nexc, exc, partial, bytes;
    int pass, passes;         // queries of a count_tiles pass, passes of a full group
    int64_t rec_cap, chunk;   // window records of a pass, groups bucketed at a time
    int64_t recs, roff;
    int n_pre;
};

static CtPlan ct_plan(const gkm_index *ix, int64_t B, int64_t W)
{
    CtPlan p = {};
    const int wt = ix->spec.weighted ? 4 : 2;
    // 32 queries a group: 64- or (weighted) 128-byte rows; the narrowest rows that
    // hold a smaller batch
    p.rb = wt * 32;
    while (p.rb > 32 && p.rb / wt / 2 >= B) p.rb /= 2;
    p.qg = p.rb / wt;
    p.groups = (B + p.qg - 1) / p.qg;
    p.rows = ct_table_rows(ix);
    const int per_sm = ix->spec.weighted ? G_BLOCKS_W : G_BLOCKS;
    p.blocks = gkm_query_blocks() * per_sm;
    auto up = [](int64_t n) { return (n + 255) & ~(int64_t)255; };
    p.table = up((p.rows + 2) * p.rb);
    p.self = up(B * 4 * 8);
    p.nexc = up(p.groups * 4);
    p.exc = ix->spec.weighted ? up(8 * CT_EXC * (B < p.qg ? B : p.qg)) : 0;
    p.dirty = up(ix->S * p.qg / 8 + 8);
    p.c = up(ix->S * p.qg * 16);
    p.partial = up(p.groups * gkm_sm_count() * per_sm * p.qg * 8);  // (a grid limit only lowers p.blocks)
    // windows by bucket: the groups whose records fit 64 MB, at least one
    p.pass = ix->spec.weighted ? CT_SLOTS : 2 * CT_SLOTS;
    p.passes = p.qg / p.pass > 0 ? p.qg / p.pass : 1;
    p.n_pre = 1 << (2 * (ix->spec.l - 6));
    p.rec_cap = (int64_t)p.pass * W * ix->strands;
    p.chunk = (64LL << 20) / (4 * p.rec_cap * p.passes);
    if (p.chunk < 1) p.chunk = 1;
    if (p.chunk > p.groups) p.chunk = p.groups;
    p.recs = up(4 * p.rec_cap * p.passes * p.chunk);
    p.roff = up(4 * (int64_t)(p.n_pre + 1) * p.passes * p.chunk);
    p.bytes = p.table + p.self + p.nexc + p.dirty + p.c + p.partial + p.recs + p.roff + p.exc;
    return p;
}

// Microseconds of a query, measured on B200 (l = 11, 300 .. 72,000 SVs of 200 ..
// 500 bp, 1 .. 1,024 rows of 30 .. 2,000 bp).  Count tables: a tile pass on one SM
// costs CT_ITEM_US plus CT_WINDOW_US per window of its longest row, the gather
// reads the SVs' table rows at CT_GATHER_BYTES_US.  Index walk: its lookups and
// hits, at least WALK_FLOOR_US (a few rows leave most SMs idle and a row's masks
// are a serial walk).
constexpr double CT_CALL_US = 60.0, CT_ITEM_US = 12.8, CT_WINDOW_US = 0.0125, CT_GATHER_BYTES_US = 9.0e6;
constexpr double WALK_FLOOR_US = 400.0, WALK_LOOKUP_US[2] = {8.0e-6, 5.8e-6}, WALK_HIT_US[2] = {1.1e-6, 2.0e-6};

// Whether a query over B rows of W window slots, `windows` windows in all, may
// take the count tables: the index has gather lists, no (row, SV, level) count
// reaches 2^32, the shared counters rarely overflow, and the estimated time is
// below the index walk's.
static bool ct_applies(const gkm_index *ix, int64_t B, int64_t W, int64_t windows)
{
    if (!ix->ct_ids || B < 1 || W < 1 || W > 60000 || B * ix->tiles > 0x7FFFFFFFLL) return false;
    const bool wt = ix->spec.weighted != 0;
    // (row, SV) weight products summed over every pair of windows
    const uint64_t wx = wt ? gkm_weight_sum(ix, W) : (uint64_t)W, wy = wt ? gkm_weight_sum(ix, ix->W) : (uint64_t)ix->W;
    if (!wx || !wy || wx >= (1ull << 32) / ((uint64_t)ix->strands * wy)) return false;
    // the mean count of a table row at level dmax: fields of 31 (unweighted, over
    // which a tile is recounted) hold the AT-rich rows of five times the mean
    double reach = 1.0;
    for (int m = 0; m < ix->spec.dmax; m++) reach *= 3.0 * (ix->spec.l - m) / (m + 1);
    const double mean = (double)ix->strands * (double)wx * reach / (double)ix->n_lmers;
    if (mean > (wt ? 80.0 : 4.6)) return false;
    if (windows <= 0) windows = B * W / 2;  // lengths unknown: rows padded to W
    const CtPlan p = ct_plan(ix, B, W);
    const int64_t items = p.rows / CT_ROWS * p.passes;
    const double row = (double)windows / B < W ? (double)windows / B : (double)W, waves = (double)((items + gkm_sm_count() - 1) / gkm_sm_count());
    const double table = CT_CALL_US + p.groups * (waves * (CT_ITEM_US + CT_WINDOW_US * row) +
                                                  (double)ix->ct_entries * p.rb / CT_GATHER_BYTES_US);
    double walk = (double)windows * (ix->n_masks * (double)ix->tiles * WALK_LOOKUP_US[wt] +
                                     (double)ix->entries * ix->n_masks / ix->n_lmers * WALK_HIT_US[wt]);
    if (walk < WALK_FLOOR_US) walk = WALK_FLOOR_US;
    return table < 0.9 * walk;
}

extern "C" int gkm_count_table_workspace(const gkm_index_t *ix, int64_t B, int64_t W, int64_t windows, int64_t *bytes)
{
    if (!ix || !bytes) return gkm_fail(GKM_ERR_INVALID, "null argument");
    *bytes = ct_applies(ix, B, W, windows) ? ct_plan(ix, B, W).bytes : 0;
    return GKM_OK;
}

extern "C" int gkm_count_table_query(const gkm_index_t *ix, const uint32_t *bx, const int32_t *cx, int64_t B,
                                     int64_t W, const int32_t *order, int32_t normalize, const double *inv_dx,
                                     double *diag, int64_t diag_offset, double *raw, const double *inv_ds,
                                     const double *coef, double gamma, int32_t rbf, double bias, double *scores,
                                     void *workspace, int64_t workspace_bytes, gkm_stream_t stream)
{
    if (!ix || !bx || !cx) return gkm_fail(GKM_ERR_INVALID, "null index or rows");
    if (!raw && !scores) return gkm_fail(GKM_ERR_INVALID, "no output");
    if (raw && scores) return gkm_fail(GKM_ERR_INVALID, "raw and scores are separate calls");
    if (scores && (!inv_ds || !coef)) return gkm_fail(GKM_ERR_INVALID, "scores need inv_ds and coef");
    if (order && diag_offset >= 0) return gkm_fail(GKM_ERR_INVALID, "a self-Gram takes rows in order");
    if (B < 0 || W < 1) return gkm_fail(GKM_ERR_INVALID, "rows %lld, windows per row %lld", (long long)B, (long long)W);
    if (B == 0) return GKM_OK;
    // (counts stay below 2^32 only where gkm_count_table_workspace says so)
    if (!ix->ct_ids || W > 60000) return gkm_fail(GKM_ERR_UNSUPPORTED, "this index or shape has no count tables");
    const CtPlan p = ct_plan(ix, B, W);
    if (!workspace || ((uintptr_t)workspace & 255) || workspace_bytes < p.bytes)
        return gkm_fail(GKM_ERR_CAPACITY, "count tables need a 256-byte aligned workspace of %lld bytes", (long long)p.bytes);
    cudaStream_t st = (cudaStream_t)stream;
    const bool wt = ix->spec.weighted != 0;
    CtArgs a = {};
    a.bx = bx;
    a.cx = cx;
    a.W = W;
    a.order = order;
    a.qg = p.qg;
    a.rb = p.rb;
    a.sh = ct_shape(ix);
    a.lists = ix->ct_lists;
    uint8_t *w = (uint8_t *)workspace;
    // the zero row, self counts, excess list lengths, dirty bits and excess counts start at zero
    a.T = w;
    uint8_t *z0 = w + p.rows * p.rb;
    w += p.table;
    a.self = (unsigned long long *)w;
    w += p.self;
    unsigned int *nexc = (unsigned int *)w;
    w += p.nexc;
    a.dirty = (uint32_t *)w;
    w += p.dirty;
    a.C = (unsigned long long *)w;
    w += p.c;
    double *partial = (double *)w;
    w += p.partial;
    uint32_t *recs = (uint32_t *)w;
    w += p.recs;
    uint32_t *roff = (uint32_t *)w;
    w += p.roff;
    a.exc = (unsigned long long *)w;
    a.cap_exc = (unsigned)(p.exc / 8);
    cudaError_t e = cudaMemsetAsync(z0, 0, (size_t)((uint8_t *)partial - z0), st);
    if (e != cudaSuccess) return gkm_cuda_status(e, "count table workspace");
    a.wd = ix->spec.wd;
    a.off = ix->offsets;
    a.ent = ix->ent;
    a.ent16 = ix->ent16;
    a.n_lmers = ix->n_lmers;
    a.tiles = ix->tiles;
    a.tile_svs = ix->tile_svs;
    a.ids = ix->ct_ids;
    a.wts = ix->ct_wts;
    a.goff = ix->ct_off;
    a.perm = ix->ct_perm;
    a.S = ix->S;
    for (int t = 0; t < 4; t++) a.h[t] = t <= a.sh.D ? ix->spec.h[a.sh.D - t] : 0.0;
    a.normalize = normalize;
    a.inv_dx = inv_dx;
    a.diag = diag;
    a.inv_ds = inv_ds;
    a.coef = coef;
    a.gamma = gamma;
    a.rbf = rbf;
    a.raw = raw;
    a.diag_offset = diag_offset;
    a.ball = ix->ct_lists + 32 * (CT_R2 + CT_R3);
    for (int m = 0; m < 4; m++) a.nball[m] = m <= a.sh.D ? ct_ball(a.sh.l - 6, m, nullptr) : 0;
    a.n_pre = p.n_pre;
    a.rec_cap = p.rec_cap;
    for (int64_t g = 0; g < p.groups; g++) {
        a.r0 = g * p.qg;
        a.nq = (int)(B - a.r0 < p.qg ? B - a.r0 : p.qg);
        a.partial = partial + g * p.blocks * p.qg;
        a.nexc = nexc + g;
        if (g % p.chunk == 0) {
            a.recs = recs;
            a.roff = roff;
            a.pass0 = (int)(g * p.passes);
            const int64_t rows = B - a.r0 < p.chunk * p.qg ? B - a.r0 : p.chunk * p.qg;
            const unsigned n = (unsigned)((rows + p.pass - 1) / p.pass);
            if (wt) ct_buckets<true><<<n, CT_THREADS, 0, st>>>(a, B);
            else ct_buckets<false><<<n, CT_THREADS, 0, st>>>(a, B);
            GKM_CHECK_LAUNCH("ct_buckets");
        }
        a.recs = recs + (g % p.chunk) * p.passes * p.rec_cap;
        a.roff = roff + (g % p.chunk) * p.passes * (p.n_pre + 1);
        const int nqp = a.nq < p.pass ? a.nq : p.pass;
        // two queries (or the one there is) x four levels for the 32-bit recount
        int words = wt ? nqp : (nqp + 1) / 2;
        if (words < 4 * (nqp < 2 ? nqp : 2)) words = 4 * (nqp < 2 ? nqp : 2);
        a.words = words;
        a.rec_smem = (int)(p.rec_cap < CT_RECS ? p.rec_cap : CT_RECS);
        const size_t smem = sizeof(uint32_t) * ((size_t)CT_ROWS * (words + 1) + a.rec_smem);  // + alignment
        a.passes = (a.nq + p.pass - 1) / p.pass;
        a.items = (int)(p.rows / CT_ROWS) * a.passes;
        // a block keeps its pass (its windows stay in L1), the passes of a tile
        // run side by side (their parts of a table row meet in L2)
        const int sms = gkm_query_blocks();
        const int fit = sms / a.passes > 0 ? sms / a.passes * a.passes : a.passes;
        const unsigned grid = (unsigned)(a.items < fit ? a.items : fit);
        if (wt) {
            cudaFuncSetAttribute(count_tiles<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            count_tiles<true><<<grid, CT_THREADS, smem, st>>>(a);
        } else {
            cudaFuncSetAttribute(count_tiles<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            count_tiles<false><<<grid, CT_THREADS, smem, st>>>(a);
        }
        GKM_CHECK_LAUNCH("count_tiles");
        if (wt) {
            spill_excess<<<(unsigned)gkm_sm_count() * 4, 256, 0, st>>>(a);
            GKM_CHECK_LAUNCH("spill_excess");
        }
#define GKM_GATHER_AS(RB, WT, RAW)                                                                        \
    do {                                                                                                  \
        gather_kernel<RB, WT, RAW><<<p.blocks, G_THREADS, 0, st>>>(a);                                   \
    } while (0)
#define GKM_GATHER(RB, WT)                                                                                \
    do {                                                                                                  \
        if (raw) GKM_GATHER_AS(RB, WT, true);                                                             \
        else GKM_GATHER_AS(RB, WT, false);                                                                \
    } while (0)
        if (p.rb == 32 && wt) GKM_GATHER(32, true);
        else if (p.rb == 32) GKM_GATHER(32, false);
        else if (p.rb == 64 && wt) GKM_GATHER(64, true);
        else if (p.rb == 64) GKM_GATHER(64, false);
        else GKM_GATHER(128, true);
#undef GKM_GATHER
#undef GKM_GATHER_AS
        GKM_CHECK_LAUNCH("gather_kernel");
    }
    if (scores) {
        const int per = p.qg < 32 ? p.qg : 32;
        ct_scores<<<(unsigned)(p.groups * (p.qg / per)), 1024, 0, st>>>(partial, p.blocks, p.qg, order, B, bias, scores);
        GKM_CHECK_LAUNCH("ct_scores");
    }
    return GKM_OK;
}
