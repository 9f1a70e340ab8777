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
// its query self-kernels): 1,000 x 300 bp, t=3: 43.5 -> 8.5 ms; 2,048 rows of 50 ..
// 2,000 bp: 135 -> 20.2 ms; 512 of them, weighted t=5: 77.8 -> 8.2 ms; one 300 bp
// row: 1.3 -> 0.2 ms.
//
// Entries are exact.  Unweighted entries take 16 bits (5, 4, 4 and 3 for levels
// dmax, dmax - 1, ...: t = dmax - m indexes the fields), weighted ones and those of
// long unweighted rows (weights of 1) four bytes, one per level.  They are counted in shared memory in fields of those widths
// (weighted: 9 / 8 / 8 / 7 bits).  A weighted count past its byte is clipped and
// the excess added to the (SV, query) counts of that l-mer's SVs through the
// index's buckets (spill_excess: C and its dirty bits, read back by the gather).
// A tile whose shared fields overflowed (its decoded fields do not sum to the
// adds made) is counted again with 32-bit counters, one level of one query each,
// and clipped alike.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdlib.h>

#include <type_traits>

#include "gkm_common.cuh"

namespace {

constexpr int CT_POS = 5;          // positions of a tile's suffix
constexpr int CT_ROWS = 1 << (2 * CT_POS);  // table rows per tile
constexpr int CT_THREADS = 512;
constexpr int CT_WARPS = CT_THREADS / 32;
constexpr int CT_BLOCKS = 2;      // count_tiles blocks per SM
constexpr int CT_SLOTS = 16;      // counter words per table row a block holds (64 KB)
constexpr int CT_LIST = 256;      // entries of a tile a block queues for a second look
constexpr int CB_THREADS = 1024;  // ct_buckets
constexpr int CT_PRE = 4096;      // most values of the other positions
constexpr int64_t CT_EXC = 4096;   // clipped counts a group queues, per query (weighted)
// unweighted counter halves (and entries): fields of 5 / 4 / 4 / 3 bits for t = 0
// .. 3, placed so that two byte dot products sum all of them
constexpr uint32_t CT_F0 = 0, CT_F1 = 8, CT_F2 = 12, CT_F3 = 5;
constexpr int CT_R2 = 4, CT_R3 = 20;  // rounds of 32 lanes over the 106 / 376 neighbour masks of budgets 2 / 3
constexpr int CT_ROUNDS = 1 + CT_R2 + CT_R3;
constexpr int CT_BALL = 694;      // masks of up to six positions within three mismatches
constexpr int CT_WLIST = 128;     // windows of budgets 1 and 2 a warp lists at a time
constexpr int G_THREADS = 128;
constexpr int G_BLOCKS = 4, G_BLOCKS_W = 6;   // gather blocks per SM, unweighted / weighted

// Shared-memory position of the table row with suffix s (10 bits): a linear
// bijection, its own inverse, chosen so that the 16 masks of budget 1 lie on 16 of
// the 32 banks, the 106 of budget 2 on all of them (at most 4 on one) and the 376 of
// budget 3 at most 20 on one: lane b takes the masks of bank class b, so a warp's
// adds around any one window hit different banks.
__host__ __device__ constexpr __forceinline__ uint32_t ct_phys(uint32_t s)
{
    return s ^ (((s >> 5) & 1u ? 15u : 0u) ^ ((s >> 6) & 1u ? 20u : 0u) ^ ((s >> 7) & 1u ? 10u : 0u) ^
                ((s >> 8) & 1u ? 18u : 0u) ^ ((s >> 9) & 1u ? 5u : 0u));
}

// Counter plane j keeps its positions with bits 3 and 4 exchanged by its quarter, so
// that the four lanes that write a table row's quarters read different banks.
__device__ __forceinline__ uint32_t ct_swap(uint32_t plane)
{
    return (plane >> 2) << 3;
}

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
    gkm_rows sh;
    const uint32_t *lists;  // neighbour masks of the six suffix positions by bank class
    const uint32_t *ball;   // masks of the other positions by mismatches
    int nball[4];           // how many of each
    // windows of the call's rows by the bases outside the suffix (ct_buckets):
    // records [pass][rec_cap], bucket offsets [pass][n_pre + 1]
    uint8_t *recs;
    uint32_t *roff;
    int64_t rec_cap;
    int n_pre;
    int pass0;  // pass of the group's first row
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
    int split;             // lane groups that share an SV's windows
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
// buckets, so v <= rc(v) stands for both; a palindrome's bucket holds every window of an
// SV twice, the forward ones in window order and then mirrored (w1 w2 w2 w1: entry_gen's
// order, kept by the stable sort), so that every second entry is every window once.
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
            const uint64_t w = WT && a.wd ? en >> 24 : 1;
            const int64_t at = s * a.qg + q;
            const unsigned long long c0 = w * ex[0] | (w * ex[1]) << 32, c1 = w * ex[2] | (w * ex[3]) << 32;
            if (c0) atomicAdd(a.C + 2 * at, c0);
            if (c1) atomicAdd(a.C + 2 * at + 1, c1);
            atomicOr(a.dirty + (at >> 5), 1u << (at & 31));
        }
    }
}

__device__ __forceinline__ void ct_fa(uint32_t &s, uint32_t &c, uint32_t a, uint32_t b)
{
    const uint32_t x = s;
    s = x ^ a ^ b;
    c = (x & a) | (x & b) | (a & b);
}

// plain add to shared memory (byte address) where a < b, no value returned;
// predicated rather than branched around
__device__ __forceinline__ void ct_add(uint32_t a, uint32_t b, uint32_t addr, uint32_t v)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.u32 p, %0, %1;\n\t@p red.shared.add.u32 [%2], %3;\n\t}" ::"r"(a), "r"(b),
                 "r"(addr), "r"(v)
                 : "memory");
}

template <bool WT>
__host__ __device__ __forceinline__ uint32_t ct_shift(uint32_t t)
{
    return WT ? (t ? 8u * t + 1u : 0u) : t == 0 ? CT_F0 : t == 1 ? CT_F1 : t == 2 ? CT_F2 : CT_F3;
}

// How ct_buckets hands a window to count_tiles: its counter (plane of the query,
// position of the suffix) and above its 14 bits its weight or (unweighted: 16 bits)
// the query's half of the word.
template <bool WT>
using ct_rec = std::conditional_t<WT, uint32_t, uint16_t>;

template <bool WT>
__device__ __forceinline__ ct_rec<WT> ct_record(const gkm_rows &sh, uint32_t v, int q, uint32_t w, uint32_t *pre)
{
    uint32_t c = v;  // the l-mer without its middle base, which goes on top (fold)
    if (sh.fold) {
        const uint32_t low = (1u << (2 * sh.mid)) - 1u;
        c = (v & low) | ((v >> 2) & ~low & ((1u << (2 * (sh.l - 1))) - 1u)) | (((v >> (2 * sh.mid)) & 3u) << (2 * (sh.l - 1)));
    }
    *pre = c >> (2 * CT_POS);
    const uint32_t plane = WT ? (uint32_t)q : (uint32_t)q >> 1;
    return (ct_rec<WT>)(plane * CT_ROWS + (ct_phys(c & (CT_ROWS - 1u)) ^ ct_swap(plane)) | (WT ? w : (uint32_t)(q & 1)) << 14);
}

// One block per pass of queries: their windows (both strands) sorted by the
// bases outside the suffix (counting sort in shared memory), so
// that a tile visits the buckets within D mismatches of it and tests nothing.
template <bool WT>
__global__ void __launch_bounds__(CB_THREADS) ct_buckets(CtArgs a, int64_t B)
{
    constexpr int PASS = WT ? CT_SLOTS : 2 * CT_SLOTS;
    constexpr int EACH = CT_PRE / CB_THREADS;
    __shared__ __align__(16) uint32_t hist[CT_PRE];
    __shared__ uint32_t wtot[32];
    const int64_t pass = a.pass0 + blockIdx.x;
    const int64_t q0 = pass * PASS;
    const int nq = (int)min((int64_t)PASS, B - q0);
    ct_rec<WT> *recs = (ct_rec<WT> *)a.recs + (int64_t)blockIdx.x * a.rec_cap;
    uint32_t *roff = a.roff + (int64_t)blockIdx.x * (a.n_pre + 1);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ((uint4 *)hist)[threadIdx.x] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    for (int phase = 0; phase < 2; phase++) {
        for (int q = warp; q < nq * 4; q += CB_THREADS / 32) {  // four warps a row
            const int64_t r = a.order ? (int64_t)a.order[q0 + (q >> 2)] : q0 + (q >> 2);
            const int n = a.cx[r];
            for (int i = (q & 3) * 32 + lane; i < n; i += 128) {
                uint32_t v = __ldg(a.bx + r * a.W + i);
                const uint32_t w = WT && a.wd ? gkm_wt(a.wd, n, i) : 1u;
                for (int st = 0; st < a.sh.strands; st++) {
                    if (st) v = gkm_rc_word(v, a.sh.l);
                    uint32_t pre;
                    const ct_rec<WT> rec = ct_record<WT>(a.sh, v, q >> 2, w, &pre);
                    const uint32_t at = atomicAdd(&hist[pre], 1u);
                    if (phase) recs[at] = rec;
                }
            }
        }
        __syncthreads();
        if (phase) break;
        // exclusive scan: the buckets' first records (four neighbours a thread)
        const uint4 c = ((const uint4 *)hist)[threadIdx.x];
        static_assert(EACH == 4, "four buckets a thread");
        const uint32_t own = c.x + c.y + c.z + c.w;
        uint32_t x = own;
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
        x = x - own + (warp ? wtot[warp - 1] : 0u);
        const uint32_t first[EACH + 1] = {x, x + c.x, x + c.x + c.y, x + c.x + c.y + c.z, x + own};
#pragma unroll
        for (int k = 0; k < EACH; k++) {
            const int pre = threadIdx.x * EACH + k;
            hist[pre] = first[k];
            if (pre < a.n_pre) roff[pre] = first[k];
            if (pre == a.n_pre - 1) roff[a.n_pre] = first[k + 1];
        }
        __syncthreads();
    }
}

// Items of (tile, pass of queries): a tile is the l-mers that agree outside the
// five suffix positions.  Windows whose other positions differ from the tile's at
// dp <= D places reach the suffixes within budget D - dp of their own: one row
// (budget 0), 16, 106 or 376.  Their buckets are dealt to the warps; a warp copies
// its buckets of budgets 1 and 2 to a list (they hold a few windows each) and adds a
// window at a time with a lane on each bank (no two of its adds conflict), two of
// budget 1.  Budget 0 is a bucket per lane.
//
// Shared counters: unweighted, one word per two queries (fields: CT_F0 ..);
// weighted, one word per query with 9 / 8 / 8 / 7 bits (entry: a byte each).
//
// Bound by instruction issue and the latency of the short chains between barriers.  A
// pass holds the 64 bytes of 32 unweighted (16 weighted) queries, so that rows are
// written 64 bytes at a time, and two blocks share an SM, so that one counts while the
// other writes.  Tiles of six positions and passes of half as many queries, one block
// of 1,024 threads per SM, a window per lane for budget 1: 110 us a group of 32 x 300
// bp, this 86 us (weighted: 268 and 184).
template <bool WT>
__global__ void __launch_bounds__(CT_THREADS, CT_BLOCKS) count_tiles(CtArgs a)
{
    constexpr int PASS = WT ? CT_SLOTS : 2 * CT_SLOTS;
    extern __shared__ __align__(16) uint8_t ct_smem[];
    __shared__ uint2 l3[CT_R3 * 32];
    __shared__ uint16_t ball_s[CT_BALL];
    __shared__ uint32_t list_s[CT_WARPS * (CT_WLIST + 8)];  // (up to eight more are read)
    __shared__ uint32_t slot_s[CT_WARPS * 32];
    // by tile parity: the entries that need a second look, and the fields' sum and
    // the adds made
    __shared__ uint16_t list_at[2][CT_LIST];
    __shared__ uint32_t list_w[2][CT_LIST];
    __shared__ int nlist[2];
    __shared__ uint32_t chk[2][2];
    // counters [words][CT_ROWS], aligned to a word's plane so that a neighbour's
    // address is an exclusive or
    constexpr uint32_t PLANE = 4 * CT_ROWS;
    const uint32_t raw0 = (uint32_t)__cvta_generic_to_shared(ct_smem), cbase = (raw0 + PLANE - 1u) & ~(PLANE - 1u);
    uint32_t *cnt = (uint32_t *)(ct_smem + (cbase - raw0));
    const int lane = threadIdx.x & 31, warp = __shfl_sync(GKM_FULL, threadIdx.x >> 5, 0);  // (known to be uniform)
    const gkm_rows sh = a.sh;
    const int D = sh.D;
    // a mask: byte offset and increment (0: none in this round)
    auto entry = [&](uint32_t e) -> uint2 {
        return (e >> 31) ? make_uint2((uint32_t)lane * 4u, 0u)
                         : make_uint2((e & 0xFFFu) * 4u, 1u << ct_shift<WT>((e >> 12) & 3u));
    };
    const uint2 e1 = entry(a.lists[lane]);
    uint2 e2[CT_R2];
#pragma unroll
    for (int k = 0; k < CT_R2; k++) e2[k] = entry(a.lists[(1 + k) * 32 + lane]);
    for (int k = threadIdx.x; k < CT_R3 * 32; k += CT_THREADS) l3[k] = entry(a.lists[(1 + CT_R2) * 32 + k]);
    const int pass = blockIdx.x % a.passes;  // grid: a multiple of passes
    const ct_rec<WT> *recs = (const ct_rec<WT> *)a.recs + (int64_t)pass * a.rec_cap;
    const uint32_t *off = a.roff + (int64_t)pass * (a.n_pre + 1);
    // A record in use: its counter's address (18 bits), and above it its weight or the
    // shift of the query's half.  (The pass's records stay in L1.)
    auto load_rec = [&](uint32_t k) -> uint32_t {
        const uint32_t r = __ldg(recs + k);
        return cbase + ((r & 0x3FFFu) << 2) + (r >> 14 << (WT ? 18 : 22));
    };
    for (int k = threadIdx.x; k < CT_BALL; k += CT_THREADS) ball_s[k] = (uint16_t)a.ball[k];
    const int q0 = pass * PASS;
    const int nqp = min(PASS, a.nq - q0);
    const int words = WT ? nqp : (nqp + 1) >> 1;
    // buckets by budget, their masks in ball_s one budget after the other
    const int nb3 = D >= 3 ? a.nball[D - 3] : 0, nb2 = D >= 2 ? a.nball[D - 2] : 0, nb1 = D >= 1 ? a.nball[D - 1] : 0,
              nb0 = a.nball[D];
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
    // What a clipped entry's fields do not hold, x of query q of the pass in table row
    // `row`, where over: to the group's list (weighted, level t = 0), else to the row's
    // SVs at once by the whole warp.  All lanes call it.
    auto spill = [&](bool over, uint32_t row, int q, const uint32_t (&x)[4]) {
        const bool listed = WT && over && !(x[1] | x[2] | x[3]);
        const uint32_t some = __ballot_sync(GKM_FULL, listed);
        if (some) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(a.nexc, (unsigned)__popc(some));
            const uint32_t pos = __shfl_sync(GKM_FULL, base, 0) + __popc(some & ((1u << lane) - 1u));
            if (listed && pos < a.cap_exc) {
                a.exc[pos] = row | (unsigned long long)(q0 + q) << 22 | (unsigned long long)x[0] << 32;
                over = false;
            }
        }
        for (uint32_t rest = __ballot_sync(GKM_FULL, over); rest; rest &= rest - 1) {
            const int j = __ffs(rest) - 1;
            const uint64_t ex[4] = {__shfl_sync(GKM_FULL, x[0], j), __shfl_sync(GKM_FULL, x[1], j),
                                    __shfl_sync(GKM_FULL, x[2], j), __shfl_sync(GKM_FULL, x[3], j)};
            ct_excess<WT>(a, sh.lmer(__shfl_sync(GKM_FULL, row, j)), q0 + __shfl_sync(GKM_FULL, q, j), ex, lane, 32);
            __syncwarp();
        }
    };
    // A second look at counter word w, `at` = j * CT_ROWS + position of a tile, one
    // query per lane (unweighted: two neighbouring lanes share the word): the
    // query's self-kernel part and, weighted, a clipped count's entry and excess.  All
    // lanes call it.
    auto look = [&](uint32_t tl, bool in, uint32_t at, uint32_t w) {
        const uint32_t j = at / CT_ROWS, q = WT ? j : 2 * j + (lane & 1);
        const uint32_t v = !in ? 0u : WT ? w : (w >> (16 * (lane & 1))) & 0xFFFFu;
        uint32_t c[4];
        fields(v, c);
        if (v & slow_mask) self_part(c, q);
        if constexpr (WT) {
            const bool over = (v & 0x100u) != 0;
            uint32_t x[4] = {0, 0, 0, 0};
            const uint32_t row = tl * CT_ROWS + ct_phys((at & (CT_ROWS - 1)) ^ ct_swap(j));
            if (over) ((uint32_t *)(a.T + (size_t)row * a.rb))[q0 + q] = clip(c, x);
            spill(over, row, (int)q, x);
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

    if (__ldg(off + a.n_pre) == 0) return;  // rows of length 0 pad a batch: the gather reads nothing of them
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

    // counts the windows of queries qa .. qb - 1 (safe: the recount of four
    // queries with 32-bit counters, plane (q - qa) * 4 + t; else all)
    auto count_buckets = [&](auto SAFE, int qa, int qb) -> uint32_t {
        constexpr bool safe = decltype(SAFE)::value;
        uint32_t adds = 0;
        auto weight = [&](uint32_t rec) -> uint32_t { return WT ? rec >> 18 : 1u; };
        // one window's counter address and what its increments are multiplied by
        // (unweighted: shifted; safe: 0 if it is not counted)
        auto where = [&](uint32_t rec, uint32_t &sa, uint32_t &inc) {
            if (safe) {
                const uint32_t at = (rec & 0x3FFFFu) - cbase, plane = at / PLANE;
                const int q = WT ? plane : 2 * plane + (rec >> 22);
                const bool in = q >= qa && q < qb;
                sa = cbase + (in ? (q - qa) * 4 * PLANE + ((at & (PLANE - 1u)) ^ (ct_swap(plane) << 2)) : 0u);
                inc = in ? weight(rec) : 0u;
            } else {
                sa = rec & 0x3FFFFu;
                inc = rec >> 18;
            }
        };
        // add at the neighbour with byte offset x, field increment f = 1 << ct_shift(t),
        // where i < n
        auto add = [&](uint32_t sa, uint32_t x, uint32_t f, uint32_t inc, uint32_t i, uint32_t n) {
            if (safe) {
                const uint32_t t = f == 1u ? 0u : f == 1u << ct_shift<WT>(1) ? 1u : f == 1u << ct_shift<WT>(2) ? 2u : 3u;
                ct_add(i, f && inc ? n : 0u, (sa ^ x) + t * PLANE, inc);
            } else {
                ct_add(i, n, sa ^ x, WT ? f * inc : f << inc);
            }
        };
        auto bucket = [&](int k, uint32_t &beg, uint32_t &end) {
            const uint32_t pre = (uint32_t)tile ^ ball_s[k];
            beg = __ldg(off + pre);
            end = __ldg(off + pre + 1);
        };
        // budget 3: a warp takes every CT_WARPS-th window of the bucket
        if (nb3) {
            uint32_t r, e;
            bucket(0, r, e);
            for (r += warp; r < e; r += CT_WARPS) {
                const uint32_t rec = load_rec(r);
                uint32_t sa, inc;
                where(rec, sa, inc);
                if (lane == 0) adds += 376u * weight(rec);
#pragma unroll 10
                for (int k = 0; k < CT_R3; k++) {
                    const uint2 x = l3[k * 32 + lane];
                    add(sa, x.x, x.y, inc, r, e);
                }
            }
        }
        // The windows of the lanes' buckets beg .. beg + len - 1 as one list: f(lane's
        // record, index of lane 0's, windows in all), 32 at a time.
        auto flatten = [&](uint32_t beg, uint32_t len, auto f) {
            uint32_t upto = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(GKM_FULL, upto, o);
                if (lane >= o) upto += y;
            }
            const uint32_t all = __shfl_sync(GKM_FULL, upto, 31), start = upto - len;
            if (all == 0) return;
            // the buckets that hold windows, side by side: window h of the list is
            // record slot + h (in 32 bits: a slot may lie below zero)
            uint32_t *slot = slot_s + 32 * warp;
            const uint32_t some = __ballot_sync(GKM_FULL, len != 0);
            if (len) slot[__popc(some & ((1u << lane) - 1u))] = beg - start;
            __syncwarp();
            // a window's bucket is the last one that starts at or before it
            uint32_t begun = 0;
            auto fetch = [&](uint32_t c) -> uint32_t {
                const uint32_t at = start - c, starts = __reduce_or_sync(GKM_FULL, len && at < 32u ? 1u << at : 0u);
                const uint32_t own = begun + __popc(starts & (0xFFFFFFFFu >> (31 - lane))) - 1u;
                begun += __popc(starts);
                return load_rec(c + lane < all ? slot[own & 31u] + (c + lane) : 0u);
            };
            uint32_t rec = fetch(0);
            for (uint32_t c = 0; c < all; c += 32) {
                const uint32_t now = rec;
                if (c + 32 < all) rec = fetch(c + 32);  // in flight meanwhile
                f(now, c, all);
            }
            __syncwarp();
        };
        const int near = nb3 + nb2 + nb1;
        for (int b = CT_WARPS - 1 - warp; b * 32 < nb0; b += CT_WARPS) {
            uint32_t r = 0, e = 0;
            if (b * 32 + lane < nb0) bucket(near + b * 32 + lane, r, e);
            if (!WT) adds += e - r;
            flatten(r, e - r, [&](uint32_t rec, uint32_t c, uint32_t all) {
                uint32_t sa, inc;
                where(rec, sa, inc);
                add(sa, 0u, 1u, inc, c + lane, all);
                if (WT && c + lane < all) adds += weight(rec);
            });
        }
        // budgets 1 and 2: lanes 0 .. n1 - 1 and n1 .. n1 + n2 - 1 have the warp's buckets
        if (nb1) {
            const int n1 = (nb1 + CT_WARPS - 1) / CT_WARPS;
            const bool is1 = lane < n1;
            const int k = is1 ? nb3 + nb2 + warp + CT_WARPS * lane : nb3 + warp + CT_WARPS * (lane - n1);
            uint32_t r = 0, e = 0;
            if (k < (is1 ? near : nb3 + nb2)) bucket(k, r, e);
            if (!WT) adds += (is1 ? 16u : 106u) * (e - r);
            const uint32_t ones = __reduce_add_sync(GKM_FULL, is1 ? e - r : 0u);  // windows of budget 1
            uint32_t *list = list_s + warp * (CT_WLIST + 8);
            flatten(r, e - r, [&](uint32_t rec, uint32_t c, uint32_t all) {
                const uint32_t at = c % CT_WLIST;
                list[at + lane] = rec;
                if (WT && c + lane < all) adds += (c + lane < ones ? 16u : 106u) * weight(rec);
                if (at + 32 < CT_WLIST && c + 32 < all) return;
                // a full list, or the last
                __syncwarp();
                const uint32_t from = c - at, n = min((uint32_t)CT_WLIST, all - from), n_1 = min(n, ones > from ? ones - from : 0u);
                for (uint32_t j = lane >> 4; j < n_1 + (lane >> 4); j += 8) {  // half a warp per window
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        uint32_t sa, inc;
                        where(list[j + 2 * i], sa, inc);
                        add(sa, e1.x, e1.y, inc, j + 2 * i, n_1);
                    }
                }
#pragma unroll 2
                for (uint32_t j = n_1; j < n; j++) {
                    uint32_t sa, inc;
                    where(list[j], sa, inc);
#pragma unroll
                    for (int i = 0; i < CT_R2; i++) add(sa, e2[i].x, e2[i].y, inc, j, n);
                }
                __syncwarp();
            });
        }
        return adds;
    };

    const uint32_t adds = count_buckets(std::false_type{}, 0, nqp);
    __syncthreads();
    // The tile's entries, the words that need more queued, and the fields' sum: it
    // equals the adds made unless some field carried into the next.  Four lanes, eight
    // apart, write the quarters of a row, so that a store writes eight rows side by
    // side.  The words are summed by carry-save adders (two logic operations a word)
    // and the fields of the six sums added up.
    // sum of a word's fields (unweighted: t = 0 and 1 are the bytes' low fields, t = 3
    // and 2 the high ones, 32 and 16 times too large)
    auto field_sum = [](uint32_t w) -> uint32_t {
        return WT ? __dp4a(w >> 9, 0x00010101u, w & 0x1FFu)
                  : __dp4a(w & 0x0F1F0F1Fu, 0x01010101u, __dp4a(w & 0xF0E0F0E0u, 0x02010201u, 0u) >> 5);
    };
    auto queue = [&](uint32_t at, uint32_t w) {
        const int n = atomicAdd(&nlist[par], 1);
        if (n < CT_LIST) {
            list_at[par][n] = (uint16_t)at;
            list_w[par][n] = w;
        }
    };
    auto check = [&](uint32_t sum) {
        const uint32_t wsum = __reduce_add_sync(GKM_FULL, sum), wadds = __reduce_add_sync(GKM_FULL, adds);
        if (lane == 0) {
            atomicAdd(&chk[par][0], wsum);
            atomicAdd(&chk[par][1], wadds);
        }
    };
    // narrow rows (a few queries): a row per thread
    auto write_few = [&]() {
        uint32_t sum = 0;
#pragma unroll
        for (int i = 0; i < CT_ROWS / CT_THREADS; i++) {
            const uint32_t p = i * CT_THREADS + threadIdx.x;
            uint32_t w[4], any = 0;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                w[j] = j < words ? cnt[j * CT_ROWS + p] : 0u;
                sum += field_sum(w[j]);
                any |= w[j];
            }
            if (any & slow_mask)
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (w[j] & slow_mask) queue(j * CT_ROWS + p, w[j]);
            if (WT)
#pragma unroll
                for (int j = 0; j < 4; j++) w[j] = (w[j] & 0xFFu) | ((w[j] >> 1) & 0xFFFFFF00u);
            uint8_t *T = a.T + ((size_t)tile * CT_ROWS + ct_phys(p)) * a.rb;
            if (a.rb == 8) *(uint2 *)T = make_uint2(w[0], w[1]);
            else *(uint4 *)T = make_uint4(w[0], w[1], w[2], w[3]);
        }
        check(sum);
    };
    auto write_tile = [&](auto FULL) {
        constexpr bool full = decltype(FULL)::value;  // every word of a row is counted and stored
        const int part = (lane >> 3) & 3, j0 = 4 * part;
        uint8_t *T = a.T + (size_t)tile * CT_ROWS * a.rb + q0 * (WT ? 4 : 2) + 16 * part;
        const bool write = full || 16 * part < a.rb;  // (narrow rows: fewer quarters)
        const uint32_t row0 = ct_phys(threadIdx.x & ~24u) * a.rb;
        const uint32_t *mine = cnt + j0 * CT_ROWS;
        uint32_t ones = 0, twos = 0, fours = 0, e[4];
        static_assert(CT_ROWS == 2 * CT_THREADS && CT_SLOTS == 16, "32 words per thread");
#pragma unroll
        for (int i = 0; i < 4; i++) {
            uint32_t t[4], f[2];
#pragma unroll
            for (int g = 0; g < 2; g++) {
                // the row of position (i / 2) * CT_THREADS + threadIdx.x with bits 3 and 4 = h
                const uint32_t h = (i & 1) * 2 + g, at = (i >> 1) * CT_THREADS;
                uint32_t w[4];
#pragma unroll
                for (int j = 0; j < 4; j++) w[j] = full || j0 + j < words ? mine[j * CT_ROWS + ((at + threadIdx.x) ^ (8u * h))] : 0u;
                ct_fa(ones, t[2 * g], w[0], w[1]);
                ct_fa(ones, t[2 * g + 1], w[2], w[3]);
                if (WT)
#pragma unroll
                    for (int j = 0; j < 4; j++) w[j] = (w[j] & 0xFFu) | ((w[j] >> 1) & 0xFFFFFF00u);
                const uint32_t row = row0 ^ ((ct_phys(at) ^ (8u * h)) * a.rb);
                if (write) *(uint4 *)(T + row) = make_uint4(w[0], w[1], w[2], w[3]);
            }
            ct_fa(twos, f[0], t[0], t[1]);
            ct_fa(twos, f[1], t[2], t[3]);
            ct_fa(fours, e[i], f[0], f[1]);
        }
        uint32_t eights = 0, s0, s1;
        ct_fa(eights, s0, e[0], e[1]);
        ct_fa(eights, s1, e[2], e[3]);
        const uint32_t sums[6] = {ones, twos, fours, eights, s0 ^ s1, s0 & s1};
        uint32_t sum = 0, any = 0;
#pragma unroll
        for (int k = 0; k < 6; k++) {
            const uint32_t w = sums[k];
            any |= w;
            sum += field_sum(w) << k;
        }
        // a lane that saw such a word: its 32 words again, one per lane
        for (uint32_t some = __ballot_sync(GKM_FULL, (any & slow_mask) != 0); some; some &= some - 1) {
            const int from = __ffs(some) - 1;
            const int j = ((from >> 3) & 3) * 4 + (lane & 3),
                      pos = ((lane >> 4) * CT_THREADS + warp * 32 + from) ^ (2 * (lane & 12));
            const uint32_t w = j < words ? cnt[j * CT_ROWS + pos] : 0u;
            if (w & slow_mask) queue(j * CT_ROWS + pos, w);
        }
        check(sum);
    };
    if (words <= 4 && a.rb <= 16) write_few();
    else if (words == CT_SLOTS && a.rb >= 4 * CT_SLOTS) write_tile(std::true_type{});
    else write_tile(std::false_type{});
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
        // a field overflowed: 32-bit counters, four queries x four levels at a time
        for (int qa = 0; qa < nqp; qa += 4) {
            const int nb = min(4, nqp - qa);
            __syncthreads();
            for (int k = threadIdx.x; k < 4 * nb * CT_ROWS; k += CT_THREADS) cnt[k] = 0;
            __syncthreads();
            count_buckets(std::true_type{}, qa, qa + nb);
            __syncthreads();
            for (int p = threadIdx.x; p < CT_ROWS; p += CT_THREADS) {
                const uint32_t suf = ct_phys(p);
                uint8_t *T = a.T + ((size_t)tile * CT_ROWS + suf) * a.rb + q0 * (WT ? 4 : 2);
                for (int q = 0; q < nb; q++) {
                    const uint32_t *cq = cnt + q * 4 * CT_ROWS + p;
                    const uint32_t c[4] = {cq[0], cq[CT_ROWS], cq[2 * CT_ROWS], cq[3 * CT_ROWS]};
                    self_part(c, qa + q);
                    uint32_t x[4];
                    const uint32_t v = clip(c, x);
                    if (WT)
                        ((uint32_t *)T)[qa + q] = v;
                    else
                        ((uint16_t *)T)[qa + q] = (uint16_t)v;
                    spill((x[0] | x[1] | x[2] | x[3]) != 0, tile * CT_ROWS + suf, qa + q, x);
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

__device__ __forceinline__ void ct_load(uint32_t (&r)[4], const uint8_t *p)
{
    const uint4 v = __ldg((const uint4 *)p);
    r[0] = v.x, r[1] = v.y, r[2] = v.z, r[3] = v.w;
}

__device__ __forceinline__ void ct_load(uint32_t (&r)[2], const uint8_t *p)
{
    const uint2 v = __ldg((const uint2 *)p);
    r[0] = v.x, r[1] = v.y;
}

// RB-byte rows, 16 bytes (RB = 8: 8) per lane, RB / 16 lanes per SV; persistent blocks take
// SVs round robin in gather order (long SVs first); where there are fewer SVs than
// lane groups, `split` groups share an SV's windows.  Bound by L1's line lookups where
// L2 holds the table (24.5M rows at one per clock and SM are 87 us; one query 112 us),
// by the row pieces in flight past it (32 queries: 172 us in 64-byte, weighted 290 us in
// 128-byte rows; 64 KB per SM at ~1 us, with HBM at 45 % and L2 at 57 %).
template <int RB, bool WT, bool RAW, bool SPLIT>
__global__ void __launch_bounds__(G_THREADS, WT ? G_BLOCKS_W : G_BLOCKS) gather_kernel(CtArgs a)
{
    constexpr int NW = RB < 16 ? RB / 4 : 4;     // words a lane loads of a row
    constexpr int NQ = WT ? NW : 2 * NW;         // queries a lane owns
    constexpr int LPG = RB / (4 * NW), QG = LPG * NQ;
    const int split = SPLIT ? a.split : 1, lanes = LPG * split, GPB = G_THREADS / lanes;  // lanes per SV, SVs per block
    __shared__ uint4 rows_s[4 * G_THREADS];
    __shared__ double inv_dx[QG];
    __shared__ uint32_t empty_s[QG];  // a query without windows (its columns may hold another group's counts)
    __shared__ double part_s[G_THREADS / 32][QG];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = threadIdx.x % LPG, j0 = sub * NQ;
    const uint32_t turn = SPLIT ? threadIdx.x / LPG % split : 0;  // the lane group's stages: turn, turn + split, ..
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
    const uint8_t *base = a.T + sub * 4 * NW;
    const int64_t rounds = (a.S + (int64_t)gridDim.x * GPB - 1) / ((int64_t)gridDim.x * GPB);
    for (int64_t it = 0; it < rounds; it++) {
        const int64_t g = (it * gridDim.x + blockIdx.x) * GPB + threadIdx.x / lanes;
        bool live = g < a.S;
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
        load_ids(turn);
        uint32_t acc[4 * NW];  // WT: [query][t]; else [word][t], two 16-bit sums each
#pragma unroll
        for (int k = 0; k < 4 * NW; k++) acc[k] = 0;
        // 16 bits per query: carry-save adders over the 32-bit words sum rows with
        // ~2 logic operations per row and word whatever the fields; every 32 rows the
        // carries of weight 32 are added field by field into 16-bit sums (31 x 2,048
        // rows < 2^16).  (p8, p16: carries waiting for the second of a pair)
        uint32_t ones[NW] = {}, twos[NW] = {}, fours[NW] = {}, eights[NW] = {}, s16[NW] = {}, p8[NW] = {}, p16[NW] = {};
        for (uint32_t k = turn, n = 0; k < nst; k += split, n++) {
            uint32_t r[8][NW];
#pragma unroll
            for (int j = 0; j < 8; j++) ct_load(r[j], base + (size_t)id[j] * RB);
            uint2 wt = make_uint2(0x01010101u, 0x01010101u);
            if (WT && a.wts) wt = __ldg((const uint2 *)(a.wts + p0) + k);
            load_ids(k + split);
            if constexpr (!WT) {
                uint32_t f[2][NW];
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int w = 0; w < NW; w++) {
                        uint32_t t0, t1;
                        ct_fa(ones[w], t0, r[4 * h][w], r[4 * h + 1][w]);
                        ct_fa(ones[w], t1, r[4 * h + 2][w], r[4 * h + 3][w]);
                        ct_fa(twos[w], f[h][w], t0, t1);
                    }
#pragma unroll
                for (int w = 0; w < NW; w++) {
                    uint32_t e;
                    ct_fa(fours[w], e, f[0][w], f[1][w]);
                    if ((n & 1) == 0) {
                        p8[w] = e;
                        continue;
                    }
                    uint32_t c;
                    ct_fa(eights[w], c, p8[w], e);
                    p8[w] = 0;
                    if ((n & 2) == 0) {
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
                    const uint32_t *w0 = r[4 * h], *w1 = r[4 * h + 1], *w2 = r[4 * h + 2], *w3 = r[4 * h + 3];
#pragma unroll
                    for (int q = 0; q < NW; q++) {
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
            for (int w = 0; w < NW; w++) {
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
        if (SPLIT) {  // the groups' sums, in the first
#pragma unroll
            for (int k = 0; k < 4 * NW; k++)
                for (int o = LPG; o < lanes; o <<= 1) acc[k] += __shfl_xor_sync(GKM_FULL, acc[k], o);
            live = live && turn == 0;
        }
        // epilogue, four queries at a time (the sums wait in the lane's slots, so
        // that the loop above has the registers).  Weighted: two lanes share a byte
        // of dirty bits.
        const int64_t dat = s * a.qg + j0;
        uint8_t *db = (uint8_t *)a.dirty + (dat >> 3);
        const uint32_t dirty = live ? (*db >> (dat & 7)) & ((1u << NQ) - 1u) : 0u;
        const double z = RAW || !live ? 0.0 : a.inv_ds[s], coef = RAW || !live ? 0.0 : a.coef[s];
        __syncwarp();
        if (dirty) {
            if (QG < 8) atomicAnd(a.dirty + (dat >> 5), ~(((1u << NQ) - 1u) << (dat & 31)));  // two SVs share the byte
            else *db = 0;
        }
        uint4 *sums = rows_s + threadIdx.x;
#pragma unroll
        for (int k = 0; k < NW; k++) sums[k * G_THREADS] = make_uint4(acc[4 * k], acc[4 * k + 1], acc[4 * k + 2], acc[4 * k + 3]);
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
__global__ void ct_rows(gkm_rows sh, const uint32_t *__restrict__ fwd, const int32_t *__restrict__ counts, int64_t W,
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

// Neighbour masks of the suffix positions with 0 .. b mismatches for b = 1 ..
// 3, arranged so that lane k of every round holds a mask of bank class k (budget 1:
// the 16 masks twice): position | t << 12, or bit 31.
static void ct_lists(uint32_t *out)
{
    const int rounds[4] = {0, 1, CT_R2, CT_R3};
    uint32_t *p = out;
    for (int b = 1; b <= 3; b++) {
        int used[32] = {0}, n = 0;
        for (int k = 0; k < rounds[b] * 32; k++) p[k] = 0x80000000u;
        for (uint32_t x = 0; x < CT_ROWS; x++) {
            const int m = __builtin_popcount((x | (x >> 1)) & 0x55555555u), cls = ct_phys(x) & 31;
            const uint32_t e = ct_phys(x) | (uint32_t)(b - m) << 12;
            if (m > b) continue;
            if (b == 1) {
                p[n] = p[n + 16] = e;
                n++;
            } else {
                p[32 * used[cls]++ + cls] = e;
            }
        }
        p += rounds[b] * 32;
    }
}

// Masks of n positions (l - CT_POS of them) with m mismatches; returns how many.
static int ct_ball(int n, int m, uint32_t *out)
{
    int k = 0;
    for (uint32_t x = 0; x < (1u << (2 * n)); x++)
        if (__builtin_popcount((x | (x >> 1)) & 0x55555555u) == m) out[k++] = x;
    return k;
}

// How many: C(n, m) 3^m.  (Every call asks; looking through the masks took 20 us of host
// time for two levels at l = 11 and 44 for four.)
static int ct_ball_size(int n, int m)
{
    int c = 1;
    for (int k = 0; k < m; k++) c = c * 3 * (n - k) / (k + 1);
    return c;
}

// 16-bit gather sums (31 x windows) and the in-block sort bound the SV rows; weighted
// entries are bytes: three windows of the largest weight fit.
static bool ct_limits(const gkm_index *ix)
{
    const int l = ix->spec.l, D = ix->spec.dmax;
    return l >= 8 && l <= 11 && D >= 0 && D <= 3 && ix->W <= 2048 && ix->S >= 64 && ix->wmax <= 85;
}

int gkm_ct_build(gkm_index *ix, const uint32_t *fwd, const int32_t *counts, cudaStream_t st)
{
    ix->ct_ids = nullptr;
    const gkm_rows sh = gkm_rows_of(ix);
    if (!ct_limits(ix)) return GKM_OK;
    const int64_t S = ix->S;
    uint32_t *k0 = nullptr, *k1 = nullptr, *v1 = nullptr;
    int s = GKM_OK;
    uint32_t total = 0;
    do {
        if (cudaMalloc(&ix->ct_perm, sizeof(uint32_t) * S) != cudaSuccess ||
            cudaMalloc(&ix->ct_off, sizeof(uint32_t) * (S + 1)) != cudaSuccess ||
            cudaMalloc(&ix->ct_lists, sizeof(uint32_t) * (32 * CT_ROUNDS + CT_BALL)) != cudaSuccess ||
            cudaMallocAsync(&k0, sizeof(uint32_t) * (S + 1), st) != cudaSuccess ||
            cudaMallocAsync(&k1, sizeof(uint32_t) * (S + 1), st) != cudaSuccess ||
            cudaMallocAsync(&v1, sizeof(uint32_t) * (S + 1), st) != cudaSuccess) {
            s = gkm_fail(GKM_ERR_OOM, "gather lists");
            break;
        }
        uint32_t lists[32 * CT_ROUNDS + CT_BALL] = {};
        ct_lists(lists);
        for (int m = 0, k = 32 * CT_ROUNDS; m <= sh.D; m++) k += ct_ball(sh.l - CT_POS, m, lists + k);
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
            sh, fwd, counts, ix->W, ix->ct_perm, ix->ct_off, (uint32_t)gkm_row_count(ix),
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
    ix->ct_ids = ix->ct_off = ix->ct_perm = ix->ct_lists = nullptr;
    ix->ct_wts = nullptr;
    ix->ct_entries = 0;
}

// How a call is laid out: the row width and the workspace's parts.
struct CtPlan {
    bool wide;                // four bytes per query (weighted kernels, dense rows), else two
    int rb, qg, blocks, split;
    int64_t groups, rows, table, c, dirty, self, nexc, exc, partial, bytes;
    int pass, passes;         // queries of a count_tiles pass, passes of a full group
    int64_t rec_cap, chunk;   // window records of a pass, groups bucketed at a time
    int64_t recs, roff;
    int n_pre;
};

// Known average rows past this mean take wide entries: below it two bytes a query cost
// less (l = 10, 72,000 SVs: 10.2 against 13.5 us a 500 bp row; l = 11: 18.2 against 22.3
// at 1,800 bp), above it most tiles are counted twice (600 bp: 19.8 against 14.2; 2,000
// bp: 29.9 against 23.2).
constexpr double WIDE_MEAN = 3.4;

// The mean count of a table row at level dmax for rows of W window slots.
static double ct_mean(const gkm_index *ix, int64_t W)
{
    double reach = 1.0;
    for (int m = 0; m < ix->spec.dmax; m++) reach *= 3.0 * (ix->spec.l - m) / (m + 1);
    const double wx = ix->spec.weighted ? (double)gkm_weight_sum(ix, W) : (double)W;
    return (double)ix->strands * wx * reach / (double)ix->n_lmers;
}

static CtPlan ct_plan(const gkm_index *ix, int64_t B, int64_t W, int64_t windows)
{
    CtPlan p = {};
    // fields of 5 bits hold the AT-rich rows of five times a mean of 4.6 (a tile with a
    // larger count is counted again); past it, and for average rows past WIDE_MEAN,
    // unweighted rows, too, take the weighted ones' bytes, all weights 1
    p.wide = ix->spec.weighted || ct_mean(ix, W) > 4.6 || (windows > 0 && ct_mean(ix, windows / B < W ? windows / B : W) > WIDE_MEAN);
    const int wt = p.wide ? 4 : 2;
    // 32 queries a group: 64- or (weighted) 128-byte rows; the narrowest rows that
    // hold a smaller batch
    p.rb = wt * 32;
    while (p.rb > 4 * wt && p.rb / wt / 2 >= B) p.rb /= 2;
    p.qg = p.rb / wt;
    p.groups = (B + p.qg - 1) / p.qg;
    p.rows = gkm_row_count(ix);
    const int per_sm = p.wide ? G_BLOCKS_W : G_BLOCKS;
    p.blocks = gkm_query_blocks() * per_sm;
    // a power of two of lane groups within a warp for each SV, until every lane has
    // work (2,000 SVs of 200 .. 500 bp: 94 -> 47 us per group of 32 weighted queries, 36
    // -> 12 us unweighted; one query against 72,000: 125 -> 112 us)
    const int lanes = p.rb < 16 ? 1 : p.rb / 16;
    p.split = 1;
    while (lanes * p.split < 32 && ix->S * lanes * p.split < (int64_t)p.blocks * G_THREADS) p.split *= 2;
    auto up = [](int64_t n) { return (n + 255) & ~(int64_t)255; };
    p.table = up((p.rows + 2) * p.rb);
    p.self = up(B * 4 * 8);
    p.nexc = up(p.groups * 4);
    p.exc = p.wide ? up(8 * CT_EXC * (B < p.qg ? B : p.qg)) : 0;
    p.dirty = up(ix->S * p.qg / 8 + 8);
    p.c = up(ix->S * p.qg * 16);
    p.partial = up(p.groups * gkm_sm_count() * per_sm * p.qg * 8);  // (a grid limit only lowers p.blocks)
    // windows by bucket: the groups whose records fit 64 MB, at least one
    p.pass = p.wide ? CT_SLOTS : 2 * CT_SLOTS;
    p.passes = p.qg / p.pass > 0 ? p.qg / p.pass : 1;
    p.n_pre = 1 << (2 * (ix->spec.l - CT_POS));
    p.rec_cap = (int64_t)p.pass * W * ix->strands;
    const int64_t rec = p.wide ? sizeof(ct_rec<true>) : sizeof(ct_rec<false>);
    p.chunk = (64LL << 20) / (rec * p.rec_cap * p.passes);
    if (p.chunk < 1) p.chunk = 1;
    if (p.chunk > p.groups) p.chunk = p.groups;
    p.recs = up(rec * p.rec_cap * p.passes * p.chunk);
    p.roff = up(4 * (int64_t)(p.n_pre + 1) * p.passes * p.chunk);
    p.bytes = p.table + p.self + p.nexc + p.dirty + p.c + p.partial + p.recs + p.roff + p.exc;
    return p;
}

// Microseconds of a query, measured on B200 (l = 8 .. 11, d = 0 .. 3, 64 .. 72,000 SVs
// of 200 .. 350 bp, 1 .. 1,024 rows of 30 .. 2,000 bp).  Count tables: a wave of tile
// passes costs CT_ITEM_US plus CT_WINDOW_US per window of the pass's rows, the gather
// reads the SVs' table rows at CT_GATHER_BYTES_US.  Short l-mers have few positions
// outside the suffix, so most windows lie in the buckets of budget 0, which the warps
// share 32 buckets at a time: at l = 8, d = 2 one warp lists 27 of 37 parts of a pass's
// windows, CT_LIST_US per round of 32 (1,024 x 2,000 bp against 64 SVs: 13.0 ms, the
// walk 5.9).  And weighted counts past a mean of CT_RECOUNT_MEAN overflow the shared
// fields of most of their few tiles, which are then counted CT_RECOUNT times (the same
// rows, weighted: 61.7 against 5.3 ms).  Index walk: its lookups and hits, at least
// WALK_FLOOR_US (a few rows leave most SMs idle and a row's masks are a serial walk).
// Of 4,450 measured shapes 3,022 take the tables by these, 3 of them slower so (by up to
// 1.21; without the two terms for short l-mers 51, by up to 11.5).  At 72,000 SVs, t=3,
// the tables win from one 300 bp row (1.3 -> 0.2 ms) on; at 30 bp rows from 64 at a time
// the walk does (1,024 rows: 7.5 against 4.0 ms).
constexpr double CT_CALL_US = 45.0, CT_ITEM_US = 12.0, CT_WINDOW_US = 8.5e-4, CT_GATHER_BYTES_US = 8.0e6;
// K_raw rows (form): the walk of whole rows allocates nothing and starts at WALK_RAW_US; rows
// that it splits over the SMs cost at least WALK_FLOOR_US, for their counts.  By the scores'
// rule 81 of 1,896 measured shapes took the tables although slower, by up to 4.4 (256 rows of
// 30 bp against 64 SVs, l = 8, d = 2: 366 against 83 us), by this form's 6 do, by up to 1.26.
// A Gram matrix's index makes its lists first, CT_LISTS_US (50 to 460 measured), and its
// weighted counts at l = 10 are counted again the oftener the nearer their mean comes to
// CT_RECOUNT_MEAN10 (2,000 bp rows: 968 us a group where one count takes 273).
// A self-Gram's walk never splits rows: its longest row on one SM is its least (64 rows of up
// to 1,000 bp, l = 11, d = 3, weighted: 3,577 us, tables and lists 620).  Where the walk packs
// its counters it takes WALK_GRAM_PACKED times as long as other rows (100 rows of up to
// 400 bp, l = 11, d = 3: 5,400 us, tables and lists 490).
constexpr double WALK_RAW_US = 60.0, CT_LISTS_US = 100.0, CT_RECOUNT_MEAN10 = 55.0, WALK_GRAM_PACKED = 2.2;
constexpr double CT_LIST_US = 0.3, CT_RECOUNT = 4.0, CT_RECOUNT_MEAN = 24.0;
constexpr double WALK_FLOOR_US = 400.0, WALK_LOOKUP_US[2] = {8.0e-6, 5.8e-6}, WALK_HIT_US[2] = {1.1e-6, 2.0e-6};

// Whether every count stays below 2^32: the (row, SV) weight products of rows of W
// windows, summed over every pair of windows.
static bool ct_exact(const gkm_index *ix, int64_t W)
{
    const bool wt = ix->spec.weighted != 0;
    const uint64_t wx = wt ? gkm_weight_sum(ix, W) : (uint64_t)W, wy = wt ? gkm_weight_sum(ix, ix->W) : (uint64_t)ix->W;
    return wx && wy && wx < (1ull << 32) / ((uint64_t)ix->strands * wy);
}

// Whether a query over B rows of W window slots, `windows` windows in all, may
// take the count tables: the index has gather lists or is within their limits, no (row,
// SV, level) count reaches 2^32, the shared counters rarely overflow, and the estimated
// time is below the index walk's.
static bool ct_applies(const gkm_index *ix, int64_t B, int64_t W, int64_t windows, int form = GKM_ROWS_SCORES)
{
    if (!ct_limits(ix) || B < 1 || W < 1 || W > 60000 || B * ix->tiles > 0x7FFFFFFFLL) return false;
    if (!ct_exact(ix, W)) return false;
    const bool wt = ix->spec.weighted != 0;
    // bytes hold the AT-rich rows of three times this mean
    if (ct_mean(ix, W) > 80.0) return false;
    const int64_t known = windows;
    if (windows <= 0) windows = B * W / 2;  // lengths unknown: rows padded to W
    const CtPlan p = ct_plan(ix, B, W, known);
    const int64_t items = p.rows / CT_ROWS * p.passes;
    const double row = (double)windows / B < W ? (double)windows / B : (double)W, waves = (double)((items + gkm_sm_count() * CT_BLOCKS - 1) / (gkm_sm_count() * CT_BLOCKS));
    const double queries = (double)(B < p.pass ? B : p.pass);
    // rounds of 32 windows that a warp lists from the buckets of budget 0
    const double far = ct_ball_size(ix->spec.l - CT_POS, ix->spec.dmax);
    const double warps = far > 32.0 * CT_WARPS ? CT_WARPS : ceil(far / 32.0);
    const double list = ix->strands * row * queries * far / p.n_pre / 32.0 / warps;
    const double window = CT_WINDOW_US * row * queries;
    double slow = CT_ITEM_US + (window > CT_LIST_US * list ? window : CT_LIST_US * list);
    if (wt && ix->spec.l <= 9 && ct_mean(ix, W) > CT_RECOUNT_MEAN) slow *= CT_RECOUNT;
    if (wt && ix->spec.l == 10 && form == GKM_ROWS_GRAM) {
        const double x = ct_mean(ix, W) / CT_RECOUNT_MEAN10;
        slow *= 1.0 + (CT_RECOUNT - 1.0) * (x < 1.0 ? x * x : 1.0);
    }
    // (lists not made yet: four windows of padding an SV)
    const double entries = ix->ct_ids ? (double)ix->ct_entries : (double)ix->entries / ix->strands + 4.0 * ix->S;
    const double gather = entries * p.rb / CT_GATHER_BYTES_US;
    const double table = CT_CALL_US + p.groups * (waves * (CT_ITEM_US + window) + gather),
                 table_slow = CT_CALL_US + p.groups * (waves * slow + gather);
    double walk = (double)windows * (ix->n_masks * (double)ix->tiles * WALK_LOOKUP_US[wt] +
                                     (double)ix->entries * ix->n_masks / ix->n_lmers * WALK_HIT_US[wt]);
    double raw = walk;
    if (walk < WALK_FLOOR_US) walk = WALK_FLOOR_US;
    if (form == GKM_ROWS_SCORES) return table < 0.9 * walk && table_slow < walk;
    // K_raw rows: whole rows leave the last of their waves of SMs partly idle
    const double rows = (double)B * ix->tiles, sms = gkm_sm_count();
    const double longest = raw / (double)windows * W * sms / ix->tiles;
    if (form == GKM_ROWS_GRAM || !gkm_walk_splits(ix, B, W)) raw = WALK_RAW_US + raw * ceil(rows / sms) * sms / rows;
    if (form == GKM_ROWS_GRAM) {
        // rows are never split, so the longest one bounds it
        if (raw < WALK_RAW_US + longest) raw = WALK_RAW_US + longest;
        walk = ix->packed ? WALK_GRAM_PACKED * raw : raw;
    } else if (raw < walk && !gkm_walk_splits(ix, B, W)) {
        walk = raw;
    }
    const double lists = ix->ct_ids ? 0.0 : CT_LISTS_US;
    return table + lists < 0.9 * walk && table_slow + lists < walk;
}

extern "C" int gkm_count_table_workspace(const gkm_index_t *ix, int64_t B, int64_t W, int64_t windows, int64_t *bytes)
{
    if (!ix || !bytes) return gkm_fail(GKM_ERR_INVALID, "null argument");
    *bytes = ix->ct_ids && ct_applies(ix, B, W, windows) ? ct_plan(ix, B, W, windows).bytes : 0;
    return GKM_OK;
}

extern "C" int gkm_count_table_pays(const gkm_index_t *ix, int64_t B, int64_t W, int64_t windows, int32_t form,
                                    int32_t *pays)
{
    if (!ix || !pays) return gkm_fail(GKM_ERR_INVALID, "null argument");
    if (form < GKM_ROWS_SCORES || form > GKM_ROWS_GRAM) return gkm_fail(GKM_ERR_INVALID, "form %d", form);
    // (the workspace call goes by the scores' rule)
    *pays = ct_applies(ix, B, W, windows) && ct_applies(ix, B, W, windows, form) ? 1 : 0;
    return GKM_OK;
}

extern "C" int gkm_count_table_query(const gkm_index_t *ix, const uint32_t *bx, const int32_t *cx, int64_t B,
                                     int64_t W, int64_t windows, const int32_t *order, int32_t normalize,
                                     const double *inv_dx, double *diag, int64_t diag_offset, double *raw, const double *inv_ds,
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
    if (!ix->ct_ids || W > 60000) return gkm_fail(GKM_ERR_UNSUPPORTED, "this index or shape has no count tables");
    if (!ct_exact(ix, W))
        return gkm_fail(GKM_ERR_UNSUPPORTED, "a pair count of rows of %lld windows could pass 2^32", (long long)W);
    const CtPlan p = ct_plan(ix, B, W, windows);
    if (!workspace || ((uintptr_t)workspace & 255) || workspace_bytes < p.bytes)
        return gkm_fail(GKM_ERR_CAPACITY, "count tables need a 256-byte aligned workspace of %lld bytes", (long long)p.bytes);
    cudaStream_t st = (cudaStream_t)stream;
    const bool wt = p.wide;
    CtArgs a = {};
    a.bx = bx;
    a.cx = cx;
    a.W = W;
    a.order = order;
    a.qg = p.qg;
    a.rb = p.rb;
    a.sh = gkm_rows_of(ix);
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
    uint8_t *recs = w;
    w += p.recs;
    uint32_t *roff = (uint32_t *)w;
    w += p.roff;
    a.exc = (unsigned long long *)w;
    a.cap_exc = (unsigned)(p.exc / 8);
    cudaError_t e = cudaMemsetAsync(z0, 0, (size_t)((uint8_t *)partial - z0), st);
    if (e != cudaSuccess) return gkm_cuda_status(e, "count table workspace");
    a.wd = ix->spec.weighted ? ix->spec.wd : nullptr;
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
    a.split = p.split;
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
    a.ball = ix->ct_lists + 32 * CT_ROUNDS;
    for (int m = 0; m < 4; m++) a.nball[m] = m <= a.sh.D ? ct_ball_size(a.sh.l - CT_POS, m) : 0;
    a.n_pre = p.n_pre;
    a.rec_cap = p.rec_cap;
    auto count = wt ? count_tiles<true> : count_tiles<false>;
    // two blocks' shared memory, the rest of the SM's for L1
    GKM_ALLOW_SHARED(count, sizeof(uint32_t) * CT_ROWS * (CT_SLOTS + 1));
    cudaFuncSetAttribute(count, cudaFuncAttributePreferredSharedMemoryCarveout, 86);
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
            if (wt) ct_buckets<true><<<n, CB_THREADS, 0, st>>>(a, B);
            else ct_buckets<false><<<n, CB_THREADS, 0, st>>>(a, B);
            GKM_CHECK_LAUNCH("ct_buckets");
        }
        a.recs = recs + (g % p.chunk) * p.passes * p.rec_cap * (wt ? sizeof(ct_rec<true>) : sizeof(ct_rec<false>));
        a.roff = roff + (g % p.chunk) * p.passes * (p.n_pre + 1);
        const int nqp = a.nq < p.pass ? a.nq : p.pass;
        // four queries (or those there are) x four levels for the 32-bit recount
        int words = wt ? nqp : (nqp + 1) / 2;
        if (words < 4 * (nqp < 4 ? nqp : 4)) words = 4 * (nqp < 4 ? nqp : 4);
        const size_t smem = sizeof(uint32_t) * (size_t)CT_ROWS * (words + 1);  // + alignment
        a.passes = (a.nq + p.pass - 1) / p.pass;
        a.items = (int)(p.rows / CT_ROWS) * a.passes;
        // a block keeps its pass (its windows stay in L1), the passes of a tile
        // run side by side (their parts of a table row meet in L2)
        const int fit = gkm_query_blocks() * CT_BLOCKS / a.passes * a.passes;
        const unsigned grid = (unsigned)(a.items < fit ? a.items : fit > 0 ? fit : a.passes);
        count<<<grid, CT_THREADS, smem, st>>>(a);
        GKM_CHECK_LAUNCH("count_tiles");
        if (wt) {
            spill_excess<<<(unsigned)gkm_sm_count() * 4, 256, 0, st>>>(a);
            GKM_CHECK_LAUNCH("spill_excess");
        }
#define GKM_GATHER_AS(RB, WT, RAW)                                                                        \
    do {                                                                                                  \
        if (p.split > 1) gather_kernel<RB, WT, RAW, true><<<p.blocks, G_THREADS, 0, st>>>(a);             \
        else gather_kernel<RB, WT, RAW, false><<<p.blocks, G_THREADS, 0, st>>>(a);                        \
    } while (0)
#define GKM_GATHER(RB, WT)                                                                                \
    do {                                                                                                  \
        if (raw) GKM_GATHER_AS(RB, WT, true);                                                             \
        else GKM_GATHER_AS(RB, WT, false);                                                                \
    } while (0)
        if (p.rb == 8) GKM_GATHER(8, false);
        else if (p.rb == 16 && wt) GKM_GATHER(16, true);
        else if (p.rb == 16) GKM_GATHER(16, false);
        else if (p.rb == 32 && wt) GKM_GATHER(32, true);
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
