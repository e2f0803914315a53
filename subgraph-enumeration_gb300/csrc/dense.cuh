// The dense-root path of the counting launch: roots whose ends share
// neighbours are counted on bitsets instead of sorted lists.
//
// A plan whose level 2 closes a triangle on the root edge and whose later
// levels all touch the root takes every candidate from one small universe
// U(root): N(m0) ∩ N(m1), N(m0), N(m1) or their union.  For such a root the
// launch builds one bit row per vertex of U (its neighbours inside U).  A
// level's candidates are then the AND of a few rows, its bounds are masks, and
// the last level is a population count: 32 candidates a word, with no
// per-element search.  The rows are shared by every plan of the launch (per
// root edge and universe); the tasks are (root, plan and orientation, level-2
// candidate, part of its level-3 list), and a warp runs one at a time.
//
// U is laid out in three segments, each sorted by id and padded to a word:
// the common neighbours, the other neighbours of u, the other neighbours of v.
// A level whose parents hold both root ends then lives in the first words
// only, and the membership masks of N(u) and N(v) are whole segments.
//
// Bound by instruction issue and L1 latency of the warp's depth-first steps;
// the rows of a root (at most 0.5 MB) stay in L1/L2.  Kernel time, lists ->
// rows: 78 seven-vertex patterns (16-19 edges) on 488 root edges of R-MAT 2^22
// 1,010 -> 17 ms; 16 six-vertex patterns on 976 root edges of R-MAT 2^20
// 20.7 -> 2.0 ms; K5 over every root of R-MAT 2^14 172 -> 97 ms.
//
// Included by engine.cu inside its anonymous namespace.
#pragma once

constexpr uint32_t DENSE_MAX_U = 2048;   // vertices of a universe (padded segments): 64 words a row, two per lane
constexpr uint32_t DENSE_WORDS = DENSE_MAX_U / 32;
constexpr uint32_t DENSE_MAX_K = 8;      // levels the running masks in shared memory are sized for
constexpr uint32_t DENSE_MAX_T = 3;      // inclusion–exclusion tail levels (2^T counters per lane)
constexpr uint32_t DENSE_ROWS = 256;     // rows per build item
constexpr uint32_t DENSE_MIN_N2 = 8, DENSE_MIN_DEG = 64, DENSE_MIN_WORDS = 3;   // see dense_worth
constexpr int DENSE_SPLIT_LOG2 = 9;      // a level-2 candidate is split once |U|^2 n2 passes 2^19
constexpr uint32_t DENSE_CAND = 16;      // level-2 candidates per task of a small root
// Universe classes of a root edge (u, v), u < v.
enum { DENSE_BOTH = 0, DENSE_U = 1, DENSE_V = 2, DENSE_UNION = 3 };
constexpr uint32_t DENSE_NONE = 0xFFFFFFFFu;

// One root edge with its universes: off[c] is the arena offset (in 16-byte
// units) of class c, DENSE_NONE when it is absent.
struct DenseRec {
    uint32_t u, v, n2, du, dv;   // n2 = |N(u) ∩ N(v)|
    uint32_t off[4];
};
// A class in the arena: a header, the ranks of each position (by position),
// and one row of `pitch` words per position.
struct DenseHead {
    // elements of U with an id <= u's, per segment, and the segment that holds u (3: none); the same for v
    uint16_t ucnt[4], vcnt[4];
};
static_assert(sizeof(DenseHead) == 16, "one arena unit");

// One (plan, orientation) of the launch.
struct DensePO {
    uint32_t plan;
    uint32_t cls;    // universe class for this orientation
    uint32_t swap;   // 1: m0 = v, m1 = u
};

struct DenseBuf {
    uint32_t *hdr;             // [0] records, [1] build queue, [2..3] arena units in use, [4..5] task queue, [6..7] tasks per (plan, orientation)
    DenseRec *recs;
    uint32_t *order;           // records, largest first
    unsigned long long *pre;   // exclusive prefix of their task counts in that order
    uint8_t *skip;             // per sampled root edge: bit c = counted here for class c
    uint4 *arena;
    const DensePO *po;
    unsigned long long arena_units;  // 16-byte units
    uint32_t rec_cap, npo, need;     // need: classes any plan of the launch uses
    uint32_t rows_both;              // classes whose plans only read rows of N(u) ∩ N(v)
    uint32_t rich;                   // classes of plans that lists serve badly: rows for all roots but the smallest
};

// Segment sizes of class c and the word each segment starts at.
struct DenseShape {
    uint32_t n[3];     // common, only N(u), only N(v)
    uint32_t w1, w2, w3, pitch;
};
__host__ __device__ inline DenseShape dense_shape(uint32_t c, uint32_t n2, uint32_t du, uint32_t dv) {
    DenseShape s;
    s.n[0] = n2;
    s.n[1] = (c == DENSE_U || c == DENSE_UNION) ? du - n2 : 0u;
    s.n[2] = (c == DENSE_V || c == DENSE_UNION) ? dv - n2 : 0u;
    s.w1 = (s.n[0] + 31u) / 32u;
    s.w2 = s.w1 + (s.n[1] + 31u) / 32u;
    s.w3 = s.w2 + (s.n[2] + 31u) / 32u;
    s.pitch = (s.w3 + 3u) & ~3u;
    return s;
}
// 16-byte units of a class: header, 8 bytes of ranks and a row per position
__host__ __device__ inline unsigned long long dense_units(uint32_t words) {
    const uint32_t pitch = (words + 3u) & ~3u;
    return 1ull + 16ull * words + 32ull * words * (pitch / 4u);
}
struct DenseView {
    const DenseHead *head;
    const uint2 *rank;     // per position: (cnt0 | cnt1 << 16, cnt2 | segment << 16), counts of ids <= its own
    const uint32_t *rows;
    DenseShape s;
};
__device__ __forceinline__ DenseView dense_view(const DenseBuf &D, const DenseRec &R, uint32_t c) {
    DenseView v;
    v.s = dense_shape(c, R.n2, R.du, R.dv);
    v.head = reinterpret_cast<const DenseHead *>(D.arena + R.off[c]);
    v.rank = reinterpret_cast<const uint2 *>(v.head + 1);
    v.rows = reinterpret_cast<const uint32_t *>(v.rank + 32u * v.s.w3);
    return v;
}
// Roots that take the path.  Building U and a task cost some 10 us of a warp,
// which a root with few common neighbours and no wider universe earns back
// only from about 8 of them on (K5 over every root of a 7,100-vertex
// Chung-Lu graph: lists 9.2 ms, from 2 on 8.3 ms, 8 on 7.1 ms, 24 on 6.4 ms;
// of a 1,500-vertex one: 0.73, 0.27, 0.24, 0.50 ms), and not while both lists
// are one step of a warp (a ring lattice of degree 24: 39 ms, with rows 45).
// The list path knows only the degrees before it starts: it splits a root
// between two large lists into thousands of tasks even when one common
// neighbour is in them, and with a wider universe it scans N(m0) or N(m1) below
// every partial match, so there one common neighbour pays (78 seven-vertex
// patterns on R-MAT 2^22: 21 ms, from 8 on 46 ms, 24 on 72 ms, lists 1,010 ms).
// Where edges share few neighbours, lists are not split and every level is cut
// by two of them (D.rich clear), a plan matches some n2^2 / 2 prefixes, which
// have to make up for |U| rows (octahedra and 4-wheels on a Chung-Lu graph of
// mean degree 7: lists 1.8 and 2.1 ms, rows for all 14.7 and 15.3).
__device__ __forceinline__ bool dense_worth(const DenseBuf &D, uint32_t c, uint32_t n2, uint32_t du, uint32_t dv,
                                            uint32_t words) {
    if (!((D.rich >> c) & 1u)) return n2 >= DENSE_MIN_N2 && max(du, dv) > 32u && (c == DENSE_BOTH || n2 * n2 >= 32u * words);
    return min(du, dv) >= DENSE_MIN_DEG || (n2 >= DENSE_MIN_N2 && max(du, dv) > 32u) ||
           (c != DENSE_BOTH && (n2 >= 2 || words >= DENSE_MIN_WORDS));
}
// Tasks of a record per (plan, orientation): large universes split each
// level-2 candidate into 2^s parts of its level-3 list (the positions = q mod
// 2^s), small ones take DENSE_CAND candidates at a time.  s grows with the
// work under one candidate, about |U|^2.
__device__ __forceinline__ uint32_t dense_parts_log2(const DenseBuf &D, const DenseRec &R) {
    uint32_t words = 0;
    for (uint32_t c = 0; c < 4; ++c)
        if (R.off[c] != DENSE_NONE) words = max(words, dense_shape(c, R.n2, R.du, R.dv).w3);
    const unsigned long long est = (unsigned long long)words * words * R.n2;   // |U|^2 n2 / 2^10
    const int s = 63 - __clzll(est | 1ull) - DENSE_SPLIT_LOG2;
    return s <= 0 ? 0u : min((uint32_t)s, 5u);
}
__device__ __forceinline__ uint32_t dense_tasks(uint32_t n2, uint32_t ps) {
    return ps ? n2 << ps : (n2 + DENSE_CAND - 1) / DENSE_CAND;
}

// Selects the dense roots: one warp per sampled root edge intersects the two
// lists (the shorter one scanned), and the edge gets a record and arena space
// for every class that fits and is worth it.  Bound by the list loads, as a triangle count of the sample.
// The launch's time budget starts here (flags + 2 holds the start).
__global__ void __launch_bounds__(256) dense_select_kernel(DevGraph g, unsigned long long root_offset,
                                                           unsigned long long root_stride, unsigned long long nedges,
                                                           uint32_t maxdeg, DenseBuf D, unsigned long long deadline_ns,
                                                           uint32_t *flags) {
    const uint32_t lane = lane_id();
    const unsigned long long nw = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
    Ctx<MODE_PLAIN> c;
    c.flags = flags;
    c.deadline = deadline_ns;
    unsigned long long t0 = 0;
    if (lane == 0) {
        volatile unsigned long long *slot = reinterpret_cast<volatile unsigned long long *>(flags + 2);
        if (blockIdx.x == 0 && threadIdx.x == 0) *slot = globaltimer_ns();
        if (deadline_ns) t0 = *slot;
        if (!t0) t0 = globaltimer_ns();   // (block 0 has not begun)
    }
    c.tstart = __shfl_sync(FULL_MASK, t0, 0);
    for (unsigned long long j = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; j < nedges; j += nw) {
        if (out_of_time(c)) break;
        const uint2 e = g.edges[root_offset + j * root_stride];
        const uint32_t *pu, *pv;
        uint32_t du, dv;
        nbr(g, e.x, pu, du);
        nbr(g, e.y, pv, dv);
        if (min(du, dv) > DENSE_MAX_U || (D.need == 1u << DENSE_BOTH && min(du, dv) < DENSE_MIN_N2)) continue;
        if (maxdeg && max(du, dv) > maxdeg) continue;
        const bool sw = dv < du;
        const uint32_t *a = sw ? pv : pu, *b = sw ? pu : pv;
        const uint32_t na = min(du, dv), nb = max(du, dv);
        const int32_t hs = hub_slot_of(g, sw ? e.x : e.y, nb);
        uint32_t n2 = 0;
        for (uint32_t i = 0; i < na; i += 32) {
            bool ok = i + lane < na;
            if (ok) {
                const uint32_t y = a[i + lane];
                ok = hs >= 0 ? hub_has(g, hs, y) : contains(b, nb, y);
            }
            n2 += __popc(__ballot_sync(FULL_MASK, ok));
        }
        __syncwarp();
        if (lane != 0) continue;
        if (n2 == 0) { D.skip[j] = (uint8_t)D.need; continue; }   // no level-2 candidate: nothing to count
        unsigned long long units = 0;
        uint32_t have = 0;
        for (uint32_t c = 0; c < 4; ++c) {
            const uint32_t words = dense_shape(c, n2, du, dv).w3;
            if (((D.need >> c) & 1u) && words <= DENSE_WORDS && dense_worth(D, c, n2, du, dv, words)) { units += dense_units(words); have |= 1u << c; }
        }
        if (!have) continue;
        unsigned long long at = atomicAdd(reinterpret_cast<unsigned long long *>(D.hdr + 2), units);
        if (at + units > D.arena_units) continue;   // no room: the list path counts this root
        const uint32_t slot = atomicAdd(D.hdr, 1u);
        if (slot >= D.rec_cap) continue;
        DenseRec R;
        R.u = e.x;
        R.v = e.y;
        R.n2 = n2;
        R.du = du;
        R.dv = dv;
        for (uint32_t c = 0; c < 4; ++c) {
            R.off[c] = DENSE_NONE;
            if ((have >> c) & 1u) { R.off[c] = (uint32_t)at; at += dense_units(dense_shape(c, n2, du, dv).w3); }
        }
        D.recs[slot] = R;
        D.skip[j] = (uint8_t)have;
    }
}

// Exclusive prefix sum of one value per thread over a 256-thread block.
__device__ __forceinline__ uint32_t block_prefix256(uint32_t v, uint32_t *ws, uint32_t &total) {
    const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(FULL_MASK, incl, o);
        if (lane >= o) incl += t;
    }
    __syncthreads();
    if (lane == 31) ws[w] = incl;
    __syncthreads();
    uint32_t before = 0;
    total = 0;
    for (uint32_t q = 0; q < 8; ++q) {
        if (q < w) before += ws[q];
        total += ws[q];
    }
    return before + incl - v;
}

// Fills one class of one record, DENSE_ROWS rows per item: the universe in
// shared memory, then a warp per row.  A hub's row is gathered from its
// bitmap (one load per bit, 32 bits a ballot); a shorter list is scanned and
// each neighbour looked up in U; a long list without a bitmap is searched.
__global__ void __launch_bounds__(256) dense_build_kernel(DevGraph g, DenseBuf D, unsigned long long deadline_ns,
                                                          uint32_t *flags) {
    __shared__ uint32_t Us[DENSE_MAX_U];         // the universe, sorted by id
    __shared__ uint32_t C[DENSE_MAX_U];          // common neighbours before index i of the shorter list; then counts
    __shared__ uint32_t Up[DENSE_MAX_U];         // the universe by position (DENSE_NONE: padding)
    __shared__ uint16_t pos[DENSE_MAX_U];        // position of Us[i]
    __shared__ uint32_t row[8][DENSE_WORDS];
    __shared__ uint32_t ws[8];
    __shared__ uint32_t item_s;
    constexpr uint32_t PARTS = DENSE_MAX_U / DENSE_ROWS, PER = DENSE_MAX_U / 256u;
    const uint32_t lane = lane_id(), wib = threadIdx.x >> 5, i0 = threadIdx.x * PER;
    const uint32_t ncls = __popc(D.need), nitems = min(D.hdr[0], D.rec_cap) * ncls * PARTS;
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) {
            bool late = false;
            if (deadline_ns) late = globaltimer_ns() - *reinterpret_cast<volatile unsigned long long *>(flags + 2) > deadline_ns;
            if (late) atomicOr(flags, FLAG_TIMEOUT);   // (the count kernel then takes no task)
            item_s = late ? 0xFFFFFFFFu : atomicAdd(D.hdr + 1, 1u);
        }
        __syncthreads();
        const uint32_t item = item_s;
        if (item >= nitems) break;
        const DenseRec &R = D.recs[item / (ncls * PARTS)];
        const uint32_t c = __fns(D.need, 0, (int)((item / PARTS) % ncls) + 1), part = item % PARTS;
        if (R.off[c] == DENSE_NONE) continue;
        const DenseView V = dense_view(D, R, c);
        const bool only_both = (D.rows_both >> c) & 1u;
        const uint32_t nrows = only_both ? R.n2 : V.s.w3 * 32u;
        if (part && part * DENSE_ROWS >= nrows) continue;
        const uint32_t pitch = V.s.pitch, nus = V.s.n[0] + V.s.n[1] + V.s.n[2];
        const uint32_t *pu, *pv;
        uint32_t du, dv;
        nbr(g, R.u, pu, du);
        nbr(g, R.v, pv, dv);
        const int32_t hu = hub_slot_of(g, R.u, du), hv = hub_slot_of(g, R.v, dv);
        auto in_u = [&](uint32_t y) { return c == DENSE_U || c == DENSE_BOTH || (hu >= 0 ? hub_has(g, hu, y) : contains(pu, du, y)); };
        auto in_v = [&](uint32_t y) { return c == DENSE_V || c == DENSE_BOTH || (hv >= 0 ? hub_has(g, hv, y) : contains(pv, dv, y)); };
        // 1. the universe, sorted
        if (c == DENSE_U || c == DENSE_V) {
            const uint32_t *p = c == DENSE_U ? pu : pv;
            for (uint32_t i = threadIdx.x; i < nus; i += 256) Us[i] = p[i];
        } else {
            const bool sw = dv < du;
            const uint32_t *a = sw ? pv : pu, *b = sw ? pu : pv;
            const uint32_t na = min(du, dv), nb = max(du, dv);
            const int32_t hb = sw ? hu : hv;
            uint32_t fl = 0, mine = 0, total = 0;
            for (uint32_t q = 0; q < PER; ++q)
                if (i0 + q < na) {
                    const uint32_t y = a[i0 + q];
                    if (hb >= 0 ? hub_has(g, hb, y) : contains(b, nb, y)) { fl |= 1u << q; ++mine; }
                }
            uint32_t at = block_prefix256(mine, ws, total);
            for (uint32_t q = 0; q < PER; ++q)
                if (i0 + q < na) {
                    const uint32_t y = a[i0 + q];
                    C[i0 + q] = at;
                    if (c == DENSE_BOTH) {
                        if ((fl >> q) & 1u) Us[at] = y;
                    } else {
                        Us[i0 + q + lb(b, nb, y) - at] = y;   // union: rank in both lists, common ones once
                    }
                    at += (fl >> q) & 1u;
                }
            __syncthreads();
            if (c == DENSE_UNION)
                for (uint32_t i = threadIdx.x; i < nb; i += 256) {
                    const uint32_t y = b[i], r = lb(a, na, y);
                    if (r < na && a[r] == y) continue;
                    Us[i + r - (r < na ? C[r] : total)] = y;
                }
        }
        for (uint32_t i = threadIdx.x; i < V.s.w3 * 32u; i += 256) Up[i] = DENSE_NONE;
        __syncthreads();
        // 2. segments: position and ranks of every element (C[i] = common ones up to i | only-u ones << 16)
        {
            uint32_t mine = 0, total = 0, seg = 0;
            for (uint32_t q = 0; q < PER; ++q)
                if (i0 + q < nus) {
                    const uint32_t y = Us[i0 + q];
                    const bool iu = in_u(y), iv = in_v(y);
                    seg |= (iu && iv ? 0u : iu ? 1u : 2u) << (2 * q);
                    mine += iu && iv ? 1u : iu ? 1u << 16 : 0u;
                }
            uint32_t at = block_prefix256(mine, ws, total);
            uint2 *rank = const_cast<uint2 *>(V.rank);
            for (uint32_t q = 0; q < PER; ++q)
                if (i0 + q < nus) {
                    const uint32_t i = i0 + q, sg = (seg >> (2 * q)) & 3u;
                    const uint32_t n0 = at & 0xFFFFu, n1 = at >> 16, n2 = i - n0 - n1;
                    const uint32_t p = sg == 0 ? n0 : sg == 1 ? V.s.w1 * 32u + n1 : V.s.w2 * 32u + n2;
                    at += sg == 0 ? 1u : sg == 1 ? 1u << 16 : 0u;
                    C[i] = at;
                    pos[i] = (uint16_t)p;
                    Up[p] = Us[i];
                    if (part == 0) rank[p] = make_uint2(at, (i + 1 - (at & 0xFFFFu) - (at >> 16)) | (sg << 16));
                }
        }
        __syncthreads();
        if (part == 0 && threadIdx.x < 2) {
            DenseHead *hd = const_cast<DenseHead *>(V.head);
            const uint32_t x = threadIdx.x ? R.v : R.u, r = ub(Us, nus, x);
            uint16_t *o = threadIdx.x ? hd->vcnt : hd->ucnt;
            const uint32_t at = r ? C[r - 1] : 0u;
            o[0] = (uint16_t)(at & 0xFFFFu);
            o[1] = (uint16_t)(at >> 16);
            o[2] = (uint16_t)(r - (at & 0xFFFFu) - (at >> 16));
            const bool in = r && Us[r - 1] == x;
            const uint32_t w = in ? pos[r - 1] >> 5 : 0u;
            o[3] = in ? (w < V.s.w1 ? 0 : w < V.s.w2 ? 1 : 2) : 3;
        }
        // 3. rows
        const uint32_t r1 = min(nrows, (part + 1) * DENSE_ROWS);
        for (uint32_t i = part * DENSE_ROWS + wib; i < r1; i += 8) {
            const uint32_t x = Up[i];
            if (x == DENSE_NONE) continue;
            const uint32_t *px;
            uint32_t dx;
            nbr(g, x, px, dx);
            const int32_t hx = hub_slot_of(g, x, dx);
            uint32_t w0 = 0, w1 = 0;   // words lane and lane + 32 of the row
            if (hx < 0 && dx <= 2u * nus) {
                uint32_t *rw = row[wib];
                for (uint32_t w = lane; w < pitch; w += 32) rw[w] = 0;
                __syncwarp();
                for (uint32_t e = lane; e < dx; e += 32) {
                    const uint32_t y = px[e], k = lb(Us, nus, y);
                    if (k < nus && Us[k] == y) {
                        const uint32_t p = pos[k];
                        atomicOr(&rw[p >> 5], 1u << (p & 31u));
                    }
                }
                __syncwarp();
                if (lane < pitch) w0 = rw[lane];
                if (lane + 32 < pitch) w1 = rw[lane + 32];
                __syncwarp();
            } else {
                for (uint32_t w = 0; w < V.s.w3; ++w) {
                    const uint32_t y = Up[w * 32 + lane];
                    bool ok = y != DENSE_NONE;
                    if (ok) ok = hx >= 0 ? hub_has(g, hx, y) : contains(px, dx, y);
                    const uint32_t b = __ballot_sync(FULL_MASK, ok);
                    if ((w & 31u) == lane) { if (w < 32) w0 = b; else w1 = b; }
                }
            }
            uint32_t *o = const_cast<uint32_t *>(V.rows) + (size_t)i * pitch;
            if (lane < pitch) o[lane] = w0;
            if (lane + 32 < pitch) o[lane + 32] = w1;
        }
    }
}

// Orders the records by falling work (the largest roots start first, so that
// none of them ends the launch alone) and numbers their tasks; one block.
__global__ void __launch_bounds__(256) dense_prefix_kernel(DenseBuf D) {
    constexpr uint32_t BINS = 256;   // work in eighths of a power of two
    __shared__ uint32_t bin[BINS];
    __shared__ uint32_t ws[8];
    const uint32_t n = min(D.hdr[0], D.rec_cap);
    auto bin_of = [&](uint32_t i) {
        const DenseRec &R = D.recs[i];
        uint32_t words = 0;
        for (uint32_t c = 0; c < 4; ++c)
            if (R.off[c] != DENSE_NONE) words = max(words, dense_shape(c, R.n2, R.du, R.dv).w3);
        const uint32_t est = max(words * words * R.n2, 8u), e = 31u - __clz(est);
        return BINS - 1u - min(e * 8u + ((est >> (e - 3u)) & 7u), BINS - 1u);
    };
    bin[threadIdx.x] = 0;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += 256) atomicAdd(&bin[bin_of(i)], 1u);
    __syncthreads();
    uint32_t total = 0;
    const uint32_t first = block_prefix256(bin[threadIdx.x], ws, total);
    bin[threadIdx.x] = first;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += 256) D.order[atomicAdd(&bin[bin_of(i)], 1u)] = i;
    __syncthreads();
    unsigned long long run = 0;
    for (uint32_t b = 0; b < n; b += 256) {
        const uint32_t i = b + threadIdx.x;
        uint32_t v = 0;
        if (i < n) {
            const DenseRec &R = D.recs[D.order[i]];
            v = dense_tasks(R.n2, dense_parts_log2(D, R));
        }
        const uint32_t at = block_prefix256(v, ws, total);
        if (i < n) D.pre[i] = run + at;
        run += total;
    }
    if (threadIdx.x == 0) *reinterpret_cast<unsigned long long *>(D.hdr + 6) = run;
}

// Per-warp shared memory of the dense count, with as many running rows as the
// launch's longest plan uses (dense_slots), which decides the resident warps:
// 24 per SM with all 20 slots and counters per lane beside them, 32 for
// seven-vertex plans with the counters in registers (78 such plans on 976 root
// edges of R-MAT 2^22: the launch sequence 35.8 -> 33.5 ms; then a level's masks
// as one word and no local arrays in the loops, 32.3 ms).
struct alignas(16) DenseWarp {
    uint16_t ylist[DENSE_MAX_U / 2];
    uint32_t lev[DENSE_MAX_K];   // level i in entry i - 1: parents | lower << 8 | upper << 16
    // Behind the struct, slot s = dense_slot(d, i): candidates of level i after
    // matching level d (word w of lane w % 32), for d = 1..ne-2 and i = d+1..k-1.
    __device__ __forceinline__ uint32_t *run(uint32_t s) {
        return reinterpret_cast<uint32_t *>(this + 1) + s * DENSE_WORDS;
    }
};
// Slots for k = DENSE_MAX_K: six levels after the root, five after level 2, ...
__host__ __device__ constexpr uint32_t dense_slot(uint32_t d, uint32_t i) {
    const uint32_t r = d - 1;                        // rows d' < d hold 6, 5, 4, ... slots
    return r * (2u * (DENSE_MAX_K - 2u) - r + 1u) / 2u + (i - d - 1u);
}
// Slots a k-vertex plan uses: the prefix ends at level ne-2 <= k-3.
__host__ __device__ constexpr uint32_t dense_slots(uint32_t k) { return dense_slot(k - 3, k - 1) + 1u; }
__host__ __device__ constexpr size_t dense_warp_bytes(uint32_t slots) {
    return sizeof(DenseWarp) + slots * DENSE_WORDS * sizeof(uint32_t);
}

// Word of a segment: its ranks from `c` on (t = c - the word's first rank).
__device__ __forceinline__ uint32_t dense_from(int t) { return __funnelshift_lc(0u, 0xFFFFFFFFu, (uint32_t)max(t, 0)); }

// A lane's view of word w: its segment and the rank of its first position.
struct DenseLane {
    uint32_t seg;
    int first;
};
__device__ __forceinline__ DenseLane dense_lane(const DenseShape &s, uint32_t w) {
    DenseLane l;
    l.seg = w < s.w1 ? 0u : w < s.w2 ? 1u : 2u;
    l.first = (int)((w - (l.seg == 0 ? 0u : l.seg == 1 ? s.w1 : s.w2)) * 32u);
    return l;
}
// Elements of the lane's segment with an id <= that of the vertex whose ranks
// are r, from the word's first on.
__device__ __forceinline__ int dense_rank(const DenseLane &l, uint2 r) {
    return (int)(l.seg == 0 ? r.x & 0xFFFFu : l.seg == 1 ? r.x >> 16 : r.y & 0xFFFFu) - l.first;
}
// Positions of the word with an id above / below that of the vertex whose
// ranks are r (uint2 of DenseView::rank).
__device__ __forceinline__ void dense_sides(const DenseLane &l, uint2 r, uint32_t &above, uint32_t &below) {
    const int c = dense_rank(l, r);
    above = dense_from(c);
    below = ~dense_from(c - ((r.y >> 16) == l.seg ? 1 : 0));
}

// What a level's bounds against the vertex leave of the word (f: the level's
// entry of DenseWarp::lev, shifted by that vertex's level).
__device__ __forceinline__ uint32_t dense_bound(uint32_t f, uint32_t above, uint32_t below) {
    return (f & 0x100u) ? above : (f & 0x10000u) ? below : above | below;
}

// Matches level d at position p: running masks of every later level.
__device__ __forceinline__ void dense_match(DenseWarp &S, const DenseView &V, uint32_t k, uint32_t d, uint32_t p) {
    const uint32_t lane = lane_id();
    const uint32_t *r = V.rows + (size_t)p * V.s.pitch;
    const uint2 rk = __ldg(V.rank + p);
    const bool row = (S.lev[DENSE_MAX_K - 1] >> d) & 1u;
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
        const uint32_t w = lane + 32 * h;
        if (w >= V.s.pitch) break;
        const uint32_t rw = row ? __ldg(r + w) : 0u;
        uint32_t above, below;
        dense_sides(dense_lane(V.s, w), rk, above, below);
        for (uint32_t i = d + 1; i < k; ++i) {
            uint32_t m = S.run(dense_slot(d - 1, i))[w];
            const uint32_t f = S.lev[i - 1] >> d;
            m &= (f & 1u) ? rw : 0xFFFFFFFFu;
            m &= dense_bound(f, above, below);
            S.run(dense_slot(d, i))[w] = m;
        }
    }
    __syncwarp();
}

// Takes the first position out of a mask (all lanes get it; DENSE_NONE: empty).
__device__ __forceinline__ uint32_t dense_pop(uint32_t *m, uint32_t pitch) {
    const uint32_t lane = lane_id();
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
        const uint32_t w = lane + 32 * h;
        const uint32_t x = w < pitch ? m[w] : 0u;
        const uint32_t b = __ballot_sync(FULL_MASK, x != 0);
        if (b) {
            const uint32_t src = __ffs(b) - 1;
            const uint32_t bits = __shfl_sync(FULL_MASK, x, src);
            if (lane == src) m[w] = x & (x - 1);
            __syncwarp();
            return (src + 32 * h) * 32 + __ffs(bits) - 1;
        }
        if (pitch <= 32) break;
    }
    return DENSE_NONE;
}

// Positions of 32 words' set bits (word `lane`: x) into the list; their number.
__device__ __forceinline__ uint32_t dense_list(uint16_t *out, uint32_t x, uint32_t first) {
    const uint32_t lane = lane_id();
    uint32_t incl = __popc(x);
    const uint32_t c = incl;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(FULL_MASK, incl, o);
        if (lane >= o) incl += t;
    }
    uint32_t at = incl - c;
    while (x) {
        out[at++] = (uint16_t)(first + __ffs(x) - 1);
        x &= x - 1;
    }
    const uint32_t n = __shfl_sync(FULL_MASK, incl, 31);
    __syncwarp();
    return n;
}

// The last enumerated level y = ne-1 and the tail, for the prefix matched up
// to level d = ne-2.  Adds to this lane's share of the sum.
__device__ __forceinline__ void dense_leaf(const DevPlan &P, DenseWarp &S, const DenseView &V, uint32_t d,
                                           unsigned long long &acc, uint32_t *flags) {
    const uint32_t lane = lane_id(), y = d + 1, ne = y + 1, k = P.k;
    const uint32_t *ym = S.run(dense_slot(d, y));
    // words the tail can have: the first segment when every tail level holds both root ends
    bool both = true;
    for (uint32_t i = ne; i < k; ++i) both &= (S.lev[i - 1] & 3u) == 3u;
    const uint32_t zw = both ? V.s.w1 : V.s.w3;
    if (P.tail_mode == SGE_TAIL_SINGLE) {
        const uint32_t *zm = S.run(dense_slot(d, ne));
        const uint32_t f = S.lev[ne - 1] >> y;
        const bool par = f & 1u, lo = f & 0x100u, up = f & 0x10000u;
        if (!par && !lo && !up) {
            // the tail does not depend on y: |Y|·|Z| pairs less those with z = y
            uint32_t ny = 0, nz = 0, nyz = 0;
            for (uint32_t w = lane; w < V.s.pitch; w += 32) {
                const uint32_t a = ym[w], b = zm[w];
                ny += __popc(a);
                nz += __popc(b);
                nyz += __popc(a & b);
            }
            ny = __reduce_add_sync(FULL_MASK, ny);
            nz = __reduce_add_sync(FULL_MASK, nz);
            acc -= nyz;
            if (lane == 0) acc += (unsigned long long)ny * nz;
            return;
        }
        // every y's row is ANDed with the tail's mask 16 bytes a lane, `lp`
        // lanes a row, so a warp takes 32 / lp rows at a time
        const uint32_t quads = (zw + 3u) / 4u, rq = V.s.pitch / 4u;
        const uint32_t lp = quads <= 1 ? 1u : 1u << (32 - __clz(quads - 1));
        const uint32_t ql = lane & (lp - 1), grp = lane / lp, step = 32 / lp;
        uint32_t z[4] = {0, 0, 0, 0};
        DenseLane l[4];
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            if (ql < quads) z[q] = zm[4 * ql + q];
            l[q] = dense_lane(V.s, 4 * ql + q);
        }
        const uint4 *rows = reinterpret_cast<const uint4 *>(V.rows);
        const uint32_t flip = up ? 0xFFFFFFFFu : 0u;   // below = not from y on
        uint32_t sum = 0;
        for (uint32_t h = 0; h * 32 < V.s.pitch; ++h) {
            const uint32_t w = lane + 32 * h;
            const uint32_t n = dense_list(S.ylist, w < V.s.pitch ? ym[w] : 0u, w * 32);
            for (uint32_t b = grp; b < n; b += step) {
                const uint32_t p = S.ylist[b];
                uint32_t m[4] = {z[0], z[1], z[2], z[3]};
                if (par) {
                    uint4 r = make_uint4(0, 0, 0, 0);
                    if (ql < quads) r = __ldg(rows + (size_t)p * rq + ql);
                    m[0] &= r.x; m[1] &= r.y; m[2] &= r.z; m[3] &= r.w;
                }
                if (lo || up) {
                    const uint2 rk = __ldg(V.rank + p);
                    const uint32_t own = up ? rk.y >> 16 : 3u;   // y itself is not below y
#pragma unroll
                    for (uint32_t q = 0; q < 4; ++q)
                        m[q] &= dense_from(dense_rank(l[q], rk) - (own == l[q].seg ? 1 : 0)) ^ flip;
                }
                sum += __popc(m[0]) + __popc(m[1]) + __popc(m[2]) + __popc(m[3]);
            }
            __syncwarp();
        }
        acc += sum;
        return;
    }
    // CHOOSE / inclusion–exclusion: a lane per y counts the sizes S[A] of the
    // intersections of the tail levels A, then takes the plan's sum over them
    const uint32_t T = P.tail_mode == SGE_TAIL_CHOOSE ? 1u : P.T;
    uint32_t f[DENSE_MAX_T];
    const uint32_t *tm[DENSE_MAX_T];
#pragma unroll
    for (uint32_t t = 0; t < DENSE_MAX_T; ++t) {
        f[t] = t < T ? S.lev[ne + t - 1] >> y : 0u;
        tm[t] = S.run(dense_slot(d, ne + (t < T ? t : 0u)));
    }
    for (uint32_t h = 0; h * 32 < V.s.pitch; ++h) {
        const uint32_t w = lane + 32 * h;
        const uint32_t n = dense_list(S.ylist, w < V.s.pitch ? ym[w] : 0u, w * 32);
        for (uint32_t b = lane; b < n; b += 32) {
            const uint32_t p = S.ylist[b];
            const uint32_t *r = V.rows + (size_t)p * V.s.pitch;
            const uint2 rk = __ldg(V.rank + p);
            uint32_t cnt[1u << DENSE_MAX_T] = {};
            for (uint32_t q = 0; q < zw; ++q) {
                uint32_t above, below, z[DENSE_MAX_T];
                dense_sides(dense_lane(V.s, q), rk, above, below);
                const uint32_t rw = __ldg(r + q);
#pragma unroll
                for (uint32_t t = 0; t < DENSE_MAX_T; ++t)
                    z[t] = t < T ? tm[t][q] & ((f[t] & 1u) ? rw : 0xFFFFFFFFu) & dense_bound(f[t], above, below) : 0u;
#pragma unroll
                for (uint32_t A = 1; A < (1u << DENSE_MAX_T); ++A)
                    cnt[A] += __popc(((A & 1u) ? z[0] : 0xFFFFFFFFu) & ((A & 2u) ? z[1] : 0xFFFFFFFFu) &
                                     ((A & 4u) ? z[2] : 0xFFFFFFFFu));
            }
            if (P.tail_mode == SGE_TAIL_CHOOSE) {
                acc += choose_leaf(cnt[1], P.T, P.choose_wrap, flags);
            } else {
                for (uint32_t q = 0; q < P.nparts; ++q) {
                    unsigned long long term = (unsigned long long)(long long)P.part_coef[q];
                    for (uint32_t bk = 0; bk < P.part_nblocks[q]; ++bk) {
                        uint32_t v = 0;   // cnt[part_block], without an indexed array
#pragma unroll
                        for (uint32_t A = 1; A < (1u << DENSE_MAX_T); ++A) v = P.part_block[q][bk] == A ? cnt[A] : v;
                        term *= v;
                    }
                    acc += term;
                }
            }
        }
        __syncwarp();
    }
}

// Counts every task, a warp at a time.
__global__ void __launch_bounds__(128, 8) dense_count_kernel(const DevPlan *__restrict__ plans, DenseBuf D,
                                                             unsigned long long *counts, unsigned long long *ptime,
                                                             unsigned long long deadline_ns, uint32_t *flags,
                                                             uint32_t slots) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const uint32_t lane = lane_id();
    DenseWarp &S = *reinterpret_cast<DenseWarp *>(smem_raw + (threadIdx.x >> 5) * dense_warp_bytes(slots));
    Ctx<false> c;
    c.flags = flags;
    c.deadline = deadline_ns;
    c.tstart = *reinterpret_cast<volatile unsigned long long *>(flags + 2);
    const uint32_t nrec = min(D.hdr[0], D.rec_cap);
    const unsigned long long total = *reinterpret_cast<unsigned long long *>(D.hdr + 6) * D.npo;
    unsigned long long *queue = reinterpret_cast<unsigned long long *>(D.hdr + 4);
    if (deadline_ns && (*reinterpret_cast<volatile uint32_t *>(flags) & FLAG_TIMEOUT)) return;   // (rows may not be built)
    while (true) {
        unsigned long long t = 0;
        if (lane == 0) t = atomicAdd(queue, 1ull);
        t = __shfl_sync(FULL_MASK, t, 0);
        if (t >= total || out_of_time(c)) break;
        // the record holding task t: the last with pre[r] * npo <= t
        uint32_t r = 0, len = nrec;
        while (len > 0) {
            const uint32_t half = len >> 1;
            if (__ldg(D.pre + r + half) * D.npo <= t) { r += half + 1; len -= half + 1; }
            else len = half;
        }
        --r;
        const DenseRec &R = D.recs[D.order[r]];
        const uint32_t ps = dense_parts_log2(D, R), per = dense_tasks(R.n2, ps);
        const unsigned long long local = t - D.pre[r] * D.npo;
        const uint32_t task = (uint32_t)(local % per);
        const DensePO po = D.po[local / per];
        if (R.off[po.cls] == DENSE_NONE) continue;   // counted by the list path
        const uint32_t c0 = ps ? task >> ps : task * DENSE_CAND, c1 = ps ? c0 + 1 : min(R.n2, c0 + DENSE_CAND);
        const DevPlan &P = plans[po.plan];
        const DenseView V = dense_view(D, R, po.cls);
        const unsigned long long began = globaltimer_ns();
        const uint32_t k = P.k, ne = P.ne;
        // the plan's masks; the last entry holds the levels some later level has as a parent
        __syncwarp();
        if (lane < DENSE_MAX_K - 1) {
            const bool on = lane + 1 < k;
            S.lev[lane] = on ? (P.parents[lane + 1] & 0xFFu) | (P.lower[lane + 1] & 0xFFu) << 8 |
                                   (P.upper[lane + 1] & 0xFFu) << 16
                             : 0u;
        }
        if (lane == 0) {
            uint32_t any = 0;
            for (uint32_t i = 2; i < k; ++i) any |= P.parents[i];
            S.lev[DENSE_MAX_K - 1] = any;
        }
        __syncwarp();
        {   // candidates given the root: segments and the bounds against m0, m1
            const uint4 hd = *reinterpret_cast<const uint4 *>(V.head);
            const uint2 ru = make_uint2(hd.x, hd.y), rv = make_uint2(hd.z, hd.w);
            for (uint32_t w = lane; w < V.s.pitch; w += 32) {
                const DenseLane l = dense_lane(V.s, w);
                const uint32_t valid = w < V.s.w3 ? ~dense_from((int)(l.seg == 0 ? V.s.n[0] : l.seg == 1 ? V.s.n[1] : V.s.n[2]) - l.first) : 0u;
                const uint32_t xu = l.seg != 2 ? valid : 0u, xv = l.seg != 1 ? valid : 0u;
                const uint32_t x0 = po.swap ? xv : xu, x1 = po.swap ? xu : xv;
                uint32_t gt0, lt0, gt1, lt1;
                dense_sides(l, po.swap ? rv : ru, gt0, lt0);
                dense_sides(l, po.swap ? ru : rv, gt1, lt1);
                for (uint32_t i = 2; i < k; ++i) {
                    const uint32_t pr = S.lev[i - 1], lo = pr >> 8, up = pr >> 16;
                    uint32_t m = ((pr & 1u) ? x0 : 0xFFFFFFFFu) & ((pr & 2u) ? x1 : 0xFFFFFFFFu);
                    m &= (lo & 1u) ? gt0 : (up & 1u) ? lt0 : (gt0 | lt0);
                    m &= (lo & 2u) ? gt1 : (up & 2u) ? lt1 : (gt1 | lt1);
                    S.run(dense_slot(1, i))[w] = m;
                }
            }
        }
        __syncwarp();
        // this part's level-3 candidates
        uint32_t pat = 0xFFFFFFFFu;
        if (ps) {
            pat = 1u << (task & ((1u << ps) - 1u));
            for (uint32_t o = 1u << ps; o < 32; o <<= 1) pat |= pat << o;
            uint32_t *l3 = S.run(dense_slot(1, 3));
            for (uint32_t w = lane; w < V.s.pitch; w += 32) l3[w] &= pat;
            __syncwarp();
        }
        unsigned long long acc = 0;
        bool ok = true;
        for (uint32_t p2 = c0; p2 < c1 && ok; ++p2) {   // (common neighbours are the first positions)
            if (!((S.run(dense_slot(1, 2))[p2 >> 5] >> (p2 & 31u)) & 1u)) continue;
            // (the leaves under one candidate's part, a few hundred at most, are not
            // cut: a look at the clock at each cost 0.4 % of a batch)
            if (out_of_time(c)) { ok = false; break; }
            dense_match(S, V, k, 2, p2);
            if (ne == 4) {
                dense_leaf(P, S, V, 2, acc, flags);
                continue;
            }
            uint32_t lv = 3;
            while (true) {
                const uint32_t p = dense_pop(S.run(dense_slot(lv - 1, lv)), V.s.pitch);
                if (p == DENSE_NONE) {
                    if (--lv < 3) break;
                    continue;
                }
                dense_match(S, V, k, lv, p);
                if (lv + 2 == ne) {
                    dense_leaf(P, S, V, lv, acc, flags);
                    continue;
                }
                if (out_of_time(c)) { ok = false; break; }
                ++lv;
            }
        }
        acc = warp_sum_u64(acc);
        if (lane == 0) {
            if (ok && acc) atomicAdd(counts + po.plan, acc);
            atomicAdd(ptime + po.plan, globaltimer_ns() - began);
        }
        if (!ok) return;
    }
}

// Host: the universe class of a plan (0..3: N(m0) ∩ N(m1), N(m0), N(m1), union), -1 when the path
// does not take it.  Level 2 must close a triangle on the root edge and every later level must touch
// the root; plans with a level bounded above and below the same vertex stay on lists, where nothing
// fits it (the masks take one bound per pair of levels).  With three enumerated levels, or four and a tail whose list does not depend on the last
// of them, the rows of a root are read about once each: the list path does that without building them.
inline int dense_class(const DevPlan &d) {
    if (d.vlab || d.ntrie || d.k > DENSE_MAX_K || d.ne < 4 || (d.parents[2] & 3u) != 3u) return -1;
    if (d.tail_mode == SGE_TAIL_IEP && d.T > DENSE_MAX_T) return -1;
    bool all0 = true, all1 = true, dep = false;
    for (uint32_t i = 2; i < d.k; ++i) {
        if (!(d.parents[i] & 3u) || (d.lower[i] & d.upper[i])) return -1;
        all0 &= (d.parents[i] & 1u) != 0;
        all1 &= (d.parents[i] & 2u) != 0;
        dep |= i >= d.ne && ((d.parents[i] >> (d.ne - 1)) & 1u);
    }
    if (d.ne == 4 && !dep) return -1;
    return all0 && all1 ? DENSE_BOTH : all0 ? DENSE_U : all1 ? DENSE_V : DENSE_UNION;
}
// Whether a level below the root enumerates all of N(m0) or N(m1).
inline bool dense_wide(const DevPlan &d) {
    for (uint32_t i = 3; i < d.ne; ++i)
        if (d.parents[i] == 1u || d.parents[i] == 2u) return true;
    return false;
}
// Whether every level whose row is read lies in N(m0) ∩ N(m1).
inline bool dense_rows_both(const DevPlan &d) {
    uint32_t any = 0;
    for (uint32_t i = 2; i < d.k; ++i) any |= d.parents[i];
    for (uint32_t i = 2; i < d.k; ++i)
        if (((any >> i) & 1u) && (d.parents[i] & 3u) != 3u) return false;
    return true;
}
// The edge's class for a plan class: N(m0) is N(v) when the root runs reversed.
inline uint32_t dense_edge_class(uint32_t plan_cls, bool swap) {
    return swap && (plan_cls == DENSE_U || plan_cls == DENSE_V) ? 3u - plan_cls : plan_cls;
}
