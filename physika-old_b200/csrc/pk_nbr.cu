// pk_nbr.cu -- neighbour rows over the cell-sorted particles.
//
// Reference: K_ComputeNeighborFixed (NeighborQuery.cu:514-581) keeps, per
// particle, the `cap` nearest hits with d < h by replacing the current
// farthest entry; K_CalNeighborSize/K_GetNeighborElements (:245-276,337-367)
// build the uncapped list.  A capped list is asymmetric (j in N(i) does not
// imply i in N(j)) and DensityPBD scatters each pair's displacement to both
// ends (DensityPBD.cu:161-173).  To solve that with gathers only, each solver
// row holds N(i) plus {j : i in N(j)} with two flag bits, so a pair's
// multiplicity in i's displacement is known without atomics.
//
//   k_build (one warp per occupied cell): the candidates of the 27 neighbour
//     cells that lie within the radius of the cell's bounding box are staged
//     once in shared memory, in the reference's visiting order; passes of up to
//     8 of the cell's particles, held in registers by every lane, test one
//     candidate of each 32-wide chunk per lane, two particles per packed
//     instruction, and one ballot per particle appends the chunk's hits to
//     the particle's staged row, which is written out in whole quads.  The hit
//     test compares the rounded squared distance with the precomputed float T
//     (sqrt_rn(d2) < h  <=>  d2 < T, sqrt_rn being monotone), so no square root
//     is taken.  For a capped list the warp then takes tau_i, the cap-th
//     smallest key (d2, sorted index) of the row, from the staged row: the
//     order of sqrt_rn(d2) agrees with the reference's distance order except
//     among hits at exactly equal distance, which the reference orders by
//     arrival.  Cells with more candidates than the stage holds, and rows
//     longer than it, take an unstaged sweep, where hits past the row capacity
//     go to the particle's segment of the spill pool, so a row of any length
//     is in candidate order.  Bound by its chains of dependent steps, half of
//     the issue slots used: 1.39 ms at 2M particles, 127 us at 152k, 14.5 us at
//     1k with the selection, where the sweep and a selection kernel of its own,
//     each reading the rows back, took 1.83 ms, 158 us and 41 us; dynamic, 70 us
//     at 99k (89 before).  On the same box: passes of 4 particles 1.36 ms and 45
//     us at 32k (8: 43 us), of 16 2.6 ms; a lane per particle 1.70 ms and 24.6
//     us at 1k; two selections at a time 1.70 ms.
//   k_emit (capped lists, one thread per particle; k_emit_lanes, 8 lanes per
//     particle, in small scenes): walks the hit row, marks
//     a = key <= tau_i (j in N(i)) and b = key' <= tau_j (i in N(j)), and
//     writes the solver row with a-entries first, then b-only entries.  A
//     dynamic list holds every hit, so k_build writes its solver rows itself.
//   k_export copies the rows' a-entries to the public NeighborList in caller
//     ids.
// Distances use the explicit roundings of exact_norm3's squared sum, so every
// d < h decision and every ordering is bit-identical for (i, j) and (j, i)
// and matches the CPU restatement.
#include <algorithm>
#include <cmath>

#include "pk_kernels.cuh"

namespace pk {

constexpr int kBuildWarps = 4;
constexpr int kBins = 32;                // histogram of d2 over [0, T)
constexpr unsigned kFull = 0xffffffffu;

// Rounded squared distance of exact_norm3 (before its square root).
__device__ __forceinline__ float exact_sum2(float dx, float dy, float dz)
{
#if PK_NORM_VARIANT == 0
    return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
#elif PK_NORM_VARIANT == 2
    return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
#else
    return __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
#endif
}
__device__ __forceinline__ float exact_d2(const float4& a, const float4& b)
{
    return exact_sum2(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z));
}
// The same for two particles against one candidate given as its negated
// coordinates (a packed add rounds as the subtraction does).
__device__ __forceinline__ float2 exact_d2x2(float2 px, float2 py, float2 pz, float2 nx, float2 ny, float2 nz)
{
    const float2 dx = __fadd2_rn(px, nx), dy = __fadd2_rn(py, ny), dz = __fadd2_rn(pz, nz);
#if PK_NORM_VARIANT == 0
    return __fadd2_rn(__fadd2_rn(__fmul2_rn(dx, dx), __fmul2_rn(dy, dy)), __fmul2_rn(dz, dz));
#elif PK_NORM_VARIANT == 2
    return __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
#else
    return __ffma2_rn(dz, dz, __ffma2_rn(dx, dx, __fmul2_rn(dy, dy)));
#endif
}

struct BuildArgs {
    const float4* xs;   // positions the list is built on (sorted)
    const int* start;   // starts of the occupied cells
    const int* count;   // particles per cell
    const int2* items;  // (begin, end) sorted ranges sharing one cell
    const int* nitems;
    Grid g;
    int n, row_cap, cap;
    int split;          // log2 of the warps that share a cell's passes
    float T;            // d2 threshold of d < h
    int flags;          // set in every entry of a dynamic list's solver rows
    int* hits;          // rows of sorted indices, candidate order, laid out as solver rows
    int* hcnt;          // hits per particle (sorted order), past the row capacity too
    int2* rcnt;         // dynamic lists: the solver rows' counts, else null
    int* count_c;       // hits per particle in caller order (dynamic public list), or null
    float4* xt;         // capped lists: (position, tau's d2; negated where tau_id decides a tie)
    int* tau_id;
    const int* perm;
    int* err;
    // spill pool (pool_cap 0: none, a row past the capacity is an error)
    long long pool_cap;
    unsigned long long* spill;  // entries handed out
    int* ovf;
    int* hpool;
};

// Entries past the row capacity: a segment of round4(count - row_cap) entries
// of the spill pool.
__device__ __forceinline__ int claim_spill(const BuildArgs& A, int s, int count)
{
    if (A.pool_cap <= 0) {
        atomicOr(A.err, kErrRowOverflow);
        return -1;
    }
    const unsigned long long need = (unsigned long long)((count - A.row_cap + 3) & ~3);
    const unsigned long long off = atomicAdd(A.spill, need);
    const int o = off + need <= (unsigned long long)A.pool_cap ? (int)off : -1;
    A.ovf[s] = o;
    if (o < 0) atomicOr(A.err, kErrHitOverflow);
    return o;
}

struct SelSmem {
    int hist[kBins];
    uint2 slot[32];
};

// The stage of a warp in shared memory: candidates (negated position, sorted
// index), the pass's rows of 16-bit candidate numbers, and the non-empty
// neighbour ranges.  A row that outgrows its place runs into what follows it,
// the next rows and the pad at the end, and the pass is done again unstaged, so
// the sweep needs no bound check.  104 entries and 384 candidates hold the rows
// and the reach of a cell at up to 1.2 times the rest density of the usual ratio
// of radius to spacing (2.5: about 65 hits of 320) and leave room for 24 warps
// per SM: the build waits on its own chains of dependent steps, and 20 warps
// took 10% longer, 16 another 9%.  Lists with long rows (dynamic ones, large
// caps) get 192 and 640, enough at a ratio of 3 (about 113 of 560).
template <int KPB, bool kLong>
struct Stage {
    static constexpr int kCand = kLong ? 640 : 384;
    static constexpr int kRows = kLong ? 192 : 104;
    static constexpr int kStride = kRows + 12;  // entries: whole 8-byte quads, rows on different banks
    float4 cand[kCand];
    unsigned short row[KPB * kStride + kCand - kRows];
    int delta[32];  // sorted index - candidate number of each non-empty range
    SelSmem sel;
};

// The 27 neighbour ranges of a cell (lane o < 27 owns offset o of the
// reference's visiting order), packed in that order: candidate g of the cell
// is sorted particle g + delta[r], r the range holding g.
struct Ranges {
    int len, off;  // this lane's range
    int total;
};
__device__ __forceinline__ Ranges sweep_ranges(const BuildArgs& A, int* delta, int s, int lane, unsigned lt)
{
    const float4 x0 = A.xs[s];
    const int3 c = cell3(A.g, x0.x, x0.y, x0.z);
    const int base = scene_key_base(A.g, __ldg(A.perm + s));
    int beg = 0;
    Ranges R;
    R.len = 0;
    if (lane < 27) {
        const int key = cell_key(A.g, c.x + kOffset27[lane][0], c.y + kOffset27[lane][1], c.z + kOffset27[lane][2]);
        if (key >= 0) {
            beg = __ldg(A.start + base + key);  // not written, and not used, where the cell is empty
            R.len = __ldg(A.count + base + key);
        }
    }
    int incl = R.len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += y;
    }
    R.off = incl - R.len;
    R.total = __shfl_sync(kFull, incl, 31);
    const unsigned ne = __ballot_sync(kFull, R.len > 0);
    __syncwarp();
    if (R.len > 0) delta[__popc(ne & lt)] = beg - R.off;
    __syncwarp();
    return R;
}

// Sorted index of candidate g0 + lane, chunks taken in order; started counts
// the ranges begun before the chunk.  The ranges that begin in the chunk are
// marked in one word (an OR over the lanes), so a lane's range is a popcount
// away.  Past the end: -1.
__device__ __forceinline__ int chunk_index(const Ranges& R, const int* delta, int g0, int lane, unsigned lt,
                                           int& started)
{
    const bool here = R.len > 0 && R.off >= g0 && R.off < g0 + 32;
    const unsigned marks = __reduce_or_sync(kFull, here ? 1u << (R.off - g0) : 0u);
    const int r = started + __popc(marks & (lt | (1u << lane))) - 1;
    started += __popc(marks);
    const int g = g0 + lane;
    return g < R.total ? g + delta[r] : -1;
}

__device__ __forceinline__ float4 load_cand(const float4* __restrict__ xs, int t)
{
    return t >= 0 ? __ldg(xs + t) : make_float4(3.0e38f, 3.0e38f, 3.0e38f, 0.f);
}

// Smallest / largest value of the warp (NaN ignored), one instruction on sm_100.
__device__ __forceinline__ float warp_min(float v)
{
    float r;
    asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v)
{
    float r;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// Stages the candidates within the radius of the bounding box of the sorted
// particles [b, e), filled up to whole chunks with far ones, and returns how
// many there are (more than kCand: the stage does not hold them).  The box
// distance is formed with the pair test's roundings, each of which is monotone,
// so no candidate with a hit is dropped.
template <class St>
__device__ __forceinline__ int stage_candidates(const BuildArgs& A, St& S, const Ranges& R, int b, int e, int lane,
                                                unsigned lt)
{
    float lo[3] = {3.0e38f, 3.0e38f, 3.0e38f}, hi[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
    for (int p = b + lane; p < e; p += 32) {
        const float4 q = __ldg(A.xs + p);
        lo[0] = fminf(lo[0], q.x);
        lo[1] = fminf(lo[1], q.y);
        lo[2] = fminf(lo[2], q.z);
        hi[0] = fmaxf(hi[0], q.x);
        hi[1] = fmaxf(hi[1], q.y);
        hi[2] = fmaxf(hi[2], q.z);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        lo[k] = warp_min(lo[k]);
        hi[k] = warp_max(hi[k]);
    }
    int n = 0, started = 0;
    int t = chunk_index(R, S.delta, 0, lane, lt, started);
    float4 q = load_cand(A.xs, t);
    for (int g0 = 0; g0 < R.total; g0 += 32) {
        const int tc = t;
        const float4 c = q;
        t = chunk_index(R, S.delta, g0 + 32, lane, lt, started);  // the next chunk's loads in flight
        q = load_cand(A.xs, t);
        const float dx = fmaxf(fmaxf(__fsub_rn(lo[0], c.x), __fsub_rn(c.x, hi[0])), 0.0f);
        const float dy = fmaxf(fmaxf(__fsub_rn(lo[1], c.y), __fsub_rn(c.y, hi[1])), 0.0f);
        const float dz = fmaxf(fmaxf(__fsub_rn(lo[2], c.z), __fsub_rn(c.z, hi[2])), 0.0f);
        const bool keep = tc >= 0 && exact_sum2(dx, dy, dz) < A.T;
        const unsigned bal = __ballot_sync(kFull, keep);
        const int pos = n + __popc(bal & lt);
        if (keep && pos < St::kCand) S.cand[pos] = make_float4(-c.x, -c.y, -c.z, __int_as_float(tc));
        n += __popc(bal);
    }
    if (n + lane < ((n + 31) & ~31) && n + lane < St::kCand)
        S.cand[n + lane] = make_float4(-3.0e38f, -3.0e38f, -3.0e38f, 0.f);
    __syncwarp();
    return n;
}

// A pass's particles in registers, two per packed value (absent ones far away).
template <int KPB>
struct PassPos {
    float2 x[KPB / 2], y[KPB / 2], z[KPB / 2];
    __device__ __forceinline__ void load(const float4* __restrict__ xs, int p0, int m)
    {
        const float4 far = make_float4(-3.0e38f, -3.0e38f, -3.0e38f, 0.f);
#pragma unroll
        for (int k = 0; k < KPB / 2; ++k) {
            const float4 a = 2 * k < m ? __ldg(xs + p0 + 2 * k) : far;
            const float4 b = 2 * k + 1 < m ? __ldg(xs + p0 + 2 * k + 1) : far;
            x[k] = make_float2(a.x, b.x);
            y[k] = make_float2(a.y, b.y);
            z[k] = make_float2(a.z, b.z);
        }
    }
};

// One chunk of candidates (this lane's negated position in q) against the
// pass's first NP pairs: put(p, rank, hit) receives every particle's hits of
// lower lanes and whether this lane's candidate is one; cnt[p] += kUnit per hit.
template <int NP, int kUnit, int KPB, class Put>
__device__ __forceinline__ void sweep_chunk(const PassPos<KPB>& P, const float4& q, float T, int (&cnt)[KPB],
                                            unsigned lt, const Put& put)
{
    const float2 nx = make_float2(q.x, q.x), ny = make_float2(q.y, q.y), nz = make_float2(q.z, q.z);
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        const float2 d2 = exact_d2x2(P.x[k], P.y[k], P.z[k], nx, ny, nz);
        const bool h0 = d2.x < T, h1 = d2.y < T;
        const unsigned b0 = __ballot_sync(kFull, h0), b1 = __ballot_sync(kFull, h1);
        put(2 * k, cnt[2 * k] + kUnit * __popc(b0 & lt), h0);
        put(2 * k + 1, cnt[2 * k + 1] + kUnit * __popc(b1 & lt), h1);
        cnt[2 * k] += kUnit * __popc(b0);
        cnt[2 * k + 1] += kUnit * __popc(b1);
    }
}

// The staged sweep of a pass of np pairs; cnt in bytes of a row (two per hit).
template <int NP, int KPB, bool kLong>
__device__ __forceinline__ void sweep_staged(const PassPos<KPB>& P, Stage<KPB, kLong>& S, int np, int nc, float T,
                                             int (&cnt)[KPB], int lane, unsigned lt)
{
    if constexpr (NP > 1) {
        if (np < NP) {  // warp-uniform
            sweep_staged<NP - 1>(P, S, np, nc, T, cnt, lane, lt);
            return;
        }
    }
    char* const rows = reinterpret_cast<char*>(S.row);
    for (int c0 = 0; c0 < nc; c0 += 32) {
        const unsigned short number = (unsigned short)(c0 + lane);
        sweep_chunk<NP, 2>(P, S.cand[c0 + lane], T, cnt, lt, [&](int p, int at, bool hit) {
            if (hit) *reinterpret_cast<unsigned short*>(rows + p * (2 * Stage<KPB, kLong>::kStride) + at) = number;
        });
    }
}

// ---- tau_i: the cap-th smallest key (d2, sorted index) of a hit row.

// Hit e of a particle's row in memory as (sorted index, d2 bits): the main
// array up to the row capacity, then the particle's spill segment.
struct HitRow {
    const int* row;   // row_slot(s, 0)
    const int* pool;  // the particle's spill segment (null when none)
    const float4* xs;
    float4 xi;
    int rc;
    __device__ __forceinline__ uint2 at(int e) const
    {
        if (e >= rc && !pool) return make_uint2(0u, 0xffffffffu);
        const int t = (e < rc ? row[(e >> 2) * 128 + (e & 3)] : pool[e - rc]) & kRowIndexMask;
        return make_uint2((unsigned)t, __float_as_uint(exact_d2(xi, __ldg(xs + t))));
    }
};

__device__ __forceinline__ int sel_bin(unsigned db, float lo, float scale)
{
    return min(max((int)((__uint_as_float(db) - lo) * scale), 0), kBins - 1);
}

// Rank rr (0-based) among the c keys of a row in memory, one warp: any length,
// any ties.  The hits in play always form an interval [plo, phi] of d2 values
// (initially all of them).  While more than 32 are in play, a 32-bin histogram
// over the interval locates the bin holding the rank, and that bin's smallest
// and largest d2 become the next interval.  Bins are monotone in d2, so an
// interval's hits are exactly its bin's hits, and plo falls in bin 0 while phi
// falls in the last bin: every level shrinks the set.  At most 32 hits left are
// ranked exactly by (d2, index); more than 32 hits at one d2 value are ranked
// by index.
__device__ __noinline__ uint2 select_rank(const HitRow row, int c, int rr, float T, SelSmem& S, int lane)
{
    const unsigned lt = (1u << lane) - 1u;
    const int nch = (c + 31) / 32;
    auto src = [&](int k) {
        const int e = k * 32 + lane;
        return e < c ? row.at(e) : make_uint2(0u, 0xffffffffu);
    };
    unsigned plo = 0u, phi = __float_as_uint(T);  // [0, T]: every hit
    float lo = 0.f, scale = (float)kBins / T;
    int np = c;
    while (np > 32 && plo != phi) {
        S.hist[lane] = 0;
        __syncwarp();
        for (int k = 0; k < nch; ++k) {
            const uint2 v = src(k);
            if (v.y >= plo && v.y <= phi) atomicAdd(&S.hist[sel_bin(v.y, lo, scale)], 1);
        }
        __syncwarp();
        const int hb = S.hist[lane];
        int incl = hb;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += y;
        }
        const int B = __ffs(__ballot_sync(kFull, incl > rr)) - 1;
        np = __shfl_sync(kFull, hb, B);
        rr -= __shfl_sync(kFull, incl - hb, B);
        // the chosen bin's extreme values
        unsigned mn = 0xffffffffu, mx = 0u;
        for (int k = 0; k < nch; ++k) {
            const uint2 v = src(k);
            if (v.y >= plo && v.y <= phi && sel_bin(v.y, lo, scale) == B) {
                mn = min(mn, v.y);
                mx = max(mx, v.y);
            }
        }
        plo = __reduce_min_sync(kFull, mn);
        phi = __reduce_max_sync(kFull, mx);
        lo = __uint_as_float(plo);
        const float width = __uint_as_float(phi) - lo;
        scale = width > 0.f ? (float)kBins / width : 0.f;
        __syncwarp();
    }
    uint2 mine = make_uint2(0u, 0x7fffffffu);
    if (np <= 32) {
        int k = 0;
        for (int q = 0; q < nch; ++q) {
            const uint2 v = src(q);
            const bool in = v.y >= plo && v.y <= phi;
            const unsigned bal = __ballot_sync(kFull, in);
            if (in) S.slot[k + __popc(bal & lt)] = v;
            k += __popc(bal);
        }
        __syncwarp();
        if (lane < k) {
            const uint2 me = S.slot[lane];
            int rank = 0;
            for (int u = 0; u < k; ++u) {
                const uint2 o = S.slot[u];
                rank += (o.y < me.y || (o.y == me.y && o.x < me.x)) ? 1 : 0;
            }
            if (rank == rr) mine = make_uint2(me.y, me.x);
        }
    } else {
        // more than 32 hits at one d2 value: the rr-th smallest index
        for (int e = lane; e < c; e += 32) {
            const uint2 v = row.at(e);
            if (v.y != plo) continue;
            int rank = 0;
            for (int u = 0; u < c; ++u) {
                const uint2 o = row.at(u);
                rank += (o.y == plo && o.x < v.x) ? 1 : 0;
            }
            if (rank == rr) mine = make_uint2(v.y, v.x);
        }
    }
    const unsigned f = __ballot_sync(kFull, mine.y != 0x7fffffffu);
    const int sl = f ? __ffs(f) - 1 : 0;
    __syncwarp();
    return make_uint2(__shfl_sync(kFull, mine.x, sl), __shfl_sync(kFull, mine.y, sl));
}

// tau's d2 for a row of c <= 32 NQ hits whose d2 the lanes hold, entry 32 q +
// lane in k[q] (+inf past the end).  A first guess takes the hits as uniform in
// the ball, so about cap of them lie below T (1 - 2/3 (c - cap)/c); the count
// below the guess says how many rounds of the warp's largest key below it, or
// smallest above it, lead to the cap-th.  Returns false where equal distances
// upset that count or straddle the cap: then the sorted index decides.
template <int NQ>
__device__ __forceinline__ bool select_tau(const float (&k)[NQ], int c, int cap, float T, float& tau)
{
    auto count = [&](float t) {
        int n = 0;
#pragma unroll
        for (int q = 0; q < NQ; ++q) n += __popc(__ballot_sync(kFull, k[q] <= t));
        return n;
    };
    float t = T * (1.0f - 0.6666667f * (float)(c - cap) / (float)c);
    int le = count(t);
    for (int it = 0; it < 3 && abs(le - cap) > 4; ++it) {
        t = fminf(fmaxf(t * (1.0f + 0.6666667f * (float)(cap - le) / (float)max(le, cap / 4 + 1)), 0.0f), T);
        le = count(t);
    }
    if (le >= cap) {
        float ub = __int_as_float(__float_as_int(t) + 1);  // k < ub  <=>  k <= t
        for (int need = le - cap + 1; need > 0; --need) {
            float m = -1.0f;
#pragma unroll
            for (int q = 0; q < NQ; ++q) m = fmaxf(m, k[q] < ub ? k[q] : -1.0f);
            ub = warp_max(m);
        }
        tau = ub;
    } else {
        float lb = t;
        for (int need = cap - le; need > 0; --need) {
            float m = __int_as_float(0x7f800000);
#pragma unroll
            for (int q = 0; q < NQ; ++q) m = fminf(m, k[q] > lb ? k[q] : __int_as_float(0x7f800000));
            lb = warp_min(m);
        }
        tau = lb;
    }
    return tau >= 0.0f && tau < T && count(tau) == cap;
}

// The same from a staged row (c <= 128).
template <int NQ, int KPB, bool kLong>
__device__ __forceinline__ bool select_staged(const Stage<KPB, kLong>& S, const float4& xi, int p, int c, int cap, float T,
                                              int lane, float& tau)
{
    float k[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int e = 32 * q + lane;
        k[q] = __int_as_float(0x7f800000);
        if (e < c) {
            const float4 n = S.cand[S.row[p * Stage<KPB, kLong>::kStride + e]];
            k[q] = exact_sum2(__fadd_rn(xi.x, n.x), __fadd_rn(xi.y, n.y), __fadd_rn(xi.z, n.z));
        }
    }
    return select_tau<NQ>(k, c, cap, T, tau);
}

// Resident blocks per SM asked of the register allocator, as many as the short
// stage's shared memory lets in.
template <int KPB, bool kLong>
constexpr int build_min_blocks()
{
    return kLong || KPB > 8 ? 1 : 6;
}

template <int KPB, bool kLong, bool kCapped>
__global__ void __launch_bounds__(kBuildWarps * 32, build_min_blocks<KPB, kLong>()) k_build(const BuildArgs A)
{
    using St = Stage<KPB, kLong>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    St& S = reinterpret_cast<St*>(smem_raw)[w];
    const unsigned nwork = (unsigned)*A.nitems << A.split;  // at most 2^29 items, split where they are few
    const unsigned gw = blockIdx.x * kBuildWarps + w, nw = gridDim.x * kBuildWarps;
    for (unsigned work = gw; work < nwork; work += nw) {
        const int2 rng = A.items[work >> A.split];
        const int sub = (int)(work & ((1u << A.split) - 1u));
        if (rng.x + sub * KPB >= rng.y) continue;
        const Ranges R = sweep_ranges(A, S.delta, rng.x, lane, lt);
        const int nc = stage_candidates(A, S, R, rng.x, rng.y, lane, lt);
        for (int p0 = rng.x + sub * KPB; p0 < rng.y; p0 += KPB << A.split) {
            const int m = min(KPB, rng.y - p0);
            PassPos<KPB> P;
            P.load(A.xs, p0, m);
            int cnt[KPB];
#pragma unroll
            for (int p = 0; p < KPB; ++p) cnt[p] = 0;
            bool staged = nc <= St::kCand;
            if (staged) {
                sweep_staged<KPB / 2>(P, S, (m + 1) >> 1, nc, A.T, cnt, lane, lt);
                int most = 0;
#pragma unroll
                for (int p = 0; p < KPB; ++p) {
                    cnt[p] >>= 1;
                    most = max(most, cnt[p]);
                }
                staged = most <= min(St::kRows, A.row_cap);
            }
            if (!staged) {
                // more candidates, or longer rows, than the stage holds
#pragma unroll
                for (int p = 0; p < KPB; ++p) cnt[p] = 0;
                int started = 0;
                for (int g0 = 0; g0 < R.total; g0 += 32) {
                    const int t = chunk_index(R, S.delta, g0, lane, lt, started);
                    float4 q = load_cand(A.xs, t);
                    q = make_float4(-q.x, -q.y, -q.z, 0.f);
                    sweep_chunk<KPB / 2, 1>(P, q, A.T, cnt, lt, [&](int p, int pos, bool hit) {
                        if (hit && pos < A.row_cap) A.hits[row_slot(p0 + p, pos, A.row_cap)] = t | A.flags;
                    });
                }
            }
            int c_l = 0;  // lane p: the hits of the pass's particle p
#pragma unroll
            for (int p = 0; p < KPB; ++p)
                if (lane == p) c_l = cnt[p];
            int off_l = -1;  // and its spill segment
            float4 x_l = make_float4(0.f, 0.f, 0.f, 0.f);
            if (lane < m) {
                const int s = p0 + lane;
                x_l = __ldg(A.xs + s);
                A.hcnt[s] = c_l;
                if (A.count_c) A.count_c[__ldg(A.perm + s)] = c_l;
                if (c_l > A.row_cap) off_l = claim_spill(A, s, c_l);
                if (!kCapped) {
                    const int keep = c_l > A.row_cap && off_l < 0 ? A.row_cap : c_l;
                    A.rcnt[s] = make_int2(keep, keep);
                }
            }
            __syncwarp();
            if (staged) {
                // rows out: lane l takes quads l / KPB, l / KPB + 32 / KPB, ... of
                // particle l % KPB, so consecutive lanes write consecutive quads
                const int p = lane % KPB, c = __shfl_sync(kFull, c_l, p);
                const ushort4* const from = reinterpret_cast<const ushort4*>(S.row + p * St::kStride);
                int4* const to = reinterpret_cast<int4*>(A.hits + row_slot(p0 + p, 0, A.row_cap));
                for (int quad = lane / KPB; 4 * quad < c; quad += 32 / KPB) {
                    const ushort4 e = from[quad];
                    const int last = c - 4 * quad;  // entries of the quad
                    int4 v;
                    v.x = __float_as_int(S.cand[e.x].w) | A.flags;
                    v.y = last > 1 ? __float_as_int(S.cand[e.y].w) | A.flags : 0;
                    v.z = last > 2 ? __float_as_int(S.cand[e.z].w) | A.flags : 0;
                    v.w = last > 3 ? __float_as_int(S.cand[e.w].w) | A.flags : 0;
                    to[32LL * quad] = v;
                }
                __syncwarp();
            } else {
                unsigned longer = __ballot_sync(kFull, off_l >= 0);
                while (longer) {  // the hits past the row capacity, in the same order
                    const int p = __ffs(longer) - 1;
                    longer &= longer - 1;
                    const int off = __shfl_sync(kFull, off_l, p);
                    const float4 xi = __ldg(A.xs + p0 + p);
                    int c = 0, started = 0;
                    for (int g0 = 0; g0 < R.total; g0 += 32) {
                        const int t = chunk_index(R, S.delta, g0, lane, lt, started);
                        const bool hit = t >= 0 && exact_d2(xi, load_cand(A.xs, t)) < A.T;
                        const unsigned b = __ballot_sync(kFull, hit);
                        const int pos = c + __popc(b & lt);
                        if (hit && pos >= A.row_cap) A.hpool[off + (pos - A.row_cap)] = t | A.flags;
                        c += __popc(b);
                    }
                }
            }
            if (kCapped) {
                float tau_l = __int_as_float(0x7f800000);  // every hit is in N(i)
                unsigned need = __ballot_sync(kFull, c_l > A.cap);
                __syncwarp();  // the rows just written are read back by select_rank
                while (need) {
                    const int p = __ffs(need) - 1;
                    need &= need - 1;
                    const int c = __shfl_sync(kFull, c_l, p), s = p0 + p;
                    const float4 xi = make_float4(__shfl_sync(kFull, x_l.x, p), __shfl_sync(kFull, x_l.y, p),
                                                  __shfl_sync(kFull, x_l.z, p), 0.f);
                    float tau = 0.f;
                    bool plain = false;
                    if (staged && c <= 96)
                        plain = select_staged<3>(S, xi, p, c, A.cap, A.T, lane, tau);
                    else if (staged && c <= 128)
                        plain = select_staged<4>(S, xi, p, c, A.cap, A.T, lane, tau);
                    if (!plain) {
                        HitRow hr{A.hits + row_slot(s, 0, A.row_cap), nullptr, A.xs, xi, A.row_cap};
                        const int off = __shfl_sync(kFull, off_l, p);
                        if (off >= 0) hr.pool = A.hpool + off;
                        const uint2 r = select_rank(hr, c, A.cap - 1, A.T, S.sel, lane);
                        tau = -__uint_as_float(r.x);
                        if (lane == 0) A.tau_id[s] = (int)r.y;
                    }
                    if (lane == p) tau_l = tau;
                }
                if (lane < m) A.xt[p0 + lane] = make_float4(x_l.x, x_l.y, x_l.z, tau_l);
            }
            __syncwarp();  // the stage's rows are written again by the next pass
        }
        __syncwarp();
    }
}

// ---- solver rows of a capped list: one thread per particle walks its hit
// row as the Jacobi passes walk the solver rows (a warp reads 512 contiguous
// bytes per quad and gathers from a few neighbour cells).  |N(i)| is
// min(hits, cap), so the b-only entries' place is known before the first is
// met and the row is written in one walk.  Bound by L1 (the gathers of 4-float
// tau entries): 395 us at 2M particles, 34 us at 152k, where 8 lanes per
// particle on rows of 8-byte keys took 642 and 52 us.
constexpr int kEmitBlock = 128;

struct EmitArgs {
    const int* hcnt;
    const int* hits;
    const int* hpool;  // null: no spill pool
    const int* ovf;
    const float4* xt;  // position, tau's d2 (negated: tau_id decides ties)
    const int* tau_id;
    int n, cap, rc;
    int* rows;
    int* rpool;
    int2* rcnt;
};

// The a-entries pass through a ring of two quads per thread in shared memory,
// so the rows are written in whole quads with no branch per entry (a quad of
// hits completes at most one); the first kStash b-only entries wait beside it.
constexpr int kStash = 6;
__global__ void __launch_bounds__(kEmitBlock) k_emit(const EmitArgs A)
{
    __shared__ int ring[8][kEmitBlock];
    __shared__ int stash[kStash][kEmitBlock];
    const int tid = threadIdx.x;
    const int s = blockIdx.x * kEmitBlock + tid;
    if (s >= A.n) return;
    const float4 xi = __ldg(A.xt + s);
    const float td = fabsf(xi.w);
    const int my_id = __float_as_int(xi.w) < 0 ? __ldg(A.tau_id + s) : 0x7fffffff;
    int cnt = A.hcnt[s];
    const int* pool = nullptr;
    int* out_pool = nullptr;
    if (cnt > A.rc) {
        const int o = A.hpool ? __ldg(A.ovf + s) : -1;
        if (o >= 0) {
            pool = A.hpool + o;
            out_pool = A.rpool + o;
        } else {
            cnt = A.rc;  // no segment could be had: cut short, the error is latched
        }
    }
    int* const row = A.rows + row_slot(s, 0, A.rc);
    const int nA = min(cnt, A.cap);
    auto entry = [&](int q) { return q < A.rc ? row + (q >> 2) * 128 + (q & 3) : out_pool + (q - A.rc); };
    int na = 0, nb = 0, out = 0;  // a- and b-only entries met, a-entries written
    auto take = [&](int t, const float4& xj, bool in) {
        // a: key <= tau_i; b: (d2, s) <= tau_t
        const float d2 = exact_d2(xi, xj);
        const bool a = in && (d2 < td || (d2 == td && t <= my_id));
        bool b = in && d2 <= fabsf(xj.w);
        if (d2 == -xj.w) b = in && (__float_as_int(xj.w) >= 0 || s <= __ldg(A.tau_id + t));
        const int v = t | (a ? kRowFlagA : 0) | (b ? kRowFlagB : 0);
        if (a) ring[na & 7][tid] = v;
        const bool bo = b && !a;
        if (bo) {
            if (nb < kStash)
                stash[nb][tid] = v;
            else
                *entry(nA + nb) = v;
        }
        na += a ? 1 : 0;
        nb += bo ? 1 : 0;
    };
    auto flush = [&]() {
        if (na - out >= 4) {
            const int r = out & 4;
            *reinterpret_cast<int4*>(entry(out)) = make_int4(ring[r][tid], ring[r + 1][tid], ring[r + 2][tid],
                                                             ring[r + 3][tid]);
            out += 4;
        }
    };
    const int m = min(cnt, A.rc), nq = (m + 3) >> 2;
    const int4* hq = reinterpret_cast<const int4*>(A.hits + row_slot(s, 0, A.rc));
    int4 nxt = nq > 0 ? __ldcs(hq) : make_int4(0, 0, 0, 0);
    for (int q = 0; q < nq; ++q) {
        const int left = m - 4 * q;  // entries past the row's end are stale: not gathered
        const int4 h = make_int4(nxt.x, left > 1 ? nxt.y : 0, left > 2 ? nxt.z : 0, left > 3 ? nxt.w : 0);
        const float4 x0 = __ldg(A.xt + h.x), x1 = __ldg(A.xt + h.y), x2 = __ldg(A.xt + h.z), x3 = __ldg(A.xt + h.w);
        if (q + 1 < nq) nxt = __ldcs(hq + 32LL * (q + 1));
        take(h.x, x0, true);
        take(h.y, x1, left > 1);
        take(h.z, x2, left > 2);
        take(h.w, x3, left > 3);
        flush();
    }
    for (int e = m; e < cnt; ++e) {
        const int t = pool[e - m];
        take(t, __ldg(A.xt + t), true);
        flush();
    }
    for (int k = out; k < na; ++k) *entry(k) = ring[k & 7][tid];
    for (int k = 0; k < min(nb, kStash); ++k) *entry(nA + k) = stash[k][tid];
    A.rcnt[s] = make_int2(na, nA + nb);
}

// The same rows by 8 lanes per particle, a quad of hits per lane and step, each
// entry placed by a scan over the lanes: for scenes whose particles alone leave
// most of the chip idle, where k_emit is one long chain of a row's loads.  Lanes
// against threads: 5.0 and 16 us at 1k particles, 15.6 and 18 at 32k; 26 and 22
// at 65k, 52 and 34 at 152k.
constexpr int kEmitLanesMax = 40000;
__global__ void __launch_bounds__(kEmitBlock) k_emit_lanes(const EmitArgs A)
{
    const int gid = blockIdx.x * kEmitBlock + threadIdx.x, l = gid & 7;
    const bool valid = (gid >> 3) < A.n;
    const int s = valid ? gid >> 3 : A.n - 1;
    int cnt = valid ? A.hcnt[s] : 0;
    const float4 xi = __ldg(A.xt + s);
    const float td = fabsf(xi.w);
    const int my_id = __float_as_int(xi.w) < 0 ? __ldg(A.tau_id + s) : 0x7fffffff;
    const int* pool = nullptr;
    int* out_pool = nullptr;
    if (cnt > A.rc) {
        const int o = A.hpool ? __ldg(A.ovf + s) : -1;
        if (o >= 0) {
            pool = A.hpool + o;
            out_pool = A.rpool + o;
        } else {
            cnt = A.rc;  // as in k_emit
        }
    }
    int* const row = A.rows + row_slot(s, 0, A.rc);
    auto entry = [&](int q) { return q < A.rc ? row + (q >> 2) * 128 + (q & 3) : out_pool + (q - A.rc); };
    const int* const hits = A.hits + row_slot(s, 0, A.rc);
    auto load = [&](int e) {  // the quad of hits e to e + 3 (segments are whole quads)
        if (e >= cnt) return make_int4(0, 0, 0, 0);
        return __ldcs(reinterpret_cast<const int4*>(e < A.rc ? hits + 32LL * e : pool + (e - A.rc)));
    };
    const int nA = min(cnt, A.cap);
    const int steps = __reduce_max_sync(kFull, (cnt + 31) >> 5);
    int na = 0, nb = nA;  // places of the next a- and b-only entries
    int4 nxt = load(4 * l);
    for (int k = 0; k < steps; ++k) {
        const int e = 32 * k + 4 * l, left = cnt - e;  // entries past the row's end are stale: not gathered
        const int h[4] = {left > 0 ? nxt.x : 0, left > 1 ? nxt.y : 0, left > 2 ? nxt.z : 0, left > 3 ? nxt.w : 0};
        float4 x[4];
#pragma unroll
        for (int z = 0; z < 4; ++z) x[z] = __ldg(A.xt + h[z]);
        nxt = load(e + 32);
        bool a[4], b[4];
        int mine = 0;  // a-entries, b-only entries << 16
#pragma unroll
        for (int z = 0; z < 4; ++z) {
            const float d2 = exact_d2(xi, x[z]);
            const bool in = left > z;
            a[z] = in && (d2 < td || (d2 == td && h[z] <= my_id));
            b[z] = in && d2 <= fabsf(x[z].w);
            if (d2 == -x[z].w) b[z] = in && (__float_as_int(x[z].w) >= 0 || s <= __ldg(A.tau_id + h[z]));
            mine += a[z] ? 1 : (b[z] ? 1 << 16 : 0);
        }
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const int t = __shfl_up_sync(kFull, incl, o, 8);
            if (l >= o) incl += t;
        }
        const int all = __shfl_sync(kFull, incl, 7, 8);
        int pa = na + ((incl - mine) & 0xffff), pb = nb + ((incl - mine) >> 16);
#pragma unroll
        for (int z = 0; z < 4; ++z)
            if (a[z] || b[z])
                *entry(a[z] ? pa++ : pb++) = h[z] | (a[z] ? kRowFlagA : 0) | (b[z] ? kRowFlagB : 0);
        na += all & 0xffff;
        nb += all >> 16;
    }
    if (valid && l == 0) A.rcnt[s] = make_int2(na, nb);
}

// The public list: 8 lanes per particle copy its row's a-entries in caller
// ids, 8 consecutive entries (one 32-byte sector) at a time.  Bound by the
// gathers of perm: 20 us for a dynamic list of 99k particles, 47 as part of the
// row kernel before.
__global__ void __launch_bounds__(256)
    k_export(const int* __restrict__ rows, const int* __restrict__ rpool, const int* __restrict__ ovf,
             const int2* __restrict__ rcnt, const int* __restrict__ perm, const int* __restrict__ offs, int n, int cap,
             int rc, int* __restrict__ index, int* __restrict__ elements, long long capacity, int* __restrict__ err)
{
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int s = (int)(gid >> 3), sub = (int)(gid & 7);
    if (s >= n) return;
    const int ps = perm[s], m = rcnt[s].x;
    const long long o = cap > 0 ? (long long)ps * cap : (long long)offs[ps];
    if (sub == 0) index[ps] = cap > 0 ? m : (int)o;
    if (!elements) return;
    const RowView row{rows, rpool, ovf, rc};
    bool over = false;
    for (int e = sub; e < m; e += 8) {
        if (o + e < capacity)
            elements[o + e] = __ldg(perm + (row.at(s, e) & kRowIndexMask));
        else
            over = true;
    }
    if (over) atomicOr(err, kErrPublicOverflow);
}

// Smallest float T with sqrt_rn(T) >= h: for every float d2, sqrt_rn(d2) < h
// exactly when d2 < T (host sqrtf is correctly rounded, as __fsqrt_rn is).
static float radius_threshold(float h)
{
    float T = h * h;
    while (std::sqrt(T) < h) T = std::nextafter(T, INFINITY);
    while (T > 0.0f && std::sqrt(std::nextafter(T, 0.0f)) >= h) T = std::nextafter(T, 0.0f);
    return T;
}

template <int KPB, bool kLong, bool kCapped>
static void launch_stage(const BuildArgs& A, int blocks_wanted, int sms, cudaStream_t st)
{
    // a resident grid
    const size_t smem = kBuildWarps * sizeof(Stage<KPB, kLong>);
    cudaFuncSetAttribute(k_build<KPB, kLong, kCapped>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_build<KPB, kLong, kCapped>, kBuildWarps * 32, smem);
    k_build<KPB, kLong, kCapped>
        <<<std::min(blocks_wanted, sms * std::max(per_sm, 1)), kBuildWarps * 32, smem, st>>>(A);
}
template <int KPB>
static void launch_build(const BuildArgs& A, bool capped, int blocks_wanted, int sms, cudaStream_t st)
{
    if (A.row_cap > 128)
        capped ? launch_stage<KPB, true, true>(A, blocks_wanted, sms, st)
               : launch_stage<KPB, true, false>(A, blocks_wanted, sms, st);
    else
        capped ? launch_stage<KPB, false, true>(A, blocks_wanted, sms, st)
               : launch_stage<KPB, false, false>(A, blocks_wanted, sms, st);
}

int build_rows(pk_ctx* c, int n, const Grid& g, float h, int cap, int row_cap, int* pub_index,
               int* pub_elements, long long pub_capacity, cudaStream_t st, bool spill)
{
    if (n <= 0) return 0;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
    const int pbn = c->tune.build_pb;
    int launches = 0;
    const bool dyn_pub = cap <= 0 && pub_index != nullptr;
    const bool capped = cap > 0;
    BuildArgs A;
    A.xs = c->xs_pre;
    A.start = c->cell_start;
    A.items = c->items;
    A.count = c->cell_cnt;
    A.nitems = c->counters;
    A.g = g;
    A.n = n;
    A.row_cap = row_cap;
    A.cap = cap;
    A.T = radius_threshold(h);
    A.flags = capped ? 0 : (kRowFlagA | kRowFlagB);
    A.hits = capped ? c->hits : c->rows;
    A.hcnt = c->hcnt;
    A.rcnt = capped ? nullptr : c->rcnt;
    A.count_c = dyn_pub ? c->count_c : nullptr;
    A.xt = c->xa;
    A.tau_id = c->tau_id;
    A.perm = c->perm;
    A.err = c->d_err;
    A.pool_cap = spill ? c->pool_cap : 0;
    A.spill = c->spill;
    A.ovf = c->ovf;
    A.hpool = capped ? c->hpool : c->rpool;
    // cells are few in a small scene: their passes are spread over more warps
    A.split = n <= 12288 ? 2 : (n <= 24576 ? 1 : 0);
    const long long warps = (long long)n << A.split;
    const int blocks = (int)std::min<long long>((warps + kBuildWarps - 1) / kBuildWarps, 1 << 20);
    prof_begin(c, PK_PROF_SELECT, st);
    if (c->tune.on) cudaEventRecord(c->tune.ev[0], st);
    if (pbn == 8)
        launch_build<8>(A, capped, blocks, sms, st);
    else if (pbn == 4)
        launch_build<4>(A, capped, blocks, sms, st);
    else
        launch_build<16>(A, capped, blocks, sms, st);
    if (c->tune.on) cudaEventRecord(c->tune.ev[1], st);
    ++launches;
    prof_end(c, PK_PROF_SELECT, st);
    prof_begin(c, PK_PROF_EMIT, st);
    if (capped) {
        EmitArgs E;
        E.hcnt = c->hcnt;
        E.hits = c->hits;
        E.hpool = A.pool_cap > 0 ? c->hpool : nullptr;
        E.ovf = c->ovf;
        E.xt = c->xa;
        E.tau_id = c->tau_id;
        E.n = n;
        E.cap = cap;
        E.rc = row_cap;
        E.rows = c->rows;
        E.rpool = c->rpool;
        E.rcnt = c->rcnt;
        const unsigned nb = (unsigned)(((long long)n + kEmitBlock - 1) / kEmitBlock);
        if (n <= kEmitLanesMax)
            k_emit_lanes<<<(unsigned)(((long long)n * 8 + kEmitBlock - 1) / kEmitBlock), kEmitBlock, 0, st>>>(E);
        else
            k_emit<<<nb, kEmitBlock, 0, st>>>(E);
        ++launches;
    } else if (dyn_pub) {
        exclusive_scan(c->count_c, n, c->offs, c->scan_part, st);
        launches += scan_launches();
    }
    if (pub_index) {
        k_export<<<(unsigned)(((long long)n * 8 + 255) / 256), 256, 0, st>>>(
            c->rows, c->rpool, c->ovf, c->rcnt, c->perm, c->offs, n, cap, row_cap, pub_index, pub_elements,
            pub_capacity, c->d_err);
        ++launches;
    }
    prof_end(c, PK_PROF_EMIT, st);
    return launches;
}

}  // namespace pk
