// Pair counting for corruscant's pair_count (kdquery.c:62-113, :165-249),
// batched over all bin edges at once.
//
// Semantics kept from the reference: the reference traversal counts, for
// every query point q and every tree node t, weight(t) if fl(d2) < fl(r*r),
// where d2 is evaluated as
//     dx = t.x - q.x, ...;  d2 = dx*dx;  d2 = fma(dy,dy,d2);  d2 = fma(dz,dz,d2)
// (kdquery.c:39-47 as the reference build compiles it), and its pruning
// (kdquery.c:96-104) never drops such a pair.  Here a pair lands in bin e, the
// first sorted squared edge with d2 < rsq[e]; cumulative sums over e give the
// reference's per-radius counts.
//
// Work decomposition (B200-first, not the reference's per-query recursion):
//   k_traverse : one warp per query block (<= 128 points) walks the tree-side
//                counting tree with box-box distance bounds.  Node pairs
//                beyond the last edge are pruned, node pairs inside one bin
//                are accepted as count(block) x count(node), and leaf pairs
//                become tile records (tree run, active edge range).  Run twice:
//                once to count the tiles, once to write them.
//   k_tiles    : one CTA per query block, its queries as eight tiles of 16,
//                walks the block's tile records.  Each query tile is compared
//                with a run's points only against the edges that its own box
//                and the leaf's allow.  Mixed mode: FP32 distances relative to
//                the block centre from the tensor pipe, binned against those
//                edges with a saturating ramp that is exactly 0 or 1 outside an
//                error band; a query with any pair of the run inside the band is
//                recounted in FP64 with the reference's operation order.  FP64
//                mode: every distance in FP64 (boxes decide in FP32 with margins
//                for every rounding, in both modes).  Per-query counters live in
//                shared memory and are reduced per own field into the global
//                (bin, qfield, tfield) histogram, tree field by tree field.

#include <algorithm>
#include <exception>
#include <new>
#include <climits>
#include <cstdlib>
#include <cstring>
#include <cmath>
#include <mutex>
#include <vector>

#include <cuda_fp16.h>

#include "kd_cuda_util.cuh"
#include "kd_sort.cuh"

namespace kd {

constexpr int kTravWarps = 4;
// Node-pair stack per traversal warp.  A round pops the top min(sp, 32)
// entries and pushes at most two children for each, so the stack grows by at
// most 32 entries per tree level: at most 32 * D + 64 entries for a counting
// tree of depth D <= 27 (928).  A push past the end stops the count with
// KD_EINTERNAL instead of writing out of bounds.  4 KB per warp (rather
// than 8) lets the count pass run more warps per SM: the traversal of the
// clustered 1M / 20M batch takes 16.3 ms instead of 19.5.
constexpr int kStack = 1024;
static_assert(kStack >= 32 * 27 + 64, "stack bound of a depth-27 counting tree");
constexpr int kShardChunk = 32;  // blocks per interleaved shard chunk

struct TreeSide {
    const double *box;
    const int *count, *tf, *leaf_run, *leaf_pos;
    const int *run_start, *run_len, *run_tf;
    int D, nleaves;
};

struct QuerySide {
    const double *x, *y, *z;
    const int *qf;
    const int *blk_start, *blk_len, *blk_qf;
    const double *blk_box;
};

// One (tree, query tree) count of a batch.  A batch numbers the query blocks
// of all its jobs consecutively: job j owns global blocks [jblk[j], jblk[j+1]).
struct JobDesc {
    TreeSide T;
    QuerySide Q;
    const double *tx, *ty, *tz;  // tree points, FP64, counting order
    const float4 *t4;            // tree points: -2 t_r, t_r relative to the leaf's centre
    const kd_leaf *leaf;         // leaf boxes: centre and half-extents
    double hT;                   // largest leaf half-diagonal, with margin
    unsigned long long *H;       // (ne + 1) x Fqe x Fte bin histogram
    // Symmetric job (tree and query are one catalog whose points all have own
    // field == tree field): a block counts only tree points at or after its
    // own first point; points inside the block as ordered pairs into H, points
    // after it once into H2, and the host adds H2 and its field transpose.
    unsigned long long *H2;
    int Fqe, Fte;
    int sym, pad_;
};
static_assert(sizeof(JobDesc) % 8 == 0, "JobDesc is copied in 8-byte words");

// the job owning global block g: the last j with jblk[j] <= g (an empty job
// shares its start with the next one, which is then the one found)
__device__ __forceinline__ int job_of(const int *__restrict__ jblk, int njobs, int g)
{
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jblk[mid] <= g) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Bins a pair of boxes can reach: pairs land in bins elo..ehi (ne = beyond
// every edge).  The box bounds are exact for the points' true distances; the
// relative margin covers the FP64 rounding of the reference's d2 and of this
// bound computation.
__device__ __forceinline__ void bin_range(const double *a, const double *b,
                                          const double *__restrict__ rsq, int ne, int &elo,
                                          int &ehi)
{
    double dmin2 = 0.0, dmax2 = 0.0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        double g = fmax(0.0, fmax(b[d] - a[3 + d], a[d] - b[3 + d]));
        double sp = fmax(b[3 + d] - a[d], a[3 + d] - b[d]);
        dmin2 += g * g;
        dmax2 += sp * sp;
    }
    double lo = dmin2 * (1.0 - 1e-12), hi = dmax2 * (1.0 + 1e-12);
    int l = 0, h = ne;  // first e with rsq[e] > lo
    while (l < h) {
        int m = (l + h) >> 1;
        if (rsq[m] > lo) h = m;
        else l = m + 1;
    }
    elo = l;
    h = ne;  // first e with rsq[e] > hi
    while (l < h) {
        int m = (l + h) >> 1;
        if (rsq[m] > hi) h = m;
        else l = m + 1;
    }
    ehi = l;
}

// A tile record: x = run start, y = leaf, z = run length | tree field << 8 |
// first active edge << 16 | active edge count << 24.
struct TravOut {
    const int *gmap;         // shard-local block index -> global block (NULL: identity)
    int *count;              // COUNT pass: tiles per block
    const long long *off;    // FILL pass: launch-relative tile offsets
    uint4 *rec;              // FILL: tile records
    unsigned long long *accepted;
    int *err;
};

// one warp per shard-local block index i in [g0, g1) (global block o.gmap[i])
template <bool FILL>
__global__ void __launch_bounds__(32 * kTravWarps) k_traverse(const JobDesc *__restrict__ jobs,
                                                             const int *__restrict__ jblk,
                                                             int njobs,
                                                             const double *__restrict__ g_rsq,
                                                             int ne, int g0, int g1, TravOut o)
{
    __shared__ int stack[kTravWarps][kStack];
    __shared__ double rsq[KD_MAX_EDGES];
    __shared__ double wb[kTravWarps][6];
    for (int k = threadIdx.x; k < ne; k += blockDim.x) rsq[k] = g_rsq[k];
    __syncthreads();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int li = g0 + blockIdx.x * kTravWarps + w;
    if (li >= g1) return;
    const int g = o.gmap ? o.gmap[li] : li;
    const int j = job_of(jblk, njobs, g);
    const int b = g - jblk[j];
    const TreeSide T = jobs[j].T;
    const QuerySide Q = jobs[j].Q;
    unsigned long long *const H = jobs[j].H, *const H2 = jobs[j].H2;
    const int Fqe = jobs[j].Fqe, Fte = jobs[j].Fte;
    const bool sym = jobs[j].sym != 0;
    const int alen = Q.blk_len[b], aqf = Q.blk_qf[b];
    const int qb0 = Q.blk_start[b], qb1 = qb0 + alen;  // the block's raw positions
    double *bb = wb[w];
    if (lane < 6) bb[lane] = Q.blk_box[6 * (size_t)b + lane];
    int *st = stack[w];
    if (lane == 0) st[0] = 1;
    __syncwarp();
    int sp = 1;
    long long emitted = 0;
    const long long base = FILL ? o.off[li - g0] : 0;
    unsigned long long acc_pairs = 0, blocked_pairs = 0;
    long long guard = 4LL * T.nleaves + 64;
    while (sp > 0) {
        if (--guard < 0) {
            if (lane == 0) atomicCAS(o.err, 0, KD_EINTERNAL);
            break;
        }
        const int nb = min(sp, 32);
        const int h = lane < nb ? st[sp - nb + lane] : 0;
        __syncwarp();
        sp -= nb;
        int act = 0, nr = 0, leaf = 0, elo = 0, ehi = 0;
        if (h) {
            // symmetric jobs: the node's raw positions [nlo, nhi) against the
            // block's [qb0, qb1): before it -> nothing (the other side's block
            // counts these pairs), after it -> once into H2, overlapping ->
            // descend, runs cut at the block's ends
            int nlo = 0, nhi = 0;
            if (sym) {
                const int sh = T.D - (31 - __clz(h));
                nlo = T.leaf_pos[(h << sh) - T.nleaves];
                nhi = T.leaf_pos[((h + 1) << sh) - T.nleaves];
            }
            const bool after = sym && nlo >= qb1;
            if (sym && nhi <= qb0) {
                act = 0;
            } else {
                bin_range(bb, T.box + 6 * (size_t)h, rsq, ne, elo, ehi);
                const bool whole = !sym || after || (nlo >= qb0 && nhi <= qb1);
                if (elo >= ne) {
                    act = 0;
                } else if (whole && elo == ehi && aqf >= 0 && T.tf[h] >= 0) {
                    if (FILL) {
                        const unsigned long long c =
                            (unsigned long long)alen * (unsigned long long)T.count[h];
                        atomicAdd(&(after ? H2 : H)[((size_t)elo * Fqe + aqf) * Fte + T.tf[h]], c);
                        acc_pairs += c;
                    }
                } else if (h >= T.nleaves) {
                    // pairs of a node pair inside one bin that are tiled only
                    // because a side holds several fields (a per-field accept
                    // would take them without distances)
                    if (FILL && whole && elo == ehi)
                        blocked_pairs += (unsigned long long)alen * (unsigned long long)T.count[h];
                    act = 2;
                    leaf = h - T.nleaves;
                    const int r0 = T.leaf_run[leaf], r1 = T.leaf_run[leaf + 1];
                    if (!sym) {
                        nr = r1 - r0;
                    } else {
                        for (int r = r0; r < r1; r++) {
                            const int a = T.run_start[r], e = a + T.run_len[r];
                            nr += (max(a, qb0) < min(e, qb1)) + (max(a, qb1) < e);
                        }
                    }
                } else {
                    act = 1;
                }
            }
        }
        int ps = act == 1 ? 2 : 0;
        for (int off = 1; off < 32; off <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, ps, off);
            if (lane >= off) ps += v;
        }
        const int ptot = __shfl_sync(0xffffffffu, ps, 31);
        if (sp + ptot > kStack) {
            if (lane == 0) atomicCAS(o.err, 0, KD_EINTERNAL);
            break;
        }
        if (act == 1) {
            st[sp + ps - 2] = 2 * h + 1;
            st[sp + ps - 1] = 2 * h;
        }
        sp += ptot;
        int es = act == 2 ? nr : 0;
        for (int off = 1; off < 32; off <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, es, off);
            if (lane >= off) es += v;
        }
        const int etot = __shfl_sync(0xffffffffu, es, 31);
        if (FILL && act == 2) {
            const unsigned code = (unsigned)elo | ((unsigned)(ehi - elo) << 8);
            const int r0 = T.leaf_run[leaf], r1 = T.leaf_run[leaf + 1];
            long long idx = base + emitted + es - nr;
            // record: start, leaf, length | tree field << 8 | edges << 16, and
            // w = 1 for the once-counted (H2) part of a symmetric job
            auto put = [&](int a, int len, int tf, unsigned once) {
                o.rec[idx++] = make_uint4((unsigned)a, (unsigned)leaf,
                                          (unsigned)len | ((unsigned)tf << 8) | (code << 16), once);
            };
            for (int r = r0; r < r1; r++) {
                const int a = T.run_start[r], e = a + T.run_len[r];
                if (!sym) {
                    put(a, e - a, T.run_tf[r], 0u);
                } else {
                    const int ia = max(a, qb0), ib = min(e, qb1), aa = max(a, qb1);
                    if (ia < ib) put(ia, ib - ia, T.run_tf[r], 0u);
                    if (aa < e) put(aa, e - aa, T.run_tf[r], 1u);
                }
            }
        }
        emitted += etot;
        __syncwarp();
    }
    if (!FILL && lane == 0) o.count[li - g0] = (int)emitted;
    if (FILL) {
        for (int off = 16; off; off >>= 1) {
            acc_pairs += __shfl_xor_sync(0xffffffffu, acc_pairs, off);
            blocked_pairs += __shfl_xor_sync(0xffffffffu, blocked_pairs, off);
        }
        if (lane == 0 && acc_pairs) atomicAdd(o.accepted, acc_pairs);
        if (lane == 0 && blocked_pairs) atomicAdd(o.accepted + 4, blocked_pairs);
    }
}

// ---------------------------------------------------------------- tiles
//
// One CTA of four warps per query block.  Its 128 queries are eight tiles of
// 16; the warps take the block's tile records (each a run of up to 64 points
// of one leaf) in chunks of 4 to 32, one tree field after the other, and share
// the queries' operands and the counters.  For every record each query tile
// has its own window: the edges that the distances between the tile's box and
// the leaf's box allow, found by one lane per (query tile, record) for four
// records at a time.  A query tile without an edge in its window costs one
// counter; the others run over the run's points in steps of 16 queries x 8
// points, against the edges of their window only.  With one window per block
// and leaf, a pair of the clustered 1M / 20M batch is compared with 3.0 edges;
// with one per 16 queries it is 1.5, and a quarter of the pairs needs none.
//
// Mixed mode: the squared distances of a step are one mma.m16n8k16 (F16 in,
// FP32 out): each coordinate of query and point is split into two halves, so
// that all four half products of the three coordinates are 12 of the 16 terms,
// and N = |t|^2 - Rref as two halves times 1 are two more; the accumulator
// starts at |q|^2 + Rref - R of the window's first edge.  The products are
// exact, and the result x = d2 - R is small where the decision is made: its
// error is 0.59 to 1.09 u (sqrt(d2) + Rq)^2 RMS (u = 2^-24) at radii of 2 to 10
// block radii Rq and 0.25 at half a block radius, where the FP32 FMA chain it
// replaces has 0.59 to 1.16 and 0.23.
// FP64 mode: a query tile at a time, each half of the warp with half of the
// run's points, every distance in the reference's operation order, up to six
// edges per distance (two tiles at a time, with one window for both, and four
// edges: 7% and 4% slower; compares as integers, on the ALU: 4%).  Bound by
// the issue slots, then the FP64 pipe (76% and 55% used).
//
// Bound: the issue slots (73% used) and the FP32 pipe (51%), by the binning (a
// ramp, a count and a check per pair and edge: 15 clocks per 128 pairs and edge
// in isolation, 20 here) and the per-pass work around it: 289 instructions per
// 16 queries x 50 points and two edges, 120 of them the binning.  More code is
// slower (loops unrolled by two or four: 15 to 35%), the instruction cache
// decides.  Seven CTAs per SM: what is uniform over a block lives in shared
// memory so that 72 registers do.  In the counting layout of that time, 3M
// uniform points and 21 edges took 36.2 ms in the former kernel (a warp per
// block, four queries per lane, one window), 31.5 with four warps per scheduler
// and 128 registers, 23.8 with seven; 1 edge 10.8 against 16.4; FP64 mode 37.3
// against 51.0.  CTA per block instead of warp per block also gives small
// counts four times the warps: 0.31 against 1.72 ms for DD + DR + RR of
// 4k / 80k points.
// Measured and left out: tcgen05 with the batch's distances in TMEM (free
// distances, but 128 queries in step and the same binning: 45.7 ms); items of
// one query tile and one edge, four at a time, repeating the MMA (39.3); two
// query tiles per pass where their windows agree on two edges (24.1); six and
// eight CTAs per SM (3% and 1% slower); four to sixteen records a fetch (0 to
// 7% slower).

constexpr int kMT = 16;                       // queries per tile (MMA rows)
constexpr int kMTiles = KD_BLOCK_MAX / kMT;   // query tiles per block
constexpr int kNT = 8;                        // points per step (MMA columns)
constexpr int kGroup = 32 / kMTiles;          // records whose windows are found together
constexpr int kTileWarps = 4;
constexpr int kTileThreads = 32 * kTileWarps;
constexpr int kTilesPerSm = 7;                // CTAs per SM the registers are held to
constexpr int kPStride = 136;                 // counters per edge (128 queries + bank shift)
constexpr unsigned kWideCount = 1u << 27;     // 32 counters below it sum to 32 bits
static_assert(kMTiles == 8 && kTileThreads == KD_BLOCK_MAX, "lane layouts below");

// FP32 tiles only where every staged value and square stays far inside FP32
// range: tree and query points within kFp32Span of the block centre (their
// squares and products below 1e30 < FLT_MAX) and squared edges below 1e30.
// Records beyond that (coordinates or radii of 1e15 and more) are counted
// by the exact FP64 path.
constexpr double kFp32Span = 1e15;
constexpr double kFp32MaxR = 1e30;

// Half-width E of the band around edge R inside which the MMA's decision is
// not trusted: a pair whose computed d2 - R is at least E away from zero is
// on the side that the FP64 reference puts it on.
// Geometry: query q and tree point t relative to the block centre, |q| <= Rq;
// t is staged as t' = fl32(fl32(t - c) + fl32(c - o)) (c: its leaf's centre,
// |t - c| <= hT), both scaled by a power of two S.  The MMA sums
//   x = C + N - 2 q.t',  N = |t'|^2 - Rref,  C = |q|^2 + Rref - R0,
// with the cross term's factors and N as two halves each (products exact).
// The decision is on x - (R - R0).  With u = 2^-24, P = sqrt(1.2 R) + Rq >=
// |t'| for every pair with d2 <= 1.2 R, and M = P^2 + R:
//   coordinates  2 (P + Rq) u (2P + 2hT + Rq)   as two roundings of t
//   N            3u M as an FMA chain, 2u M its two halves
//   cross term   8u Rq P      (2^-23 relative for each split factor)
//   C, edges     2u (Rq^2 + R) + 3u R
//   ramp         4u R         (its offset and slope)
//   accumulation 17u max(M, 2 Rq P), with |N|, |C| <= M, |2 q t'| <= 2 Rq P
// plus the halves' absolute floor, 2^-25 of the scaled values, and the
// rounding of the FP64 reference itself; 25% on top.
// All but the accumulation is derived.  How the tensor core aligns, cuts and
// rounds the 17 terms PTX leaves open, so that term is an assumption.  It rests
// on a measurement: over 2.5M sums each of eight kinds (spread exponents, equal
// magnitudes, a large term, cancelling ones) the error was at most 2.1u of the
// largest term where the sum cancels, and else 2u of the result besides, which
// here stays below 3 max(M, 2 Rq P): 8u in all, where an FP32 FMA chain had up to
// 12u where the sum cancels.  (x as a whole: at most 6u (sqrt(d2) + Rq)^2
// measured, about 70u allowed.)  Pairs with d2 > 1.2 R: their error grows with
// (sqrt(d2) + Rq)^2 while x - (R - R0) >= d2 / 6, so the sign is right
// unless d2 is so small beside Rq^2 that E's Rq terms cover the error.
__device__ __forceinline__ double band_halfwidth(double R, double Rq, double hT, double S)
{
    const double u = 5.9604644775390625e-08;  // 2^-24
    const double P = sqrt(1.2 * R) + Rq, M = P * P + R;
    const double e = 2.0 * (P + Rq) * (2.0 * P + 2.0 * hT + Rq) + 5.0 * M + 8.0 * Rq * P +
                     2.0 * (Rq * Rq + R) + 7.0 * R + 17.0 * fmax(M, 2.0 * Rq * P);
    const double f = 1.1920928955078125e-07 / S;  // 2^-23 / S
    return 1.25 * u * e + 1e-15 * R + f * (P + Rq) + f / S;
}

// reference-order FP64 distance (kdquery.c:39-47 as compiled)
__device__ __forceinline__ double d2_ref(double tx, double ty, double tz, double qx, double qy,
                                         double qz)
{
    const double dx = __dsub_rn(tx, qx), dy = __dsub_rn(ty, qy), dz = __dsub_rn(tz, qz);
    double s = __dmul_rn(dx, dx);
    s = __fma_rn(dy, dy, s);
    return __fma_rn(dz, dz, s);
}

struct TileArgs {
    const JobDesc *jobs;
    const int *jblk;
    int njobs;
    const double *rsq;
    int ne;
    int g0, g1;                 // shard-local block indices of this launch
    const int *gmap;            // shard-local index -> global block (NULL: identity)
    const long long *off;       // launch-relative tile offsets
    const uint4 *rec;
    int *work;
    unsigned long long *stats;  // tested, rechecked, accepted, wide, edge-pairs, tiles
};

// saturating FMA: clamp(a*b + c, 0, 1) in one instruction (NaN -> 0)
__device__ __forceinline__ float fma_sat(float a, float b, float c)
{
    float d;
    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// d = A (16 x 16, row) B (16 x 8, col) + c, rows g = lane / 4 and g + 8 at
// columns 2 (lane % 4) and + 1 (c0, c1: the rows' start values)
__device__ __forceinline__ void mma_16x8x16(float (&d)[4], const uint4 &a, uint32_t b, float c0,
                                            float c1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, "
        "{%4, %5, %6, %7}, {%8, %8}, {%9, %9, %10, %10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b), "f"(c0), "f"(c1));
}

// v as two halves hi + lo (lo rounds what hi left over)
__device__ __forceinline__ uint32_t split_halves(float v)
{
    const __half hi = __float2half_rn(v);
    const __half lo = __float2half_rn(v - __half2float(hi));
    return (uint32_t)__half_as_ushort(hi) | ((uint32_t)__half_as_ushort(lo) << 16);
}

// FP64 mode: a query's pairs with np pairs of staged points (a missing one is
// NaN: its distance is below no edge, while any number could be a query's own
// place) below the ne first edges of R (ne <= K <= kFpEdges)
constexpr int kFpEdges = 6;
template <int K>
__device__ __forceinline__ void fp64_run(const double2 *__restrict__ tx,
                                         const double2 *__restrict__ ty,
                                         const double2 *__restrict__ tz, int np, double qx, double qy,
                                         double qz, const double *R, int ne, unsigned (&cnt)[kFpEdges])
{
    double r[K];
#pragma unroll
    for (int k = 0; k < K; k++) r[k] = k < ne ? R[k] : 0.0;  // (no distance is below zero)
#pragma unroll 4
    for (int j = 0; j < np; j++) {
        const double2 x = tx[j], y = ty[j], z = tz[j];
        const double a = d2_ref(x.x, y.x, z.x, qx, qy, qz), b = d2_ref(x.y, y.y, z.y, qx, qy, qz);
#pragma unroll
        for (int k = 0; k < K; k++) cnt[k] += (unsigned)(a < r[k]) + (unsigned)(b < r[k]);
    }
}

// Shared memory of a CTA (what is the same for all threads of a block lives
// here rather than in registers: warps in flight are what the kernel needs).
//   F[e * kMTiles + m]: points of records below edges e, e + 1, ... for every
//     query of tile m
//   P[e * kPStride + q], behind it: pairs of query q below edge e, over the
//     records whose window for q's tile holds e
//   behind P, in the general variant: the edge table of small leaves
struct TileCommon {
    JobDesc job;  // the job of the block being counted
    double R[KD_MAX_EDGES];
    double o[3];                             // block centre
    float Rup[KD_MAX_EDGES], Rdn[KD_MAX_EDGES];  // R rounded up / down
    float qc[kMTiles][3], qh[kMTiles][3];    // the query tiles' boxes: centre, half-extents
    unsigned F[(KD_MAX_EDGES + 1) * kMTiles];
    unsigned keys[16];                       // the block's flush keys, a bit each
    unsigned long long stats[5];             // tested, rechecked, wide, edge-pairs, tiles
    long long eoff;                          // the block's records: first, number
    int ecnt, chunk;
    int qs, qlen;                            // its queries: first, number
    int next, item, kmin, kmax, kfp;
    float Rq, hT, S;
    // of the general variant
    float hSmall, hcap;                      // half-extents' sum of leaves with the smaller band, with any
    int points, bqf;                         // of the block's runs; its single own field, -1 when mixed
};
template <int MODE> struct TileSmem;
template <> struct TileSmem<KD_MODE_MIXED> : TileCommon {
    alignas(16) uint4 qa[kMTiles][32];       // MMA A fragments of the query tiles
    float2 qn[kMTiles][kMT / 2];             // |q|^2 S^2 of rows g and g + 8
    float2 edge[KD_MAX_EDGES];               // R S^2 and 0.4545 / (E S^2)
    alignas(16) uint32_t bs[kTileWarps][KD_RUN_MAX / kNT * 32];  // MMA B fragments of the staged runs
};
template <> struct TileSmem<KD_MODE_FP64> : TileCommon {
    alignas(16) double pt[kTileWarps][3][KD_RUN_MAX];  // the staged runs
};

// The MMA operands of the block's queries (relative to the block centre o) and
// the edge tables, at scale S, by the whole CTA.  Lane (g, t) of a query
// tile's fragment holds, for t < 3, coordinate t of rows g and g + 8: the
// halves of v = -2 q_t S as (hi, hi) against the point's (hi, lo), and (lo,
// lo) against the same; for t = 3, (1, 1) against the halves of N, and (0, 0).
template <bool GENERAL> __device__ __noinline__ void set_scale(TileSmem<KD_MODE_MIXED> &s, float2 *small, int ne, int tid)
{
    const double S = (double)s.S, Rq = (double)s.Rq;
    const int qs = s.qs, qlen = s.qlen;
    for (int i = tid; i < kMTiles * 32; i += kTileThreads) {
        const int m = i >> 5, g = (i & 31) >> 2, t = i & 3;
        uint32_t hh[2] = {0x3C003C00u, 0x3C003C00u}, ll[2] = {0u, 0u};
        if (t < 3) {
            const double *const src = t == 0 ? s.job.Q.x : (t == 1 ? s.job.Q.y : s.job.Q.z);
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int q = kMT * m + g + 8 * r;
                const double v = q < qlen ? -2.0 * (src[qs + q] - s.o[t]) * S : 0.0;
                const __half h = __double2half(v), l = __double2half(v - (double)__half2float(h));
                hh[r] = (uint32_t)__half_as_ushort(h) * 0x10001u;
                ll[r] = (uint32_t)__half_as_ushort(l) * 0x10001u;
            }
        }
        s.qa[m][i & 31] = make_uint4(hh[0], hh[1], ll[0], ll[1]);
    }
    {
        double n = 0.0;
        if (tid < qlen) {
            const double x = (s.job.Q.x[qs + tid] - s.o[0]) * S, y = (s.job.Q.y[qs + tid] - s.o[1]) * S,
                         z = (s.job.Q.z[qs + tid] - s.o[2]) * S;
            n = x * x + y * y + z * z;
        }
        float2 &q = s.qn[tid / kMT][tid % 8];
        if (tid % kMT < 8) q.x = (float)n;
        else q.y = (float)n;
    }
    for (int b = 0; b < (GENERAL && small ? 2 : 1); b++) {
        float2 *const edge = b ? small : s.edge;
        for (int k = tid; k < ne; k += kTileThreads)
            edge[k] = make_float2(
                (float)(s.R[k] * S * S),
                (float)(0.5 / 1.1 / (band_halfwidth(s.R[k], Rq, b ? (double)s.hSmall : (double)s.hT, S) * S * S)));
    }
}
template <bool GENERAL> __device__ __forceinline__ void set_scale(TileSmem<KD_MODE_FP64> &, float2 *, int, int) {}

// A whole block whose runs are a point or two each (many labels that interleave
// in space), by the whole CTA: a warp per record, four queries a lane, every
// distance in FP64 in the reference's order, and the pairs of each bin straight
// into the histogram.  A tile pass per (16 queries, point) and a flush per tree
// field take several times the instructions there, for many fields of few pairs
// each.  Bound by the issue slots (71% at 64 labels: a compare per pair and edge)
// and the adds' wavefronts (69%).  ONE, for a block with one own field, adds a
// run's pairs at once; the others add every pair, which needs enough pairs of
// fields to keep the adds apart.  400k points, 21 edges, tile passes -> this:
// labels of 64 kinds at random with themselves 24.7 -> 6.5 ms, of 250 kinds 48.1 ->
// 6.4; 8 kinds against 64 (512 pairs of fields) 42.7 -> 24.9, 8 against 40 31.9 ->
// 39.8; 16 kinds with themselves (runs of 4 points) 8.4 -> 24.  No labels against
// 64 kinds 34.6 -> 11.3, against 20 13.6 -> 10.0, 16 10.9 -> 9.7, 12 (runs of 5)
// 8.1 -> 9.5.
constexpr float kDirectRun = 2.5f, kDirectRunOne = 5.0f;  // points per run, on average
constexpr int kDirectCells = 512;                         // pairs of fields
template <bool ONE>
__device__ __noinline__ void count_direct(TileCommon &s, const uint4 *__restrict__ recs, int ne, int tid)
{
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int NQ = KD_BLOCK_MAX / 32;
    const int lane = tid & 31, one = ONE ? s.bqf : 0;
    const JobDesc &J = s.job;
    double qx[NQ], qy[NQ], qz[NQ];
    int qf[NQ];
#pragma unroll
    for (int g = 0; g < NQ; g++) {
        const int q = 32 * g + lane, i = s.qs + min(q, s.qlen - 1);
        qx[g] = J.Q.x[i];
        qy[g] = J.Q.y[i];
        qz[g] = J.Q.z[i];
        qf[g] = q < s.qlen ? (ONE ? one : J.Q.qf[i]) : -1;
    }
    unsigned long long pairs = 0, wide = 0, edges = 0, tiles = 0;
    while (true) {
        int c0 = 0;
        if (lane == 0) c0 = atomicAdd(&s.next, s.chunk);
        c0 = __shfl_sync(FULL, c0, 0);
        const int nr = min(s.chunk, s.ecnt - c0);
        if (nr <= 0) break;
        const uint4 mine = __ldg(recs + c0 + min(lane, nr - 1));
        for (int r = 0; r < nr; r++) {
            const int rs = __shfl_sync(FULL, (int)mine.x, r);
            const unsigned z = __shfl_sync(FULL, mine.z, r);
            const int n = z & 0xFF, tf = (z >> 8) & 0xFF, k0 = (z >> 16) & 0xFF, K = z >> 24;
            unsigned long long *const Hd = (__shfl_sync(FULL, mine.w, r) ? J.H2 : J.H) + tf;
            auto bin = [&](int e, int f) { return &Hd[((size_t)e * J.Fqe + f) * J.Fte]; };
            if constexpr (ONE) {
                // a lane per edge holds the run's pairs below it
                unsigned below = 0;  // the edge before these 32
                for (int kb = k0; kb < k0 + K; kb += 32) {
                    const int kn = min(32, k0 + K - kb);
                    unsigned cum = 0;
                    for (int j = 0; j < n; j++) {
                        const double x = __ldg(J.tx + rs + j), y = __ldg(J.ty + rs + j), zz = __ldg(J.tz + rs + j);
#pragma unroll
                        for (int g = 0; g < NQ; g++) {
                            const double d2 = d2_ref(x, y, zz, qx[g], qy[g], qz[g]);
                            for (int k = 0; k < kn; k++) {
                                const unsigned c = __popc(__ballot_sync(FULL, d2 < s.R[kb + k] && qf[g] >= 0));
                                if (lane == k) cum += c;
                            }
                        }
                    }
                    unsigned prev = __shfl_up_sync(FULL, cum, 1);
                    if (lane == 0) prev = below;
                    if (lane < kn && cum != prev) atomicAdd(bin(kb + lane, one), (unsigned long long)(cum - prev));
                    below = __shfl_sync(FULL, cum, kn - 1);
                }
                const unsigned rest = (unsigned)(n * s.qlen) - below;
                if (lane == 0 && k0 + K < ne && rest) atomicAdd(bin(k0 + K, one), (unsigned long long)rest);
            } else {
                for (int j = 0; j < n; j++) {
                    const double x = __ldg(J.tx + rs + j), y = __ldg(J.ty + rs + j), zz = __ldg(J.tz + rs + j);
#pragma unroll
                    for (int g = 0; g < NQ; g++) {
                        const double d2 = d2_ref(x, y, zz, qx[g], qy[g], qz[g]);
                        int e = k0;
                        for (int k = k0; k < k0 + K; k++) e += !(d2 < s.R[k]);
                        if (qf[g] >= 0 && e < ne) atomicAdd(bin(e, qf[g]), 1ull);
                    }
                }
            }
            const unsigned np = K ? (unsigned)(n * s.qlen) : 0u;
            pairs += np;
            edges += (unsigned long long)np * K;
            wide += K > 4 ? np : 0u;
            tiles += K ? (s.qlen + kMT - 1) / kMT : 0;
        }
    }
    if (lane == 0) {
        atomicAdd(&s.stats[0], pairs);
        atomicAdd(&s.stats[2], wide);
        atomicAdd(&s.stats[3], edges);
        atomicAdd(&s.stats[4], tiles);
    }
}

// Exact counts of the flagged rows of query tile m (rows: bit per row) over
// the run [rs, rs + n) for kn (<= 4) edges from kk on, added to their counters
// less what the lanes (g, t < kn) added before: v, rows g and g + 8.  The
// run's points stay in registers, two per lane.
__device__ __noinline__ void recount_rows(TileCommon &s, unsigned *P, unsigned rows, int m, int rs, int n,
                                          int kk, int kn, unsigned v, int lane)
{
    static_assert(KD_RUN_MAX <= 64, "two points per lane");
    const JobDesc &J = s.job;
    const int g = lane >> 2, t = lane & 3;
    rows &= (2u << (min(kMT, s.qlen - kMT * m) - 1)) - 1u;
    if (lane == 0) atomicAdd(&s.stats[1], (unsigned long long)(__popc(rows) * n));
    double x[2], y[2], z[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int j = rs + min(lane + 32 * h, n - 1);
        x[h] = __ldg(J.tx + j);
        y[h] = __ldg(J.ty + j);
        z[h] = __ldg(J.tz + j);
    }
    while (rows) {
        const int row = __ffs(rows) - 1;
        rows &= rows - 1;
        const int qi = s.qs + kMT * m + row;
        const double qx = __ldg(J.Q.x + qi), qy = __ldg(J.Q.y + qi), qz = __ldg(J.Q.z + qi);
        unsigned part = 0;  // counts of four edges, a byte each (n <= 64)
#pragma unroll
        for (int h = 0; h < 2; h++)
            if (lane + 32 * h < n) {
                const double d2 = d2_ref(x[h], y[h], z[h], qx, qy, qz);
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (k < kn) part += (unsigned)(d2 < s.R[kk + k]) << (8 * k);
            }
        const unsigned c = (__reduce_add_sync(0xffffffffu, part) >> (8 * t)) & 0xFFu;
        if (g == (row & 7) && t < kn)
            atomicAdd(&P[(kk + t) * kPStride + kMT * m + row], c - (row < 8 ? v & 0xFFFFu : v >> 16));
    }
}

// M query tiles against a staged run (nt steps of 8 points) and the K edges
// from kk on (K * M <= 4).  Each pair gives c = sat(a_k - 0.4545 x / E): exactly
// 0 or 1 where |x| is 10% beyond the band, in [1/22, 21/22] inside it.  Per
// tile, row and lane, sum_k acc_k equals sq = sum c^2 bit for bit when every c
// is 0 or 1; a band pair makes them differ by at least 0.04, far above the
// FP32 rounding of these short sums (at most 4 * 16 terms in [0, 1]).  Rows g
// and g + 8 travel as a pair through the packed FP32 pipe (FADD2 / FFMA2); the
// saturating ramp has no packed form.
template <int K, int M>
__device__ __forceinline__ void tile_pass(TileSmem<KD_MODE_MIXED> &s, unsigned *P, const int (&mt)[2],
                                          int kk, const float2 *edges, int nt, float ref, int rs, int n, int lane,
                                          const uint32_t *__restrict__ bs)
{
    static_assert(K * M <= 4 && M <= 2, "an item per lane of a row");
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int NI = K * M;  // item i: edge kk + i % K of tile mt[i / K]
    const int g = lane >> 2, t = lane & 3;
    const float2 *const edge = edges + kk;
    const float e0 = edge[0].x, nsl = -edge[K - 1].y;
    float a[K];
    a[0] = 0.5f;
#pragma unroll
    for (int k = 1; k < K; k++) a[k] = fmaf(e0 - edge[k].x, nsl, 0.5f);
    uint4 qa[M];
    float c0[M], c1[M];
    float2 acc[M][K], sq[M][2];
#pragma unroll
    for (int i = 0; i < M; i++) {
        qa[i] = s.qa[mt[i]][lane];
        const float2 qn = s.qn[mt[i]][g];
        c0[i] = qn.x + (ref - e0);
        c1[i] = qn.y + (ref - e0);
        sq[i][0] = sq[i][1] = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int k = 0; k < K; k++) acc[i][k] = make_float2(0.0f, 0.0f);
    }
    auto bin = [&](const float (&x)[4], int i) {
#pragma unroll
        for (int k = 0; k < K; k++) {
            const float2 c = make_float2(fma_sat(x[0], nsl, a[k]), fma_sat(x[2], nsl, a[k]));
            const float2 d = make_float2(fma_sat(x[1], nsl, a[k]), fma_sat(x[3], nsl, a[k]));
            acc[i][k] = __fadd2_rn(acc[i][k], c);
            sq[i][0] = __ffma2_rn(c, c, sq[i][0]);
            acc[i][k] = __fadd2_rn(acc[i][k], d);
            sq[i][1] = __ffma2_rn(d, d, sq[i][1]);
        }
    };
    if constexpr (M == 1) {
        for (; nt >= 2; nt -= 2, bs += 64) {
            float x[4], y[4];
            mma_16x8x16(x, qa[0], bs[0], c0[0], c1[0]);
            mma_16x8x16(y, qa[0], bs[32], c0[0], c1[0]);
            bin(x, 0);
            bin(y, 0);
        }
        if (nt) {
            float x[4];
            mma_16x8x16(x, qa[0], bs[0], c0[0], c1[0]);
            bin(x, 0);
        }
    } else {
        for (; nt; nt--, bs += 32) {
            float x[M][4];
#pragma unroll
            for (int i = 0; i < M; i++) mma_16x8x16(x[i], qa[i], bs[0], c0[i], c1[i]);
#pragma unroll
            for (int i = 0; i < M; i++) bin(x[i], i);
        }
    }
    // counts without the conversion unit: v + 1.5 * 2^23 has round(v) in the
    // low bits of its pattern (the bias's low half is zero); rows g | g + 8 << 16
    unsigned pc[4] = {0u, 0u, 0u, 0u};
    bool b0[M], b1[M], any = false;
#pragma unroll
    for (int i = 0; i < M; i++) {
        const float2 q = __fadd2_rn(sq[i][0], sq[i][1]);
        float2 tot = acc[i][0];
#pragma unroll
        for (int k = 0; k < K; k++) {
            if (k) tot = __fadd2_rn(tot, acc[i][k]);
            const float2 b = __fadd2_rn(acc[i][k], make_float2(12582912.0f, 12582912.0f));
            pc[i * K + k] = __byte_perm(__float_as_uint(b.x), __float_as_uint(b.y), 0x5410);
        }
        b0[i] = tot.x != q.x;
        b1[i] = tot.y != q.y;
        any = any || b0[i] || b1[i];
    }
    // sums over a row's four lanes, item i ending in lane i of the row
    unsigned v;
    if constexpr (NI == 1) {
        v = pc[0] + __shfl_xor_sync(FULL, pc[0], 1);
        v += __shfl_xor_sync(FULL, v, 2);
    } else {
        const bool odd = t & 1, high = t & 2;
        v = (odd ? pc[1] : pc[0]) + __shfl_xor_sync(FULL, odd ? pc[0] : pc[1], 1);
        if constexpr (NI == 2) {
            v += __shfl_xor_sync(FULL, v, 2);
        } else {
            const unsigned u = (odd ? pc[3] : pc[2]) + __shfl_xor_sync(FULL, odd ? pc[2] : pc[3], 1);
            const unsigned give = high ? v : u;
            v = (high ? u : v) + __shfl_xor_sync(FULL, give, 2);
        }
    }
    const int my = M == 1 ? mt[0] : (t / K == 0 ? mt[0] : mt[1]);
    unsigned *const at = P + (kk + t % K) * kPStride + kMT * my + g;
    if (t < NI) {
        atomicAdd(at, v & 0xFFFFu);
        atomicAdd(at + 8, v >> 16);
    }
    if (__any_sync(FULL, any)) {
#pragma unroll
        for (int i = 0; i < M; i++) {
            const unsigned lo = __ballot_sync(FULL, b0[i]), hi = __ballot_sync(FULL, b1[i]);
            if (!(lo | hi)) continue;
            unsigned rows = 0;
#pragma unroll
            for (int r = 0; r < 8; r++)
                rows |= (((lo >> (4 * r)) & 0xFu) ? 1u << r : 0u) | (((hi >> (4 * r)) & 0xFu) ? 256u << r : 0u);
            const unsigned vi = i == 0 ? v : __shfl_sync(FULL, v, (lane & 28) | ((t + K) & 3));
            recount_rows(s, P, rows, mt[i], rs, n, kk, K, vi, lane);
        }
    }
}

// GENERAL: with what labels that interleave in space, counters of 2^27 and more and
// leaves of very different sizes need besides (see TileKernel)
template <int MODE, bool GENERAL>
__global__ void __launch_bounds__(kTileThreads, kTilesPerSm) k_tiles(TileArgs A)
{
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr unsigned FULL = 0xffffffffu;
    TileSmem<MODE> &s = *(TileSmem<MODE> *)smem;
    const int ne = A.ne;
    unsigned *const P = (unsigned *)(smem + sizeof(TileSmem<MODE>));
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int wm = lane & (kMTiles - 1), wr = lane / kMTiles;  // this lane's window: tile, record
    for (int k = tid; k < ne; k += kTileThreads) {
        const double r = A.rsq[k];
        s.R[k] = r;
        s.Rup[k] = __double2float_ru(r);
        s.Rdn[k] = __double2float_rd(r);
    }
    for (int k = tid; k < ne * kPStride; k += kTileThreads) P[k] = 0;
    for (int k = tid; k < (KD_MAX_EDGES + 1) * kMTiles; k += kTileThreads) s.F[k] = 0;
    if (tid < 5) s.stats[tid] = 0;

    while (true) {
        __syncthreads();
        if (tid == 0) s.item = atomicAdd(A.work, 1);
        if (tid < 16) s.keys[tid] = 0;
        if (tid == 0) {
            if constexpr (GENERAL) s.points = s.next = 0;
            s.kmin = ne;
            s.kmax = 0;
            s.kfp = -1;
        }
        __syncthreads();
        const int li = A.g0 + s.item;
        if (li >= A.g1) break;
        {
            const long long eoff = A.off[li - A.g0];
            const int ecnt = (int)(A.off[li - A.g0 + 1] - eoff);
            if (ecnt == 0) continue;
            const int g = A.gmap ? A.gmap[li] : li;
            const int jb = job_of(A.jblk, A.njobs, g);
            const unsigned long long *src = (const unsigned long long *)(A.jobs + jb);
            unsigned long long *dst = (unsigned long long *)&s.job;
            for (int u = tid; u < (int)(sizeof(JobDesc) / 8); u += kTileThreads) dst[u] = src[u];
            // the records' keys and edges
            int points = 0;
            for (int i = tid; i < ecnt; i += kTileThreads) {
                const uint4 r = __ldg(A.rec + eoff + i);
                const unsigned key = ((r.z >> 8) & 0xFF) | (r.w << 8);
                const int k0 = (r.z >> 16) & 0xFF, k1 = k0 + (int)(r.z >> 24);
                atomicOr(&s.keys[key >> 5], 1u << (key & 31));
                atomicMin(&s.kmin, k0);
                atomicMax(&s.kmax, k1);
                if (k1 > k0 && s.R[k1 - 1] < kFp32MaxR) atomicMax(&s.kfp, k1 - 1);
                if constexpr (GENERAL) points += r.z & 0xFF;
            }
            if constexpr (GENERAL) {
                points = __reduce_add_sync(FULL, points);
                if (lane == 0) atomicAdd(&s.points, points);
            }
            __syncthreads();
            const JobDesc &J = s.job;
            const int b = g - A.jblk[jb];
            const int qlen = J.Q.blk_len[b], qs = J.Q.blk_start[b];
            const double *bx = J.Q.blk_box + 6 * (size_t)b;
            const double ox = 0.5 * (bx[0] + bx[3]), oy = 0.5 * (bx[1] + bx[4]), oz = 0.5 * (bx[2] + bx[5]);
            const double hx = 0.5 * (bx[3] - bx[0]), hy = 0.5 * (bx[4] - bx[1]), hz = 0.5 * (bx[5] - bx[2]);
            const float Rq = __double2float_ru(sqrt(hx * hx + hy * hy + hz * hz) * (1.0 + 1e-12));
            float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
            if (tid < qlen) {
                lo[0] = hi[0] = (float)(J.Q.x[qs + tid] - ox);
                lo[1] = hi[1] = (float)(J.Q.y[qs + tid] - oy);
                lo[2] = hi[2] = (float)(J.Q.z[qs + tid] - oz);
            }
#pragma unroll
            for (int d = 0; d < 3; d++) {
#pragma unroll
                for (int o = kMT / 2; o; o >>= 1) {
                    lo[d] = fminf(lo[d], __shfl_xor_sync(FULL, lo[d], o));
                    hi[d] = fmaxf(hi[d], __shfl_xor_sync(FULL, hi[d], o));
                }
                if ((tid & (kMT - 1)) == 0) {
                    s.qc[tid / kMT][d] = 0.5f * (lo[d] + hi[d]);
                    s.qh[tid / kMT][d] = 0.5f * (hi[d] - lo[d]);
                }
            }
            const float far = s.kfp >= 0 ? sqrtf(s.Rup[s.kfp]) * 1.0001f : 0.0f;
            float hT = __double2float_ru(J.hT), hSmall = 0.0f;
            if constexpr (GENERAL) {
                // The error band allows for the rounding of a point relative to
                // its leaf's centre, so it grows with the leaf, and beside leaves
                // that span the catalog (around a far point, between tight groups)
                // it would cover every pair.  So leaves of no more than a few
                // times what this block and its edges span have a band of their
                // own, and leaves with which the scale could not resolve the block
                // take the exact path.
                hT = fminf(hT, 16384.0f * (Rq + sqrtf(s.Rup[min(s.kmin, ne - 1)])) + 4.0f * far);
                hSmall = fminf(hT, 4.0f * (far + Rq));
            }
            // every coordinate and edge root of a record with pairs below edge
            // kfp stays below Bm: scaled values below 240, squares below 65504
            float S = 0.0f;
            const float Bm = far + 2.1f * hT + 4.0f * Rq;
            if (Bm > 0.0f && Bm < (float)kFp32Span) {
                int ex;
                frexpf(Bm, &ex);  // Bm in [2^(ex-1), 2^ex)
                S = ldexpf(1.0f, max(-60, min(60, 7 - ex)));
            }
            if (tid == 0) {
                s.o[0] = ox;
                s.o[1] = oy;
                s.o[2] = oz;
                s.eoff = eoff;
                s.ecnt = ecnt;
                // records a warp takes at a time: a few, where the block has few
                s.chunk = ecnt >= 1024 ? 32 : (ecnt >= 512 ? 16 : (ecnt >= 128 ? 8 : 4));
                if constexpr (GENERAL) s.bqf = J.Q.blk_qf[b];
                s.qs = qs;
                s.qlen = qlen;
                s.Rq = Rq;
                s.hT = hT;
                if constexpr (GENERAL) {
                    s.hSmall = hSmall;
                    s.hcap = J.hT <= (double)hT ? INFINITY : hT;  // (J.hT may be NaN)
                }
                s.S = S;
            }
            __syncthreads();
            if constexpr (GENERAL)
                if (s.bqf >= 0 ? (float)s.points <= kDirectRunOne * (float)ecnt
                               : (float)s.points <= kDirectRun * (float)ecnt &&
                                     (long long)J.Fqe * J.Fte >= kDirectCells) {
                    if (s.bqf >= 0) count_direct<true>(s, A.rec + eoff, ne, tid);
                    else count_direct<false>(s, A.rec + eoff, ne, tid);
                    continue;
                }
            if (MODE == KD_MODE_MIXED && S > 0.0f)
                set_scale<GENERAL>(s, GENERAL && hSmall < hT ? (float2 *)(P + ne * kPStride) : nullptr, ne, tid);
        }
        // ---- one flush key after the other (tree field | 256 for the
        // once-counted part of a symmetric job)
        for (int key = 0; key < 512; key++) {
            const unsigned kw = s.keys[key >> 5] >> (key & 31);
            if (!kw) {
                key |= 31;
                continue;
            }
            key += __ffs(kw) - 1;
            __syncthreads();  // the last key's counters are clear
            if (tid == 0) s.next = 0;
            __syncthreads();
            while (true) {
                int c0 = 0;
                if (lane == 0) c0 = atomicAdd(&s.next, s.chunk);
                c0 = __shfl_sync(FULL, c0, 0);
                if (c0 >= s.ecnt) break;
                const uint4 *const crec = A.rec + s.eoff + c0;
                unsigned mine;
                {
                    uint2 r = make_uint2(0, 0);
                    const bool in = lane < s.chunk && c0 + lane < s.ecnt;
                    if (in) r = __ldg(reinterpret_cast<const uint2 *>(crec + lane) + 1);
                    mine = __ballot_sync(FULL, in && (((r.x >> 8) & 0xFF) | (r.y << 8)) == (unsigned)key);
                }
                while (mine) {
                    // ---- the next four records: lane (wm, wr) has record wr
                    const unsigned m1 = mine & (mine - 1), m2 = m1 & (m1 - 1), m3 = m2 & (m2 - 1);
                    const unsigned sel = wr == 0 ? mine : (wr == 1 ? m1 : (wr == 2 ? m2 : m3));
                    const bool have = sel != 0;
                    const int nr = min(kGroup, __popc(mine));
                    mine = m3 & (m3 - 1);
                    const int from = have ? __ffs(sel) - 1 : 0;
                    const uint4 rec = __ldg(crec + from);
                    const int r_rs = (int)rec.x;
                    const unsigned r_z = have ? rec.z : 0u;
                    const int rl = r_z & 0xFF, rk0 = (r_z >> 16) & 0xFF, rK = r_z >> 24;
                    // ---- windows: edges [k0, k1) may separate pairs of query
                    // tile wm and the record; every pair lies below the edges
                    // from k1 on
                    int k0 = rk0, k1 = rk0 + rK;
                    bool ok = have && rK != 0, fast_ok = false, small = false;  // windows, FP32 distances, band
                    float dx, dy, dz;
                    {
                        const double2 *geo = reinterpret_cast<const double2 *>(s.job.leaf + rec.y);
                        const double2 ga = __ldg(geo), gb = __ldg(geo + 1);
                        const float hx = __int_as_float(__double2loint(gb.y)),
                                    hy = __int_as_float(__double2hiint(gb.y)),
                                    hz = __ldg(reinterpret_cast<const float *>(geo + 2));
                        dx = (float)(ga.x - s.o[0]);
                        dy = (float)(ga.y - s.o[1]);
                        dz = (float)(gb.x - s.o[2]);
                        // B >= |t'| of every point of a leaf of the FP32 path and
                        // sqrt of every edge of the record
                        const float B = sqrtf(dx * dx + dy * dy + dz * dz) * 1.0001f + s.hT + 2.0f * s.Rq;
                        ok = ok && B < (float)kFp32Span && s.R[k1 - 1] < kFp32MaxR;
                        if constexpr (GENERAL) {  // (a window needs no scale)
                            const float h = hx + hy + hz;
                            fast_ok = ok && s.S > 0.0f && B * s.S <= 240.0f && h <= s.hcap;
                            small = h <= s.hSmall && s.hSmall < s.hT;
                        } else {
                            ok = ok && (MODE == KD_MODE_FP64 || (s.S > 0.0f && B * s.S <= 240.0f));
                        }
                        if (ok) {
                            // rounding of the staged coordinates and of the tile box
                            const float mg = 4.8e-7f * (fabsf(dx) + fabsf(dy) + fabsf(dz) + hx + hy + hz +
                                                        2.0f * (s.Rq + s.hT));
                            const float ax = fabsf(dx - s.qc[wm][0]), ay = fabsf(dy - s.qc[wm][1]),
                                        az = fabsf(dz - s.qc[wm][2]);
                            const float ex = hx + s.qh[wm][0] + mg, ey = hy + s.qh[wm][1] + mg,
                                        ez = hz + s.qh[wm][2] + mg;
                            const float gx = fmaxf(ax - ex, 0.0f), gy = fmaxf(ay - ey, 0.0f),
                                        gz = fmaxf(az - ez, 0.0f);
                            const float sx = ax + ex, sy = ay + ey, sz = az + ez;
                            // (squares below FLT_MIN are cut to multiples of
                            // 2^-149: a few of those steps, within 1e-40)
                            const float lo2 = fmaf(gx * gx + gy * gy + gz * gz, 1.0f - 4e-6f, -1e-40f);
                            const float hi2 = fmaf(sx * sx + sy * sy + sz * sz, 1.0f + 4e-6f, 1e-40f);
                            int below = 0, upto = 0;  // edges below / not above the pairs
                            for (int k = rk0; k < rk0 + rK; k++) {
                                below += s.Rup[k] <= lo2;
                                upto += s.Rdn[k] <= hi2;
                            }
                            k0 = rk0 + below;
                            k1 = rk0 + max(below, upto);
                        }
                    }
                    const int mval = max(0, min(kMT, s.qlen - kMT * wm));  // queries of tile wm
                    const int K = have && mval ? k1 - k0 : 0;
                    const unsigned win = (unsigned)k0 | ((unsigned)K << 8) | (GENERAL && small ? 1u << 16 : 0u);
                    const unsigned actm = __ballot_sync(FULL, K != 0), okm = __ballot_sync(FULL, GENERAL ? fast_ok : ok);
                    if (have && mval) atomicAdd(&s.F[k1 * kMTiles + wm], (unsigned)rl);
                    {
                        const unsigned q = K ? (unsigned)(mval * rl) : 0u;
                        const unsigned np = __reduce_add_sync(FULL, q), nk = __reduce_add_sync(FULL, q * (unsigned)K),
                                       nw = __reduce_add_sync(FULL, K > 4 ? q : 0u);
                        if (lane < 4) {
                            const unsigned v = lane == 0 ? np : (lane == 1 ? nw : (lane == 2 ? nk : __popc(actm)));
                            atomicAdd(&s.stats[lane == 0 ? 0 : lane + 1], (unsigned long long)v);
                        }
                    }
                    // ---- record by record
                    float4 npt[2];
                    double px[2], py[2], pz[2];
                    auto load_points = [&](int r) {
                        const int rs = __shfl_sync(FULL, r_rs, r * kMTiles);
                        const int n = __shfl_sync(FULL, rl, r * kMTiles);
#pragma unroll
                        for (int h = 0; h < 2; h++)
                            if (lane + 32 * h < n) {
                                const int j = rs + lane + 32 * h;
                                if constexpr (MODE == KD_MODE_MIXED) {
                                    npt[h] = __ldg(s.job.t4 + j);
                                } else {
                                    px[h] = __ldg(s.job.tx + j);
                                    py[h] = __ldg(s.job.ty + j);
                                    pz[h] = __ldg(s.job.tz + j);
                                }
                            }
                    };
                    load_points(0);
                    for (int r = 0; r < nr; r++) {
                        const int src = r * kMTiles;
                        const int n = __shfl_sync(FULL, rl, src), rs = __shfl_sync(FULL, r_rs, src);
                        unsigned act = (actm >> src) & 0xFFu;
                        if constexpr (MODE == KD_MODE_MIXED) {
                            const bool fast = (okm >> src) & 1;
                            const float ref = s.edge[(__shfl_sync(FULL, r_z, src) >> 16) & 0xFF].x, S = s.S;
                            const float Dx = __shfl_sync(FULL, dx, src), Dy = __shfl_sync(FULL, dy, src),
                                        Dz = __shfl_sync(FULL, dz, src);
                            // ---- stage the run: lane (g, t) of step j reads
                            // word t of point 8 j + g
                            if (act && fast) {
#pragma unroll
                                for (int h = 0; h < 2; h++) {
                                    const int j = lane + 32 * h;
                                    if (j < ((n + kNT - 1) & ~(kNT - 1))) {
                                        // t' = t_r + (c - o); -0.5 * (-2 t_r) is exact
                                        const float x = fmaf(-0.5f, npt[h].x, Dx) * S,
                                                    y = fmaf(-0.5f, npt[h].y, Dy) * S,
                                                    zz = fmaf(-0.5f, npt[h].z, Dz) * S;
                                        const float N = fmaf(zz, zz, fmaf(y, y, fmaf(x, x, -ref)));
                                        uint4 v = make_uint4(split_halves(x), split_halves(y),
                                                             split_halves(zz), split_halves(N));
                                        // columns without a point lie above every edge
                                        if (j >= n) v = make_uint4(0u, 0u, 0u, 0x7BFF7BFFu);
                                        *reinterpret_cast<uint4 *>(s.bs[w] + 4 * j) = v;
                                    }
                                }
                            }
                            if (r + 1 < nr) load_points(r + 1);
                            __syncwarp();
                            const int nt = (n + kNT - 1) / kNT;
                            const uint32_t *const bs = s.bs[w] + lane;
                            while (act) {
                                int mt[2];
                                mt[0] = __ffs(act) - 1;
                                act &= act - 1;
                                mt[1] = act ? __ffs(act) - 1 : mt[0];
                                const unsigned wv = __shfl_sync(FULL, win, src + mt[0]),
                                               wv2 = __shfl_sync(FULL, win, src + mt[1]);
                                int kk = wv & 0xFF, left = GENERAL ? (wv >> 8) & 0xFF : wv >> 8;
                                const float2 *const edges = GENERAL && wv >> 16 ? (const float2 *)(P + ne * kPStride) : s.edge;
                                if (fast) {
                                    // two tiles with one window go together
                                    if (left == 1 && act && wv2 == wv) {
                                        act &= act - 1;
                                        tile_pass<1, 2>(s, P, mt, kk, edges, nt, ref, rs, n, lane, bs);
                                        continue;
                                    }
                                    for (; left > 4; left -= 4, kk += 4)
                                        tile_pass<4, 1>(s, P, mt, kk, edges, nt, ref, rs, n, lane, bs);
                                    switch (left) {
                                    case 1: tile_pass<1, 1>(s, P, mt, kk, edges, nt, ref, rs, n, lane, bs); break;
                                    case 2: tile_pass<2, 1>(s, P, mt, kk, edges, nt, ref, rs, n, lane, bs); break;
                                    case 3: tile_pass<3, 1>(s, P, mt, kk, edges, nt, ref, rs, n, lane, bs); break;
                                    default: tile_pass<4, 1>(s, P, mt, kk, edges, nt, ref, rs, n, lane, bs); break;
                                    }
                                } else {  // out of FP32 range: every row exactly
                                    for (; left > 0; left -= 4, kk += 4)
                                        recount_rows(s, P, 0xFFFFu, mt[0], rs, n, kk, min(4, left), 0u, lane);
                                }
                            }
                        } else {
                            if (act) {
#pragma unroll
                                for (int h = 0; h < 2; h++) {
                                    const int j = lane + 32 * h;
                                    if (j < ((n + 3) & ~3)) {
                                        s.pt[w][0][j] = j < n ? px[h] : NAN;
                                        s.pt[w][1][j] = j < n ? py[h] : NAN;
                                        s.pt[w][2][j] = j < n ? pz[h] : NAN;
                                    }
                                }
                            }
                            if (r + 1 < nr) load_points(r + 1);
                            __syncwarp();
                            const double2 *X = reinterpret_cast<const double2 *>(s.pt[w][0]),
                                          *Y = reinterpret_cast<const double2 *>(s.pt[w][1]),
                                          *Z = reinterpret_cast<const double2 *>(s.pt[w][2]);
                            // a query tile at a time, each half of the warp
                            // with half of the points (two and two)
                            const int np = (n + 3) / 4, at = (lane >> 4) * np;
                            for (; act; act &= act - 1) {
                                const int m = __ffs(act) - 1, q = kMT * m + (lane & (kMT - 1));
                                const unsigned wv = __shfl_sync(FULL, win, src + m);
                                const bool v = q < s.qlen;
                                const double qx = v ? s.job.Q.x[s.qs + q] : s.o[0],
                                             qy = v ? s.job.Q.y[s.qs + q] : s.o[1],
                                             qz = v ? s.job.Q.z[s.qs + q] : s.o[2];
                                for (int kk = wv & 0xFF, left = GENERAL ? (wv >> 8) & 0xFF : wv >> 8; left > 0; left -= kFpEdges, kk += kFpEdges) {
                                    unsigned cnt[kFpEdges] = {};
                                    switch (left) {
                                    case 1: fp64_run<1>(X + at, Y + at, Z + at, np, qx, qy, qz, s.R + kk, 1, cnt); break;
                                    case 2: fp64_run<2>(X + at, Y + at, Z + at, np, qx, qy, qz, s.R + kk, 2, cnt); break;
                                    case 3: fp64_run<3>(X + at, Y + at, Z + at, np, qx, qy, qz, s.R + kk, 3, cnt); break;
                                    case 4: fp64_run<4>(X + at, Y + at, Z + at, np, qx, qy, qz, s.R + kk, 4, cnt); break;
                                    default: fp64_run<kFpEdges>(X + at, Y + at, Z + at, np, qx, qy, qz, s.R + kk, left, cnt); break;
                                    }
#pragma unroll
                                    for (int k = 0; k < kFpEdges; k++)
                                        if (k < left) {
                                            const unsigned c = cnt[k] + __shfl_xor_sync(FULL, cnt[k], kMT);
                                            if (lane < kMT) atomicAdd(&P[(kk + k) * kPStride + q], c);
                                        }
                                }
                            }
                        }
                        __syncwarp();
                    }
                }
            }
            __syncthreads();
            // ---- the key's counters to the global histogram: thread = query
            {
                const JobDesc &J = s.job;
                unsigned long long *const Hd = (key >> 8) ? J.H2 : J.H;
                const int tf = key & 0xFF, kmin = s.kmin, kmax = s.kmax;
                const int qf = tid < s.qlen ? J.Q.qf[s.qs + tid] : -1;
                unsigned run = 0, before = 0, vm = __ballot_sync(FULL, qf >= 0);
                unsigned alone = 0;  // the bits of its counters that a query adds by itself
                if constexpr (GENERAL) {
                    // Up to KD_FEW_FIELDS own fields are summed over the warp, a
                    // round each; with more, every query adds its own counts.
                    // 400k points, symmetric, 21 edges, labels at random: 4
                    // fields 2.9 ms by rounds and 4.7 by query, 5 3.45 and 3.45,
                    // 16 10.2 and 8.2.
                    const unsigned peers = __match_any_sync(FULL, qf);
                    const bool many = __popc(__ballot_sync(FULL, qf >= 0 && lane == __ffs(peers) - 1)) > KD_FEW_FIELDS;
                    if (qf >= 0) alone = many ? FULL : ~(kWideCount - 1);
                    if (many) vm = 0;
                }
                for (int e = kmin; e < min(kmax + 1, ne); e++) {
                    run += s.F[e * kMTiles + tid / kMT];
                    const unsigned cum = run + P[e * kPStride + tid];
                    P[e * kPStride + tid] = 0;
                    unsigned v = cum - before;
                    before = cum;
                    if constexpr (GENERAL) {
                        if (v & alone)
                            atomicAdd(&Hd[((size_t)e * J.Fqe + qf) * J.Fte + tf], (unsigned long long)(v & alone));
                        v &= ~alone;
                    }
                    unsigned rem = vm;
                    while (rem) {  // one round per distinct own field of the warp
                        const int from = __ffs(rem) - 1;
                        const int f = __shfl_sync(FULL, qf, from);
                        const bool same = qf == f;
                        const unsigned sum = __reduce_add_sync(FULL, same ? v : 0u);
                        if (lane == from && sum)
                            atomicAdd(&Hd[((size_t)e * J.Fqe + f) * J.Fte + tf], (unsigned long long)sum);
                        rem &= ~__ballot_sync(FULL, same);
                    }
                }
                __syncthreads();
                for (int i = kmin * kMTiles + tid; i < (kmax + 1) * kMTiles; i += kTileThreads) s.F[i] = 0;
            }
        }
    }
    // (the loop ends behind a barrier)
    if (tid == 0) {
        if (s.stats[0]) atomicAdd(&A.stats[0], s.stats[0]);
        if (s.stats[1]) atomicAdd(&A.stats[1], s.stats[1]);
        if (s.stats[2]) atomicAdd(&A.stats[3], s.stats[2]);
        if (s.stats[3]) atomicAdd(&A.stats[4], s.stats[3]);
        if (s.stats[4]) atomicAdd(&A.stats[5], s.stats[4]);
    }
}

static size_t tile_smem(int ne, int mode, bool general)
{
    const size_t fixed = mode == KD_MODE_MIXED ? sizeof(TileSmem<KD_MODE_MIXED>)
                                               : sizeof(TileSmem<KD_MODE_FP64>);
    static_assert(kPStride % 2 == 0 && sizeof(TileSmem<KD_MODE_MIXED>) % 8 == 0, "the table behind P is aligned");
    return fixed + sizeof(unsigned) * (size_t)ne * kPStride + (general ? sizeof(float2) * (size_t)ne : 0);
}

// The kernel for these counts.  Its general variant costs all others 2 to 3% (the
// code: 3M uniform points in 21 edges 5.66 and 5.80 ms), so it is taken only where
// labels interleave (a tree's runs are short, or a query warp's own fields many),
// where a counter could reach 2^27, or where the leaves' sizes differ so much that
// one error band is too wide.  In the last case: 1M points, 20 groups 1e-6 wide,
// radii 1e-8 and 1e-7, 3.13 -> 0.86 ms; one point at 1e12 3.78 -> 2.03, at infinity
// 3.13 -> 1.27; twelve decades of |x| 29 -> 7.3.
struct TileKernel {
    void (*run)(TileArgs);
    size_t smem;
    int ctas;  // per SM

    TileKernel(const kd_catalog *const *tcs, const kd_catalog *const *qcs, int njobs, int ne, int mode)
    {
        bool general = false;
        for (int j = 0; j < njobs; j++)
            general = general || tcs[j]->short_runs || qcs[j]->many_fields || tcs[j]->n_raw >= (int)kWideCount ||
                      (mode == KD_MODE_MIXED && tcs[j]->uneven_leaves);
        run = mode == KD_MODE_MIXED ? (general ? k_tiles<KD_MODE_MIXED, true> : k_tiles<KD_MODE_MIXED, false>)
                                    : (general ? k_tiles<KD_MODE_FP64, true> : k_tiles<KD_MODE_FP64, false>);
        smem = tile_smem(ne, mode, general);
        check(cudaFuncSetAttribute(run, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
              "smem attribute");
        check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, run, kTileThreads, smem), "occupancy");
        ctas = std::max(ctas, 1);
    }
};

struct Events {
    cudaEvent_t e[8];
    Events()
    {
        for (auto &x : e) check(cudaEventCreate(&x), "cudaEventCreate");
    }
    ~Events()
    {
        for (auto &x : e) cudaEventDestroy(x);
    }
};

static float elapsed(cudaEvent_t a, cudaEvent_t b)
{
    float ms = 0;
    cudaEventElapsedTime(&ms, a, b);
    return ms;
}

// the traversal and tile views of one (tree, query tree) job
static JobDesc job_desc(const kd_catalog *tc, const kd_catalog *qc, unsigned long long *H)
{
    JobDesc d;
    memset(&d, 0, sizeof d);
    d.T.box = tc->d_box;
    d.T.count = tc->d_ncount;
    d.T.tf = tc->d_ntf;
    d.T.leaf_run = tc->d_leaf_run;
    d.T.leaf_pos = tc->d_leaf_pos;
    d.T.run_start = tc->d_run_start;
    d.T.run_len = tc->d_run_len;
    d.T.run_tf = tc->d_run_tf;
    d.T.D = tc->depth;
    d.T.nleaves = tc->nleaves;
    d.Q.x = qc->d_x;
    d.Q.y = qc->d_y;
    d.Q.z = qc->d_z;
    d.Q.qf = qc->d_qf;
    d.Q.blk_start = qc->d_blk_start;
    d.Q.blk_len = qc->d_blk_len;
    d.Q.blk_qf = qc->d_blk_qf;
    d.Q.blk_box = qc->d_blk_box;
    d.tx = tc->d_x;
    d.ty = tc->d_y;
    d.tz = tc->d_z;
    d.t4 = (const float4 *)tc->d_t4;
    d.leaf = tc->d_leaf;
    d.hT = tc->leaf_hdiag * (1.0 + 1e-12);
    d.H = H;
    d.H2 = nullptr;
    d.Fqe = qc->max_qf + 1;
    d.Fte = tc->max_tf + 1;
    d.sym = 0;
    return d;
}

// An autocorrelation count (one catalog on both sides) whose points all keep
// their own field on the tree side can count each unordered pair once: the
// distance of (q, t) and of (t, q) is the same double (t - q and q - t differ
// only in sign, so every square, product and FMA is identical), and the pair's
// second orientation lands in the transposed field cell.
static bool symmetric_job(const kd_catalog *tc, const kd_catalog *qc)
{
    return tc == qc && !tc->fields_split && tc->max_qf == tc->max_tf;
}

static size_t hist_size(const kd_catalog *tc, const kd_catalog *qc, int ne)
{
    return (size_t)(ne + 1) * (size_t)(qc->max_qf + 1) * (size_t)(tc->max_tf + 1);
}

// Every job's query blocks (this shard's share of them) in one traversal and
// one persistent tile launch per record batch, over a shared work counter.
static void count_batch_impl(const kd_catalog *const *tcs, const kd_catalog *const *qcs,
                             int njobs, const double *h_rsq, int ne, int mode, int shard,
                             int nshards, long long *const *hists, kd_count_stats *stats)
{
    const int device = tcs[0]->device;
    for (int j = 0; j < njobs; j++)
        if (tcs[j]->device != device || qcs[j]->device != device)
            raise(KD_EINVAL, "the catalogs of a count are on different devices");
    check(cudaSetDevice(device), "cudaSetDevice");
    init_device();
    Stream st;
    cudaStream_t s = st.s;
    Pool pool(s, true);
    Events ev;
    int launches = 0, tile_launches = 0;

    // job table, histogram offsets, global block numbering
    std::vector<size_t> hoff(njobs + 1, 0);
    std::vector<int> hblk(njobs + 1, 0);
    std::vector<char> sym(njobs);
    for (int j = 0; j < njobs; j++) {
        sym[j] = symmetric_job(tcs[j], qcs[j]);
        // a symmetric job has its once-counted histogram H2 right after H
        hoff[j + 1] = hoff[j] + (sym[j] ? 2 : 1) * hist_size(tcs[j], qcs[j], ne);
        if ((long long)hblk[j] + qcs[j]->nblocks > INT_MAX) raise(KD_EINVAL, "too many query blocks in one count");
        hblk[j + 1] = hblk[j] + qcs[j]->nblocks;
    }
    const size_t hsz = hoff[njobs];
    unsigned long long *H = pool.alloc<unsigned long long>(hsz);
    std::vector<JobDesc> hj(njobs);
    for (int j = 0; j < njobs; j++) {
        hj[j] = job_desc(tcs[j], qcs[j], H + hoff[j]);
        if (sym[j]) {
            hj[j].sym = 1;
            hj[j].H2 = H + hoff[j] + hist_size(tcs[j], qcs[j], ne);
        }
    }
    JobDesc *jobs = pool.alloc<JobDesc>(njobs);
    int *jblk = pool.alloc<int>(njobs + 1);
    unsigned long long *dstats = pool.alloc<unsigned long long>(8);
    int *err = pool.alloc<int>(1);
    int *work = pool.alloc<int>(1);
    double *rsq = pool.alloc<double>(std::max(ne, 1));
    check(cudaEventRecord(ev.e[0], s), "event");
    check(cudaMemsetAsync(H, 0, sizeof(unsigned long long) * hsz, s), "memset");
    check(cudaMemsetAsync(dstats, 0, sizeof(unsigned long long) * 8, s), "memset");
    check(cudaMemsetAsync(err, 0, sizeof(int), s), "memset");
    check(cudaMemcpyAsync(rsq, h_rsq, sizeof(double) * ne, cudaMemcpyHostToDevice, s), "H2D");
    check(cudaMemcpyAsync(jobs, hj.data(), sizeof(JobDesc) * njobs, cudaMemcpyHostToDevice, s), "H2D");
    check(cudaMemcpyAsync(jblk, hblk.data(), sizeof(int) * (njobs + 1), cudaMemcpyHostToDevice, s),
          "H2D");

    // this shard's global blocks
    const int NB = hblk[njobs];
    // this shard's blocks: interleaved chunks of kShardChunk global blocks
    // (chunk c belongs to shard c mod nshards), so that every shard gets an
    // even mix of early and late blocks (a symmetric job's block only counts
    // tree points after its own, so early blocks carry more work)
    std::vector<int> gl;
    if (nshards > 1)
        for (int c = shard * kShardChunk; c < NB; c += nshards * kShardChunk)
            for (int g = c; g < std::min(NB, c + kShardChunk); g++) gl.push_back(g);
    const int G0 = 0;
    const int G1 = nshards > 1 ? (int)gl.size() : NB;
    const int nb = G1 - G0;
    int *gmap = nullptr;
    if (nshards > 1 && nb > 0) {
        gmap = pool.alloc<int>(nb);
        check(cudaMemcpyAsync(gmap, gl.data(), sizeof(int) * (size_t)nb, cudaMemcpyHostToDevice, s),
              "H2D");
    }
    int *cnt = pool.alloc<int>(std::max(nb, 1));
    TravOut to;
    memset(&to, 0, sizeof to);
    to.gmap = gmap;
    to.count = cnt;
    to.accepted = dstats + 2;
    to.err = err;
    if (nb > 0) {
        k_traverse<false><<<blocks_for(nb, kTravWarps), 32 * kTravWarps, 0, s>>>(jobs, jblk, njobs,
                                                                                  rsq, ne, G0, G1, to);
        launches++;
    }
    KD_LAUNCH_CHECK("k_traverse(count)");
    std::vector<int> hcnt(std::max(nb, 1));
    check(cudaMemcpyAsync(hcnt.data(), cnt, sizeof(int) * (size_t)nb, cudaMemcpyDeviceToHost, s),
          "D2H");
    int herr = 0;
    check(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, s), "D2H");
    st.sync();
    if (herr) raise(herr, "node-pair traversal exceeded its stack");

    // batches of global blocks whose tile records fit the buffer: up to 2^30
    // records (16 GiB) or a quarter of the free memory, so that on a B200 a
    // full DD + DR + RR batch of 20M-point catalogs runs as one launch
    long long total = 0, maxblk = 0;
    for (int i = 0; i < nb; i++) {
        total += hcnt[i];
        maxblk = std::max<long long>(maxblk, hcnt[i]);
    }
    // (asked for only where it can matter: not below 2^20 records, nor where
    // the record pool's idle memory holds them all.  The driver answers in
    // milliseconds, at times tens of them, on a machine whose other GPUs keep
    // it busy: a count of 4k / 80k points took 0.7 ms, and now and then 16 or 89)
    // free memory: the driver's, plus what the record pool and the default
    // pool hold cached (reusable without asking the driver)
    const cudaMemPool_t rpool = side_pool(kPoolRecords);
    long long cap = 1LL << 30;
    uint4 *rec = nullptr;
    // KD_TILE_RECORD_CAP (records, > 0) lowers the batch size: it exercises
    // the multi-batch path on small counts
    const char *const env = getenv("KD_TILE_RECORD_CAP");
    const long long set = env ? atoll(env) : 0;
    if (set <= 0 && total > 1 << 20 && total <= cap && (size_t)total * sizeof(uint4) <= pool_idle_bytes(rpool))
        rec = pool.try_alloc_from<uint4>(rpool, total);
    if (rec) {
        cap = total;
    } else {
        if (total > 1 << 20) {
            size_t freeb = 0, totb = 0;
            cudaMemGetInfo(&freeb, &totb);
            freeb += pool_idle_bytes(rpool);
            cudaMemPool_t dpool = nullptr;
            if (cudaDeviceGetDefaultMemPool(&dpool, device) == cudaSuccess && dpool != rpool)
                freeb += pool_idle_bytes(dpool);
            cudaGetLastError();
            cap = std::max<long long>(1 << 20, std::min<long long>(cap, (long long)(freeb / 4 / sizeof(uint4))));
        }
        if (set > 0) cap = set;
        // every batch holds at least one whole block: the buffer must take the
        // largest block's records (a failed allocation is reported, not overrun)
        cap = std::max(cap, maxblk);
        cap = std::min<long long>(cap, std::max<long long>(total, 1));
        rec = pool.alloc_from<uint4>(rpool, cap);
    }
    long long *off = pool.alloc<long long>(nb + 1);
    std::vector<long long> hoffs(nb + 1);

    const TileKernel kern(tcs, qcs, njobs, ne, mode);
    int nsm = 148;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);

    float ms_trav = 0, ms_tiles = 0;
    int b0 = 0;  // shard-relative
    while (b0 < nb) {
        long long acc = 0;
        int b1 = b0;
        hoffs[0] = 0;
        while (b1 < nb && (b1 == b0 || acc + hcnt[b1] <= cap)) {
            acc += hcnt[b1];
            b1++;
            hoffs[b1 - b0] = acc;
        }
        check(cudaMemcpyAsync(off, hoffs.data(), sizeof(long long) * (size_t)(b1 - b0 + 1),
                              cudaMemcpyHostToDevice, s), "H2D");
        TravOut tf = to;
        tf.count = nullptr;
        tf.off = off;
        tf.rec = rec;
        check(cudaEventRecord(ev.e[1], s), "event");
        k_traverse<true><<<blocks_for(b1 - b0, kTravWarps), 32 * kTravWarps, 0, s>>>(
            jobs, jblk, njobs, rsq, ne, G0 + b0, G0 + b1, tf);
        launches++;
        KD_LAUNCH_CHECK("k_traverse(fill)");
        check(cudaEventRecord(ev.e[2], s), "event");
        TileArgs ta;
        ta.jobs = jobs;
        ta.jblk = jblk;
        ta.njobs = njobs;
        ta.rsq = rsq;
        ta.ne = ne;
        ta.g0 = G0 + b0;
        ta.g1 = G0 + b1;
        ta.gmap = gmap;
        ta.off = off;
        ta.rec = rec;
        ta.work = work;
        ta.stats = dstats;
        check(cudaMemsetAsync(work, 0, sizeof(int), s), "memset");
        const int grid = (int)std::min<long long>(b1 - b0, (long long)nsm * kern.ctas);
        kern.run<<<grid, kTileThreads, kern.smem, s>>>(ta);
        launches++;
        tile_launches++;
        KD_LAUNCH_CHECK("k_tiles");
        check(cudaEventRecord(ev.e[3], s), "event");
        st.sync();
        ms_trav += elapsed(ev.e[1], ev.e[2]);
        ms_tiles += elapsed(ev.e[2], ev.e[3]);
        b0 = b1;
    }
    check(cudaEventRecord(ev.e[4], s), "event");
    std::vector<unsigned long long> hh(std::max<size_t>(hsz, 1));
    unsigned long long hs[8];
    check(cudaMemcpyAsync(hh.data(), H, sizeof(unsigned long long) * hsz, cudaMemcpyDeviceToHost, s),
          "D2H");
    check(cudaMemcpyAsync(hs, dstats, sizeof hs, cudaMemcpyDeviceToHost, s), "D2H");
    check(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, s), "D2H");
    st.sync();
    if (herr) raise(herr, "node-pair traversal exceeded its stack");
    for (int j = 0; j < njobs; j++) {
        const size_t n1 = hist_size(tcs[j], qcs[j], ne);
        const unsigned long long *h1 = hh.data() + hoff[j];
        for (size_t i = 0; i < n1; i++) hists[j][i] = (long long)h1[i];
        if (sym[j]) {  // both orientations of the once-counted pairs
            const unsigned long long *h2 = h1 + n1;
            const size_t F = (size_t)hj[j].Fqe;
            for (int e = 0; e <= ne; e++)
                for (size_t a = 0; a < F; a++)
                    for (size_t c = 0; c < F; c++)
                        hists[j][((size_t)e * F + a) * F + c] +=
                            (long long)(h2[((size_t)e * F + a) * F + c] +
                                        h2[((size_t)e * F + c) * F + a]);
        }
    }
    if (stats) {
        stats->pairs_tested = (long long)hs[0];
        stats->pairs_rechecked = (long long)hs[1];
        stats->pairs_accepted = (long long)hs[2];
        stats->pairs_one_bin_multifield = (long long)hs[6];
        stats->pairs_wide = (long long)hs[3];
        stats->edge_pairs = (long long)hs[4];
        stats->warp_tiles = (long long)hs[5];
        stats->entries = total;
        stats->ms_traverse = ms_trav;
        stats->ms_tiles = ms_tiles;
        stats->ms_total = elapsed(ev.e[0], ev.e[4]);
        stats->tile_launches = tile_launches;
        stats->launches = launches;
    }
}

// ------------------------------------------------------------------------
// Count without any allocation (kd_count_radii_static).
//
// For callers that cannot allocate device memory at count time: every
// per-call buffer of a count (bin histogram, tile records, block offsets,
// scan workspace, counters, the final per-radius matrices) is carved out of
// one file-scope device array.  Every GPU that loads the library holds this
// array until the process exits.  All calls on a device share it and it keeps
// the previous call's contents, so everything that must start at zero is
// cleared at the start of a call, and two calls that overlap on the same GPU
// race.  Jobs whose tile records do not fit are counted in as many batches as
// it takes.

constexpr size_t kStaticScratchBytes = size_t(32) << 20;
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_static_mu;
void *g_static_ptr[kMaxDevices];  // device address of g_static_scratch, per device
}  // namespace

// Device address of the scratch array on the current device.  Host code
// cannot use the symbol itself (on the host it names a host-side stand-in),
// so the address is looked up once per device with that device current and
// kept for the life of the process (a device reset through this library's
// runtime would invalidate it; the entry point's contract excludes that).
static unsigned char *static_scratch(int device)
{
    if (device < 0 || device >= kMaxDevices) raise(KD_ENODEV, "device index out of range");
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (!g_static_ptr[device]) {
        void *ptr = nullptr;
        check(cudaGetSymbolAddress(&ptr, g_static_scratch), "cudaGetSymbolAddress(scratch)");
        g_static_ptr[device] = ptr;
    }
    return (unsigned char *)g_static_ptr[device];
}

// last block b1 > b0 such that blocks [b0, b1) have at most cap tile records
// (at least one block); records of block b0 alone above cap: b1 = -1
__global__ void k_static_batch(const long long *off, int nb, int b0, long long cap, int *b1_out,
                               long long *rel, int rel_cap)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        int lo = b0 + 1, hi = nb;
        if (off[b0 + 1] - off[b0] > cap) {
            *b1_out = -1;
            return;
        }
        while (lo < hi) {  // largest b1 in [b0+1, nb] with off[b1] - off[b0] <= cap
            const int mid = (lo + hi + 1) / 2;
            if (off[mid] - off[b0] <= cap) lo = mid;
            else hi = mid - 1;
        }
        *b1_out = min(lo, b0 + rel_cap - 1);
    }
    __syncthreads();
    const int b1 = *b1_out;
    for (int i = threadIdx.x; b1 > b0 && i <= b1 - b0; i += blockDim.x)
        rel[i] = off[b0 + i] - off[b0];
}

// hist[e][qf][tf] -> out[k][qf*Fq + tf]: the pairs with d2 < rsq of radius k
// (cumulative over sorted edges), in the reference's counter layout.  out is
// zeroed on the stream before the launch (several (qf, tf) can share a slot
// of that layout, so the slots are accumulated atomically): any grid works.
__global__ void k_static_out(const unsigned long long *H, int ne, int Fqe, int Fte,
                             const int *edge_of, int nradii, int Fq, int Ft, long long *out)
{
    const int nrow = Fq * Ft;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nradii * Fqe * Fte;
         i += gridDim.x * blockDim.x) {
        const int k = i / (Fqe * Fte), qf = (i / Fte) % Fqe, tf = i % Fte;
        const int e = edge_of[k];
        if (e < 0) continue;
        unsigned long long v = 0;
        for (int j = 0; j <= e; j++) v += H[((size_t)j * Fqe + qf) * Fte + tf];
        atomicAdd((unsigned long long *)&out[(size_t)k * nrow + qf * Fq + tf], v);
    }
}

// int tile counts per block (staged in the offsets' storage) widened to int64
__global__ void k_gather_widen(const int *in, int n, long long *out)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = in[i];
}

static size_t align_up(size_t x) { return (x + 255) & ~size_t(255); }

static void count_static_impl(const kd_catalog *tc, int Ft, const kd_catalog *qc, int Fq,
                              const double *rsq_sorted, int ne, const int *edge_of, int nradii,
                              int mode, long long *h_out)
{
    if (tc->device != qc->device) raise(KD_EINVAL, "tree and query catalogs on different devices");
    check(cudaSetDevice(tc->device), "cudaSetDevice");
    unsigned char *base = static_scratch(tc->device);
    const cudaStream_t s = 0;  // legacy default stream: nothing is created

    const int nb = qc->nblocks;
    const int Fqe = qc->max_qf + 1, Fte = tc->max_tf + 1;
    const size_t hsz = (size_t)(ne + 1) * Fqe * Fte;

    // carve the scratch
    size_t at = 0;
    auto take = [&](size_t bytes) {
        unsigned char *p = base + at;
        at = align_up(at + bytes);
        return p;
    };
    auto *H = (unsigned long long *)take(sizeof(unsigned long long) * hsz);
    auto *job = (JobDesc *)take(sizeof(JobDesc));
    auto *jblk = (int *)take(sizeof(int) * 2);
    auto *misc = (unsigned long long *)take(sizeof(unsigned long long) * 8);  // stats
    auto *err = (int *)take(sizeof(int) * 4);  // err, work, b1
    auto *rsq = (double *)take(sizeof(double) * KD_MAX_EDGES);
    auto *eo = (int *)take(sizeof(int) * KD_MAX_EDGES);
    auto *out = (long long *)take(sizeof(long long) * (size_t)nradii * Fq * Ft);
    auto *cnt = (long long *)take(sizeof(long long) * ((size_t)nb + 1));
    auto *off = (long long *)take(sizeof(long long) * ((size_t)nb + 1));
    const size_t scan_bytes = sort::scan_temp_bytes<long long>(nb + 1);
    void *scan_tmp = take(scan_bytes);
    const int rel_cap = 4096;  // blocks per batch
    auto *rel = (long long *)take(sizeof(long long) * (rel_cap + 1));
    if (at + 16 * 64 > kStaticScratchBytes)
        raise(KD_EINVAL, "count too large for the static scratch (needs more than 32 MiB for "
                         "its histogram and block tables)");
    const long long cap = (long long)((kStaticScratchBytes - at) / sizeof(uint4));
    auto *rec = (uint4 *)(base + at);

    check(cudaMemsetAsync(H, 0, sizeof(unsigned long long) * hsz, s), "memset");
    check(cudaMemsetAsync(misc, 0, sizeof(unsigned long long) * 8, s), "memset");
    check(cudaMemsetAsync(err, 0, sizeof(int) * 4, s), "memset");
    check(cudaMemsetAsync(cnt, 0, sizeof(long long) * ((size_t)nb + 1), s), "memset");
    check(cudaMemcpyAsync(rsq, rsq_sorted, sizeof(double) * ne, cudaMemcpyHostToDevice, s), "H2D");
    check(cudaMemcpyAsync(eo, edge_of, sizeof(int) * nradii, cudaMemcpyHostToDevice, s), "H2D");
    const JobDesc hjob = job_desc(tc, qc, H);
    const int hjblk[2] = {0, nb};
    check(cudaMemcpyAsync(job, &hjob, sizeof hjob, cudaMemcpyHostToDevice, s), "H2D");
    check(cudaMemcpyAsync(jblk, hjblk, sizeof hjblk, cudaMemcpyHostToDevice, s), "H2D");

    // tile counts per block (the traversal writes int counts; widen in place)
    TravOut to;
    memset(&to, 0, sizeof to);
    to.count = (int *)off;  // int counts, staged in off's storage
    to.accepted = misc + 2;
    to.err = err;
    if (nb > 0)
        k_traverse<false><<<blocks_for(nb, kTravWarps), 32 * kTravWarps, 0, s>>>(job, jblk, 1, rsq,
                                                                                  ne, 0, nb, to);
    KD_LAUNCH_CHECK("k_traverse(count)");
    k_gather_widen<<<blocks_for(nb, 256), 256, 0, s>>>((const int *)off, nb, cnt);
    check(sort::scan<long long, sort::SumOp, false>(scan_tmp, cnt, off, nb + 1, sort::SumOp(), s),
          "scan");

    const TileKernel kern(&tc, &qc, 1, ne, mode);
    int nsm = 148;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, tc->device);
    int b0 = 0;
    while (b0 < nb) {
        k_static_batch<<<1, 256, 0, s>>>(off, nb, b0, cap, err + 2, rel, rel_cap);
        KD_LAUNCH_CHECK("k_static_batch");
        int b1 = 0;
        check(cudaMemcpyAsync(&b1, err + 2, sizeof(int), cudaMemcpyDeviceToHost, s), "D2H");
        check(cudaStreamSynchronize(s), "sync");
        if (b1 < 0) raise(KD_EINVAL, "a query block has more tile records than the static scratch holds");
        TravOut tf = to;
        tf.count = nullptr;
        tf.off = rel;
        tf.rec = rec;
        k_traverse<true><<<blocks_for(b1 - b0, kTravWarps), 32 * kTravWarps, 0, s>>>(job, jblk, 1,
                                                                                      rsq, ne, b0, b1, tf);
        KD_LAUNCH_CHECK("k_traverse(fill)");
        TileArgs ta;
        ta.jobs = job;
        ta.jblk = jblk;
        ta.njobs = 1;
        ta.rsq = rsq;
        ta.ne = ne;
        ta.g0 = b0;
        ta.g1 = b1;
        ta.gmap = nullptr;
        ta.off = rel;
        ta.rec = rec;
        ta.work = err + 1;
        ta.stats = misc;
        check(cudaMemsetAsync(err + 1, 0, sizeof(int), s), "memset");
        const int grid = (int)std::min<long long>(b1 - b0, (long long)nsm * kern.ctas);
        kern.run<<<grid, kTileThreads, kern.smem, s>>>(ta);
        KD_LAUNCH_CHECK("k_tiles");
        b0 = b1;
    }
    check(cudaMemsetAsync(out, 0, sizeof(long long) * (size_t)nradii * Fq * Ft, s), "memset");
    k_static_out<<<blocks_for((long long)nradii * Fqe * Fte, 256), 256, 0, s>>>(H, ne, Fqe, Fte, eo,
                                                                                 nradii, Fq, Ft, out);
    KD_LAUNCH_CHECK("k_static_out");
    int herr = 0;
    check(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, s), "D2H");
    check(cudaMemcpyAsync(h_out, out, sizeof(long long) * (size_t)nradii * Fq * Ft,
                          cudaMemcpyDeviceToHost, s), "D2H");
    check(cudaStreamSynchronize(s), "sync");
    if (herr) raise(herr, "node-pair traversal exceeded its stack");
}

}  // namespace kd

extern "C" int kdg_count_static(const kd_catalog *tree, int Ft, const kd_catalog *query, int Fq,
                                const double *rsq_sorted, int ne, const int *edge_of,
                                int nradii, int mode, long long *out)
{
    if (ne < 0 || ne > KD_MAX_EDGES || nradii < 0 || nradii > KD_MAX_EDGES) {
        kd_set_error(KD_EINVAL, "at most %d radii", KD_MAX_EDGES);
        return KD_EINVAL;
    }
    try {
        kd::count_static_impl(tree, Ft, query, Fq, rsq_sorted, ne, edge_of, nradii, mode, out);
        return KD_OK;
    } catch (const kd::Error &e) {
        kd_set_error(e.code, "%s", e.msg);
        return e.code;
    } catch (const std::bad_alloc &) {
        kd_set_error(KD_ENOMEM, "out of host memory");
        return KD_ENOMEM;
    } catch (const std::exception &e) {
        kd_set_error(KD_EINTERNAL, "host error: %s", e.what());
        return KD_EINTERNAL;
    }
}

extern "C" int kdg_set_device(int device)
{
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || device < 0 || device >= n) {
        cudaGetLastError();
        kd_set_error(KD_ENODEV, "no CUDA device %d (%d visible)", device, n);
        return KD_ENODEV;
    }
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) {
        kd_set_error(KD_ECUDA, "cudaSetDevice: %s", cudaGetErrorString(e));
        return KD_ECUDA;
    }
    return KD_OK;
}

extern "C" int kdg_count_batch(const kd_catalog *const *trees, const kd_catalog *const *queries,
                               int njobs, const double *rsq, int ne, int mode, int shard,
                               int nshards, long long *const *hists, kd_count_stats *stats)
{
    if (nshards < 1 || shard < 0 || shard >= nshards) {
        kd_set_error(KD_EINVAL, "shard %d of %d", shard, nshards);
        return KD_EINVAL;
    }
    if (ne < 1 || ne > KD_MAX_EDGES) {
        kd_set_error(KD_EINVAL, "between 1 and %d distinct radii per count", KD_MAX_EDGES);
        return KD_EINVAL;
    }
    if (njobs < 1) {
        kd_set_error(KD_EINVAL, "a batch needs at least one job");
        return KD_EINVAL;
    }
    try {
        kd::count_batch_impl(trees, queries, njobs, rsq, ne, mode, shard, nshards, hists, stats);
        return KD_OK;
    } catch (const kd::Error &e) {
        kd_set_error(e.code, "%s", e.msg);
        return e.code;
    } catch (const std::bad_alloc &) {
        kd_set_error(KD_ENOMEM, "out of host memory");
        return KD_ENOMEM;
    } catch (const std::exception &e) {
        kd_set_error(KD_EINTERNAL, "host error: %s", e.what());
        return KD_EINTERNAL;
    }
}

extern "C" int kdg_count(const kd_catalog *tree, const kd_catalog *query, const double *rsq,
                         int ne, int mode, int shard, int nshards, long long *hist,
                         kd_count_stats *stats)
{
    return kdg_count_batch(&tree, &query, 1, rsq, ne, mode, shard, nshards, &hist, stats);
}
