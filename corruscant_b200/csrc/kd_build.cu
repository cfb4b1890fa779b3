// GPU tree build for corruscant's tree_construct (kdbuild.c:451-537).
//
// Produces, on the device, the same node array and in-order permutation the
// reference's recursive presort-median build produces (semantic fields:
// coordinates, field, weight, has_lchild, has_rchild, dim), and from that tree
// the counting layout used by kd_count.cu (see kd_internal.h).
//
// Reference semantics reproduced (kdbuild.c line numbers):
//   dedup            : stable lexicographic (x,y,z) sort with '==' compares
//                      (so -0.0 == +0.0), first occurrence keeps its field,
//                      weight = run length, >= 256 copies is an error
//                      (:82-96, :98-152, :479-511)
//   argsorts         : the three cyclic superkey orders of the unique points
//                      (:59-80, :158-243)
//   median           : (l+r+1)/2, rounding right (:52-55)
//   split dimension  : max_variance_dim over subtrees of 4+ points: per
//                      dimension a sequential sum in that dimension's superkey
//                      order, mean by division, sequential fused
//                      multiply-add sum of squared deviations, first strict
//                      maximum wins (:308-351, :383-386)
//   partition        : stable split of the other orders around the median
//                      (:251-291)
//   base cases       : sizes 1, 2, 3 taken from the superkey-0 order (:402-418)
//   heap layout      : root 1, children 2p and 2p+1, memsize = pow2ceil (:435-449)
//
// GPU formulation (not the reference's recursion): all subtrees of one depth
// are processed together.  Positions of the three superkey-ordered index arrays
// are grouped in contiguous segments, one per subtree.  A level computes every
// segment's split dimension, writes the level's nodes, then moves every
// position to its child segment with a stable segmented partition; segments of
// up to kSubCap points go through all their remaining levels in one block's
// shared memory.  Split dimensions of segments of more than kSubSeq points come
// from a parallel variance with a rigorous error interval around the value the
// reference's sequential sums produce; only when the intervals of the best and
// another dimension overlap is the sequential computation run.

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <condition_variable>
#include <cstdio>
#include <exception>
#include <memory>
#include <new>
#include <cmath>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#if defined(__x86_64__)
#include <immintrin.h>
#endif

#include "kd_cuda_util.cuh"
#include "kd_sort.cuh"

namespace kd {

struct alignas(8) NodeRec {
    double v[3];
    uint32_t fw;    // field:8 | weight:8 << 8  (kdtree.h:15-16)
    uint32_t pad0;
    uint32_t flags; // has_lchild:1 | has_rchild:1 << 1 | dim:8 << 2 (kdtree.h:21-24)
    uint32_t pad1;
};
static_assert(sizeof(NodeRec) == 40, "node_t is 40 bytes");

static const int TPB = 256;

// Positions and threads per block in the parallel variance kernels.  Fewer
// than the smallest segment of the level loop, so that a block meets at most
// two of them.
constexpr int kVarChunk = 512;
constexpr int kVarThreads = 128;

// Once per device (any thread may get here first; doing it twice is harmless):
// keep freed stream-ordered allocations in the device's pool instead of
// returning them to the driver at every synchronisation.
void init_device()
{
    static std::atomic<unsigned long long> done{0};
    int dev = 0;
    check(cudaGetDevice(&dev), "cudaGetDevice");
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
    if (bit && (done.load() & bit)) return;
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
        uint64_t thr = UINT64_MAX;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr);
    }
    cudaGetLastError();
    done.fetch_or(bit);
}

// Order-preserving 64-bit key of a double; -0.0 maps to +0.0's key so that
// key equality is C '==' equality for non-NaN values.
__device__ __forceinline__ uint64_t okey(double v)
{
    if (v == 0.0) v = 0.0;
    uint64_t b = (uint64_t)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

__device__ __forceinline__ void set_err(int *err, int code) { atomicCAS(err, 0, code); }

// ------------------------------------------------------------ dedup stage

// value of a key (the +0.0 key gives +0.0)
__host__ __device__ __forceinline__ double okey_value(uint64_t k)
{
    const uint64_t b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
    double v;
    memcpy(&v, &b, sizeof v);
    return v;
}

// What the points' keys span, per coordinate: the OR of (key xor first key),
// i.e. the bits that vary, the largest key and the largest ~key.
struct KeySpan {
    unsigned long long vary[3], hi[3], inv_lo[3];
};

template <bool KEYS>
__global__ void __launch_bounds__(TPB) k_prep(const double *__restrict__ xyz, int n, uint64_t *kx,
                                              uint64_t *ky, uint64_t *kz, int *iota, int *err,
                                              KeySpan *span)
{
    __shared__ unsigned long long red[9];
    if (threadIdx.x < 9) red[threadIdx.x] = 0;
    __syncthreads();
    uint64_t *const out[3] = {kx, ky, kz};
    unsigned long long first[3], m[9];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        first[d] = okey(xyz[d]);
        m[d] = m[3 + d] = m[6 + d] = 0;
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        bool bad = false;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const double v = xyz[3 * (size_t)i + d];
            const unsigned long long k = okey(v);
            bad = bad || isnan(v);
            if (KEYS) out[d][i] = k;
            m[d] |= k ^ first[d];
            m[3 + d] = max(m[3 + d], k);
            m[6 + d] = max(m[6 + d], ~k);
        }
        if (bad) set_err(err, KD_ENAN);
        if (KEYS) iota[i] = i;
    }
#pragma unroll
    for (int k = 0; k < 9; k++) {
        for (int o = 16; o; o >>= 1) {
            const unsigned long long v = __shfl_xor_sync(0xffffffffu, m[k], o);
            m[k] = k < 3 ? m[k] | v : max(m[k], v);
        }
        if ((threadIdx.x & 31) == 0) {
            if (k < 3) atomicOr(&red[k], m[k]);
            else atomicMax(&red[k], m[k]);
        }
    }
    __syncthreads();
    if (threadIdx.x < 9) {
        unsigned long long *g = span->vary + threadIdx.x;
        if (threadIdx.x < 3) atomicOr(g, red[threadIdx.x]);
        else atomicMax(g, red[threadIdx.x]);
    }
}

// A coordinate's 32-bit sort key, weakly increasing in its 64-bit key: the
// bits that vary where 32 hold them all, else the position within [lo, hi] in
// steps of 2^-bits (rounding keeps the order), else, for an infinite or
// overflowing range, the 32 highest bits that vary.
struct KeyMap {
    double lo, scale, top;
    int shift, bits, exact;
    __device__ __forceinline__ unsigned operator()(uint64_t k) const
    {
        if (scale > 0.0) return __double2uint_rd(fmin((okey_value(k) - lo) * scale, top));
        const unsigned v = (unsigned)(k >> shift);
        return bits < 32 ? v & ((1u << bits) - 1u) : v;
    }
};

__global__ void k_map_keys(const uint64_t *__restrict__ k, const int *__restrict__ perm, int n, KeyMap map,
                           unsigned *out)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = map(k[perm ? perm[i] : i]);
}

// Finish a stable sort made by 32-bit keys: runs of equal 32-bit keys are put
// in order of the NK 64-bit keys (k[0] first), in place in `out`, which starts
// as a copy of the permutation `in`.  The thread at a run's first inversion
// sorts the run; a run of more than kFixRun points that is out of order sets
// *too_long instead.
constexpr int kFixRun = 32;
struct Keys3 {
    const uint64_t *k[3];
};
template <int NK>
__global__ void k_fix_runs(const unsigned *__restrict__ s32, int n, Keys3 keys, const int *__restrict__ in,
                           int *__restrict__ out, int *too_long)
{
    auto less = [&](int a, int b) {
#pragma unroll
        for (int j = 0; j < NK; j++) {
            const uint64_t x = keys.k[j][a], y = keys.k[j][b];
            if (x != y) return x < y;
        }
        return false;
    };
    for (int i = blockIdx.x * blockDim.x + threadIdx.x + 1; i < n; i += gridDim.x * blockDim.x) {
        const unsigned key = s32[i];
        if (s32[i - 1] != key || !less(in[i], in[i - 1])) continue;
        int h = i - 1, e = i + 1;
        bool first = true;
        while (h > 0 && s32[h - 1] == key && i - h < kFixRun) {
            if (less(in[h], in[h - 1])) {
                first = false;
                break;
            }
            h--;
        }
        if (!first) continue;
        while (e < n && s32[e] == key && e - h <= kFixRun) e++;
        if (e - h > kFixRun || i - h >= kFixRun) {
            *too_long = 1;
            continue;
        }
        int a[kFixRun];
        for (int j = h; j < e; j++) {
            const int p = in[j];
            int q = j - h;
            for (; q > 0 && less(p, a[q - 1]); q--) a[q] = a[q - 1];
            a[q] = p;
        }
        for (int j = h; j < e; j++) out[j] = a[j - h];
    }
}

__global__ void k_gather_u64(const uint64_t *__restrict__ src, const int *__restrict__ idx, int n,
                             uint64_t *dst)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        dst[i] = src[idx[i]];
}

// first: points sorted by 32-bit keys of x, where two equal points share one
// (null: not sorted so); spares most gathers (0.13 ms at 5M points, so 0.02)
__global__ void k_heads(const int *__restrict__ p, const unsigned *__restrict__ first, const uint64_t *kx,
                        const uint64_t *ky, const uint64_t *kz, int n, int *head)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int h = 1;
        if (i > 0 && (!first || first[i] == first[i - 1])) {
            int a = p[i], b = p[i - 1];
            h = (kx[a] != kx[b]) | (ky[a] != ky[b]) | (kz[a] != kz[b]);
        }
        head[i] = h;
    }
}

struct UniqueArrays {
    double *ux, *uy, *uz;
    int *ufield, *uw, *urep, *uhead;
    uint64_t *uky, *ukz;
};

// cls[i] = 1-based class number of dedup-sorted position i
__global__ void k_unique(const int *__restrict__ p, const int *__restrict__ head,
                         const int *__restrict__ cls, int n, const double *__restrict__ xyz,
                         const int *__restrict__ fin, UniqueArrays u, int n_u)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (!head[i]) continue;
        int c = cls[i] - 1, r = p[i];
        const double x = xyz[3 * (size_t)r], y = xyz[3 * (size_t)r + 1], z = xyz[3 * (size_t)r + 2];
        u.ux[c] = x;
        u.uy[c] = y;
        u.uz[c] = z;
        u.ufield[c] = fin ? (fin[r] & 0xFF) : 0;
        u.urep[c] = r;
        u.uhead[c] = i;
        u.uky[c] = okey(y);  // (gathered, like that of x: 0.41 ms at 5M points, so 0.16)
        u.ukz[c] = okey(z);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) u.uhead[n_u] = n;
}

struct FieldInfo {
    int min_qf, max_qf, max_tf, split;
};

__global__ void k_weights(UniqueArrays u, int n_u, const int *__restrict__ p,
                          const int *__restrict__ cls, const int *__restrict__ fin, int n,
                          int *err, FieldInfo *fi)
{
    int maxtf = 0;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n_u; c += gridDim.x * blockDim.x) {
        int w = u.uhead[c + 1] - u.uhead[c];
        u.uw[c] = w;
        if (w > 255) set_err(err, KD_EDUP);
        maxtf = max(maxtf, u.ufield[c]);
    }
    int minq = 0x7fffffff, maxq = -0x7fffffff, split = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int qf = fin ? fin[p[i]] : 0;
        int tf = u.ufield[cls[i] - 1];
        minq = min(minq, qf);
        maxq = max(maxq, qf);
        split |= (qf != tf);
    }
    for (int o = 16; o; o >>= 1) {
        maxtf = max(maxtf, __shfl_xor_sync(0xffffffffu, maxtf, o));
        minq = min(minq, __shfl_xor_sync(0xffffffffu, minq, o));
        maxq = max(maxq, __shfl_xor_sync(0xffffffffu, maxq, o));
        split |= __shfl_xor_sync(0xffffffffu, split, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&fi->max_tf, maxtf);
        atomicMin(&fi->min_qf, minq);
        atomicMax(&fi->max_qf, maxq);
        atomicOr(&fi->split, split);
    }
}

// ------------------------------------------------------------ level loop

struct Segs {
    int *p, *l, *r;   // heap id and in-order range of each segment
    int *count;       // device count
};

struct LevelBufs {
    int *tdim;                  // split dimension
    double *acc;                // S0 S1 S2 A0 A1 A2 V0 V1 V2
    int *mid;                   // the median point's rank in the split order
    const int *rank1, *rank2;   // ranks of the points in orders 1 and 2
};

__global__ void k_first_seg(Segs sg, int n_u)
{
    sg.count[0] = sg.p[0] = 1;
    sg.l[0] = 0;
    sg.r[0] = n_u - 1;
}

// One level's buffers cleared, and the next level's segments (the largest of the
// level loop holds more than kSubCap points and no other more than one fewer, so
// all of them split).
__global__ void k_seg_setup(Segs sg, int ub, LevelBufs lb, Segs nxt)
{
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= ub) return;
    const int ns = *sg.count;
    if (s == 0) *nxt.count = 2 * ns;
    if (s >= ns) return;
    const int p = sg.p[s], l = sg.l[s], r = sg.r[s], med = (l + r + 1) / 2;
    for (int k = 0; k < 9; k++) lb.acc[9 * (size_t)s + k] = 0.0;
    nxt.p[2 * s] = 2 * p;
    nxt.l[2 * s] = l;
    nxt.r[2 * s] = med - 1;
    nxt.p[2 * s + 1] = 2 * p + 1;
    nxt.l[2 * s + 1] = med + 1;
    nxt.r[2 * s + 1] = r;
}

// Parallel sums per segment: pass 0 accumulates S_j = sum v_j and
// A_j = sum |v_j|; pass 1 accumulates V_j = sum (v_j - S_j/n)^2.  Bound by
// memory: 5M points in 30 us and 34 (with 256 positions per block and each
// load behind its position's segment 47 and 53).
// c0, c1, c2: the x of the point at each position of superkey order 0, the
// y along order 1, the z along order 2 (carried through the partitions), so
// a segment's coordinates are read contiguously; the parallel sums do not
// depend on the order within a segment
template <int PASS>
__global__ void __launch_bounds__(kVarThreads) k_var_par(int n_u, const int *__restrict__ pos_seg,
                                                         Segs sg, LevelBufs lb,
                                                         const double *__restrict__ c0,
                                                         const double *__restrict__ c1,
                                                         const double *__restrict__ c2)
{
    // pass 0: S0 S1 S2 A0 A1 A2; pass 1: V0 V1 V2
    constexpr int NV = PASS == 0 ? 6 : 3;
    constexpr int PER = kVarChunk / kVarThreads;
    constexpr int NW = kVarThreads / 32;
    __shared__ double wsum[NW][2][NV];
    __shared__ double mu_sh[2][3];
    __shared__ int wmin[NW];
    const int base = blockIdx.x * kVarChunk;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int seg[PER];
    double x[PER][3];
    int smin = 0x7fffffff;
#pragma unroll
    for (int k = 0; k < PER; k++) {  // (every load before the first use)
        const int i = base + threadIdx.x + kVarThreads * k, j = min(i, n_u - 1);
        seg[k] = i < n_u ? pos_seg[j] : -1;
        x[k][0] = c0[j];
        x[k][1] = c1[j];
        x[k][2] = c2[j];
    }
#pragma unroll
    for (int k = 0; k < PER; k++)
        if (seg[k] >= 0) smin = min(smin, seg[k]);
    smin = __reduce_min_sync(0xffffffffu, smin);
    if (lane == 0) wmin[w] = smin;
    __syncthreads();
    int s0 = wmin[0];
#pragma unroll
    for (int q = 1; q < NW; q++) s0 = min(s0, wmin[q]);
    if (s0 == 0x7fffffff) return;
    if (PASS == 1) {  // the means of the chunk's first two segments, once
        if (threadIdx.x < 6) {
            const int q = threadIdx.x / 3, j = threadIdx.x % 3, sq = s0 + q;
            mu_sh[q][j] = sq < *sg.count
                              ? lb.acc[9 * (size_t)sq + j] / (double)(sg.r[sq] - sg.l[sq] + 1)
                              : 0.0;
        }
        __syncthreads();
    }
    double a[2][NV];
#pragma unroll
    for (int q = 0; q < 2; q++)
#pragma unroll
        for (int j = 0; j < NV; j++) a[q][j] = 0.0;
    bool second = false;
#pragma unroll
    for (int k = 0; k < PER; k++) {
        const int s = seg[k];
        if (s < 0) continue;
        const double *const v = x[k];
        double c[NV];
        const int slot = s - s0;
        if (PASS == 0) {
#pragma unroll
            for (int j = 0; j < 3; j++) {
                c[j] = v[j];
                c[3 + j] = fabs(v[j]);
            }
        } else {
            const double n = (double)(sg.r[s] - sg.l[s] + 1);
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const double mu = slot < 2 ? mu_sh[slot][j] : lb.acc[9 * (size_t)s + j] / n;
                const double d = v[j] - mu;
                c[j] = d * d;
            }
        }
        if (slot == 0) {
#pragma unroll
            for (int j = 0; j < NV; j++) a[0][j] += c[j];
        } else if (slot == 1) {
            second = true;
#pragma unroll
            for (int j = 0; j < NV; j++) a[1][j] += c[j];
        } else {  // a third segment in one chunk: segments this small are rare
#pragma unroll
            for (int j = 0; j < NV; j++)
                atomicAdd(&lb.acc[9 * (size_t)s + (PASS == 0 ? 0 : 6) + j], c[j]);
        }
    }
    // warp sums; the second segment's only where a lane of the warp holds one
    const bool two = __any_sync(0xffffffffu, second);
#pragma unroll
    for (int q = 0; q < 2; q++) {
        if (q == 1 && !two) {
            if (lane < NV) wsum[w][1][lane] = 0.0;
            break;
        }
#pragma unroll
        for (int j = 0; j < NV; j++) {
            double v = a[q][j];
#pragma unroll
            for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) wsum[w][q][j] = v;
        }
    }
    __syncthreads();
    if (threadIdx.x < 2 * NV) {
        const int q = threadIdx.x / NV, j = threadIdx.x % NV, s = s0 + q;
        double v = wsum[0][q][j];
#pragma unroll
        for (int x = 1; x < NW; x++) v += wsum[x][q][j];
        if (v != 0.0 && s < *sg.count)
            atomicAdd(&lb.acc[9 * (size_t)s + (PASS == 0 ? 0 : 6) + j], v);
    }
}

__device__ __forceinline__ double gam(double m)
{
    const double u = 1.1102230246251565e-16;  // 2^-53
    return m * u / (1.0 - m * u);
}

// The split dimension of a segment of n points from rigorous intervals around
// the reference's rounded variances, or -1 when they overlap.  a: sums of v,
// |v| and (v - mean)^2 per dimension, in any order of summation.
__device__ __forceinline__ int decide_dim(double n, const double *a)
{
    const double u = 1.1102230246251565e-16;
    double lo[3], hi[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
        double A = a[3 + j] * (1.0 + gam(n));
        double dmu = (gam(n - 1) * (1.0 + u) + u) * A / n * (1.0 + 4 * u);
        double V = a[6 + j];
        double nd2 = n * dmu * dmu * (1.0 + 4 * u);
        double l = V / (1.0 + gam(n + 2)) - nd2;
        if (l < 0) l = 0;
        lo[j] = (1.0 - gam(n + 1)) * (1.0 - u) * (1.0 - u) * l * (1.0 - 1e-14);
        hi[j] = (1.0 + gam(n + 1)) * (1.0 + u) * (1.0 + u) * (V / (1.0 - gam(n + 2)) + nd2) *
                (1.0 + 1e-14);
    }
    int c = 0;
    if (a[7] > a[6 + c]) c = 1;
    if (a[8] > a[6 + c]) c = 2;
    bool ok = true;
#pragma unroll
    for (int j = 0; j < 3; j++)
        if (j != c && !(lo[c] > hi[j])) ok = false;
    return ok ? c : -1;
}

// max_variance_dim exactly as the reference evaluates it (kdbuild.c:308-351),
// one thread per segment; the three dimensions' chains are independent and
// are interleaved for latency hiding without changing any chain's order.
// c0, c1, c2 as for k_var_par: c_j[i] is coordinate j of the point at
// position i of superkey order j, so the sums below run over exactly the
// values, in exactly the order, of the reference's loops over args[j]
__device__ __noinline__ int seq_dim(int l, int r, const double *__restrict__ c0, const double *__restrict__ c1,
                                    const double *__restrict__ c2)
{
    const int size = r - l + 1;
    double m0 = 0.0, m1 = 0.0, m2 = 0.0;
    int i = l;
    for (; i + 4 <= r + 1; i += 4) {
        double v0[4], v1[4], v2[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v0[k] = c0[i + k];
            v1[k] = c1[i + k];
            v2[k] = c2[i + k];
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            m0 = __dadd_rn(m0, v0[k]);
            m1 = __dadd_rn(m1, v1[k]);
            m2 = __dadd_rn(m2, v2[k]);
        }
    }
    for (; i <= r; i++) {
        m0 = __dadd_rn(m0, c0[i]);
        m1 = __dadd_rn(m1, c1[i]);
        m2 = __dadd_rn(m2, c2[i]);
    }
    double nn = (double)size;
    m0 = __ddiv_rn(m0, nn);
    m1 = __ddiv_rn(m1, nn);
    m2 = __ddiv_rn(m2, nn);
    double q0 = 0.0, q1 = 0.0, q2 = 0.0;
    i = l;
    for (; i + 4 <= r + 1; i += 4) {
        double v0[4], v1[4], v2[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v0[k] = c0[i + k];
            v1[k] = c1[i + k];
            v2[k] = c2[i + k];
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            double d0 = __dsub_rn(v0[k], m0), d1 = __dsub_rn(v1[k], m1), d2 = __dsub_rn(v2[k], m2);
            q0 = __fma_rn(d0, d0, q0);
            q1 = __fma_rn(d1, d1, q1);
            q2 = __fma_rn(d2, d2, q2);
        }
    }
    for (; i <= r; i++) {
        double d0 = __dsub_rn(c0[i], m0), d1 = __dsub_rn(c1[i], m1), d2 = __dsub_rn(c2[i], m2);
        q0 = __fma_rn(d0, d0, q0);
        q1 = __fma_rn(d1, d1, q1);
        q2 = __fma_rn(d2, d2, q2);
    }
    int dim = 0;
    double mx = q0;
    if (q1 > mx) {
        mx = q1;
        dim = 1;
    }
    if (q2 > mx) dim = 2;
    return dim;
}

struct TreeOut {
    NodeRec *nodes;
    int *inorder_rep;  // input index of the point at every in-order position
    int memsize;
};

__device__ __forceinline__ void put_node(TreeOut t, const UniqueArrays &u, int hp, int pt, int dim,
                                         int hl, int hr, int pos, int *err)
{
    if (hp >= t.memsize) {
        set_err(err, KD_EINTERNAL);
        return;
    }
    NodeRec rec;
    rec.v[0] = u.ux[pt];
    rec.v[1] = u.uy[pt];
    rec.v[2] = u.uz[pt];
    rec.fw = (uint32_t)u.ufield[pt] | ((uint32_t)u.uw[pt] << 8);
    rec.pad0 = 0;
    rec.flags = (uint32_t)hl | ((uint32_t)hr << 1) | ((uint32_t)dim << 2);
    rec.pad1 = 0;
    t.nodes[hp] = rec;
    t.inorder_rep[pos] = u.urep[pt];
}

// A level's split dimensions, nodes and median ranks, one thread per segment.
__global__ void k_level_nodes(Segs sg, int ub, LevelBufs lb, const int *__restrict__ a0,
                              const int *__restrict__ a1, const int *__restrict__ a2,
                              const double *__restrict__ c0, const double *__restrict__ c1,
                              const double *__restrict__ c2, UniqueArrays u, TreeOut t, int *err)
{
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= ub || s >= *sg.count) return;
    const int l = sg.l[s], r = sg.r[s], med = (l + r + 1) / 2;
    int d = decide_dim((double)(r - l + 1), lb.acc + 9 * (size_t)s);
    if (d < 0) d = seq_dim(l, r, c0, c1, c2);
    const int pt = (d == 0 ? a0 : (d == 1 ? a1 : a2))[med];
    put_node(t, u, sg.p[s], pt, d, 1, 1, med, err);
    lb.tdim[s] = d;
    lb.mid[s] = d == 0 ? pt : (d == 1 ? lb.rank1 : lb.rank2)[pt];
}

__global__ void k_ranks(int n, const int *__restrict__ a1, const int *__restrict__ a2, int *rank1, int *rank2)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        rank1[a1[i]] = i;
        rank2[a2[i]] = i;
    }
}

// ---- Stable three-way partition of the three superkey orders, one level.
// Within every segment [l, r], median position med = (l + r + 1) / 2, the
// points of each order d go, in their order, to [l, med) when they stand before
// the median point in the order of the split dimension (side 0), to (med, r]
// when behind it (side 1), the median point itself to med; positions outside
// segments stay.  The side follows from the ranks that the points have in the
// whole sorted orders (a point's id is its rank in order 0).  The destination of a
// point is its segment's start plus the number of same-side points before it
// in the segment.  Three launches over tiles of kPtTile positions handle all
// three orders at once, with no waiting between blocks: per 32 positions, a
// bit mask of each order's left and right points, and the tile's counts from
// its last segment start on; one block scans those; the move counts bits
// below a position, in the tile and back to its segment's start or the tile's
// carry.  Lanes hold neighbouring positions, so that loads are whole lines and
// a warp's stores two runs.  Bound by memory: with eight consecutive positions
// per thread, whose stores met a line once per position, the move of 5M points
// took 150 us a level (and 20 for the next level's segments, written here),
// now 83; the counts 57 after 45 for a kernel that marked each point's side, which
// the ranks spare, now 62.
constexpr int kPtThreads = 256;
constexpr int kPtWarps = kPtThreads / 32;
constexpr int kPtRounds = 8;                      // positions per thread
constexpr int kPtTile = kPtThreads * kPtRounds;
constexpr int kPtWords = kPtTile / 32;            // words of 32 positions per tile
constexpr int kPtMasks = 6;                       // per word: order 0 left, right, order 1 left, ...

struct PartIO {
    const int *a[3];     // superkey orders (point ids by position)
    int *ao[3];          // partitioned orders
    const double *c[3];  // coordinate d of the point at each position of order d
    double *co[3];       // the same, partitioned
};

// inclusive segmented scan over the lanes of a warp: a lane's value restarts
// at a lane holding a head (f = 1)
template <int NV>
__device__ __forceinline__ void warp_seg_scan(unsigned &f, unsigned (&v)[NV], int lane)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned pf = __shfl_up_sync(0xffffffffu, f, o);
        unsigned pv[NV];
#pragma unroll
        for (int k = 0; k < NV; k++) pv[k] = __shfl_up_sync(0xffffffffu, v[k], o);
        if (lane >= o) {
            if (!f)
#pragma unroll
                for (int k = 0; k < NV; k++) v[k] += pv[k];
            f |= pf;
        }
    }
}

// masks[tile][word][kPtMasks], and per tile (a segment start in the tile?, the
// three orders' left | right << 16 counts from its last one, or from the
// tile's start when it has none).
__global__ void __launch_bounds__(kPtThreads) k_part_count(int n_u, const int *__restrict__ pos_seg,
                                                           Segs sg, const int *__restrict__ a0,
                                                           const int *__restrict__ a1,
                                                           const int *__restrict__ a2, LevelBufs lb,
                                                           unsigned *masks, uint4 *tagg)
{
    constexpr unsigned FULL = 0xffffffffu;
    static_assert(kPtWords == 64 && kPtWarps >= kPtMasks, "two words per lane, a warp per mask");
    __shared__ unsigned sm[kPtWords][kPtMasks], heads[kPtWords], tot[kPtMasks + 1];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int base = blockIdx.x * kPtTile;
    int sd[kPtRounds][3];
#pragma unroll
    for (int k = 0; k < kPtRounds; k++) {
        const int wd = w * kPtRounds + k, i = base + 32 * wd + lane;
        const int seg = i < n_u ? pos_seg[i] : -1;
        const bool in = seg >= 0;
        const int l = in ? sg.l[seg] : 0, r = in ? sg.r[seg] : 0, dim = in ? lb.tdim[seg] : 0,
                  mid = in ? lb.mid[seg] : 0, med = (l + r + 1) / 2;
        const unsigned h = __ballot_sync(FULL, in && l == i);
        if (lane == 0) heads[wd] = h;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            sd[k][d] = 3;
            if (!in) continue;
            int at = i, than = med;  // the split order itself: by place
            if (d != dim) {
                const int pt = (d == 0 ? a0 : (d == 1 ? a1 : a2))[i];
                at = dim == 0 ? pt : (dim == 1 ? lb.rank1 : lb.rank2)[pt];
                than = mid;
            }
            sd[k][d] = at < than ? 0 : (at > than ? 1 : 2);
        }
    }
#pragma unroll
    for (int k = 0; k < kPtRounds; k++)
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const unsigned l = __ballot_sync(FULL, sd[k][d] == 0), r = __ballot_sync(FULL, sd[k][d] == 1);
            if (lane == 0) {
                sm[w * kPtRounds + k][2 * d] = l;
                sm[w * kPtRounds + k][2 * d + 1] = r;
            }
        }
    __syncthreads();
    for (int i = threadIdx.x; i < kPtWords * kPtMasks; i += kPtThreads)
        masks[(size_t)blockIdx.x * (kPtWords * kPtMasks) + i] = (&sm[0][0])[i];
    if (w < kPtMasks) {
        // the last start: its word, then its bit
        const unsigned h0 = heads[lane], h1 = heads[lane + 32];
        const unsigned b0 = __ballot_sync(FULL, h0 != 0), b1 = __ballot_sync(FULL, h1 != 0);
        const int hw = b1 ? 63 - __clz(b1) : (b0 ? 31 - __clz(b0) : -1);
        const int bit = hw >= 0 ? 31 - __clz(heads[hw]) : 0;
        unsigned c = 0;
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int wd = lane + 32 * q;
            unsigned m = sm[wd][w];
            if (wd < hw) m = 0;
            if (wd == hw) m &= FULL << bit;
            c += __popc(m);
        }
        c = __reduce_add_sync(FULL, c);
        if (lane == 0) tot[w] = c;
        if (w == 0 && lane == 0) tot[kPtMasks] = hw >= 0;
    }
    __syncthreads();
    if (threadIdx.x == 0)
        tagg[blockIdx.x] = make_uint4(tot[kPtMasks], tot[0] | tot[1] << 16, tot[2] | tot[3] << 16,
                                      tot[4] | tot[5] << 16);
}

__device__ __forceinline__ void unpack_counts(const uint4 &g, unsigned (&x)[6])
{
    x[0] = g.y & 0xffffu;
    x[1] = g.y >> 16;
    x[2] = g.z & 0xffffu;
    x[3] = g.z >> 16;
    x[4] = g.w & 0xffffu;
    x[5] = g.w >> 16;
}

// One block: for every tile, the side counts (left, right for each order, 32
// bits each) from the last head before the tile: carry[2t], carry[2t+1].
__global__ void __launch_bounds__(1024) k_part_carry(int ntiles, const uint4 *__restrict__ tagg,
                                                     uint4 *carry)
{
    __shared__ unsigned sf[32], sv[32][6];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int per = (ntiles + 1023) / 1024;
    const int j0 = min(ntiles, t * per), j1 = min(ntiles, j0 + per);
    unsigned f = 0, v[6] = {0u, 0u, 0u, 0u, 0u, 0u};
    for (int j = j0; j < j1; j++) {
        const uint4 g = tagg[j];
        unsigned x[6];
        unpack_counts(g, x);
        for (int k = 0; k < 6; k++) v[k] = g.x ? x[k] : v[k] + x[k];
        f |= g.x;
    }
    unsigned fi = f, vi[6];
    for (int k = 0; k < 6; k++) vi[k] = v[k];
    warp_seg_scan<6>(fi, vi, lane);
    if (lane == 31) {
        sf[w] = fi;
        for (int k = 0; k < 6; k++) sv[w][k] = vi[k];
    }
    __syncthreads();
    // everything before this thread's tiles: the earlier warps, then the
    // earlier lanes of this warp
    unsigned pv[6] = {0u, 0u, 0u, 0u, 0u, 0u};
    for (int q = 0; q < w; q++)
        for (int k = 0; k < 6; k++) pv[k] = sf[q] ? sv[q][k] : pv[k] + sv[q][k];
    unsigned ef = __shfl_up_sync(0xffffffffu, fi, 1), ev[6];
    for (int k = 0; k < 6; k++) ev[k] = __shfl_up_sync(0xffffffffu, vi[k], 1);
    if (lane == 0) {
        ef = 0;
        for (int k = 0; k < 6; k++) ev[k] = 0;
    }
    unsigned cv[6];
    for (int k = 0; k < 6; k++) cv[k] = ef ? ev[k] : pv[k] + ev[k];
    for (int j = j0; j < j1; j++) {
        carry[2 * (size_t)j] = make_uint4(cv[0], cv[1], cv[2], cv[3]);
        carry[2 * (size_t)j + 1] = make_uint4(cv[4], cv[5], 0u, 0u);
        const uint4 g = tagg[j];
        unsigned x[6];
        unpack_counts(g, x);
        for (int k = 0; k < 6; k++) cv[k] = g.x ? x[k] : cv[k] + x[k];
    }
}

// The move: every position's point id and carried coordinate, in each of the
// three orders, to its place, and the next level's segment of every position.
__global__ void __launch_bounds__(kPtThreads) k_part_move(int n_u, const int *__restrict__ pos_seg, Segs sg,
                                                          PartIO io, const unsigned *__restrict__ masks,
                                                          const uint4 *__restrict__ carry, int *pos_next,
                                                          int *err)
{
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ unsigned sm[kPtWords][kPtMasks];
    __shared__ int pre[kPtMasks][kPtWords], car[kPtMasks];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int base = blockIdx.x * kPtTile;
    for (int i = threadIdx.x; i < kPtWords * kPtMasks; i += kPtThreads)
        (&sm[0][0])[i] = masks[(size_t)blockIdx.x * (kPtWords * kPtMasks) + i];
    if (threadIdx.x < kPtMasks)
        car[threadIdx.x] = (int)reinterpret_cast<const unsigned *>(carry + 2 * (size_t)blockIdx.x)[threadIdx.x];
    __syncthreads();
    if (w < kPtMasks) {  // points of the tile before each word
        const int c0 = __popc(sm[2 * lane][w]), c1 = __popc(sm[2 * lane + 1][w]);
        int inc = c0 + c1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(FULL, inc, o);
            if (lane >= o) inc += v;
        }
        pre[w][2 * lane] = inc - c0 - c1;
        pre[w][2 * lane + 1] = inc - c1;
    }
    __syncthreads();
#pragma unroll 2
    for (int k = 0; k < kPtRounds; k++) {
        const int wd = w * kPtRounds + k, i = base + 32 * wd + lane;
        if (i >= n_u) break;
        const int s = pos_seg[i];
        int pt[3];
        double cv[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            pt[d] = io.a[d][i];
            cv[d] = io.c[d][i];
        }
        int l = i, r = i, med = i, next = -1, at = 0;
        if (s >= 0) {
            l = sg.l[s];
            r = sg.r[s];
            med = (l + r + 1) / 2;
            if (i != med) next = 2 * s + (i > med);
            at = l - base;  // the segment's start in the tile, or before it
        }
        pos_next[i] = next;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            int dst = i;
            if (s >= 0) {
                const int sd = (sm[wd][2 * d] >> lane & 1u) ? 0 : ((sm[wd][2 * d + 1] >> lane & 1u) ? 1 : 2), q = 2 * d + sd;
                dst = med;
                if (sd < 2) {
                    int c = pre[q][wd] + __popc(sm[wd][q] & ((1u << lane) - 1u));
                    if (at >= 0) c -= pre[q][at >> 5] + __popc(sm[at >> 5][q] & ((1u << (at & 31)) - 1u));
                    else c += car[q];
                    dst = (sd == 0 ? l : med + 1) + c;
                }
                if (dst < l || dst > r) {
                    set_err(err, KD_EINTERNAL);
                    continue;
                }
            }
            io.ao[d][dst] = pt[d];
            io.co[d][dst] = cv[d];
        }
    }
}

// ------------------------------------------------------------ subtrees

// Whole subtrees of up to kSubCap points, one CTA each, from the level where
// every segment fits: the level loop's steps (split dimension, node, stable
// partition of the three orders) in shared memory, all subtrees of one depth
// together, with the points as 16-bit places in the segment's order 0.  Every
// point is read once and every node written once, where the level loop reads
// and writes ~180 bytes per point and level in twelve launches: the last ten
// levels of a 5M-point build took 3.7 ms there and take 1.6 ms here, all levels
// of a 4000-point build 0.93 and 0.39 ms.  What bounds it is the latency of its
// shared-memory gathers and the barriers between its steps (a third of the
// issue slots are used, with four blocks per SM).  1024 points: a larger cap
// would halve the blocks per SM, a smaller one would leave levels to the loop.
constexpr int kSubCap = 1024;
constexpr int kSubThreads = 256;
constexpr int kSubSeq = 48;  // segments up to this size: one thread, sequentially

struct SubSmem {
    double v[3][kSubCap];               // coordinates by place
    uint32_t fw[kSubCap];               // field | weight << 8 by place
    int rep[kSubCap];                   // input indices by place
    unsigned short o[2][3][kSubCap];    // the three orders: places by position
    short seg[2][kSubCap];              // position -> segment of the level, -1: none
    short l[2][kSubCap / 2 + 1], r[2][kSubCap / 2 + 1];  // segments: positions [l, r]
    unsigned mask[3][2][kSubCap / 32];  // positions going left / right, a bit each
    unsigned short pre[3][2][kSubCap / 32];
    unsigned char side[kSubCap];        // by place: 0 left, 1 right, 2 median
    unsigned char tdim[kSubCap / 2 + 1];
};

// max_variance_dim exactly as the reference evaluates it (kdbuild.c:308-351)
__device__ __forceinline__ int sub_var_seq(const SubSmem &s, const unsigned short (&o)[3][kSubCap], int l,
                                           int r)
{
    double m[3] = {0.0, 0.0, 0.0}, q[3] = {0.0, 0.0, 0.0};
    for (int i = l; i <= r; i++)
#pragma unroll
        for (int d = 0; d < 3; d++) m[d] = __dadd_rn(m[d], s.v[d][o[d][i]]);
    const double nn = (double)(r - l + 1);
#pragma unroll
    for (int d = 0; d < 3; d++) m[d] = __ddiv_rn(m[d], nn);
    for (int i = l; i <= r; i++)
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const double e = __dsub_rn(s.v[d][o[d][i]], m[d]);
            q[d] = __fma_rn(e, e, q[d]);
        }
    int dim = 0;
    double mx = q[0];
    if (q[1] > mx) {
        mx = q[1];
        dim = 1;
    }
    if (q[2] > mx) dim = 2;
    return dim;
}

__global__ void __launch_bounds__(kSubThreads) k_subtrees(Segs sg, const int *__restrict__ a0,
                                                         const int *__restrict__ a1,
                                                         const int *__restrict__ a2, UniqueArrays u,
                                                         TreeOut t, int *place, int *err)
{
    extern __shared__ __align__(16) unsigned char smem[];
    SubSmem &s = *reinterpret_cast<SubSmem *>(smem);
    constexpr unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, b = blockIdx.x;
    if (b >= *sg.count) return;
    const int base = sg.l[b], m = sg.r[b] - base + 1;
    const long long root = sg.p[b];
    if (m < 1) return;
    if (m > kSubCap) {
        if (tid == 0) set_err(err, KD_EINTERNAL);
        return;
    }
    // places: positions in order 0; the other orders through the point's place
    for (int i = tid; i < m; i += kSubThreads) {
        const int pt = a0[base + i];
        s.fw[i] = (uint32_t)u.ufield[pt] | ((uint32_t)u.uw[pt] << 8);
        s.rep[i] = u.urep[pt];
        s.o[0][0][i] = (unsigned short)i;
        place[pt] = i;
        s.v[0][i] = u.ux[pt];
        s.v[1][i] = u.uy[pt];
        s.v[2][i] = u.uz[pt];
        s.seg[0][i] = 0;
    }
    if (tid == 0) {
        s.l[0][0] = 0;
        s.r[0][0] = (short)(m - 1);
    }
    __syncthreads();  // (place[] of this segment's points is written by this CTA alone)
    for (int i = tid; i < m; i += kSubThreads) {
        const int p1 = place[a1[base + i]], p2 = place[a2[base + i]];
        if ((unsigned)p1 >= (unsigned)m || (unsigned)p2 >= (unsigned)m) set_err(err, KD_EINTERNAL);
        s.o[0][1][i] = (unsigned short)min(max(p1, 0), m - 1);
        s.o[0][2][i] = (unsigned short)min(max(p2, 0), m - 1);
    }
    __syncthreads();
    const int words = (m + 31) / 32;
    auto node = [&](int hp, int pl, int dim, int hl, int hr, int pos) {
        if (hp >= t.memsize) {
            set_err(err, KD_EINTERNAL);
            return;
        }
        NodeRec rec;
        rec.v[0] = s.v[0][pl];
        rec.v[1] = s.v[1][pl];
        rec.v[2] = s.v[2][pl];
        rec.fw = s.fw[pl];
        rec.pad0 = 0;
        rec.flags = (uint32_t)hl | ((uint32_t)hr << 1) | ((uint32_t)dim << 2);
        rec.pad1 = 0;
        t.nodes[hp] = rec;
        t.inorder_rep[base + pos] = s.rep[pl];
    };
    int cur = 0;
    for (int lev = 0;; lev++) {
        const int nseg = 1 << lev;
        const short *const L = s.l[cur], *const R = s.r[cur];
        auto &o = s.o[cur];
        auto &o2 = s.o[cur ^ 1];
        // ---- split dimensions: a warp per large segment, a thread per small one
        if ((m >> lev) > kSubSeq) {
            for (int g = w; g < nseg; g += kSubThreads / 32) {
                const int l = L[g], r = R[g], n = r - l + 1;
                if (n <= kSubSeq) continue;
                double a[9];
#pragma unroll
                for (int k = 0; k < 9; k++) a[k] = 0.0;
                for (int i = l + lane; i <= r; i += 32)
#pragma unroll
                    for (int d = 0; d < 3; d++) {
                        const double v = s.v[d][o[0][i]];  // (the sums' order is free)
                        a[d] += v;
                        a[3 + d] += fabs(v);
                    }
#pragma unroll
                for (int k = 0; k < 6; k++)
#pragma unroll
                    for (int f = 16; f; f >>= 1) a[k] += __shfl_xor_sync(FULL, a[k], f);
                const double mu[3] = {a[0] / (double)n, a[1] / (double)n, a[2] / (double)n};
                for (int i = l + lane; i <= r; i += 32)
#pragma unroll
                    for (int d = 0; d < 3; d++) {
                        const double e = s.v[d][o[0][i]] - mu[d];
                        a[6 + d] += e * e;
                    }
#pragma unroll
                for (int k = 6; k < 9; k++)
#pragma unroll
                    for (int f = 16; f; f >>= 1) a[k] += __shfl_xor_sync(FULL, a[k], f);
                int c = decide_dim((double)n, a);
                if (c < 0 && lane == 0) c = sub_var_seq(s, o, l, r);
                if (lane == 0) s.tdim[g] = (unsigned char)c;
            }
        }
        for (int g = tid; g < nseg; g += kSubThreads) {
            const int l = L[g], r = R[g], n = r - l + 1;
            if (n >= 4 && n <= kSubSeq) s.tdim[g] = (unsigned char)sub_var_seq(s, o, l, r);
        }
        __syncthreads();
        // ---- the level's nodes, from shared memory (with their points gathered
        // here, by the few threads that hold a segment, the kernel took a third
        // more: 1.9 ms at 5M points instead of 1.6)
        for (int g = tid; g < nseg; g += kSubThreads) {
            const int l = L[g], r = R[g], n = r - l + 1;
            const int p = (int)((root << lev) + g);
            if (n >= 4) {
                const int med = (l + r + 1) / 2, d = s.tdim[g];
                node(p, o[d][med], d, 1, 1, med);
            } else if (n == 3) {
                node(p, o[0][l + 1], 0, 1, 1, l + 1);
                node(2 * p, o[0][l], 0, 0, 0, l);
                node(2 * p + 1, o[0][r], 0, 0, 0, r);
            } else if (n == 2) {
                node(p, o[0][r], 0, 1, 0, r);
                node(2 * p, o[0][l], 0, 0, 0, l);
            } else if (n == 1) {
                node(p, o[0][l], 0, 0, 0, l);
            }
        }
        if ((m >> lev) < 4) break;  // every segment was a base case
        // ---- sides of the points of splitting segments
        for (int i = tid; i < m; i += kSubThreads) {
            const int g = s.seg[cur][i];
            if (g < 0) continue;
            const int l = L[g], r = R[g];
            if (r - l + 1 < 4) continue;
            const int med = (l + r + 1) / 2;
            s.side[o[s.tdim[g]][i]] = i < med ? 0 : (i == med ? 2 : 1);
        }
        __syncthreads();
        // ---- stable partition: prefix counts of left and right points along
        // each order, then the move
        for (int x = w; x < 3 * words; x += kSubThreads / 32) {
            const int d = x / words, wd = x % words, i = 32 * wd + lane;
            int sd = 3;
            if (i < m) {
                const int g = s.seg[cur][i];
                if (g >= 0 && R[g] - L[g] + 1 >= 4) sd = s.side[o[d][i]];
            }
            const unsigned ml = __ballot_sync(FULL, sd == 0), mr = __ballot_sync(FULL, sd == 1);
            if (lane == 0) {
                s.mask[d][0][wd] = ml;
                s.mask[d][1][wd] = mr;
            }
        }
        __syncthreads();
        if (w < 6) {
            static_assert(kSubCap / 32 <= 32, "one lane per word");
            const int c = lane < words ? __popc(s.mask[w / 2][w % 2][lane]) : 0;
            int inc = c;
#pragma unroll
            for (int f = 1; f < 32; f <<= 1) {
                const int v = __shfl_up_sync(FULL, inc, f);
                if (lane >= f) inc += v;
            }
            if (lane < words) s.pre[w / 2][w % 2][lane] = (unsigned short)(inc - c);
        }
        __syncthreads();
        for (int i = tid; i < m; i += kSubThreads) {
            const int g = s.seg[cur][i];
            int ng = -1;
            if (g >= 0) {
                const int l = L[g], r = R[g], med = (l + r + 1) / 2;
                if (r - l + 1 >= 4) {
#pragma unroll
                    for (int d = 0; d < 3; d++) {
                        const int pl = o[d][i], sd = s.side[pl];
                        int dst = med;
                        if (sd != 2) {
                            const unsigned *mk = s.mask[d][sd];
                            const unsigned short *pr = s.pre[d][sd];
                            const int at = pr[i >> 5] + __popc(mk[i >> 5] & ((1u << (i & 31)) - 1u)),
                                      from = pr[l >> 5] + __popc(mk[l >> 5] & ((1u << (l & 31)) - 1u));
                            dst = (sd == 0 ? l : med + 1) + at - from;
                        }
                        if (dst < l || dst > r) {
                            set_err(err, KD_EINTERNAL);
                            dst = i;
                        }
                        o2[d][dst] = (unsigned short)pl;
                    }
                    if (i != med) ng = 2 * g + (i > med);
                }
            }
            s.seg[cur ^ 1][i] = (short)ng;
        }
        for (int g = tid; g < nseg; g += kSubThreads) {
            const int l = L[g], r = R[g], med = (l + r + 1) / 2;
            const bool split = r - l + 1 >= 4;
            s.l[cur ^ 1][2 * g] = (short)(split ? l : 0);
            s.r[cur ^ 1][2 * g] = (short)(split ? med - 1 : -1);
            s.l[cur ^ 1][2 * g + 1] = (short)(split ? med + 1 : 0);
            s.r[cur ^ 1][2 * g + 1] = (short)(split ? r : -1);
        }
        __syncthreads();
        cur ^= 1;
    }
}

// ------------------------------------------------------------ counting layout

// The counting order.  Raw points go by cells of at most kChunk points: of a
// tree's, the cells of its own splits at the depth where they have become that
// small (they are boxes that tile the points' cloud, whatever its shape); of
// query points that have no tree, stretches of a Hilbert curve.  Within a cell
// they are split in the middle again and again (k_refine).  A cell's points are
// then cut every KD_RUN_MAX into leaves (each grouped by tree field into runs)
// and every KD_BLOCK_MAX into query blocks, so that a block is two leaves and a
// symmetric count's runs never straddle one; only a cell's last leaf and block
// are partly filled.
// Against leaves by the tree's own depth (32 to 64 points each, and blocks cut
// across them at the ends of 16-leaf subtrees), in the tile kernel: 3M uniform
// points with themselves in 21 edges 7.6 -> 5.8 ms, 5M on the sky in 16 edges
// 13.9 -> 11.2, 1M + 1M on a grid in 30 edges 25.9 -> 21.9; the layout of 5M
// points 2.8 -> 1.9 ms.  Curves instead of the tree's cells, without splits and
// with: 7.4 and 6.2 ms, 18.4 and 15.0, 25.8 and 23.1 (a curve leaves and enters
// a surface again, far away).  Leaves of 32 points: 6.5 ms for the first, but
// 647 instead of 572 ms for 1M / 20M points in edges spread over two decades.

template <class T>
__global__ void k_gather(const T *__restrict__ src, const int *__restrict__ idx, int n, T *dst)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        dst[i] = src[idx[i]];
}

// The bits of v (21 of them) three apart.
__device__ __forceinline__ uint64_t spread3(uint64_t v)
{
    v = (v | (v << 32)) & 0x001f00000000ffffull;
    v = (v | (v << 16)) & 0x001f0000ff0000ffull;
    v = (v | (v << 8)) & 0x100f00f00f00f00full;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
    return (v | (v << 2)) & 0x1249249249249249ull;
}

// Position along the Hilbert curve of 2^21 cells per side, three bits a level,
// by the transform of Skilling (AIP Conf. Proc. 707, 381, 2004): from the
// coarsest level down, each axis exchanges or inverts the finer bits of the
// first one, and a Gray code orders the eight cells of a level.
__device__ __forceinline__ uint64_t hilbert(unsigned (&c)[3])
{
#pragma unroll 1
    for (unsigned bit = 1u << 20; bit > 1; bit >>= 1) {
        const unsigned finer = bit - 1;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const unsigned swap = (c[d] & bit) ? 0u : (c[0] ^ c[d]) & finer;
            c[0] ^= (c[d] & bit) ? finer : swap;
            if (d) c[d] ^= swap;
        }
    }
    c[1] ^= c[0];
    c[2] ^= c[1];
    unsigned flip = c[2] >> 1;  // bit b: parity of the bits of c[2] above b
    flip ^= flip >> 1;
    flip ^= flip >> 2;
    flip ^= flip >> 4;
    flip ^= flip >> 8;
    flip ^= flip >> 16;
    return spread3(c[0] ^ flip) << 2 | spread3(c[1] ^ flip) << 1 | spread3(c[2] ^ flip);
}

// Position of each point along the curve through the points' cube (key), or
// its 32 highest bits (key32), and, with fi, the range of the own fields.
__global__ void __launch_bounds__(TPB) k_curve(const double *__restrict__ xyz, const int *__restrict__ fin,
                                               int n, const KeySpan *span, uint64_t *key, unsigned *key32,
                                               int *iota, FieldInfo *fi)
{
    double lo[3], ext = 0.0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        lo[d] = okey_value(~span->inv_lo[d]);
        ext = fmax(ext, okey_value(span->hi[d]) - lo[d]);
    }
    const double top = 2097151.0, scale = ext > 0.0 ? top / ext : 0.0;
    int minq = 0x7fffffff, maxq = -0x7fffffff;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        unsigned c[3];
#pragma unroll
        for (int d = 0; d < 3; d++)  // (NaN, from an infinite range: the last cell)
            c[d] = __double2uint_rd(fmin((xyz[3 * (size_t)i + d] - lo[d]) * scale, top));
        const uint64_t k = hilbert(c);
        if (key) key[i] = k;
        else key32[i] = (unsigned)(k >> 31);
        iota[i] = i;
        const int qf = fin ? fin[i] : 0;
        minq = min(minq, qf);
        maxq = max(maxq, qf);
    }
    if (!fi) return;
    minq = __reduce_min_sync(0xffffffffu, minq);
    maxq = __reduce_max_sync(0xffffffffu, maxq);
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&fi->min_qf, minq);
        atomicMax(&fi->max_qf, maxq);
    }
}

// Points of a run of more than kCellMax equal keys whose places differ.
constexpr int kCellMax = 512;
template <class K>
__global__ void k_full_cells(const K *__restrict__ srt, const int *__restrict__ perm,
                             const double *__restrict__ xyz, int n, int *full)
{
    int c = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x + kCellMax; i < n; i += gridDim.x * blockDim.x) {
        if (srt[i] != srt[i - kCellMax]) continue;
        const size_t a = perm[i], b = perm[i - kCellMax];
        c += xyz[3 * a] != xyz[3 * b] || xyz[3 * a + 1] != xyz[3 * b + 1] || xyz[3 * a + 2] != xyz[3 * b + 2];
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if (c && (threadIdx.x & 31) == 0) atomicAdd(full, c);
}

// A tree's cells: cell c holds places [start[c], start[c + 1]) of the order and
// owns 2^leaf_bits leaves, the last of them empty.
struct Cells {
    const int *start;
    int bits, leaf_bits;  // 2^bits cells
};

// The order within a cell, every kChunk points at a time: split in the middle
// along the longest side of their box, and so on down to kCut points, so that
// leaves, query tiles and halves of each are boxes that hardly overlap.  One
// CTA per chunk: keys of 20 bits of the coordinate within the segment's box
// and the point's place, sorted in every segment at once by a bitonic network
// (registers, then lanes, then shared memory); positions behind the last point
// sort last.  Bound by the latency of the network's steps and barriers.  Chunks
// (and cells) of 4096 points made the counts of large catalogs 1 to 2% faster
// (fewer partly filled leaves) and a call with 1000 points 7% slower; of 1024,
// neither.  5M points: 0.8 ms.
constexpr int kChunk = 2048;
constexpr int kCut = 16;
constexpr int kRefThreads = kChunk / 4;  // thread t: positions 4 t .. 4 t + 3
constexpr int kRefWarps = kRefThreads / 32;
struct RefineSmem {
    double v[3][kChunk];
    double box[kRefWarps][6];
    unsigned key[kChunk];
};
__global__ void __launch_bounds__(kRefThreads) k_refine(int n, const double *__restrict__ xyz, Cells cells,
                                                        const int *__restrict__ in, int *__restrict__ out)
{
    extern __shared__ __align__(16) unsigned char ref_smem[];
    RefineSmem &s = *reinterpret_cast<RefineSmem *>(ref_smem);
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int kIdBits = 12, kIdMask = (1 << kIdBits) - 1;
    static_assert(kChunk <= 1 << kIdBits && kRefWarps <= 32, "ids in a key, a lane per warp's box");
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    long long base = (long long)blockIdx.x * kChunk, end = n;
    if (cells.start) {
        const int per = max(1, (KD_RUN_MAX << cells.leaf_bits) / kChunk);  // chunks per cell
        base = cells.start[blockIdx.x / per] + (long long)(blockIdx.x % per) * kChunk;
        end = cells.start[blockIdx.x / per + 1];
    }
    const int m = (int)min((long long)kChunk, end - base);
    if (m <= 0) return;
    for (int i = t; i < m; i += kRefThreads) {
        const size_t p = in[base + i];
#pragma unroll
        for (int d = 0; d < 3; d++) s.v[d][i] = xyz[3 * p + d];
    }
    unsigned key[4];
#pragma unroll
    for (int k = 0; k < 4; k++) key[k] = 4 * t + k;
    int first = kChunk;
    while (first > kCut && first / 2 >= m) first /= 2;
    __syncthreads();
    for (int seg = first; seg > kCut; seg >>= 1) {
        // ---- the segments' boxes
        double lo[3], hi[3];
#pragma unroll
        for (int d = 0; d < 3; d++) lo[d] = INFINITY, hi[d] = -INFINITY;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int id = key[k] & kIdMask;
            if (id < m)
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    lo[d] = fmin(lo[d], s.v[d][id]);
                    hi[d] = fmax(hi[d], s.v[d][id]);
                }
        }
        for (int f = 1; f < min(32, seg / 4); f <<= 1)
#pragma unroll
            for (int d = 0; d < 3; d++) {
                lo[d] = fmin(lo[d], __shfl_xor_sync(FULL, lo[d], f));
                hi[d] = fmax(hi[d], __shfl_xor_sync(FULL, hi[d], f));
            }
        if (seg > 128) {  // several warps per segment
            if (lane == 0)
#pragma unroll
                for (int d = 0; d < 3; d++) s.box[w][d] = lo[d], s.box[w][3 + d] = hi[d];
            __syncthreads();
            const int nw = seg / 128, w0 = w & ~(nw - 1);
            const double *const b = s.box[w0 + (lane & (nw - 1))];
#pragma unroll
            for (int d = 0; d < 3; d++) lo[d] = b[d], hi[d] = b[3 + d];
            for (int f = 1; f < nw; f <<= 1)
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    lo[d] = fmin(lo[d], __shfl_xor_sync(FULL, lo[d], f));
                    hi[d] = fmax(hi[d], __shfl_xor_sync(FULL, hi[d], f));
                }
        }
        // ---- keys along the longest side (a side of infinite length first)
        const double ex = hi[0] - lo[0], ey = hi[1] - lo[1], ez = hi[2] - lo[2];
        const int dim = ex >= ey && ex >= ez ? 0 : (ey >= ez ? 1 : 2);
        const double ext = dim == 0 ? ex : (dim == 1 ? ey : ez), low = dim == 0 ? lo[0] : (dim == 1 ? lo[1] : lo[2]);
        const double top = (double)((1 << (32 - kIdBits)) - 2), scale = ext > 0.0 ? top / ext : 0.0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int id = key[k] & kIdMask;
            unsigned q = (1u << (32 - kIdBits)) - 1u;
            if (id < m) q = __double2uint_rd(fmin((s.v[dim][id] - low) * scale, top));
            key[k] = q << kIdBits | (unsigned)id;
        }
        // ---- sort every segment
        auto swap_if = [&](unsigned &a, unsigned &b, bool up) {  // a before b
            const unsigned x = min(a, b), y = max(a, b);
            a = up ? x : y;
            b = up ? y : x;
        };
        for (int k = 2; k <= seg; k <<= 1) {
            // direction of this thread's elements (k >= 4: one for all four)
            const bool up = k == seg || !((4 * t) & k);
            int j = k >> 1;
            for (; j >= 128; j >>= 1) {
                __syncthreads();
                *reinterpret_cast<uint4 *>(s.key + 4 * t) = make_uint4(key[0], key[1], key[2], key[3]);
                __syncthreads();
                const uint4 o = *reinterpret_cast<const uint4 *>(s.key + ((4 * t) ^ j));
                const bool low_half = !((4 * t) & j), take_min = low_half == up;
                key[0] = take_min ? min(key[0], o.x) : max(key[0], o.x);
                key[1] = take_min ? min(key[1], o.y) : max(key[1], o.y);
                key[2] = take_min ? min(key[2], o.z) : max(key[2], o.z);
                key[3] = take_min ? min(key[3], o.w) : max(key[3], o.w);
            }
            for (; j >= 4; j >>= 1) {
                const bool low_half = !((4 * t) & j), take_min = low_half == up;
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const unsigned o = __shfl_xor_sync(FULL, key[e], j >> 2);
                    key[e] = take_min ? min(key[e], o) : max(key[e], o);
                }
            }
            if (j == 2) {
                swap_if(key[0], key[2], up);
                swap_if(key[1], key[3], up);
                j = 1;
            }
            if (k == 2) {
                swap_if(key[0], key[1], true);
                swap_if(key[2], key[3], false);
            } else {
                swap_if(key[0], key[1], up);
                swap_if(key[2], key[3], up);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (4 * t + k < m) out[base + 4 * t + k] = in[base + (key[k] & kIdMask)];
}

// For points that the curve's cells do not resolve: the rank of each point's
// coordinates among their values, in place of the coordinates.
__global__ void k_value_heads(const uint64_t *__restrict__ key, const int *__restrict__ ord, int n, int *head)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        head[i] = i == 0 || key[ord[i]] != key[ord[i - 1]];
}

__global__ void k_scatter_rank(const int *__restrict__ cls, const int *__restrict__ ord, int n, int *rank)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        rank[ord[i]] = cls[i] - 1;
}

__global__ void k_curve_ranks(const int *__restrict__ rx, const int *__restrict__ ry,
                              const int *__restrict__ rz, int n, uint64_t *key)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int r[3] = {rx[i], ry[i], rz[i]};
        unsigned c[3];
#pragma unroll
        for (int d = 0; d < 3; d++) c[d] = (unsigned)(((unsigned long long)r[d] << 21) / (unsigned)n);
        key[i] = hilbert(c);
    }
}

// The cell (node of depth `bits`) of the point at every in-order position, by
// its input index.  A point above the cells lies on a split plane: it goes by
// the splits below its left child.
__global__ void k_cell_of(int n_u, int bits, const NodeRec *__restrict__ nodes,
                          const int *__restrict__ inorder_rep, int *cell)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_u; i += gridDim.x * blockDim.x) {
        int l = 0, r = n_u - 1, h = 1;
        for (int b = 0; b < bits; b++) {
            const int med = (l + r + 1) / 2;  // (the ranges do not depend on the data)
            if (i == med) {
                const double v[3] = {nodes[h].v[0], nodes[h].v[1], nodes[h].v[2]};
                for (h *= 2; ++b < bits;) {
                    const int d = (nodes[h].flags >> 2) & 3;
                    h = 2 * h + ((d == 0 ? v[0] : (d == 1 ? v[1] : v[2])) > nodes[h].v[d]);
                }
                break;
            }
            h = 2 * h + (i > med);
            if (i > med) l = med + 1;
            else r = med - 1;
        }
        cell[inorder_rep[i]] = h - (1 << bits);
    }
}

__global__ void k_cell_keys(int n, const int *__restrict__ p, const int *__restrict__ cls,
                            const int *__restrict__ urep, const int *__restrict__ cell, unsigned *key)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        key[i] = (unsigned)cell[urep[cls[i] - 1]];
}

// cells' first places (no cell is empty); key: sorted cells, null for one cell
__global__ void k_cell_starts(int n, int ncells, const unsigned *__restrict__ key, int *start)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        start[0] = 0;
        start[ncells] = n;
    }
    if (!key) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x + 1; i < n; i += gridDim.x * blockDim.x)
        if (key[i] != key[i - 1]) start[key[i]] = i;
}

__global__ void k_cell_max(int ncells, const int *__restrict__ start, int *largest)
{
    int m = 0;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncells; c += gridDim.x * blockDim.x)
        m = max(m, start[c + 1] - start[c]);
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) atomicMax(largest, m);
}

// cells of kChunk places each, empty ones behind the last point
__global__ void k_even_cells(int n, int ncells, int *start)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c <= ncells) start[c] = (int)min((long long)n, (long long)c * kChunk);
}

struct RawOut {
    double *x, *y, *z;
    int *qf, *tf;
};

struct Summ {
    double *box;
    int *count, *tf;
};

struct LeafOut {
    RawOut o;
    Summ sm;
    int *qf;        // single own field of the leaf, -1 when mixed
    kd_leaf *leaf;  // leaf boxes as the tile kernel reads them
    float4 *t4;     // each point in FP32 relative to its leaf's centre
    int *pos, *nruns, *blocks;  // blocks: query blocks per pair of leaves
    unsigned long long *hdiag;
};

constexpr int kBlockLeaves = KD_BLOCK_MAX / KD_RUN_MAX;
static_assert(KD_BLOCK_MAX == kBlockLeaves * KD_RUN_MAX, "blocks are whole leaves");

// One warp per leaf: its points, gathered and grouped by tree field, its box
// and summary.  tf: tree field per input point, null where it is the own field.
__global__ void __launch_bounds__(TPB) k_leaves(int n, int nleaves, Cells cells, const int *__restrict__ perm,
                                                const double *__restrict__ xyz, const int *__restrict__ fin,
                                                const int *__restrict__ tfin, LeafOut out)
{
    constexpr int PL = KD_RUN_MAX / 32;  // points per lane
    constexpr unsigned FULL = 0xffffffffu;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w > nleaves) return;
    int a = n, len = 0;
    if (w < nleaves) {
        const int c = w >> cells.leaf_bits, end = cells.start[c + 1];
        a = min(end, cells.start[c] + (w - (c << cells.leaf_bits)) * KD_RUN_MAX);
        len = min(end - a, KD_RUN_MAX);
    }
    if (lane == 0) {
        out.pos[w] = a;
        if (w % kBlockLeaves == 0 || w == nleaves) out.blocks[(w + kBlockLeaves - 1) / kBlockLeaves] = len > 0;
        if (w == nleaves) out.nruns[w] = 0;
    }
    if (w == nleaves) return;
    double v[PL][3], lo[3], hi[3];
    int qf[PL], tf[PL], rank[PL];
#pragma unroll
    for (int d = 0; d < 3; d++) lo[d] = INFINITY, hi[d] = -INFINITY;
#pragma unroll
    for (int k = 0; k < PL; k++) {
        qf[k] = tf[k] = 0;
        rank[k] = lane + 32 * k;
        if (lane + 32 * k < len) {
            const size_t p = perm[a + lane + 32 * k];
#pragma unroll
            for (int d = 0; d < 3; d++) {
                v[k][d] = xyz[3 * p + d];
                lo[d] = fmin(lo[d], v[k][d]);
                hi[d] = fmax(hi[d], v[k][d]);
            }
            if (fin) qf[k] = fin[p];
            tf[k] = tfin ? tfin[p] : qf[k];
        }
    }
    const int tf0 = __shfl_sync(FULL, tf[0], 0), qf0 = __shfl_sync(FULL, qf[0], 0);
    bool tmix = false, qmix = false;
#pragma unroll
    for (int k = 0; k < PL; k++)
        if (lane + 32 * k < len) {
            tmix = tmix || tf[k] != tf0;
            qmix = qmix || qf[k] != qf0;
        }
    tmix = __any_sync(FULL, tmix);
    qmix = __any_sync(FULL, qmix);
    int runs = len > 0 ? 1 : 0;
    if (tmix) {  // stable order by tree field, and the number of fields
        bool first[PL];
#pragma unroll
        for (int k = 0; k < PL; k++) {
            first[k] = lane + 32 * k < len;
            rank[k] = 0;
        }
#pragma unroll
        for (int m = 0; m < PL; m++)
            for (int j = 0; j < 32; j++) {
                const int at = 32 * m + j, other = __shfl_sync(FULL, tf[m], j);
                if (at >= len) break;
#pragma unroll
                for (int k = 0; k < PL; k++) {
                    const bool before = at < lane + 32 * k;
                    rank[k] += other < tf[k] || (other == tf[k] && before);
                    first[k] = first[k] && !(other == tf[k] && before);
                }
            }
        runs = 0;
#pragma unroll
        for (int k = 0; k < PL; k++) runs += __popc(__ballot_sync(FULL, first[k]));
    }
#pragma unroll
    for (int f = 16; f; f >>= 1)
#pragma unroll
        for (int d = 0; d < 3; d++) {
            lo[d] = fmin(lo[d], __shfl_xor_sync(FULL, lo[d], f));
            hi[d] = fmax(hi[d], __shfl_xor_sync(FULL, hi[d], f));
        }
    double c[3];
#pragma unroll
    for (int d = 0; d < 3; d++) c[d] = 0.5 * (lo[d] + hi[d]);
#pragma unroll
    for (int k = 0; k < PL; k++)
        if (lane + 32 * k < len) {
            const size_t i = (size_t)a + rank[k];
            out.o.x[i] = v[k][0];
            out.o.y[i] = v[k][1];
            out.o.z[i] = v[k][2];
            out.o.qf[i] = qf[k];
            if (tfin) out.o.tf[i] = tf[k];
            out.t4[i] = make_float4(-2.0f * (float)(v[k][0] - c[0]), -2.0f * (float)(v[k][1] - c[1]),
                                    -2.0f * (float)(v[k][2] - c[2]), 0.0f);
        }
    if (lane == 0) {
        const size_t h = (size_t)nleaves + w;
        double hx[3];
        kd_leaf l;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            out.sm.box[6 * h + d] = lo[d];
            out.sm.box[6 * h + 3 + d] = hi[d];
            hx[d] = fmax(hi[d] - c[d], c[d] - lo[d]);
            l.c[d] = c[d];
            l.h[d] = __double2float_ru(hx[d]);
            l.pad_[d] = 0.0f;
        }
        out.leaf[w] = l;
        out.sm.count[h] = len > 0 ? len : 0;
        out.sm.tf[h] = tmix ? -1 : tf0;
        out.qf[w] = qmix ? -1 : qf0;
        out.nruns[w] = runs;
        if (len > 0)
            atomicMax(out.hdiag, (unsigned long long)__double_as_longlong(
                                     sqrt(hx[0] * hx[0] + hx[1] * hx[1] + hx[2] * hx[2])));
    }
}

// one warp per leaf: its runs, one per tree field
__global__ void __launch_bounds__(TPB) k_leaf_runs(int nleaves, const int *__restrict__ pos,
                                                   const int *__restrict__ tf,
                                                   const int *__restrict__ leaf_run, int *run_start,
                                                   int *run_len, int *run_tf)
{
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= nleaves) return;
    const int a = pos[w], len = pos[w + 1] - a;
    constexpr int PL = KD_RUN_MAX / 32;
    unsigned long long all = 0;
    int f[PL];
#pragma unroll
    for (int k = 0; k < PL; k++) {
        const int i = lane + 32 * k;
        bool hd = false;
        f[k] = 0;
        if (i < len) {
            f[k] = tf[a + i];
            hd = i == 0 || f[k] != tf[a + i - 1];
        }
        all |= (unsigned long long)__ballot_sync(0xffffffffu, hd) << (32 * k);
    }
#pragma unroll
    for (int k = 0; k < PL; k++) {
        const int i = lane + 32 * k;
        if (!((all >> i) & 1)) continue;
        const int r = leaf_run[w] + __popcll(all & ((1ull << i) - 1));
        const unsigned long long later = i < 63 ? all >> (i + 1) : 0;
        run_start[r] = a + i;
        run_len[r] = later ? __ffsll((long long)later) : len - i;
        run_tf[r] = f[k];
    }
}

// Summaries of the levels [max(0, d0 - 8), d0), one CTA per subtree of the
// lowest of them.  Empty leaves (at the end) leave their parent to its sibling.
// leaf, where d0 is the leaves' level: also the number of leaves below 1/64 of
// the largest half-diagonal.
__global__ void __launch_bounds__(TPB) k_internal_summary(int d0, Summ sm, const kd_leaf *__restrict__ leaf,
                                                          const double *hdiag, int *small)
{
    const int top = max(0, d0 - 8);
    static_assert(TPB >= 128, "a thread per node of the first level");
    if (leaf) {  // (every thread one of the CTA's up to 256 leaves)
        static_assert(TPB >= 256, "a thread per leaf");
        const int per = 1 << (d0 - top), l = blockIdx.x * per + threadIdx.x;
        bool below = false;
        if ((int)threadIdx.x < per && sm.count[((size_t)1 << d0) + l] > 0)
            below = !(leaf[l].h[0] + leaf[l].h[1] + leaf[l].h[2] >= (float)(*hdiag / 64));
        const int n = __syncthreads_count(below);
        if (threadIdx.x == 0 && n) atomicAdd(small, n);
    }
    for (int d = d0 - 1; d >= top; d--) {
        const int cnt = 1 << (d - top);
        if ((int)threadIdx.x < cnt) {
            const size_t h = ((size_t)1 << d) + (size_t)blockIdx.x * cnt + threadIdx.x, a = 2 * h, b = 2 * h + 1;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                sm.box[6 * h + k] = fmin(sm.box[6 * a + k], sm.box[6 * b + k]);
                sm.box[6 * h + 3 + k] = fmax(sm.box[6 * a + 3 + k], sm.box[6 * b + 3 + k]);
            }
            const int nb = sm.count[b];
            sm.count[h] = sm.count[a] + nb;
            sm.tf[h] = nb == 0 || sm.tf[a] == sm.tf[b] ? sm.tf[a] : (sm.count[a] == 0 ? sm.tf[b] : -1);
        }
        __syncthreads();
    }
}

// query blocks of a tree: kBlockLeaves leaves each, where they hold a point
__global__ void k_tree_blocks(int groups, int nleaves, const int *__restrict__ pos,
                              const int *__restrict__ off, const double *__restrict__ box,
                              const int *__restrict__ leaf_qf, int *bstart, int *blen, double *bbox, int *bqf)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= groups) return;
    const int l0 = kBlockLeaves * p, l1 = min(nleaves, l0 + kBlockLeaves);
    const int start = pos[l0], len = pos[l1] - start, b = off[p];
    if (len <= 0) return;
    double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    int q = leaf_qf[l0];
    for (int l = l0; l < l1 && pos[l] < pos[l + 1]; l++) {
        const double *x = box + 6 * ((size_t)nleaves + l);
#pragma unroll
        for (int d = 0; d < 3; d++) {
            lo[d] = fmin(lo[d], x[d]);
            hi[d] = fmax(hi[d], x[3 + d]);
        }
        if (leaf_qf[l] != q) q = -1;
    }
#pragma unroll
    for (int d = 0; d < 3; d++) {
        bbox[6 * (size_t)b + d] = lo[d];
        bbox[6 * (size_t)b + 3 + d] = hi[d];
    }
    bstart[b] = start;
    blen[b] = len;
    bqf[b] = q;
}

// tree field of every input point: its coordinates' first occurrence's
__global__ void k_tree_fields(int n, const int *__restrict__ p, const int *__restrict__ cls,
                              const int *__restrict__ ufield, int *tf)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        tf[p[i]] = ufield[cls[i] - 1];
}

// one CTA of KD_BLOCK_MAX threads per query block: box and single own field;
// many, if given: warps with more than KD_MANY_FIELDS own fields
__global__ void __launch_bounds__(KD_BLOCK_MAX) k_block_boxes(int nblocks, const int *bstart,
                                                             const int *blen, RawOut o,
                                                             double *bbox, int *bqf, int *many)
{
    constexpr int W = KD_BLOCK_MAX / 32;
    __shared__ double sw[W][6];
    __shared__ int sq[W];
    int b = blockIdx.x;
    if (b >= nblocks) return;
    int t = threadIdx.x, w = t >> 5, lane = t & 31;
    int len = blen[b], s = bstart[b];
    bool valid = t < len;
    double lo[3], hi[3];
    int qf = valid ? o.qf[s + t] : 0x7fffffff;
    for (int d = 0; d < 3; d++) {
        double v = valid ? (d == 0 ? o.x[s + t] : (d == 1 ? o.y[s + t] : o.z[s + t])) : 0.0;
        lo[d] = valid ? v : INFINITY;
        hi[d] = valid ? v : -INFINITY;
    }
    int q0 = __shfl_sync(0xffffffffu, qf, 0);
    int mixed = valid && qf != q0;
    if (many) {
        const unsigned peers = __match_any_sync(0xffffffffu, qf);
        const unsigned fields = __ballot_sync(0xffffffffu, valid && lane == __ffs(peers) - 1);
        if (lane == 0 && __popc(fields) > KD_MANY_FIELDS) atomicAdd(many, 1);
    }
    for (int off = 16; off; off >>= 1)
        for (int d = 0; d < 3; d++) {
            lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], off));
            hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], off));
        }
    mixed = __any_sync(0xffffffffu, mixed);
    if (lane == 0) {
        for (int d = 0; d < 3; d++) {
            sw[w][d] = lo[d];
            sw[w][3 + d] = hi[d];
        }
        sq[w] = (32 * w >= len) ? -2 : (mixed ? -1 : q0);
    }
    __syncthreads();
    if (t == 0) {
        double L[3] = {INFINITY, INFINITY, INFINITY}, H[3] = {-INFINITY, -INFINITY, -INFINITY};
        int q = -2;
        for (int k = 0; k < W; k++) {
            for (int d = 0; d < 3; d++) {
                L[d] = fmin(L[d], sw[k][d]);
                H[d] = fmax(H[d], sw[k][3 + d]);
            }
            if (sq[k] == -2) continue;
            if (sq[k] == -1 || (q != -2 && q != sq[k])) q = -1;
            else if (q == -2) q = sq[k];
        }
        for (int d = 0; d < 3; d++) {
            bbox[6 * (size_t)b + d] = L[d];
            bbox[6 * (size_t)b + 3 + d] = H[d];
        }
        bqf[b] = q < 0 ? -1 : q;
    }
}

// ------------------------------------------------------------ helpers

// Stable radix sort of (key, value) pairs by key bits [b0, b1) and device
// scans: the project's own (kd_sort.cuh), temporaries from the call's pool.
// Keys are unsigned or non-negative.
template <class K, class V>
static void sort_pairs(Pool &pool, cudaStream_t s, const K *kin, K *kout, const V *vin, V *vout,
                       int n, int b0, int b1)
{
    char *tmp = pool.alloc<char>(sort::sort_temp_bytes<K, V>(n));
    check(sort::sort_pairs<K, V>(tmp, kin, kout, vin, vout, n, b0, b1, s), "radix sort");
}

template <class T>
static void excl_sum(Pool &pool, cudaStream_t s, const T *in, T *out, int n)
{
    char *tmp = pool.alloc<char>(sort::scan_temp_bytes<T>(n));
    check(sort::scan<T, sort::SumOp, false>(tmp, in, out, n, sort::SumOp(), s), "scan");
}

template <class T>
static void incl_sum(Pool &pool, cudaStream_t s, const T *in, T *out, int n)
{
    char *tmp = pool.alloc<char>(sort::scan_temp_bytes<T>(n));
    check(sort::scan<T, sort::SumOp, true>(tmp, in, out, n, sort::SumOp(), s), "scan");
}

static int bit_hi(unsigned long long v) { return v ? 64 - __builtin_clzll(v) : 0; }
static int bit_lo(unsigned long long v) { return v ? __builtin_ctzll(v) : 0; }

// bits: at least 4 more than number the points, in whole digits, so that few
// of them share a key.  With 8 more, a digit more at 65k to 1M points, the three
// orders took 0.45 ms at 80k points and 0.72 at 1M, so 0.38 and 0.63 (uniform,
// clustered and tightly clustered points alike).
static KeyMap key_map(unsigned long long vary, double lo, double hi, int n)
{
    KeyMap m = {lo, 0.0, 0.0, bit_lo(vary), bit_hi(vary) - bit_lo(vary), 1};
    if (m.bits <= 32) return m;
    m.exact = 0;
    int want = 8;
    while (want < 32 && (1ll << (want - 4)) < n) want += 8;
    const double top = (double)((1ll << want) - 1), scale = top / (hi - lo);
    if (std::isfinite(hi - lo) && std::isfinite(scale) && scale > 0.0) {
        m.scale = scale;
        m.top = top;
        m.bits = want;
    } else {
        m.shift = bit_hi(vary) - 32;
        m.bits = 32;
    }
    return m;
}


static unsigned grid_for(long long n)
{
    long long b = (n + TPB - 1) / TPB;
    if (b < 1) b = 1;
    if (b > 148 * 32) b = 148 * 32;
    return (unsigned)b;
}

template <class T> static T read1(const T *d, cudaStream_t s)
{
    T v;
    check(cudaMemcpyAsync(&v, d, sizeof(T), cudaMemcpyDeviceToHost, s), "D2H");
    check(cudaStreamSynchronize(s), "sync");
    return v;
}

static void copy_perm(int *dst, const int *src, int n, cudaStream_t s)
{
    check(cudaMemcpyAsync(dst, src, sizeof(int) * (size_t)n, cudaMemcpyDeviceToDevice, s), "copy");
}

// Stable sorts of points by one coordinate: vout = the order vin, sorted.  By
// 32-bit keys (four passes over 8 bytes a point instead of eight over 12) with
// the few runs of equal ones put right, or by all bits that vary.  5M uniform
// points: the first order (x, then y and z where x ties, not z, y, x) 3.4 ms by
// 64-bit keys and 1.1 ms so, the other two 1.9 and 0.9 ms.
struct CoordSort {
    Pool &pool;
    cudaStream_t s;
    unsigned *key, *srt;  // n each
    uint64_t *key64, *srt64;
    int n;

    void by_map(const uint64_t *k, const KeyMap &m, const int *perm, const int *vin, int *vout, int cnt)
    {
        k_map_keys<<<grid_for(cnt), TPB, 0, s>>>(k, perm, cnt, m, key);
        sort_pairs(pool, s, (const unsigned *)key, srt, vin, vout, cnt, 0, m.bits);
    }
    // sorted, except where a run is too long (*too_long set)
    void by_key(const uint64_t *k, const KeyMap &m, const int *vin, int *vout, int *tmp, int cnt,
                int *too_long)
    {
        by_map(k, m, vin, vin, m.exact ? vout : tmp, cnt);
        if (m.exact) return;
        copy_perm(vout, tmp, cnt, s);
        k_fix_runs<1><<<grid_for(cnt), TPB, 0, s>>>(srt, cnt, Keys3{{k, k, k}}, tmp, vout, too_long);
        KD_LAUNCH_CHECK("k_fix_runs");
    }
    void by_bits(const uint64_t *k, unsigned long long vary, const KeyMap &m, const int *vin, int *vout,
                 int cnt)
    {
        if (m.exact) {
            by_map(k, m, vin, vin, vout, cnt);
            return;
        }
        if (!key64) {
            key64 = pool.alloc<uint64_t>(n);
            srt64 = pool.alloc<uint64_t>(n);
        }
        k_gather_u64<<<grid_for(cnt), TPB, 0, s>>>(k, vin, cnt, key64);
        sort_pairs(pool, s, (const uint64_t *)key64, srt64, vin, vout, cnt, bit_lo(vary), bit_hi(vary));
    }
};

// Points in counting order, in two halves: launch() queues the order along the
// curve, and finish(), given the flag that it left (read by the caller, after
// its next synchronisation), settles cells of more points than a chunk puts in
// order: by all 63 bits, and where one point in eight is still in such a cell
// (an outlier far away, an infinite coordinate, detail below 2^-21 of the
// extent) along the curve through the ranks of the coordinates, which follows
// the points at any scale but takes three more sorts (a whole call with 5M
// points: 11.7 ms instead of 7.3).  Then it puts the chunks in order.
struct Curve {
    Pool &pool;
    cudaStream_t s;
    const double *xyz;
    int n;
    int *full;  // device, zeroed here
    const KeySpan *span;
    int *iota = nullptr, *perm = nullptr, *tmp = nullptr;

    void launch(const int *fin, FieldInfo *fi)
    {
        if (!iota) iota = pool.alloc<int>(n);
        perm = pool.alloc<int>(n);
        tmp = pool.alloc<int>(n);
        unsigned *key32 = pool.alloc<unsigned>(n), *srt = pool.alloc<unsigned>(n);
        check(cudaMemsetAsync(full, 0, sizeof *full, s), "memset");
        k_curve<<<grid_for(n), TPB, 0, s>>>(xyz, fin, n, span, nullptr, key32, iota, fi);
        KD_LAUNCH_CHECK("k_curve");
        sort_pairs(pool, s, (const unsigned *)key32, srt, (const int *)iota, tmp, n, 0, 32);
        k_full_cells<<<grid_for(n), TPB, 0, s>>>((const unsigned *)srt, tmp, xyz, n, full);
        KD_LAUNCH_CHECK("k_full_cells");
    }
    void finish(int nfull)
    {
        if (nfull) exact(nfull);
        check(cudaFuncSetAttribute(k_refine, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(RefineSmem)), "smem attribute");
        k_refine<<<blocks_for(n, kChunk), kRefThreads, sizeof(RefineSmem), s>>>(n, xyz, Cells{nullptr, 0, 0},
                                                                                tmp, perm);
        KD_LAUNCH_CHECK("k_refine");
    }
    void exact(int nfull)
    {
        uint64_t *key = pool.alloc<uint64_t>(n), *srt = pool.alloc<uint64_t>(n);
        k_curve<<<grid_for(n), TPB, 0, s>>>(xyz, nullptr, n, span, key, nullptr, iota, nullptr);
        sort_pairs(pool, s, (const uint64_t *)key, srt, (const int *)iota, tmp, n, 0, 63);
        check(cudaMemsetAsync(full, 0, sizeof *full, s), "memset");
        k_full_cells<<<grid_for(n), TPB, 0, s>>>((const uint64_t *)srt, tmp, xyz, n, full);
        KD_LAUNCH_CHECK("k_full_cells");
        if (read1(full, s) <= n / 8) return;
        uint64_t *k[3];
        int *rank[3], *head = pool.alloc<int>(n), *cls = pool.alloc<int>(n), *err = pool.alloc<int>(1);
        KeySpan *sp = pool.alloc<KeySpan>(1);
        for (int d = 0; d < 3; d++) {
            k[d] = pool.alloc<uint64_t>(n);
            rank[d] = pool.alloc<int>(n);
        }
        check(cudaMemsetAsync(err, 0, sizeof(int), s), "memset");
        check(cudaMemsetAsync(sp, 0, sizeof *sp, s), "memset");
        k_prep<true><<<grid_for(n), TPB, 0, s>>>(xyz, n, k[0], k[1], k[2], iota, err, sp);
        for (int d = 0; d < 3; d++) {
            sort_pairs(pool, s, (const uint64_t *)k[d], srt, (const int *)iota, tmp, n, 0, 64);
            k_value_heads<<<grid_for(n), TPB, 0, s>>>(k[d], tmp, n, head);
            incl_sum(pool, s, head, cls, n);
            k_scatter_rank<<<grid_for(n), TPB, 0, s>>>(cls, tmp, n, rank[d]);
        }
        k_curve_ranks<<<grid_for(n), TPB, 0, s>>>(rank[0], rank[1], rank[2], n, key);
        KD_LAUNCH_CHECK("k_curve_ranks");
        sort_pairs(pool, s, (const uint64_t *)key, srt, (const int *)iota, tmp, n, 0, 63);
    }
};

// Device -> pageable host copy of the node array returned by tree_construct
// (1.3 GB at 20M points), one queued item at a time.  A plain cudaMemcpy into
// pageable memory goes through the driver's own staging, one copy at a time
// for the whole process, and at the speed of the page faults of its one
// copying thread; it also makes every other pageable transfer of the process
// (the build's own small reads of device scalars) queue behind it.  Here the
// data goes through two pinned staging chunks (the next chunk's DMA overlaps
// the current one's host copy) and each chunk is copied into the destination
// by several threads, which take the destination's first-touch page faults in
// parallel.
namespace {
struct Staging {
    static constexpr size_t kChunk = size_t(32) << 20;
    void *pin[2] = {nullptr, nullptr};
};
// pinned staging pairs kept for the life of the process (allocating pinned
// memory per copy costs more than the copy): one per copy running at once,
// at most kMaxStaging (a batch of many small deferred builds would otherwise
// pin 64 MB per build); a copy that finds them all in use waits for one
constexpr int kMaxStaging = 4;
std::mutex g_stage_mu;
std::condition_variable g_stage_cv;
std::vector<Staging *> g_stage_free;
int g_stage_made = 0;
struct StagingLease {
    Staging *st = nullptr;
    StagingLease()
    {
        {
            std::unique_lock<std::mutex> g(g_stage_mu);
            g_stage_cv.wait(g, [] { return !g_stage_free.empty() || g_stage_made < kMaxStaging; });
            if (!g_stage_free.empty()) {
                st = g_stage_free.back();
                g_stage_free.pop_back();
                return;
            }
            g_stage_made++;  // this thread makes the next pair
        }
        std::unique_ptr<Staging> n(new Staging);
        for (int i = 0; i < 2; i++)
            if (cudaHostAlloc(&n->pin[i], Staging::kChunk, cudaHostAllocPortable) != cudaSuccess) {
                cudaGetLastError();
                for (int j = 0; j < i; j++) cudaFreeHost(n->pin[j]);
                {
                    std::lock_guard<std::mutex> g(g_stage_mu);
                    g_stage_made--;
                }
                g_stage_cv.notify_one();
                raise(KD_ENOMEM, "out of pinned host memory for the node array copy");
            }
        st = n.release();
    }
    ~StagingLease()
    {
        {
            std::lock_guard<std::mutex> g(g_stage_mu);
            g_stage_free.push_back(st);
        }
        g_stage_cv.notify_one();
    }
};
// Copy to or from a staging chunk without leaving its lines in this core's
// cache: a DMA that meets lines of a core gone idle runs at 6 GB/s instead of
// 50.  The chunk's side is aligned to 64 bytes.
static void copy_uncached(char *d, const char *f, size_t n, bool to_staging)
{
    size_t i = 0;
#if defined(__x86_64__)
    for (; i + 64 <= n; i += 64) {
        __m128i v[4];
        if (!to_staging) _mm_prefetch(f + i + 1024, _MM_HINT_NTA);
        for (int k = 0; k < 4; k++) v[k] = _mm_loadu_si128((const __m128i *)(f + i) + k);
        for (int k = 0; k < 4; k++)
            if (to_staging) _mm_stream_si128((__m128i *)(d + i) + k, v[k]);
            else _mm_storeu_si128((__m128i *)(d + i) + k, v[k]);
    }
    if (to_staging) _mm_sfence();
#endif
    std::memcpy(d + i, f + i, n - i);
}
// Host copies of a transfer's chunks fanned out over threads made once for the
// whole transfer (a 32 MB chunk takes ~1 ms; creating threads per chunk would
// cost a good part of that): one per MB of the transfer, up to 16, the calling
// thread among them.
struct FanOut {
    int nthr = 1;
    std::vector<std::thread> th;
    std::mutex mu;
    std::condition_variable go, done;
    size_t gen = 0;
    int pending = 0;
    bool stop = false;
    char *to = nullptr;
    const char *from = nullptr;
    size_t len = 0;
    bool to_staging;
    explicit FanOut(size_t bytes, bool to_staging_) : to_staging(to_staging_)
    {
        const unsigned hw = std::thread::hardware_concurrency();
        nthr = (int)std::max<size_t>(1, std::min<size_t>({16, hw ? hw : 1, bytes >> 20}));
        try {
            for (int t = 1; t < nthr; t++) th.emplace_back(&FanOut::worker, this, t);
        } catch (const std::exception &) {  // fewer threads: the rest is copied by this one
        }
    }
    void slice(int t, char *d, const char *f, size_t n)
    {
        const size_t a = n * t / nthr & ~(size_t)63, b = t == nthr - 1 ? n : n * (t + 1) / nthr & ~(size_t)63;
        copy_uncached(d + a, f + a, b - a, to_staging);
    }
    void worker(int t)
    {
        size_t seen = 0;
        std::unique_lock<std::mutex> g(mu);
        for (;;) {
            go.wait(g, [&] { return stop || gen != seen; });
            if (stop) return;
            seen = gen;
            char *d = to;
            const char *f = from;
            const size_t n = len;
            g.unlock();
            slice(t, d, f, n);
            g.lock();
            if (--pending == 0) done.notify_one();
        }
    }
    void copy(char *d, const char *f, size_t n)
    {
        {
            std::lock_guard<std::mutex> g(mu);
            to = d;
            from = f;
            len = n;
            pending = (int)th.size();
            gen++;
        }
        go.notify_all();
        // slices of the threads that could not be started are done here
        for (int t = (int)th.size() + 1; t < nthr; t++) slice(t, d, f, n);
        slice(0, d, f, n);
        std::unique_lock<std::mutex> g(mu);
        done.wait(g, [&] { return pending == 0; });
    }
    ~FanOut()
    {
        {
            std::lock_guard<std::mutex> g(mu);
            stop = true;
        }
        go.notify_all();
        for (auto &x : th) x.join();
    }
};
}  // namespace

static void copy_to_pageable(void *dst, const void *src, size_t bytes, FanOut &fan);
static void copy_from_host(void *dst, const void *src, size_t bytes, cudaStream_t s);

// Touch one byte of every 4 KiB page of [p, p + bytes), on a thread per 4 MB
// and up to 16, so that the pages are resident before they are copied into (a
// fresh page takes about 1 us, more than its copy).
static void prefault(void *p, size_t bytes)
{
    const unsigned hw = std::thread::hardware_concurrency();
    const int nthr = (int)std::max<size_t>(1, std::min<size_t>({16, hw ? hw : 1, bytes >> 22}));
    auto touch = [p, bytes, nthr](int t) {
        volatile char *c = (volatile char *)p;
        const size_t a = bytes * t / nthr, b = bytes * (t + 1) / nthr;
        for (size_t i = a & ~(size_t)4095; i < b; i += 4096)
            if (i >= a) c[i] = 0;
    };
    std::vector<std::thread> th;
    try {
        for (int t = 1; t < nthr; t++) th.emplace_back(touch, t);
    } catch (const std::exception &) {
    }
    touch(0);
    for (int t = (int)th.size() + 1; t < nthr; t++) touch(t);  // threads not started
    for (auto &x : th) x.join();
}

static double wall_ms()
{
    return std::chrono::duration<double, std::milli>(
               std::chrono::steady_clock::now().time_since_epoch()).count();
}

// The node array's way to the caller's host array (see build_impl): the
// per-level items the build queues, the copier thread that drains them, and,
// for a deferred build, the device node array it reads until it is done.
struct NodeCopy {
    kd_node_sink *sink = nullptr;
    void *host = nullptr;
    bool handed = false;
    std::thread th;
    std::mutex mu;
    std::condition_variable cv;
    struct Item {
        cudaEvent_t ev;
        size_t off, len;
    };
    std::vector<Item> items;
    size_t next = 0;     // first item the copier has not taken
    bool closed = false; // no more items
    std::vector<cudaEvent_t> events;
    int code = 0;
    char msg[160] = "";
    double ms = 0;
    // deferred builds: the device node array (freed once the copy is done)
    // and the one-time join
    void *dnodes = nullptr;
    std::once_flag joined;
    void push(cudaEvent_t ev, size_t off, size_t len)
    {
        std::lock_guard<std::mutex> g(mu);
        items.push_back({ev, off, len});
        cv.notify_one();
    }
    void close()
    {
        std::lock_guard<std::mutex> g(mu);
        closed = true;
        cv.notify_one();
    }
    ~NodeCopy()
    {
        close();
        if (th.joinable()) th.join();
        for (auto e : events) cudaEventDestroy(e);
        if (dnodes) cudaFree(dnodes);
        if (host && !handed) sink->release(host);
    }
};

static void build_impl(const double *h_xyz, const int *h_fields, int n, int num_fields,
                       kd_node_sink *sink, int deferred, kd_catalog *cat)
{
    init_device();
    Stream st;
    cudaStream_t s = st.s;
    Pool pool(s, true);  // temporaries
    Pool keep(s);     // catalog arrays (released to the catalog on success)
    // phase boundaries: start, dedup, argsorts, levels, layout, end
    cudaEvent_t ph[6] = {};
    struct EvRelease {
        cudaEvent_t *e;
        ~EvRelease()
        {
            for (int i = 0; i < 6; i++)
                if (e[i]) cudaEventDestroy(e[i]);
        }
    } ev_release{ph};
    for (auto &e : ph) check(cudaEventCreate(&e), "cudaEventCreate");
    check(cudaEventRecord(ph[0], s), "event");

    // ---- inputs
    double *xyz = pool.alloc<double>(3 * (size_t)n);
    copy_from_host(xyz, h_xyz, sizeof(double) * 3 * (size_t)n, s);
    int *fin = nullptr;
    if (h_fields) {
        fin = pool.alloc<int>(n);
        copy_from_host(fin, h_fields, sizeof(int) * (size_t)n, s);
    }
    int *err = pool.alloc<int>(1);
    KeySpan *dks = pool.alloc<KeySpan>(1), ks;
    check(cudaMemsetAsync(err, 0, sizeof(int), s), "memset");
    check(cudaMemsetAsync(dks, 0, sizeof(KeySpan), s), "memset");

    uint64_t *kx = pool.alloc<uint64_t>(n), *ky = pool.alloc<uint64_t>(n),
             *kz = pool.alloc<uint64_t>(n);
    int *iota = pool.alloc<int>(n);
    k_prep<true><<<grid_for(n), TPB, 0, s>>>(xyz, n, kx, ky, kz, iota, err, dks);
    KD_LAUNCH_CHECK("k_prep");
    check(cudaMemcpyAsync(&ks, dks, sizeof ks, cudaMemcpyDeviceToHost, s), "D2H");
    int herr = 0;
    check(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, s), "D2H");
    st.sync();
    if (herr) raise(herr, "NaN coordinate in tree points");
    KeyMap map[3];
    double maxabs = 0;
    for (int d = 0; d < 3; d++) {
        const double lo = okey_value(~ks.inv_lo[d]), hi = okey_value(ks.hi[d]);
        maxabs = std::max(maxabs, std::max(fabs(lo), fabs(hi)));
        map[d] = key_map(ks.vary[d], lo, hi, n);
    }

    check(cudaEventRecord(ph[1], s), "event");
    // ---- lexicographic order, stable: by x, ties put right in place; only
    // where many points share an x, by z, then y, then x
    CoordSort cs{pool, s, pool.alloc<unsigned>(n), pool.alloc<unsigned>(n), nullptr, nullptr, n};
    int *pa = pool.alloc<int>(n), *pb = pool.alloc<int>(n);
    const Keys3 k3 = {{kx, ky, kz}};
    int *too_long = pool.alloc<int>(1);
    check(cudaMemsetAsync(too_long, 0, sizeof(int), s), "memset");
    // (fewer x values than points / kFixRun: some run is too long)
    bool by_all = map[0].exact && map[0].bits < 31 && (n >> map[0].bits) > kFixRun;
    if (!by_all) {
        cs.by_map(kx, map[0], nullptr, iota, pb, n);
        copy_perm(pa, pb, n, s);
        k_fix_runs<3><<<grid_for(n), TPB, 0, s>>>(cs.srt, n, k3, pb, pa, too_long);
        KD_LAUNCH_CHECK("k_fix_runs");
        by_all = read1(too_long, s) != 0;
    }
    if (by_all) {
        copy_perm(pa, iota, n, s);
        for (int d = 2; d >= 0; d--) {
            if (!ks.vary[d]) continue;  // constant key: a stable sort is the identity
            cs.by_bits(k3.k[d], ks.vary[d], map[d], pa, pb, n);
            std::swap(pa, pb);
        }
    }
    int *p3 = pa;

    // ---- runs of equal points
    int *head = pool.alloc<int>(n), *cls = pool.alloc<int>(n);
    k_heads<<<grid_for(n), TPB, 0, s>>>(p3, by_all ? nullptr : cs.srt, kx, ky, kz, n, head);
    incl_sum(pool, s, head, cls, n);
    int n_u = read1(cls + (n - 1), s);

    UniqueArrays u;
    u.ux = pool.alloc<double>(n_u);
    u.uy = pool.alloc<double>(n_u);
    u.uz = pool.alloc<double>(n_u);
    u.ufield = pool.alloc<int>(n_u);
    u.uw = pool.alloc<int>(n_u);
    u.urep = pool.alloc<int>(n_u);
    u.uhead = pool.alloc<int>(n_u + 1);
    u.uky = pool.alloc<uint64_t>(n_u);
    u.ukz = pool.alloc<uint64_t>(n_u);
    k_unique<<<grid_for(n), TPB, 0, s>>>(p3, head, cls, n, xyz, fin, u, n_u);
    FieldInfo *fi = pool.alloc<FieldInfo>(1);
    FieldInfo fi0 = {0x7fffffff, -0x7fffffff, 0, 0};
    check(cudaMemcpyAsync(fi, &fi0, sizeof fi0, cudaMemcpyHostToDevice, s), "H2D");
    k_weights<<<grid_for(std::max(n, n_u)), TPB, 0, s>>>(u, n_u, p3, cls, fin, n, err, fi);
    KD_LAUNCH_CHECK("k_weights");
    FieldInfo hfi;
    check(cudaMemcpyAsync(&hfi, fi, sizeof hfi, cudaMemcpyDeviceToHost, s), "D2H");
    check(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, s), "D2H");
    st.sync();
    if (herr) raise(herr, "a point is repeated 256 or more times (the node weight is 8 bits)");

    check(cudaEventRecord(ph[2], s), "event");
    // ---- superkey argsorts of the unique points (dedup order = superkey 0)
    int *A[3], *B[3];
    for (int d = 0; d < 3; d++) {
        A[d] = pool.alloc<int>(n_u);
        B[d] = pool.alloc<int>(n_u);
    }
    check(cudaMemcpyAsync(A[0], iota, sizeof(int) * (size_t)n_u, cudaMemcpyDeviceToDevice, s),
          "copy");
    // superkey 2 = (z, x, y): stable sort of the (x, y, z) order by z;
    // superkey 1 = (y, z, x): stable sort of the (z, x, y) order by y
    check(cudaMemsetAsync(too_long, 0, sizeof(int), s), "memset");
    cs.by_key(u.ukz, map[2], iota, A[2], pb, n_u, too_long);
    cs.by_key(u.uky, map[1], A[2], A[1], pb, n_u, too_long);
    if (!(map[1].exact && map[2].exact) && read1(too_long, s)) {
        cs.by_bits(u.ukz, ks.vary[2], map[2], iota, A[2], n_u);
        cs.by_bits(u.uky, ks.vary[1], map[1], A[2], A[1], n_u);
    }
    // coordinate d of the point at every position of order d, partitioned
    // along with the order (the variance passes then read contiguously)
    double *C[3], *CB[3];
    {
        const double *uc[3] = {u.ux, u.uy, u.uz};
        for (int d = 0; d < 3; d++) {
            C[d] = pool.alloc<double>(n_u);
            CB[d] = pool.alloc<double>(n_u);
            k_gather<double><<<grid_for(n_u), TPB, 0, s>>>(uc[d], A[d], n_u, C[d]);
        }
    }

    check(cudaEventRecord(ph[3], s), "event");
    // ---- tree
    int memsize = 2;
    {
        int x = n_u, e = 1;
        while (x > 1) {
            x /= 2;
            e++;
        }
        memsize = 1 << e;
    }
    TreeOut to;
    to.memsize = memsize;
    to.nodes = keep.alloc_from<NodeRec>(side_pool(kPoolNodes), memsize);
    to.inorder_rep = keep.alloc<int>(n_u);
    check(cudaMemsetAsync(to.nodes, 0, sizeof(NodeRec) * (size_t)memsize, s), "memset");

    const int cap = n_u / (kSubCap / 4) + 16;  // segments of the level loop, and those it leaves
    Segs sg[2];
    for (int k = 0; k < 2; k++) {
        sg[k].p = pool.alloc<int>(cap);
        sg[k].l = pool.alloc<int>(cap);
        sg[k].r = pool.alloc<int>(cap);
        sg[k].count = pool.alloc<int>(1);
    }
    LevelBufs lb;
    lb.tdim = pool.alloc<int>(cap);
    lb.acc = pool.alloc<double>(9 * (size_t)cap);
    int *pos[2] = {pool.alloc<int>(n_u), pool.alloc<int>(n_u)}, *place = pool.alloc<int>(n_u);
    lb.mid = pool.alloc<int>(cap);
    if (n_u > kSubCap) {
        int *r1 = pool.alloc<int>(n_u), *r2 = pool.alloc<int>(n_u);
        k_ranks<<<grid_for(n_u), TPB, 0, s>>>(n_u, A[1], A[2], r1, r2);
        KD_LAUNCH_CHECK("k_ranks");
        lb.rank1 = r1;
        lb.rank2 = r2;
    }
    const int ntiles = (int)((n_u + (long long)kPtTile - 1) / kPtTile);
    unsigned *masks = pool.alloc<unsigned>((size_t)ntiles * (kPtWords * kPtMasks));
    uint4 *tagg = pool.alloc<uint4>(ntiles), *tcarry = pool.alloc<uint4>(2 * (size_t)ntiles);
    {
        check(cudaMemsetAsync(pos[0], 0, sizeof(int) * (size_t)n_u, s), "memset");
        k_first_seg<<<1, 1, 0, s>>>(sg[0], n_u);
        KD_LAUNCH_CHECK("k_first_seg");
    }
    // The node array goes to the caller's host array while the counting layout
    // is built: k_subtrees writes the slots of the last ten levels, so nearly all
    // of them, and is the last kernel of the tree.  (Iteration lev of the loop
    // below writes the heap slots of level lev, so once it has run, every slot
    // below 2^(lev+1) is final; those go ahead where they are worth a copy, from
    // about 70M points on.)  The build records an event and queues the slots; a
    // second host thread, which has touched the host pages meanwhile, waits for
    // each event and copies them (pinned staging, DMA on its own stream).
    std::unique_ptr<NodeCopy> ncu(new NodeCopy);
    NodeCopy &nc = *ncu;
    const size_t node_bytes = sizeof(NodeRec) * (size_t)memsize;
    size_t node_queued = sizeof(NodeRec);  // slot 0 is never written: it stays zero
    // queue the node slots [node_queued, upto) once the stream reaches here
    auto queue_nodes = [&](size_t upto) {
        if (upto <= node_queued) return;
        cudaEvent_t ev = nullptr;
        check(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming), "cudaEventCreate");
        nc.events.push_back(ev);
        check(cudaEventRecord(ev, s), "event");
        nc.push(ev, node_queued, upto - node_queued);
        node_queued = upto;
    };
    if (sink) {
        nc.sink = sink;
        nc.host = sink->alloc(node_bytes);
        if (!nc.host) raise(KD_ENOMEM, "out of host memory for the node array");
        memset(nc.host, 0, sizeof(NodeRec));
        int dev = 0;
        check(cudaGetDevice(&dev), "cudaGetDevice");
        const char *src = (const char *)to.nodes;
        NodeCopy *ncp = &nc;
        auto job = [ncp, dev, src, node_bytes] {
            const double t0 = wall_ms();
            try {
                check(cudaSetDevice(dev), "cudaSetDevice");
                // fault the whole host array in first, on parallel threads,
                // while the first levels are built: the copies then write
                // resident pages instead of taking a page fault (and the
                // kernel's zeroing of a fresh page) at every page
                prefault(ncp->host, node_bytes);
                FanOut fan(node_bytes, false);  // (its threads start before the first level is done)
                for (;;) {
                    NodeCopy::Item it;
                    {
                        std::unique_lock<std::mutex> g(ncp->mu);
                        ncp->cv.wait(g, [ncp] { return ncp->next < ncp->items.size() || ncp->closed; });
                        if (ncp->next == ncp->items.size()) break;
                        it = ncp->items[ncp->next++];
                    }
                    check(cudaEventSynchronize(it.ev), "node copy wait");
                    copy_to_pageable((char *)ncp->host + it.off, src + it.off, it.len, fan);
                }
            } catch (const Error &e) {
                ncp->code = e.code;
                snprintf(ncp->msg, sizeof ncp->msg, "node copy: %.140s", e.msg);
            } catch (const std::exception &e) {
                ncp->code = KD_EINTERNAL;
                snprintf(ncp->msg, sizeof ncp->msg, "node copy: %s", e.what());
            }
            ncp->ms = wall_ms() - t0;
        };
        try {
            nc.th = std::thread(job);
        } catch (const std::exception &) {
            // no thread to spare: the copy runs on this thread at the end
        }
    }

    check(cudaFuncSetAttribute(k_subtrees, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)sizeof(SubSmem)), "smem attribute");
    int cur = 0, nlevels = 0;
    for (int lev = 0; (1LL << lev) <= (long long)n_u; lev++) {
        nlevels = lev + 1;
        long long ub64 = std::min<long long>(1LL << lev, cap);
        int ub = (int)ub64;
        unsigned gs = blocks_for(ub, TPB);
        Segs S = sg[cur], N = sg[cur ^ 1];
        long long maxsize = (long long)n_u >> lev;
        if (maxsize <= kSubCap) {  // the rest of the tree, a CTA per segment
            while ((n_u >> (nlevels - 1)) >= 4) nlevels++;
            k_subtrees<<<ub, kSubThreads, sizeof(SubSmem), s>>>(S, A[0], A[1], A[2], u, to, place, err);
            KD_LAUNCH_CHECK("k_subtrees");
            break;
        }
        k_seg_setup<<<gs, TPB, 0, s>>>(S, ub, lb, N);
        const unsigned gv = blocks_for(n_u, kVarChunk);
        k_var_par<0><<<gv, kVarThreads, 0, s>>>(n_u, pos[cur], S, lb, C[0], C[1], C[2]);
        k_var_par<1><<<gv, kVarThreads, 0, s>>>(n_u, pos[cur], S, lb, C[0], C[1], C[2]);
        k_level_nodes<<<blocks_for(ub, 64), 64, 0, s>>>(S, ub, lb, A[0], A[1], A[2], C[0], C[1], C[2], u, to,
                                                        err);
        KD_LAUNCH_CHECK("level kernels");
        // levels 0 .. lev are final: copy their slots once they are large
        // enough to be worth a copy of their own
        {
            const size_t upto = sizeof(NodeRec) * std::min<size_t>((size_t)2 << lev, memsize);
            if (upto - node_queued >= ((size_t)4 << 20)) queue_nodes(upto);
        }
        {
            k_part_count<<<ntiles, kPtThreads, 0, s>>>(n_u, pos[cur], S, A[0], A[1], A[2], lb, masks,
                                                       tagg);
            k_part_carry<<<1, 1024, 0, s>>>(ntiles, tagg, tcarry);
            PartIO io;
            for (int d = 0; d < 3; d++) {
                io.a[d] = A[d];
                io.ao[d] = B[d];
                io.c[d] = C[d];
                io.co[d] = CB[d];
            }
            k_part_move<<<ntiles, kPtThreads, 0, s>>>(n_u, pos[cur], S, io, masks, tcarry,
                                                      pos[cur ^ 1], err);
            for (int d = 0; d < 3; d++) {
                std::swap(A[d], B[d]);
                std::swap(C[d], CB[d]);
            }
        }
        KD_LAUNCH_CHECK("partition kernels");
        cur ^= 1;
    }
    // every slot is final: queue the rest and let the copier finish it while
    // the counting layout is built
    queue_nodes(node_bytes);
    nc.close();
    if (!nc.th.joinable()) {  // no copier thread: copy here
        FanOut fan(node_bytes, false);
        for (auto &it : nc.items) {
            check(cudaEventSynchronize(it.ev), "node copy wait");
            copy_to_pageable((char *)nc.host + it.off, (const char *)to.nodes + it.off, it.len, fan);
        }
    }
    // ---- counting layout
    check(cudaEventRecord(ph[4], s), "event");
    Cells cells = {nullptr, 0, 0};
    // (points above the cells, one per cell on average, and duplicates join them)
    while ((n >> cells.bits) > kChunk - 128 && (n_u >> cells.bits) >= 128) cells.bits++;
    int *start = pool.alloc<int>(((size_t)1 << cells.bits) + 1), *perm = pool.alloc<int>(n);
    const int *order = p3;
    cells.start = start;
    int *flags = pool.alloc<int>(2), hflags[2];  // largest cell, error
    check(cudaMemsetAsync(flags, 0, sizeof(int), s), "memset");
    if (cells.bits) {
        int *cell = pool.alloc<int>(n), *ord = pool.alloc<int>(n);
        unsigned *key = pool.alloc<unsigned>(n), *skey = pool.alloc<unsigned>(n);
        k_cell_of<<<grid_for(n_u), TPB, 0, s>>>(n_u, cells.bits, to.nodes, to.inorder_rep, cell);
        k_cell_keys<<<grid_for(n), TPB, 0, s>>>(n, p3, cls, u.urep, cell, key);
        sort_pairs(pool, s, (const unsigned *)key, skey, (const int *)p3, ord, n, 0, cells.bits);
        k_cell_starts<<<grid_for(n), TPB, 0, s>>>(n, 1 << cells.bits, skey, start);
        order = ord;
    } else {
        k_cell_starts<<<1, 32, 0, s>>>(n, 1, nullptr, start);
    }
    k_cell_max<<<grid_for(1 << cells.bits), TPB, 0, s>>>(1 << cells.bits, start, flags);
    KD_LAUNCH_CHECK("cell kernels");
    check(cudaMemcpyAsync(flags + 1, err, sizeof(int), cudaMemcpyDeviceToDevice, s), "copy");
    check(cudaMemcpyAsync(hflags, flags, sizeof hflags, cudaMemcpyDeviceToHost, s), "D2H");
    st.sync();
    if (hflags[1]) raise(hflags[1], "tree build exceeded an internal bound");
    if (hflags[0] <= 4 * kChunk) {
        while (KD_RUN_MAX << cells.leaf_bits < hflags[0]) cells.leaf_bits++;
        check(cudaFuncSetAttribute(k_refine, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(RefineSmem)), "smem attribute");
        const int per = std::max(1, (KD_RUN_MAX << cells.leaf_bits) / kChunk);
        k_refine<<<per << cells.bits, kRefThreads, sizeof(RefineSmem), s>>>(n, xyz, cells, order, perm);
        KD_LAUNCH_CHECK("k_refine");
    } else {
        // points repeated so often that the tree's cells are very uneven: every
        // cell would own the largest one's leaves.  Even ones, along the curve.
        Curve cv{pool, s, xyz, n, flags, dks, iota};
        cv.launch(nullptr, nullptr);
        cv.finish(read1(flags, s));
        perm = cv.perm;
        cells.bits = 0;
        while (((long long)kChunk << cells.bits) < n) cells.bits++;
        while (KD_RUN_MAX << cells.leaf_bits < kChunk) cells.leaf_bits++;
        start = pool.alloc<int>(((size_t)1 << cells.bits) + 1);
        k_even_cells<<<blocks_for((1ll << cells.bits) + 1, TPB), TPB, 0, s>>>(n, 1 << cells.bits, start);
        KD_LAUNCH_CHECK("k_even_cells");
        cells.start = start;
    }

    const int split = hfi.split ? 1 : 0;
    int *tfin = nullptr;
    if (split) {
        tfin = pool.alloc<int>(n);
        k_tree_fields<<<grid_for(n), TPB, 0, s>>>(n, p3, cls, u.ufield, tfin);
    }
    const int D = cells.bits + cells.leaf_bits, nleaves = 1 << D;
    const int groups = std::max(1, nleaves / kBlockLeaves);
    LeafOut lf;
    RawOut &ro = lf.o;
    Summ &sm = lf.sm;
    ro.x = keep.alloc<double>(n);
    ro.y = keep.alloc<double>(n);
    ro.z = keep.alloc<double>(n);
    ro.qf = keep.alloc<int>(n);
    ro.tf = split ? keep.alloc<int>(n) : ro.qf;
    sm.box = keep.alloc<double>(6 * 2 * (size_t)nleaves);
    sm.count = keep.alloc<int>(2 * (size_t)nleaves);
    sm.tf = keep.alloc<int>(2 * (size_t)nleaves);
    lf.qf = pool.alloc<int>(nleaves);
    lf.leaf = keep.alloc<kd_leaf>(nleaves);
    lf.t4 = keep.alloc<float4>(n);
    lf.pos = keep.alloc<int>((size_t)nleaves + 1);
    lf.nruns = pool.alloc<int>((size_t)nleaves + 1);
    lf.blocks = pool.alloc<int>((size_t)groups + 1);
    lf.hdiag = pool.alloc<unsigned long long>(2);  // and the number of small leaves
    check(cudaMemsetAsync(lf.hdiag, 0, 2 * sizeof(unsigned long long), s), "memset");
    const unsigned gl = blocks_for(32 * ((long long)nleaves + 1), TPB);
    k_leaves<<<gl, TPB, 0, s>>>(n, nleaves, cells, perm, xyz, fin, tfin, lf);
    for (int d = D; d > 0; d = std::max(0, d - 8))
        k_internal_summary<<<1u << std::max(0, d - 8), TPB, 0, s>>>(d, sm, d == D ? lf.leaf : nullptr,
                                                                    (const double *)lf.hdiag, (int *)(lf.hdiag + 1));
    int *leaf_run = keep.alloc<int>((size_t)nleaves + 1);
    excl_sum(pool, s, lf.nruns, leaf_run, nleaves + 1);
    int *boff = pool.alloc<int>((size_t)groups + 1);
    excl_sum(pool, s, lf.blocks, boff, groups + 1);
    KD_LAUNCH_CHECK("layout kernels");
    struct {
        double hdiag;
        int small, pad;
    } hl;
    int nblocks;
    check(cudaMemcpyAsync(&hl, lf.hdiag, sizeof hl, cudaMemcpyDeviceToHost, s), "D2H");
    check(cudaMemcpyAsync(&nblocks, boff + groups, sizeof(int), cudaMemcpyDeviceToHost, s), "D2H");
    const int nruns = read1(leaf_run + nleaves, s);
    int *run_start = keep.alloc<int>(nruns), *run_len = keep.alloc<int>(nruns),
        *run_tf = keep.alloc<int>(nruns);
    int *bstart = keep.alloc<int>(nblocks), *blen = keep.alloc<int>(nblocks),
        *bqf = keep.alloc<int>(nblocks);
    double *bbox = keep.alloc<double>(6 * (size_t)nblocks);
    k_tree_blocks<<<blocks_for(groups, TPB), TPB, 0, s>>>(groups, nleaves, lf.pos, boff, sm.box, lf.qf, bstart,
                                                          blen, bbox, bqf);
    k_leaf_runs<<<gl, TPB, 0, s>>>(nleaves, lf.pos, ro.tf, leaf_run, run_start, run_len, run_tf);
    KD_LAUNCH_CHECK("summary kernels");
    check(cudaEventRecord(ph[5], s), "event");
    st.sync();
    kd_build_stats bs;
    memset(&bs, 0, sizeof bs);
    if (!deferred) {
        const double wait0 = wall_ms();
        if (nc.th.joinable()) nc.th.join();
        const double waited = wall_ms() - wait0;
        if (nc.code) raise(nc.code, nc.msg);
        bs.ms_node_copy = nc.ms;
        bs.ms_node_wait = waited;
    }
    {
        float ms[5] = {0, 0, 0, 0, 0}, tot = 0;
        for (int i = 0; i < 5; i++) cudaEventElapsedTime(&ms[i], ph[i], ph[i + 1]);
        cudaEventElapsedTime(&tot, ph[0], ph[5]);
        bs.ms_prep = ms[0];
        bs.ms_dedup = ms[1];
        bs.ms_argsort = ms[2];
        bs.ms_levels = ms[3];
        bs.ms_layout = ms[4];
        bs.ms_device = tot;
        bs.levels = nlevels;
        bs.n_unique = n_u;
    }

    // ---- hand the kept arrays to the catalog
    memset(cat, 0, sizeof *cat);
    check(cudaGetDevice(&cat->device), "cudaGetDevice");
    cat->n_raw = n;
    cat->n_u = n_u;
    cat->memsize = memsize;
    cat->num_fields = num_fields;
    cat->min_qf = h_fields ? hfi.min_qf : 0;
    cat->max_qf = h_fields ? hfi.max_qf : 0;
    cat->max_tf = hfi.max_tf;
    cat->fields_split = split;
    cat->short_runs = hfi.max_tf > 0 && 4LL * nruns > n;
    cat->many_fields = hfi.max_tf > 0 && 8LL * nruns > n;
    cat->uneven_leaves = 8LL * KD_RUN_MAX * hl.small > n;
    cat->max_abs = maxabs;
    // the host holds the node array; the device copy is freed with the pool,
    // or, while a deferred copy still reads it, once that is done
    sink->nodes = nc.host;
    nc.handed = true;
    nc.sink = nullptr;
    cat->d_inorder_rep = keep.keep(to.inorder_rep);
    cat->d_x = keep.keep(ro.x);
    cat->d_y = keep.keep(ro.y);
    cat->d_z = keep.keep(ro.z);
    cat->d_qf = keep.keep(ro.qf);
    cat->d_tf = split ? keep.keep(ro.tf) : ro.qf;
    cat->depth = D;
    cat->nleaves = nleaves;
    cat->d_box = keep.keep(sm.box);
    cat->d_ncount = keep.keep(sm.count);
    cat->d_ntf = keep.keep(sm.tf);
    cat->d_leaf_run = keep.keep(leaf_run);
    cat->d_leaf_pos = keep.keep(lf.pos);
    cat->nruns = nruns;
    cat->d_run_start = keep.keep(run_start);
    cat->d_run_len = keep.keep(run_len);
    cat->d_run_tf = keep.keep(run_tf);
    cat->d_t4 = keep.keep(lf.t4);
    cat->d_leaf = keep.keep(lf.leaf);
    cat->leaf_hdiag = hl.hdiag;
    cat->nblocks = nblocks;
    cat->d_blk_start = keep.keep(bstart);
    cat->d_blk_len = keep.keep(blen);
    cat->d_blk_qf = keep.keep(bqf);
    cat->d_blk_box = keep.keep(bbox);
    cat->device_bytes = keep.bytes;
    cat->bstats = bs;
    if (deferred) {
        nc.dnodes = keep.keep(to.nodes);
        cat->pending = ncu.release();
    }
}

// ------------------------------------------------------------ query points

// the points in curve order, and the query blocks' ranges
__global__ void k_query_points(const double *__restrict__ xyz, const int *__restrict__ fin,
                               const int *__restrict__ perm, int n, RawOut o, int nblocks, int *bstart,
                               int *blen)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const size_t p = perm[i];
        o.x[i] = xyz[3 * p];
        o.y[i] = xyz[3 * p + 1];
        o.z[i] = xyz[3 * p + 2];
        o.qf[i] = fin ? fin[p] : 0;
        if (i < nblocks) {
            bstart[i] = i * KD_BLOCK_MAX;
            blen[i] = min(KD_BLOCK_MAX, n - i * KD_BLOCK_MAX);
        }
    }
}

// Query points that are counted once and dropped need no tree: a count reads
// them as blocks of near points with boxes.  So they are sorted along a curve
// and cut every KD_BLOCK_MAX points, where a tree and its counting layout take
// several times the work: a whole count of 400k points in one radius took
// 4.2 ms by a tree and takes 1.8 ms so, of 1000 points 1.14 and 0.54 ms.  The
// blocks are better ones, too (no cut at the subtrees' ends, near points next
// to each other): 3M points, 21 edges, 1.58M instead of 1.80M (block, run)
// records and 9.4 instead of 12.0 ms in the tile kernel; in Z-order, whose
// jumps stretch the boxes, 2.37M records and 14.4 ms.  Where the curve's cells
// are too coarse for the points, Curve::finish follows them at any scale.
static void build_query(const double *h_xyz, const int *h_fields, int n, int num_fields, kd_catalog *cat)
{
    init_device();
    Stream st;
    cudaStream_t s = st.s;
    Pool pool(s, true), keep(s);
    double *xyz = pool.alloc<double>(3 * (size_t)n);
    copy_from_host(xyz, h_xyz, sizeof(double) * 3 * (size_t)n, s);
    int *fin = nullptr;
    if (h_fields) {
        fin = pool.alloc<int>(n);
        copy_from_host(fin, h_fields, sizeof(int) * (size_t)n, s);
    }
    struct State {
        KeySpan span;
        FieldInfo fi;
        int full, err, many;
    } h, *dstate = pool.alloc<State>(1);
    memset(&h, 0, sizeof h);
    h.fi = {0x7fffffff, -0x7fffffff, 0, 0};
    check(cudaMemcpyAsync(dstate, &h, sizeof h, cudaMemcpyHostToDevice, s), "H2D");
    k_prep<false><<<grid_for(n), TPB, 0, s>>>(xyz, n, nullptr, nullptr, nullptr, nullptr, &dstate->err,
                                              &dstate->span);
    Curve cv{pool, s, xyz, n, &dstate->full, &dstate->span};
    cv.launch(fin, &dstate->fi);
    h = read1(dstate, s);
    if (h.err) raise(h.err, "NaN coordinate in query points");
    cv.finish(h.full);

    const int nblocks = (int)blocks_for(n, KD_BLOCK_MAX);
    RawOut ro;
    ro.x = keep.alloc<double>(n);
    ro.y = keep.alloc<double>(n);
    ro.z = keep.alloc<double>(n);
    ro.qf = ro.tf = keep.alloc<int>(n);
    int *bstart = keep.alloc<int>(nblocks), *blen = keep.alloc<int>(nblocks),
        *bqf = keep.alloc<int>(nblocks);
    double *bbox = keep.alloc<double>(6 * (size_t)nblocks);
    k_query_points<<<grid_for(n), TPB, 0, s>>>(xyz, fin, cv.perm, n, ro, nblocks, bstart, blen);
    const bool fields = (long long)h.fi.max_qf - h.fi.min_qf >= KD_MANY_FIELDS;
    k_block_boxes<<<nblocks, KD_BLOCK_MAX, 0, s>>>(nblocks, bstart, blen, ro, bbox, bqf,
                                                   fields ? &dstate->many : nullptr);
    KD_LAUNCH_CHECK("k_query_points");
    if (fields)
        check(cudaMemcpyAsync(&h.many, &dstate->many, sizeof(int), cudaMemcpyDeviceToHost, s), "D2H");
    st.sync();

    memset(cat, 0, sizeof *cat);
    check(cudaGetDevice(&cat->device), "cudaGetDevice");
    cat->n_raw = n;
    cat->num_fields = num_fields;
    cat->min_qf = h.fi.min_qf;
    cat->max_qf = h.fi.max_qf;
    cat->many_fields = 2LL * h.many > (n + 31) / 32;
    for (int d = 0; d < 3; d++)
        cat->max_abs = std::max(cat->max_abs, std::max(fabs(okey_value(~h.span.inv_lo[d])),
                                                       fabs(okey_value(h.span.hi[d]))));
    cat->d_x = keep.keep(ro.x);
    cat->d_y = keep.keep(ro.y);
    cat->d_z = keep.keep(ro.z);
    cat->d_qf = cat->d_tf = keep.keep(ro.qf);
    cat->nblocks = nblocks;
    cat->d_blk_start = keep.keep(bstart);
    cat->d_blk_len = keep.keep(blen);
    cat->d_blk_qf = keep.keep(bqf);
    cat->d_blk_box = keep.keep(bbox);
    cat->device_bytes = keep.bytes;
}

}  // namespace kd

static int build_entry(const double *h_xyz, const int *h_fields, int n, int num_fields,
                       kd_node_sink *sink, int deferred, kd_catalog *cat)
{
    if (n < 1) {
        kd_set_error(KD_EINVAL, "a tree needs at least one point");
        return KD_EINVAL;
    }
    try {
        if (!sink) kd::build_query(h_xyz, h_fields, n, num_fields, cat);
        else kd::build_impl(h_xyz, h_fields, n, num_fields, sink, deferred, cat);
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

extern "C" int kdg_build(const double *h_xyz, const int *h_fields, int n, int num_fields,
                         int query_only, kd_catalog *cat)
{
    if (!query_only) {
        kd_set_error(KD_EINVAL, "kdg_build: a tree is built by kdg_build_tree");
        return KD_EINVAL;
    }
    return build_entry(h_xyz, h_fields, n, num_fields, nullptr, 0, cat);
}

extern "C" int kdg_build_tree(const double *h_xyz, const int *h_fields, int n, int num_fields,
                              kd_node_sink *sink, int deferred, kd_catalog *cat)
{
    if (!sink || !sink->alloc || !sink->release) {
        kd_set_error(KD_EINVAL, "kdg_build_tree: no node array sink");
        return KD_EINVAL;
    }
    sink->nodes = nullptr;
    return build_entry(h_xyz, h_fields, n, num_fields, sink, deferred, cat);
}

// Runs a catalog operation on the catalog's device, then restores the
// calling thread's device.
struct OnDevice {
    int prev = 0;
    explicit OnDevice(int dev)
    {
        cudaGetDevice(&prev);
        if (prev != dev) cudaSetDevice(dev);
    }
    ~OnDevice() { cudaSetDevice(prev); }
};

namespace kd {

// Host -> device copy of a build's input on stream s.  Pinned (or managed)
// memory, and anything under 4 MB (where starting the copying threads costs
// more than it saves), is one cudaMemcpyAsync.  Pageable memory otherwise
// takes the driver's own staging path at 10 to 20 GB/s (50 ms for the 560 MB of
// a 20M-point catalog, 2.0 ms for the 24 MB of 1M points); here several threads
// copy each chunk into a pinned staging buffer while the previous chunk's DMA
// runs (1M points 1.0 ms).  Returns once the last DMA has finished (the staging
// pair is then free).
static void copy_from_host(void *dst, const void *src, size_t bytes, cudaStream_t s)
{
    if (bytes == 0) return;
    bool plain = bytes < (size_t(4) << 20);
    if (!plain) {
        cudaPointerAttributes at;
        if (cudaPointerGetAttributes(&at, src) == cudaSuccess)
            plain = at.type != cudaMemoryTypeUnregistered;
        else
            cudaGetLastError();  // not known to the runtime: pageable
    }
    if (plain) {
        check(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s), "H2D");
        return;
    }
    const size_t chunk = size_t(8) << 20;  // (the first chunk's copy has no DMA to overlap)
    StagingLease lease;
    void *const *pin = lease.st->pin;
    cudaEvent_t done[2] = {nullptr, nullptr};
    struct Release {
        cudaEvent_t *ev;
        ~Release()
        {
            for (int i = 0; i < 2; i++)
                if (ev[i]) {
                    cudaEventSynchronize(ev[i]);  // no DMA may still read the staging
                    cudaEventDestroy(ev[i]);
                }
        }
    } rel{done};
    for (int i = 0; i < 2; i++)
        check(cudaEventCreateWithFlags(&done[i], cudaEventDisableTiming), "cudaEventCreate");
    FanOut fan(bytes, true);
    const size_t nch = (bytes + chunk - 1) / chunk;
    for (size_t c = 0; c < nch; c++) {
        const int b = (int)(c & 1);
        if (c >= 2) check(cudaEventSynchronize(done[b]), "H2D wait");  // its last DMA is done
        const size_t off = c * chunk, len = std::min(chunk, bytes - off);
        fan.copy((char *)pin[b], (const char *)src + off, len);
        check(cudaMemcpyAsync((char *)dst + off, pin[b], len, cudaMemcpyHostToDevice, s), "H2D");
        check(cudaEventRecord(done[b], s), "event");
    }
    for (int b = 0; b < 2; b++) check(cudaEventSynchronize(done[b]), "H2D wait");
}

static void copy_to_pageable(void *dst, const void *src, size_t bytes, FanOut &fan)
{
    const size_t chunk = Staging::kChunk;
    if (bytes == 0) return;
    StagingLease lease;
    void *const *pin = lease.st->pin;
    Stream st;
    cudaEvent_t done[2] = {nullptr, nullptr};
    struct Release {
        cudaEvent_t *ev;
        ~Release()
        {
            for (int i = 0; i < 2; i++)
                if (ev[i]) cudaEventDestroy(ev[i]);
        }
    } rel{done};
    for (int i = 0; i < 2; i++)
        check(cudaEventCreateWithFlags(&done[i], cudaEventDisableTiming), "cudaEventCreate");
    const size_t nch = (bytes + chunk - 1) / chunk;
    auto issue = [&](size_t c) {
        const size_t off = c * chunk, len = std::min(chunk, bytes - off);
        check(cudaMemcpyAsync(pin[c & 1], (const char *)src + off, len, cudaMemcpyDeviceToHost, st.s),
              "D2H");
        check(cudaEventRecord(done[c & 1], st.s), "event");
    };
    issue(0);
    for (size_t c = 0; c < nch; c++) {
        check(cudaEventSynchronize(done[c & 1]), "D2H wait");
        if (c + 1 < nch) issue(c + 1);  // into the other buffer, already drained
        const size_t off = c * chunk, len = std::min(chunk, bytes - off);
        fan.copy((char *)dst + off, (const char *)pin[c & 1], len);
    }
}

}  // namespace kd

extern "C" int kdg_copy_inorder(const kd_catalog *cat, int *h_perm)
{
    OnDevice on(cat->device);
    cudaError_t e = cudaMemcpy(h_perm, cat->d_inorder_rep, sizeof(int) * (size_t)cat->n_u,
                               cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
        kd_set_error(KD_ECUDA, "permutation copy: %s", cudaGetErrorString(e));
        return KD_ECUDA;
    }
    return KD_OK;
}

extern "C" int kdg_wait_nodes(kd_catalog *cat)
{
    kd::NodeCopy *nc = (kd::NodeCopy *)cat->pending;
    if (!nc) return KD_OK;
    std::call_once(nc->joined, [nc, cat] {
        const double w0 = kd::wall_ms();
        if (nc->th.joinable()) nc->th.join();
        cat->bstats.ms_node_wait = kd::wall_ms() - w0;
        cat->bstats.ms_node_copy = nc->ms;
        OnDevice on(cat->device);
        // the copier has finished reading it: a stream-ordered free, so that
        // a count still running on the device is not waited for
        if (nc->dnodes) cudaFreeAsync(nc->dnodes, cudaStreamPerThread);
        nc->dnodes = nullptr;
    });
    if (nc->code) {
        kd_set_error(nc->code, "%s", nc->msg);
        return nc->code;
    }
    return KD_OK;
}

extern "C" void kdg_free(kd_catalog *cat)
{
    if (cat->pending) {
        kdg_wait_nodes(cat);
        OnDevice on(cat->device);
        delete (kd::NodeCopy *)cat->pending;
        cat->pending = nullptr;
    }
    OnDevice on(cat->device);
    void *ptrs[] = {cat->d_inorder_rep, cat->d_x,    cat->d_y,
                    cat->d_z,        cat->d_qf,          cat->fields_split ? cat->d_tf : nullptr,
                    cat->d_box,      cat->d_ncount,      cat->d_ntf,
                    cat->d_leaf_run, cat->d_leaf_pos,    cat->d_run_start, cat->d_run_len,
                    cat->d_run_tf,   cat->d_t4,          cat->d_leaf,
                    cat->d_blk_start, cat->d_blk_len,    cat->d_blk_qf,  cat->d_blk_box};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    memset(cat, 0, sizeof *cat);
}
