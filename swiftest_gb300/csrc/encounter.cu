// encounter.cu -- close-encounter checks for sm_103a.
//
// Restates encounter_check_all_plpl / _plplm / _pltp (src/encounter/encounter_check.f90:14-140)
// in both of the reference's modes:
//   * TRIANGULAR (:384-570): every pair is tested with encounter_check_one (:573-621).
//     Long checks go over radius-sorted tiles instead (encounter_sorted.cu, SORTED_PAIRS).
//   * SORTSWEEP  (:143-326, :763-988): 1-D radial bounding boxes |r| +- 1.1 renc,
//     sorted by extent, ties by extent index: one system's in tiles that are merged
//     (SAS_MERGED), longer lists and ensembles by a stable radix sort (radix_sort.cu);
//     each body whose box holds >= 2 foreign extents strictly inside (the reference's
//     loverlap test) tests the bodies whose extents lie inside.
//
// The encounter decision is made in FP64 with the reference's expression order
// (this file is compiled with -fmad=false), so lists are bit-identical to the
// reference loop.  In both modes a conservative FP32 prefilter first
// rejects pairs whose closest approach over the step provably exceeds the
// encounter radius (min_t |x + v t| >= |x| - |v| |dt|; see prefilter_reject for
// the margins).  Only pairs the FP64 test could accept reach it, so the
// prefilter changes speed, never the list.
//
// Output: pairs are appended with an atomic counter (up to cap), then sorted by
// (index1, index2), packed with lvdotr into one key: up to PAIRS_BLOCK pairs in one block,
// longer lists in tiles of MERGE_TILE that are merged MERGE_WAYS at a time.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "encounter_dev.cuh"
#include "swg_internal.cuh"

namespace swg {

constexpr int ET = 128;  // partner tile / block size

// Float copies of the bodies for the prefilter, written once per check.
__global__ void k_encounter_prep(int n, const double *__restrict__ r, const double *__restrict__ v,
                                 const double *__restrict__ renc, float4 *A, float4 *B, float4 *V) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const BodyF o = load_body(r, v, renc, i);
    A[i] = o.a;
    B[i] = o.b;
    V[i] = o.v;
}

// both lists of a check in one launch
__global__ void k_encounter_prep2(int n1, const double *__restrict__ r1, const double *__restrict__ v1,
                                  const double *__restrict__ renc1, float4 *F1, int n2, const double *__restrict__ r2,
                                  const double *__restrict__ v2, const double *__restrict__ renc2, float4 *F2) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n1 + n2) return;
    const bool first = t < n1;
    const int i = first ? t : t - n1, n = first ? n1 : n2;
    const BodyF o = load_body(first ? r1 : r2, first ? v1 : v2, first ? renc1 : renc2, i);
    float4 *F = first ? F1 : F2;
    F[i] = o.a;
    F[n + i] = o.b;
    F[2 * n + i] = o.v;
}

constexpr int EP = 64;  // partners per shared-memory tile


// Receivers: list-2 bodies j in [j0, j0 + ET) (one thread each).  Partners: list-1 bodies
// i in [ibeg, iend) (i < j when `upper`, i.e. pl-pl).  A pair is written as
// (i + 1 + base1, j + 1 + base2); lists are sorted afterwards, so the tiling is invisible.
// DISCARD: the close-approach scan of swiftest_discard_pl_tp instead (list 1 = pl with
// renc1 = their radii, list 2 = the tp with status st2): the FP64 test is
// swiftest_discard_pl_close with r2crit = radius^2, and a hit sets o2[base2 + j] = 1.  The
// prefilter bound holds for it too (same closest-approach expression).
// Whole block; returns at once (block-uniformly) when the range is empty.
template <bool DISCARD>
__device__ __forceinline__ void enc_tri_tile(
    int n1, const float4 *__restrict__ A1, const float4 *__restrict__ B1, const float4 *__restrict__ V1,
    const double *__restrict__ r1, const double *__restrict__ v1, const double *__restrict__ renc1, int n2,
    const float4 *__restrict__ A2, const float4 *__restrict__ B2, const float4 *__restrict__ V2,
    const double *__restrict__ r2, const double *__restrict__ v2, const double *__restrict__ renc2, int upper, int j0,
    int ibeg, int iend, int base1, int base2, double dt, long long cap, int32_t *__restrict__ o1,
    int32_t *__restrict__ o2, int32_t *__restrict__ olv, unsigned long long *__restrict__ count,
    const int32_t *__restrict__ st2 = nullptr) {
    __shared__ float4 sa[EP], sb[EP], sv[EP];
    const int j = j0 + threadIdx.x;
    const bool active = j < n2 && (!DISCARD || st2[j] == ST_ACTIVE);
    iend = min(n1, iend);
    if (upper) iend = min(iend, j0 + ET);
    if (ibeg >= iend) return;  // whole block outside the upper triangle
    BodyF q;
    if (active) {
        q.a = A2[j];
        q.b = B2[j];
        q.v = V2[j];
    }
    const int own_end = upper ? min(iend, j) : iend;
    const float dtf = __double2float_ru(fabs(dt)) * (1.0f + 1e-6f);  // |dt| bounds either direction of time
    for (int i0 = ibeg; i0 < iend; i0 += EP) {
        if (threadIdx.x < EP && i0 + threadIdx.x < iend) {
            sa[threadIdx.x] = A1[i0 + threadIdx.x];
            sb[threadIdx.x] = B1[i0 + threadIdx.x];
            sv[threadIdx.x] = V1[i0 + threadIdx.x];
        }
        __syncthreads();
        if (active) {
            const int nt = min(EP, own_end - i0);
            for (int ii = 0; ii < nt; ii++) {
                BodyF p;
                p.a = sa[ii];
                p.b = sb[ii];
                p.v = sv[ii];
                if (prefilter_reject(p, q, dtf)) continue;
                const int i = i0 + ii;
                const double xr = r2[3 * j + 0] - r1[3 * i + 0];
                const double yr = r2[3 * j + 1] - r1[3 * i + 1];
                const double zr = r2[3 * j + 2] - r1[3 * i + 2];
                const double vxr = v2[3 * j + 0] - v1[3 * i + 0];
                const double vyr = v2[3 * j + 1] - v1[3 * i + 1];
                const double vzr = v2[3 * j + 2] - v1[3 * i + 2];
                if (DISCARD) {
                    if (d_discard_close(xr, yr, zr, vxr, vyr, vzr, dt, renc1[i] * renc1[i])) o2[base2 + j] = 1;
                    continue;
                }
                const double renc12 = renc1[i] + (renc2 ? renc2[j] : 0.0);
                int lenc, lv;
                d_encounter_one(xr, yr, zr, vxr, vyr, vzr, renc12, dt, lenc, lv);
                if (lenc) {
                    const unsigned long long k = atomicAdd(count, 1ull);
                    if ((long long)k < cap) {
                        o1[k] = i + 1 + base1;
                        o2[k] = j + 1 + base2;
                        olv[k] = lv;
                    }
                }
            }
        }
        __syncthreads();
    }
}

// One system: receivers tile blockIdx.x, partner chunk blockIdx.y.
template <bool DISCARD>
__global__ void __launch_bounds__(ET) k_encounter_tri(
    int n1, const float4 *__restrict__ A1, const float4 *__restrict__ B1, const float4 *__restrict__ V1,
    const double *__restrict__ r1, const double *__restrict__ v1, const double *__restrict__ renc1, int n2,
    const float4 *__restrict__ A2, const float4 *__restrict__ B2, const float4 *__restrict__ V2,
    const double *__restrict__ r2, const double *__restrict__ v2, const double *__restrict__ renc2, int upper,
    int shift2, double dt, int chunk, long long cap, int32_t *__restrict__ o1, int32_t *__restrict__ o2,
    int32_t *__restrict__ olv, unsigned long long *__restrict__ count, const int32_t *__restrict__ st2) {
    const int ibeg = blockIdx.y * chunk;
    enc_tri_tile<DISCARD>(n1, A1, B1, V1, r1, v1, renc1, n2, A2, B2, V2, r2, v2, renc2, upper, blockIdx.x * ET, ibeg,
                          ibeg + chunk, 0, shift2, dt, cap, o1, o2, olv, count, st2);
}

// Batched (ensemble) check: block b takes item b = (system s, first receiver j0) of a
// table sorted by cost.  List 1 is system s's pl ([off1[s], off1[s] + n1[s]) in the
// float/double arrays), list 2 its pl again (upper, pl-pl) or its tp (off2, n2).  Pairs
// are written with global 1-based indices, so the sorted list groups by system.
template <bool DISCARD>
__global__ void __launch_bounds__(ET) k_encounter_tri_batched(
    const int4 *__restrict__ items, const int32_t *__restrict__ off1, const int32_t *__restrict__ n1s,
    const float4 *__restrict__ A1, const float4 *__restrict__ B1, const float4 *__restrict__ V1,
    const double *__restrict__ r1, const double *__restrict__ v1, const double *__restrict__ renc1,
    const int32_t *__restrict__ off2, const int32_t *__restrict__ n2s, const float4 *__restrict__ A2,
    const float4 *__restrict__ B2, const float4 *__restrict__ V2, const double *__restrict__ r2,
    const double *__restrict__ v2, const double *__restrict__ renc2, int upper, double dt, long long cap,
    int32_t *__restrict__ o1, int32_t *__restrict__ o2, int32_t *__restrict__ olv,
    unsigned long long *__restrict__ count, const int32_t *__restrict__ st2) {
    const int4 w = items[blockIdx.x];
    const int s = w.x;
    const int a = off1[s], b = off2[s];
    enc_tri_tile<DISCARD>(n1s[s], A1 + a, B1 + a, V1 + a, r1 + 3 * (size_t)a, v1 + 3 * (size_t)a, renc1 + a,
                          n2s[s], A2 + b, B2 + b, V2 + b, r2 + 3 * (size_t)b, v2 + 3 * (size_t)b,
                          renc2 ? renc2 + b : nullptr, upper, w.y, 0, n1s[s], a, b, dt, cap, o1, o2, olv, count,
                          st2 ? st2 + b : nullptr);
}

// ------------------------------------------------------------------ sorting
// Ascending bitonic network over the N keys (a power of two) at sk, N / 2 threads of the block (all
// of it calls); places (optional) move along, and order equal keys.
template <bool PLACES>
__device__ __forceinline__ void blk_bitonic(int N, uint64_t *sk, uint16_t *si) {
    for (int k = 2; k <= N; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            __syncthreads();
            const int t = threadIdx.x, i = 2 * t - (t & (j - 1)), q = i + j;
            if (t >= N / 2) continue;
            const uint64_t a = sk[i], b = sk[q];
            const bool more = a > b || (PLACES && a == b && si[i] > si[q]);
            if (more == ((i & k) == 0)) {
                sk[i] = b;
                sk[q] = a;
                if (PLACES) {
                    const uint16_t x = si[i];
                    si[i] = si[q];
                    si[q] = x;
                }
            }
        }
    __syncthreads();
}
// The place of key q when each group of MERGE_WAYS sorted runs of `run` keys (a power of two) is merged:
// its place in its run plus, run by run, the count of keys before it there.  Equal keys keep their
// order: they count from the runs before the own one only.
constexpr int MERGE_WAYS = 8, MERGE_TILE = 512;
template <class I>  // I: holds n + MERGE_WAYS run
__device__ __forceinline__ I merge_place(I q, I n, I run, const uint64_t *__restrict__ keys) {
    const uint64_t key = keys[q];
    const I own = q / run, r0 = own / MERGE_WAYS * MERGE_WAYS;
    I place = r0 * run + (q - own * run);
    I lo[MERGE_WAYS - 1], beg[MERGE_WAYS - 1], end[MERGE_WAYS - 1];
    // the searches go in step: each step waits for its loads
#pragma unroll
    for (int w = 0; w < MERGE_WAYS - 1; w++) {
        const I r = r0 + w + (r0 + w >= own);  // the group's runs but the own one
        beg[w] = lo[w] = min(r * run, n);
        end[w] = min((r + 1) * run, n);
    }
#pragma unroll 1
    for (I step = run; step > 0; step >>= 1)
#pragma unroll
        for (int w = 0; w < MERGE_WAYS - 1; w++)
            // all before lo count; the next `step` do if the last of them does
            if (lo[w] + step <= end[w]) {
                const uint64_t k = keys[lo[w] + step - 1];
                if (k < key || (k == key && r0 + w < own)) lo[w] += step;
            }
#pragma unroll
    for (int w = 0; w < MERGE_WAYS - 1; w++) place += lo[w] - beg[w];
    return place;
}

// Pairs (i1, i2, lv) sorted by (i1, i2), repeats dropped (they carry the same lv, 0 or 1).  One key
// holds all three.  Up to PAIRS_BLOCK pairs in one block and launch; more in tiles and merges.
// One key-value network of four launches before: a check of 4096 pl x 40,001 tp 99.7 -> 85.8 us, a
// sort-and-sweep check of 20,000 x 500,000 969 -> 766 us.
constexpr int PAIRS_BLOCK = 2048;
__device__ __forceinline__ uint64_t pair_key(int i1, int i2, int lv) {
    return ((uint64_t)(uint32_t)i1 << 32) | ((uint64_t)(uint32_t)i2 << 1) | (uint64_t)(lv != 0);
}
__device__ __forceinline__ void write_pair(uint64_t k, int64_t o, int32_t *i1, int32_t *i2, int32_t *lv) {
    i1[o] = (int32_t)(k >> 32);
    i2[o] = (int32_t)((uint32_t)k >> 1);
    lv[o] = (int32_t)(k & 1);
}
// keep(t) of the block's elements t in [0, n) to the places after each other, whole block of 1024
template <class K, class W>
__device__ __forceinline__ int64_t blk_compact(int64_t n, K keep, W write) {
    __shared__ int cnt[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int64_t base = 0;
    for (int64_t c0 = 0; c0 < n; c0 += 1024) {
        const int64_t t = c0 + threadIdx.x;
        const bool on = t < n && keep(t);
        const unsigned m = __ballot_sync(0xffffffffu, on);
        if (lane == 0) cnt[w] = __popc(m);
        __syncthreads();
        int c = cnt[lane];
        for (int off = 1; off < 32; off <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, c, off);
            if (lane >= off) c += x;
        }
        const int before = w ? __shfl_sync(0xffffffffu, c, (w + 31) & 31) : 0, total = __shfl_sync(0xffffffffu, c, 31);
        if (on) write(t, base + before + __popc(m & ((1u << lane) - 1)));
        base += total;
        __syncthreads();
    }
    return base;
}
__global__ void __launch_bounds__(1024) k_pairs_block(int n, int N, int32_t *i1, int32_t *i2, int32_t *lv,
                                                      unsigned long long *nout) {
    __shared__ uint64_t sk[PAIRS_BLOCK];
    for (int t = threadIdx.x; t < N; t += 1024) sk[t] = t < n ? pair_key(i1[t], i2[t], lv[t]) : ~0ull;
    blk_bitonic<false>(N, sk, nullptr);
    const int64_t m = blk_compact(
        n, [&](int64_t t) { return t == 0 || (sk[t] >> 1) != (sk[t - 1] >> 1); },
        [&](int64_t t, int64_t o) { write_pair(sk[t], o, i1, i2, lv); });
    if (threadIdx.x == 0) *nout = (unsigned long long)m;
}
__global__ void __launch_bounds__(MERGE_TILE / 2) k_pairs_tiles(int64_t n, const int32_t *i1, const int32_t *i2,
                                                                const int32_t *lv, uint64_t *keys) {
    __shared__ uint64_t sk[MERGE_TILE];
    const int64_t base = blockIdx.x * (int64_t)MERGE_TILE;
    for (int l = threadIdx.x; l < MERGE_TILE; l += MERGE_TILE / 2)
        sk[l] = base + l < n ? pair_key(i1[base + l], i2[base + l], lv[base + l]) : ~0ull;
    blk_bitonic<false>(MERGE_TILE, sk, nullptr);
    for (int l = threadIdx.x; l < MERGE_TILE && base + l < n; l += MERGE_TILE / 2) keys[base + l] = sk[l];
}
template <class I>
__global__ void __launch_bounds__(256) k_pairs_merge(I n, I run, const uint64_t *__restrict__ keys, uint64_t *okeys) {
    const I q = blockIdx.x * (I)256 + threadIdx.x;
    if (q < n) okeys[merge_place(q, n, run, keys)] = keys[q];
}
__global__ void __launch_bounds__(1024) k_pairs_unique(int64_t n, const uint64_t *__restrict__ keys, int32_t *i1,
                                                       int32_t *i2, int32_t *lv, unsigned long long *nout) {
    const int64_t m = blk_compact(
        n, [&](int64_t t) { return t == 0 || (keys[t] >> 1) != (keys[t - 1] >> 1); },
        [&](int64_t t, int64_t o) { write_pair(keys[t], o, i1, i2, lv); });
    if (threadIdx.x == 0) *nout = (unsigned long long)m;
}

// scratch: two buffers of keys
size_t sort_pairs_scratch_bytes(int64_t n) { return (size_t)n * 16 + 256; }

int sort_pairs_unique(swg_ctx *c, int64_t n, int32_t *i1, int32_t *i2, int32_t *lv, void *scratch,
                      unsigned long long *d_nout) {
    if (n <= 0) return SWG_OK;
    if (n <= PAIRS_BLOCK) {
        int N = 2;
        while (N < n) N <<= 1;
        k_pairs_block<<<1, 1024, 0, c->stream>>>((int)n, N, i1, i2, lv, d_nout);
        c->launches++;
        return launch_status(c, "sort_pairs_unique");
    }
    uint64_t *from = (uint64_t *)scratch, *to = from + n;
    k_pairs_tiles<<<(int)((n + MERGE_TILE - 1) / MERGE_TILE), MERGE_TILE / 2, 0, c->stream>>>(n, i1, i2, lv, from);
    c->launches++;
    for (int64_t run = MERGE_TILE; run < n; run *= MERGE_WAYS) {
        const int grid = (int)((n + 255) / 256);
        if (n <= 1 << 27)
            k_pairs_merge<int><<<grid, 256, 0, c->stream>>>((int)n, (int)run, from, to);
        else
            k_pairs_merge<int64_t><<<grid, 256, 0, c->stream>>>(n, run, from, to);
        c->launches++;
        std::swap(from, to);
    }
    k_pairs_unique<<<1, 1024, 0, c->stream>>>(n, from, i1, i2, lv, d_nout);
    c->launches++;
    return launch_status(c, "sort_pairs_unique");
}

// ------------------------------------------------------------------ sort & sweep
// orderable bit pattern of a double (ascending numeric order)
__device__ __forceinline__ uint64_t d2key(double x) {
    if (x == 0.0) x = 0.0;  // -0.0 compares equal to +0.0: one key for both
    uint64_t u = (uint64_t)__double_as_longlong(x);
    return (u & 0x8000000000000000ull) ? ~u : (u | 0x8000000000000000ull);
}

// gfortran NORM2 (scaled sum of squares), as used for |r| in the sweep extents
__device__ __forceinline__ double d_norm2e(double a, double b, double c) {
    double scale = 0.0, ssq = 1.0;
    const double v[3] = {a, b, c};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        if (v[k] != 0.0) {
            const double absx = fabs(v[k]);
            if (scale < absx) {
                if (scale != 0.0) {  // else q = 0: ssq stays 1
                    const double q = xdiv(scale, absx);
                    ssq = 1.0 + ssq * q * q;
                }
                scale = absx;
            } else {
                const double q = xdiv(absx, scale);
                ssq = ssq + q * q;
            }
        }
    }
    return scale * xsqrt(ssq);
}

// extents: body b (0..ntot-1) -> keys[b] = rmin, keys[ntot+b] = rmax, vals = extent index
__global__ void k_sas_extents(int n1, const double *r1, const double *renc1, int n2, const double *r2,
                              const double *renc2, uint64_t *keys, uint32_t *vals) {
    const int ntot = n1 + n2;
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= ntot) return;
    const double *r = b < n1 ? &r1[3 * b] : &r2[3 * (b - n1)];
    const double rc = b < n1 ? renc1[b] : (renc2 ? renc2[b - n1] : 0.0);
    const double rmag = d_norm2e(r[0], r[1], r[2]);
    keys[b] = d2key(rmag - RSWEEP_FACTOR * rc);
    vals[b] = (uint32_t)b;
    keys[ntot + b] = d2key(rmag + RSWEEP_FACTOR * rc);
    vals[ntot + b] = (uint32_t)(ntot + b);
}

__global__ void k_sas_positions(int ntot, const uint32_t *vals, int32_t *ibeg, int32_t *iend) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= 2 * ntot) return;
    const uint32_t e = vals[k];
    if (e < (uint32_t)ntot)
        ibeg[e] = k + 1;
    else
        iend[e - ntot] = k + 1;
}

// sweep: body b with loverlap tests the bodies whose extents are strictly inside its box.
// FA/FB/FV: float copies of the ntot bodies (list 1 then list 2) for the conservative FP32
// prefilter, which drops only pairs the FP64 test is certain to reject (see
// prefilter_reject), so the list is the same.  One warp per body: its lanes take the
// entries of the body's box 32 at a time (a box holds up to hundreds of entries in a
// disk, and a thread per body left the scan latency-bound on its serial loads); the
// pairs' order in the output does not matter (the lists are sorted afterwards).
__global__ void k_sas_sweep(int n1, const double *r1, const double *v1, const double *renc1, int n2,
                            const double *r2, const double *v2, const double *renc2, int single, int shift2, double dt,
                            const uint32_t *vals, const int32_t *ibeg, const int32_t *iend, const float4 *FA,
                            const float4 *FB, const float4 *FV, long long cap, int32_t *o1, int32_t *o2, int32_t *olv,
                            unsigned long long *count) {
    const int ntot = n1 + n2;
    const int i = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);  // warp-uniform
    if (i >= ntot) return;
    if (!((ibeg[i] + 1) < (iend[i] - 1))) return;
    const bool il1 = i < n1;
    const double *ri = il1 ? &r1[3 * i] : &r2[3 * (i - n1)];
    const double *vi = il1 ? &v1[3 * i] : &v2[3 * (i - n1)];
    const double renci = il1 ? renc1[i] : (renc2 ? renc2[i - n1] : 0.0);
    const BodyF q = {FA[i], FB[i], FV[i]};
    const float dtf = __double2float_ru(fabs(dt)) * (1.0f + 1e-6f);  // |dt| bounds either direction of time
    const int pend = iend[i] - 1;
    for (int p = ibeg[i] + 1 + (int)(threadIdx.x & 31); p <= pend; p += 32) {
        int b = (int)vals[p - 1];
        if (b >= ntot) b -= ntot;
        const bool bl1 = b < n1;
        if (!single && bl1 == il1) continue;
        const BodyF f = {FA[b], FB[b], FV[b]};
        if (prefilter_reject(f, q, dtf)) continue;
        const double *rb = bl1 ? &r1[3 * b] : &r2[3 * (b - n1)];
        const double *vb = bl1 ? &v1[3 * b] : &v2[3 * (b - n1)];
        const double rencb = bl1 ? renc1[b] : (renc2 ? renc2[b - n1] : 0.0);
        int lenc, lv;
        d_encounter_one(rb[0] - ri[0], rb[1] - ri[1], rb[2] - ri[2], vb[0] - vi[0], vb[1] - vi[1], vb[2] - vi[2],
                        renci + rencb, dt, lenc, lv);
        if (!lenc) continue;
        int a, cidx;
        if (single) {
            a = min(i, b) + 1;
            cidx = max(i, b) + 1;
        } else if (il1) {
            a = i + 1;
            cidx = b - n1 + 1 + shift2;
        } else {
            a = b + 1;
            cidx = i - n1 + 1 + shift2;
        }
        const unsigned long long k = atomicAdd(count, 1ull);
        if ((long long)k < cap) {
            o1[k] = a;
            o2[k] = cidx;
            olv[k] = lv;
        }
    }
}

// The sorted order of one system's extents, up to SAS_MERGED of them: each block forms and sorts a
// tile of SAS_TILE in shared memory, then rounds of merges join up to MERGE_WAYS runs each
// (merge_place).  Ties keep the extents' order, as in the radix sort.  Bound by launches and dependent loads: two to five launches here,
// up to 24 and a host read in the radix sort.  A whole pl-tp check, radix sort and this: 314 x 2501
// bodies 168 -> 62 us, 2370 x 3650 220 -> 119, 8192 x 50,000 292 -> 198, 4000 x 200,000 462 -> 407,
// 20,000 x 500,000 1012 and 1033, hence the line.  Merges of 16 runs: 50, 122, 191, 458 us; tiles of
// 2048 took 60 us themselves.
constexpr int SAS_TILE = MERGE_TILE, SAS_T = SAS_TILE / 2;
constexpr int64_t SAS_MERGED = 524288;
__global__ void __launch_bounds__(SAS_T) k_sas_tiles(int n1, const double *r1, const double *v1, const double *renc1,
                                                     int n2, const double *r2, const double *v2, const double *renc2,
                                                     uint64_t *keys, uint32_t *ids, float4 *FA, float4 *FB,
                                                     float4 *FV) {
    __shared__ uint64_t sk[SAS_TILE];
    __shared__ uint16_t si[SAS_TILE];
    const int ntot = n1 + n2, ne = 2 * ntot, base = blockIdx.x * SAS_TILE;
    for (int l = threadIdx.x; l < SAS_TILE; l += SAS_T) {
        const int e = base + l;
        uint64_t k = ~0ull;  // beyond the last extent (after it also where its key is the same)
        if (e < ne) {
            const int b = e < ntot ? e : e - ntot;
            const bool il1 = b < n1;
            const double *r = il1 ? &r1[3 * b] : &r2[3 * (b - n1)];
            const double rc = il1 ? renc1[b] : (renc2 ? renc2[b - n1] : 0.0);
            const double rmag = d_norm2e(r[0], r[1], r[2]);
            k = d2key(e < ntot ? rmag - RSWEEP_FACTOR * rc : rmag + RSWEEP_FACTOR * rc);
            if (e < ntot) {
                const BodyF o = il1 ? load_body(r1, v1, renc1, b) : load_body(r2, v2, renc2, b - n1);
                FA[b] = o.a;
                FB[b] = o.b;
                FV[b] = o.v;
            }
        }
        sk[l] = k;
        si[l] = (uint16_t)l;
    }
    blk_bitonic<true>(SAS_TILE, sk, si);
    for (int l = threadIdx.x; l < SAS_TILE && base + l < ne; l += SAS_T) {
        keys[base + l] = sk[l];
        ids[base + l] = (uint32_t)(base + si[l]);
    }
}
// Runs of `run` extents in (keys, ids) to runs of MERGE_WAYS run in (okeys, oids), or, in the last
// round (okeys null), to the sorted order: oids and the positions of each body's two extents.
__global__ void __launch_bounds__(256) k_sas_merge(int ntot, int run, const uint64_t *__restrict__ keys,
                                                   const uint32_t *__restrict__ ids, uint64_t *okeys, uint32_t *oids,
                                                   int32_t *ibeg, int32_t *iend) {
    const int ne = 2 * ntot, q = blockIdx.x * 256 + threadIdx.x;
    if (q >= ne) return;
    const int place = merge_place(q, ne, run, keys);
    const uint32_t e = ids[q];
    oids[place] = e;
    if (okeys)
        okeys[place] = keys[q];
    else if (e < (uint32_t)ntot)
        ibeg[e] = place + 1;
    else
        iend[e - ntot] = place + 1;
}

// keys | vals | ibeg | iend | radix-sort scratch, each 256-byte aligned
static size_t align256(size_t b) { return (b + 255) & ~size_t(255); }
size_t sas_scratch_bytes(int ntot) {
    const int64_t ne = 2 * (int64_t)ntot;
    return align256((size_t)ne * 8) + align256((size_t)ne * 4) + align256((size_t)ntot * 8) +
           align256((size_t)ntot * 3 * sizeof(float4)) + radix_sort_scratch_bytes(ne) + 256;
}

// Sort-and-sweep check of one list (single, pl-pl: list 1) or two lists (pl-tp), of one
// system or, with seg_of (the system of every extent, 2 (n1 + n2) entries), of every system
// of an ensemble at once: the extents sort into per-system runs and each body sweeps only its
// own run.  Pairs land unsorted in (o1, o2, olv) with the total in *count.  host_skip: the
// radix sort reads its digit counts back to skip constant digits (synchronizes the stream).
int sas_launch(swg_ctx *c, int n1, const double *r1, const double *v1, const double *renc1, int n2, const double *r2,
               const double *v2, const double *renc2, int single, int shift2, double dt, long long cap, int32_t *o1,
               int32_t *o2, int32_t *olv, unsigned long long *count, void *scratch, const int32_t *seg_of,
               int seg_bits, bool host_skip) {
    const int nb1 = n1, nb2 = single ? 0 : n2;
    const int ntot = nb1 + nb2;
    if (ntot <= 0) return SWG_OK;
    const int64_t ne = 2 * (int64_t)ntot;
    char *p = (char *)scratch;
    uint64_t *keys = (uint64_t *)p;
    uint32_t *vals = (uint32_t *)(p += align256((size_t)ne * 8));
    int32_t *ibeg = (int32_t *)(p += align256((size_t)ne * 4));
    int32_t *iend = ibeg + ntot;
    float4 *FA = (float4 *)(p += align256((size_t)ntot * 8)), *FB = FA + ntot, *FV = FB + ntot;
    void *rs = p + align256((size_t)ntot * 3 * sizeof(float4));
    const bool merged = !seg_of && ne <= SAS_MERGED;
    if (merged) {
        uint64_t *bkeys = (uint64_t *)rs;  // the radix sort's scratch holds 16 bytes an extent
        uint32_t *bids = (uint32_t *)(bkeys + ne), *ids = bids + ne;
        const int tiles = (int)((ne + SAS_TILE - 1) / SAS_TILE), grid = (int)((ne + 255) / 256);
        k_sas_tiles<<<tiles, SAS_T, 0, c->stream>>>(nb1, r1, v1, renc1, nb2, r2, v2, renc2, keys, ids, FA, FB, FV);
        int64_t run = SAS_TILE;
        uint64_t *from = keys, *to = bkeys;
        uint32_t *idf = ids, *idt = bids;
        for (; run * MERGE_WAYS < ne; run *= MERGE_WAYS) {
            k_sas_merge<<<grid, 256, 0, c->stream>>>(ntot, (int)run, from, idf, to, idt, nullptr, nullptr);
            std::swap(from, to);
            std::swap(idf, idt);
            c->launches++;
        }
        k_sas_merge<<<grid, 256, 0, c->stream>>>(ntot, (int)run, from, idf, nullptr, vals, ibeg, iend);
        c->launches += 2;
    } else {
        k_sas_extents<<<(ntot + 127) / 128, 128, 0, c->stream>>>(nb1, r1, renc1, nb2, r2, renc2, keys, vals);
        c->launches++;
    }
    if (!merged && nb1 > 0) {
        k_encounter_prep<<<(nb1 + 255) / 256, 256, 0, c->stream>>>(nb1, r1, v1, renc1, FA, FB, FV);
        c->launches++;
    }
    if (!merged && nb2 > 0) {
        k_encounter_prep<<<(nb2 + 255) / 256, 256, 0, c->stream>>>(nb2, r2, v2, renc2, FA + nb1, FB + nb1, FV + nb1);
        c->launches++;
    }
    if (!merged) {
        // stable radix sort by extent; the extents enter in index order, so ties keep it
        SWG_TRY(radix_sort_kv(c, ne, keys, vals, rs, seg_of, seg_bits, host_skip));
        k_sas_positions<<<(int)((ne + 255) / 256), 256, 0, c->stream>>>(ntot, vals, ibeg, iend);
        c->launches++;
    }
    k_sas_sweep<<<(unsigned)((32 * (int64_t)ntot + 127) / 128), 128, 0, c->stream>>>(
        nb1, r1, v1, renc1, nb2, r2, v2, renc2, single, shift2, dt, vals, ibeg, iend, FA, FB, FV, cap, o1, o2, olv,
        count);
    c->launches++;
    return launch_status(c, "encounter_sas");
}

// Runs one encounter check; pairs land unsorted in (o1,o2,olv) (first cap of
// them) and the total in *count (device).  Caller sorts/dedups afterwards.
int encounter_launch(swg_ctx *c, int mode, int n1, const double *r1, const double *v1, const double *renc1, int n2,
                     const double *r2, const double *v2, const double *renc2, int upper, int shift2, double dt,
                     long long cap, int32_t *o1, int32_t *o2, int32_t *olv, unsigned long long *count,
                     void *sas_scratch) {
    if (mode == SWG_ENC_SORTSWEEP)  // single list when upper (pl-pl), double list otherwise
        return sas_launch(c, n1, r1, v1, renc1, n2, r2, v2, renc2, upper ? 1 : 0, shift2, dt, cap, o1, o2, olv, count,
                          sas_scratch, nullptr, 0, true);
    if (n1 <= 0 || n2 <= 0) return SWG_OK;
    // float copies for the prefilter: list 1 then (unless it is the same list) list 2
    float4 *A1 = (float4 *)sas_scratch, *B1 = A1 + n1, *V1 = B1 + n1;
    float4 *A2 = A1, *B2 = B1, *V2 = V1;
    const bool same = upper && r2 == r1;
    if (!same) {
        A2 = V1 + n1;
        B2 = A2 + n2;
        V2 = B2 + n2;
    }
    const int np = n1 + (same ? 0 : n2);
    k_encounter_prep2<<<(np + 127) / 128, 128, 0, c->stream>>>(n1, r1, v1, renc1, A1, np - n1, r2, v2, renc2, A2);
    c->launches++;
    const int bx = (n2 + ET - 1) / ET;
    const int target = 4 * (c->num_sms > 0 ? c->num_sms : 152);
    int nchunk = (target + bx - 1) / bx;
    const int maxchunk = (n1 + EP - 1) / EP;
    if (nchunk > maxchunk) nchunk = maxchunk;
    if (nchunk < 1) nchunk = 1;
    int chunk = (n1 + nchunk - 1) / nchunk;
    chunk = (chunk + EP - 1) / EP * EP;
    nchunk = (n1 + chunk - 1) / chunk;
    k_encounter_tri<false><<<dim3(bx, nchunk), ET, 0, c->stream>>>(n1, A1, B1, V1, r1, v1, renc1, n2, A2, B2, V2, r2,
                                                                   v2, renc2, upper, shift2, dt, chunk, cap, o1, o2, olv,
                                                                   count, nullptr);
    c->launches++;
    return launch_status(c, "encounter_tri");
}

// Float copies (A, B, V) of n bodies for the prefilter of the batched check.
int encounter_prep_launch(swg_ctx *c, int64_t n, const double *r, const double *v, const double *renc, float4 *A,
                          float4 *B, float4 *V) {
    if (n <= 0) return SWG_OK;
    k_encounter_prep<<<(int)((n + 255) / 256), 256, 0, c->stream>>>((int)n, r, v, renc, A, B, V);
    c->launches++;
    return launch_status(c, "encounter_prep");
}

// Batched TRIANGULAR check over an item table (see k_encounter_tri_batched); F1/F2 are
// the prepared float copies (3 arrays of float4 each, A|B|V) of list 1 and list 2.
int encounter_tri_batched(swg_ctx *c, int nitems, const int4 *items, const int32_t *off1, const int32_t *n1,
                          const float4 *F1, int64_t nf1, const double *r1, const double *v1, const double *renc1,
                          const int32_t *off2, const int32_t *n2, const float4 *F2, int64_t nf2, const double *r2,
                          const double *v2, const double *renc2, int upper, double dt, long long cap, int32_t *o1,
                          int32_t *o2, int32_t *olv, unsigned long long *count) {
    if (nitems <= 0) return SWG_OK;
    k_encounter_tri_batched<false><<<nitems, ET, 0, c->stream>>>(items, off1, n1, F1, F1 + nf1, F1 + 2 * nf1, r1, v1,
                                                                 renc1, off2, n2, F2, F2 + nf2, F2 + 2 * nf2, r2, v2,
                                                                 renc2, upper, dt, cap, o1, o2, olv, count, nullptr);
    c->launches++;
    return launch_status(c, "encounter_tri_batched");
}

// Close-approach discard scan (swiftest_discard_pl_tp, src/swiftest/swiftest_discard.f90:244-290)
// of the ACTIVE test particles of one system against its massive bodies: heliocentric
// positions and velocities, r2crit = radius^2; flag[j] = 1 for every tp that comes too
// close to some pl (flag zeroed by the caller).  F: scratch for the float copies,
// 3 * (npl + ntp) float4.
int discard_pl_tp_launch(swg_ctx *c, int32_t npl, const double *rpl, const double *vpl, const double *radius,
                         int32_t ntp, const double *rtp, const double *vtp, const int32_t *tstatus, double dt,
                         float4 *F, int32_t *flag) {
    if (npl <= 0 || ntp <= 0) return SWG_OK;
    float4 *A1 = F, *B1 = A1 + npl, *V1 = B1 + npl, *A2 = V1 + npl, *B2 = A2 + ntp, *V2 = B2 + ntp;
    k_encounter_prep<<<(npl + 255) / 256, 256, 0, c->stream>>>(npl, rpl, vpl, radius, A1, B1, V1);
    k_encounter_prep<<<(ntp + 255) / 256, 256, 0, c->stream>>>(ntp, rtp, vtp, nullptr, A2, B2, V2);
    c->launches += 2;
    const int bx = (ntp + ET - 1) / ET;
    const int target = 4 * (c->num_sms > 0 ? c->num_sms : 152);
    int nchunk = std::max(1, std::min((target + bx - 1) / bx, (npl + EP - 1) / EP));
    int chunk = (npl + nchunk - 1) / nchunk;
    chunk = (chunk + EP - 1) / EP * EP;
    nchunk = (npl + chunk - 1) / chunk;
    k_encounter_tri<true><<<dim3(bx, nchunk), ET, 0, c->stream>>>(npl, A1, B1, V1, rpl, vpl, radius, ntp, A2, B2, V2,
                                                                  rtp, vtp, nullptr, 0, 0, dt, chunk, 0, nullptr,
                                                                  flag, nullptr, nullptr, tstatus);
    c->launches++;
    return launch_status(c, "discard_pl_tp");
}

// The same scan for every system of an ensemble over its pl-tp item table; F1/F2: the
// float copies (A|B|V) of all pl (nf1 = NPL) and tp (nf2 = NTP), prepared here.
int discard_pl_tp_batched(swg_ctx *c, int nitems, const int4 *items, const int32_t *poff, const int32_t *npl,
                          int64_t NPL, const double *rpl, const double *vpl, const double *radius,
                          const int32_t *toff, const int32_t *ntp, int64_t NTP, const double *rtp, const double *vtp,
                          const int32_t *tstatus, double dt, float4 *F1, float4 *F2, int32_t *flag) {
    if (nitems <= 0) return SWG_OK;
    SWG_TRY(encounter_prep_launch(c, NPL, rpl, vpl, radius, F1, F1 + NPL, F1 + 2 * NPL));
    SWG_TRY(encounter_prep_launch(c, NTP, rtp, vtp, nullptr, F2, F2 + NTP, F2 + 2 * NTP));
    k_encounter_tri_batched<true><<<nitems, ET, 0, c->stream>>>(items, poff, npl, F1, F1 + NPL, F1 + 2 * NPL, rpl, vpl,
                                                                radius, toff, ntp, F2, F2 + NTP, F2 + 2 * NTP, rtp,
                                                                vtp, nullptr, 0, dt, 0, nullptr, flag, nullptr,
                                                                nullptr, tstatus);
    c->launches++;
    return launch_status(c, "discard_pl_tp_batched");
}

// scratch of one encounter_launch call (mode, list sizes)
size_t encounter_scratch_bytes(int mode, int n1, int n2) {
    if (mode == SWG_ENC_SORTSWEEP) return sas_scratch_bytes(n1 + n2);
    return (size_t)3 * sizeof(float4) * (size_t)(n1 + n2) + 256;
}

// shift index2 by `shift` for entries [from, to)
__global__ void k_shift_i2(long long from, long long to, int32_t *i2, int shift) {
    const long long t = from + blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t < to) i2[t] += shift;
}

int shift_index2(swg_ctx *c, long long from, long long to, int32_t *i2, int shift) {
    if (to <= from || shift == 0) return SWG_OK;
    k_shift_i2<<<(int)((to - from + 255) / 256), 256, 0, c->stream>>>(from, to, i2, shift);
    c->launches++;
    return launch_status(c, "shift_i2");
}

}  // namespace swg

namespace swg {

// From this many pair tests on, a TRIANGULAR check of one list, or of massive bodies against test
// particles, goes over radius-sorted tiles, which test a few percent of a disk's pairs but take
// two launches more; whole calls all-pairs / sorted: 300 x 20,000 66 / 67 us, 1000 x 10,000 72 / 72,
// 400 x 50,000 93 / 72, 8192 x 50,000 935 / 112.  Against fewer massive bodies than SORTED_PL the
// ordering of the test particles costs more than it saves: 8 x 1,251,251 97 / 135 us, 32 x 312,813
// 61 / 74, 48 x 2,000,001 292 / 249, 64 x 156,407 105 / 83.
constexpr int64_t SORTED_PAIRS = 10000000;
constexpr int SORTED_PL = 64;

int encounter_check_kind(swg_ctx *c, EncWork &w, int kind, int mode, int32_t n1, const double *r1,
                         const double *v1, const double *renc1, int32_t n2, const double *r2, const double *v2,
                         const double *renc2, double dt, int64_t *n_out, int32_t **o1, int32_t **o2,
                         int32_t **olv) {
    *n_out = 0;
    SWG_TRY(ensure(c, w.counters, 2 * sizeof(unsigned long long)));
    unsigned long long *d_count = (unsigned long long *)w.counters.ptr;
    if (w.rawcap < 1024) {
        w.rawcap = 1024;
        SWG_TRY(ensure(c, w.raw, (size_t)w.rawcap * 3 * sizeof(int32_t)));
    }
    const int64_t pairs = kind == 0 ? (int64_t)n1 * n1 / 2 : (int64_t)n1 * n2;
    const bool sorted = mode == SWG_ENC_TRIANGULAR && kind != 1 && n1 >= SORTED_PL && pairs >= SORTED_PAIRS;
    SWG_TRY(ensure(c, w.sort, sorted ? encounter_sorted_one_bytes(n1, kind == 0 ? 0 : n2)
                                     : encounter_scratch_bytes(mode, n1, kind == 0 ? n1 : n2)));
    unsigned long long h_count = 0;
    for (int attempt = 0; attempt < 8; attempt++) {
        int32_t *i1 = (int32_t *)w.raw.ptr, *i2 = i1 + w.rawcap, *lv = i2 + w.rawcap;
        SWG_TRY(cuda_status(c, cudaMemsetAsync(d_count, 0, sizeof(unsigned long long), c->stream), "memset"));
        if (sorted) {
            SWG_TRY(encounter_sorted_one(c, n1, r1, v1, renc1, kind == 0 ? 0 : n2, r2, v2, dt, w.rawcap, i1, i2, lv,
                                         d_count, w.sort.ptr));
        } else if (kind == 0) {
            SWG_TRY(encounter_launch(c, mode, n1, r1, v1, renc1, n1, r1, v1, renc1, 1, 0, dt, w.rawcap, i1, i2, lv,
                                     d_count, w.sort.ptr));
        } else if (kind == 1) {
            SWG_TRY(encounter_launch(c, mode, n1, r1, v1, renc1, n1, r1, v1, renc1, 1, 0, dt, w.rawcap, i1, i2, lv,
                                     d_count, w.sort.ptr));
            if (n2 > 0)
                SWG_TRY(encounter_launch(c, mode, n1, r1, v1, renc1, n2, r2, v2, renc2, 0, n1, dt, w.rawcap, i1, i2,
                                         lv, d_count, w.sort.ptr));
        } else {
            SWG_TRY(encounter_launch(c, mode, n1, r1, v1, renc1, n2, r2, v2, nullptr, 0, 0, dt, w.rawcap, i1, i2, lv,
                                     d_count, w.sort.ptr));
        }
        SWG_TRY(cuda_status(c, cudaMemcpyAsync(&h_count, d_count, sizeof(h_count), cudaMemcpyDeviceToHost, c->stream),
                            "count"));
        SWG_TRY(cuda_status(c, cudaStreamSynchronize(c->stream), "sync"));
        if ((int64_t)h_count <= w.rawcap) break;
        // grow the raw buffers and redo the check
        w.rawcap = (int64_t)h_count + h_count / 2 + 1024;
        DevBuf fresh;
        SWG_TRY(ensure(c, fresh, (size_t)w.rawcap * 3 * sizeof(int32_t)));
        cudaFree(w.raw.ptr);
        w.raw = fresh;
    }
    int32_t *i1 = (int32_t *)w.raw.ptr, *i2 = i1 + w.rawcap, *lv = i2 + w.rawcap;
    *o1 = i1;
    *o2 = i2;
    *olv = lv;
    if (h_count == 0) return SWG_OK;
    // sort by (index1, index2) and drop repeats; only the sweep repeats pairs, so only its count
    // is read again
    const size_t need = sort_pairs_scratch_bytes((int64_t)h_count);
    if (w.sort.bytes < need) SWG_TRY(ensure(c, w.sort, need));
    SWG_TRY(sort_pairs_unique(c, (int64_t)h_count, i1, i2, lv, w.sort.ptr, d_count + 1));
    if (mode == SWG_ENC_TRIANGULAR) {
        *n_out = (int64_t)h_count;
        return SWG_OK;
    }
    unsigned long long h_unique = 0;
    SWG_TRY(cuda_status(c, cudaMemcpyAsync(&h_unique, d_count + 1, sizeof(h_unique), cudaMemcpyDeviceToHost, c->stream),
                        "count"));
    SWG_TRY(cuda_status(c, cudaStreamSynchronize(c->stream), "sync"));
    *n_out = (int64_t)h_unique;
    return SWG_OK;
}

}  // namespace swg
