// kick_fp64.cu -- FP64 pair kick in the reference's exact operation order, spread over all SMs.
//
// Restates swiftest_kick_getacch_int_all_tri_* (src/swiftest/swiftest_kick.f90:165-371),
// the flat forms (:69-162) and swiftest_kick_getacch_int_all_tp (:374-415).
//
// Every per-body sum must add its terms one at a time in ascending partner order
// to reproduce the reference's rounding, which leaves no parallelism inside one
// body's sum; the terms themselves have no such constraint.  A block therefore owns RT
// receivers: each of RT term warps forms one receiver's terms, 32 partners a round (one per
// lane), and the fold warp adds the rounds' terms in order, one lane per (receiver,
// component), so that one addition of the narrow FP64 pipe serves 3 RT sums.  The terms pass
// through a ring in shared memory.
//
// Bound: the FP64 pipe, at 16 cycles per warp instruction and SM (19 for DADD, so additions
// are issued as DFMA with a factor of one: the same rounding).  The square root, the
// quotient and the products are formed outside that pipe (fp64_exact.cuh, the same bits), which
// leaves five additions per pair and 3.2 for the fold: 8.2 instructions, 131 cycles, per 32
// pairs and SM against ~40 before.  65,537 tp x 2047 pl: 10.3 -> 2.5 ms (16,384 pl: 22.6 -> 5.3 ms),
// FP64 pipe 77%, ALU pipe 60%, issue slots 68% busy (ncu): the long chains of dependent
// instructions want warps (three blocks of 56 registers per SM: 2.8 ms, two: 3.9 ms).
//
#include <cuda_runtime.h>

#include "fp64_exact.cuh"
#include "swg_internal.cuh"

namespace swg {

// Most receivers per block (which the batched forms use), and blocks per SM.  Ten receivers fill 30
// of the fold warp's 32 lanes, with four blocks of 40 registers a thread.  The test particles' forms
// spill little at 32 registers, where six blocks of nine fit: more chains of additions at a time
// (2047 pl x 65,537 tp: 2.58 -> 2.53 ms; the pl-pl forms 5.28 -> 5.34 ms; blocks of eight 2.64 and
// 5.51 ms, of seven 2.74 and 5.68 ms).
constexpr int FP64_RT = KICK_FP64_TILE, FP64_BLOCKS = 4;
constexpr int FP64_RT_TP = KICK_FP64_TP_TILE, FP64_BLOCKS_TP = 6;
constexpr int PT = 32;                   // partners per round

static_assert(3 * FP64_RT <= 32 && 3 * FP64_RT_TP <= 32, "one fold warp");
__host__ __device__ constexpr int fp64_threads(int rt) { return 32 * (rt + 1); }
// doubles per partner of a stage (odd: conflict-free columns) and bytes of the ring
__host__ __device__ constexpr int term_stride(int rt) { return (3 * rt) | 1; }

// Opaque one: an addition as fma(a, 1, b) stays a DFMA.
__constant__ double c_one = 1.0;
__constant__ double c_mone = -1.0;
__device__ __forceinline__ double add1(double a, double b) { return fma(a, c_one, b); }
__device__ __forceinline__ double sub1(double a, double b) { return fma(b, c_mone, a); }

enum { KICK_TP = 2 };  // beside KICK_DIRECT and KICK_SPLIT

// Terms of ST = 2 rounds: a ring between the term warps and the fold warp.  Barrier 1 + s:
// a round's terms are in stage s (term warps arrive, the fold warp waits); barrier 3 + s: its
// sums are made (the fold warp arrives, the term warps wait).  Three, four and six stages
// measured no faster.
constexpr int ST = 2;
template <int BASE>
__device__ __forceinline__ void bar_sync(int s, int n) {  // constant barrier numbers: five per block
    if (s) asm volatile("bar.sync %0, %1;" ::"n"(BASE + 1), "r"(n) : "memory");
    else asm volatile("bar.sync %0, %1;" ::"n"(BASE), "r"(n) : "memory");
}
template <int BASE>
__device__ __forceinline__ void bar_arrive(int s, int n) {
    if (s) asm volatile("bar.arrive %0, %1;" ::"n"(BASE + 1), "r"(n) : "memory");
    else asm volatile("bar.arrive %0, %1;" ::"n"(BASE), "r"(n) : "memory");
}
constexpr int FULL = 1, EMPTY = 3;

// A float not below 2 R^2, so that bound(R_i) + bound(R_j) >= (R_i + R_j)^2: R cut to its
// leading 24 bits and one unit more (a conversion would take the FP64 pipe), infinity out of
// range.
__device__ __forceinline__ float radius_bound(double R) {
    const int hi = __double2hiint(R), lo = __double2loint(R);
    if (!x_ok(hi)) return (hi | lo) == 0 ? 0.0f : __int_as_float(0x7f800000);
    const float f = __int_as_float(__funnelshift_l(lo, hi - ((1023 - 127) << 20), 3) + 1);
    return __fmul_ru(2.0f, __fmul_ru(f, f));
}

// Displacements outside the exact products' range, found by one test of the smallest and one of
// the largest exponent (a test per component: kick_pl_fp64's 16,384 bodies 5.47 ms, this 5.29).
// A zero component is replaced by 2^-300, whose square leaves every other square and r^2 as they
// are, and marked (bit c of the result); what else is out of range sets bad.
__device__ __forceinline__ int odd_disp(double &dx, double &dy, double &dz, bool &bad) {
    constexpr int LOW = (1023 - XR_EXP) << 20, HIGH = ((1023 + XR_EXP + 1) << 20) - 1;
    auto one = [&](double &d, int bit) {
        const int h = __double2hiint(d) & 0x7fffffff;
        if (h >= LOW) return 0;
        bad |= (h | __double2loint(d)) != 0;
        d = __hiloint2double((1023 - 300) << 20, 0);
        return bit;
    };
    const int hx = __double2hiint(dx) & 0x7fffffff, hy = __double2hiint(dy) & 0x7fffffff,
              hz = __double2hiint(dz) & 0x7fffffff;
    bad |= max(hx, max(hy, hz)) > HIGH;
    if (min(hx, min(hy, hz)) >= LOW) return 0;
    return one(dx, 1) | one(dy, 2) | one(dz, 4);
}

// Receivers [i0, i0 + RT) (those below nrecv) of one system against all its partners, whole
// block of fp64_threads(RT) threads; sh: fp64_shared(RT) bytes.  kv: the velocities that the
// finished accelerations kick (KickVel; a launch of their own took 3 us).  MODE: KICK_DIRECT and
// KICK_SPLIT (pl-pl), KICK_TP (swiftest_kick.f90:374-415: acc -= Gm_j / (r^2 sqrt r^2)
// (r_tp - r_j), masked).
template <bool RAD, int MODE>
__device__ __forceinline__ void fp64_group(int RT, int nrecv, int npart, int nplm, const double *__restrict__ rr,
                                           const double *__restrict__ rp, const double *__restrict__ Gm,
                                           const double *__restrict__ R, const int32_t *__restrict__ lmask,
                                           double *__restrict__ acc, int acc_is_zero, int i0, double *sh, const KickVel &kv = KickVel()) {
    const int nth = fp64_threads(RT), ts = term_stride(RT);
    const int w = (int)(threadIdx.x >> 5) - 1, lane = threadIdx.x & 31;
    constexpr bool plpl = MODE != KICK_TP;
    const int jmax = plpl && i0 >= nplm ? nplm : npart;  // partners of the block's receivers
    const int rounds = (jmax + PT - 1) / PT;
    if (!plpl) {  // a block without an active receiver
        const int i = i0 + (int)threadIdx.x;
        if (!__syncthreads_or((int)threadIdx.x < RT && i < nrecv && lmask[i] != 0)) {
            if (acc_is_zero)
                for (int k = threadIdx.x; k < 3 * min(RT, nrecv - i0); k += nth) acc[3 * i0 + k] = 0.0;
            return;
        }
    }
    if (w >= 0) {  // term warps: warp w + 1 of the block
        // a term that leaves the sum as it is, signed zeros included
        const double neutral = plpl ? -0.0 : 0.0;
        const int i = i0 + w;
        const bool on = i < nrecv && (plpl || lmask[i] != 0);
        double xi = 0, yi = 0, zi = 0;
        float rbi = 0;
        if (on) {
            xi = rr[3 * i + 0];
            yi = rr[3 * i + 1];
            zi = rr[3 * i + 2];
            if (RAD) rbi = radius_bound(R[i]);
        }
        const int jend = !on ? 0 : (plpl && i >= nplm ? nplm : npart);
        double *out = sh + lane * ts + 3 * w;
        for (int r = 0; r < rounds; r++) {
            const int j = r * PT + lane, st = r % ST;
            double fx = neutral, fy = neutral, fz = neutral;
            if (j < jend && (!plpl || j != i)) {
                const double g = Gm[j];
                const double xj = rp[3 * j + 0], yj = rp[3 * j + 1], zj = rp[3 * j + 2];
                double dx = plpl ? sub1(xj, xi) : sub1(xi, xj);
                double dy = plpl ? sub1(yj, yi) : sub1(yi, yj);
                double dz = plpl ? sub1(zj, zi) : sub1(zi, zj);
                bool bad = false, near = false;
                const int zero = odd_disp(dx, dy, dz, bad);
                const double r2 = add1(add1(x_sqr(dx), x_sqr(dy)), x_sqr(dz));
                const int h = __double2hiint(r2);
                bad |= !x_ok(h) || !x_ok(__double2hiint(g));
                if (RAD) near = !(__int_as_float((h - ((1023 - 127) << 20)) << 3) > __fadd_ru(rbi, radius_bound(R[j])));
                const double s = x_sqrt(r2, bad);
                const double p = x_mul(r2, s);  // within 2^+-152: g / p and the terms stay normal
                double fac;
                if (MODE == KICK_SPLIT) {
                    const XNum one = {1.0f, 0.0f, 0x3ff00000, 0};
                    fac = g * x_div(one, p, bad);
                } else {
                    fac = x_div(x_num(g), p, bad);
                }
                fx = x_mul(fac, dx);
                fy = x_mul(fac, dy);
                fz = x_mul(fac, dz);
                if (zero) {  // the products of zero displacements, with their signs
                    if (zero & 1) fx = plpl ? sub1(xj, xi) : sub1(xi, xj);
                    if (zero & 2) fy = plpl ? sub1(yj, yi) : sub1(yi, yj);
                    if (zero & 4) fz = plpl ? sub1(zj, zi) : sub1(zi, zj);
                }
                if (bad || near) {  // rare: native operations
                    dx = plpl ? sub1(xj, xi) : sub1(xi, xj);
                    dy = plpl ? sub1(yj, yi) : sub1(yi, yj);
                    dz = plpl ? sub1(zj, zi) : sub1(zi, zj);
                    const double q2 = dx * dx + dy * dy + dz * dz;
                    const double q = q2 * sqrt(q2);
                    fac = MODE == KICK_SPLIT ? g * (1.0 / q) : g / q;
                    fx = fac * dx;
                    fy = fac * dy;
                    fz = fac * dz;
                    if (RAD) {
                        const double rs = R[i] + R[j];
                        if (!(q2 > rs * rs)) fx = fy = fz = neutral;
                    }
                }
            }
            __syncwarp();
            if (r >= ST) bar_sync<EMPTY>(st, nth);
            double *o = out + st * PT * ts;
            o[0] = fx;
            o[1] = fy;
            o[2] = fz;
            __syncwarp();
            bar_arrive<FULL>(st, nth);
        }
        return;
    }
    // the fold warp: lane f owns component f % 3 of receiver f / 3
    const int f = threadIdx.x, ia = i0 + f / 3, d = f % 3;
    const bool own = f < 3 * RT && ia < nrecv, fold = own && (plpl || lmask[ia] != 0);
    double v = 0.0, vb = 0.0;
    if (MODE != KICK_SPLIT && fold && !acc_is_zero) v = acc[3 * ia + d];
    for (int r = 0; r < rounds; r++) {
        const int j0 = r * PT, np = min(PT, jmax - j0), st = r % ST;
        bar_sync<FULL>(st, nth);
        if (fold) {
            const double *t = sh + st * PT * ts + f;
#pragma unroll 8
            for (int p = 0; p < np; p++) {
                if (MODE == KICK_SPLIT && j0 + p == ia) {  // partners below, then above the receiver
                    vb = v;
                    v = 0.0;
                }
                v = MODE == KICK_TP ? sub1(v, t[p * ts]) : add1(t[p * ts], v);
            }
        }
        __syncwarp();
        if (r + ST < rounds) bar_arrive<EMPTY>(st, nth);
    }
    if (!own) return;
    if (MODE == KICK_SPLIT) {
        if (ia >= jmax) {  // no partner above the receiver
            vb = v;
            v = 0.0;
        }
        v = (acc_is_zero ? 0.0 : acc[3 * ia + d]) + v + vb;
        acc[3 * ia + d] = v;
    } else if (fold) {
        acc[3 * ia + d] = v;
    } else if (acc_is_zero) {
        acc[3 * ia + d] = 0.0;
    }
    if (kv.v && (plpl ? kv.mask[ia] != 0 : fold)) kv.v[3 * ia + d] = kv.v[3 * ia + d] + v * kv.dt;
}

template <bool RAD, int MODE>
__global__ void __launch_bounds__(fp64_threads(FP64_RT), FP64_BLOCKS)
    k_kick_plpl_fp64(int RT, int npl, int nplm, const double *__restrict__ r, const double *__restrict__ Gm,
                     const double *__restrict__ R, double *__restrict__ acc, int acc_is_zero, KickVel kv) {
    extern __shared__ double sh[];
    fp64_group<RAD, MODE>(RT, npl, npl, nplm, r, r, Gm, R, nullptr, acc, acc_is_zero, blockIdx.x * RT, sh, kv);
}

__global__ void __launch_bounds__(fp64_threads(FP64_RT_TP), FP64_BLOCKS_TP)
    k_kick_tp_fp64(int RT, int ntp, int npl, const double *__restrict__ rtp, const double *__restrict__ rpl,
                   const double *__restrict__ Gm, const int32_t *__restrict__ lmask, double *__restrict__ acc,
                   int acc_is_zero, KickVel kv) {
    extern __shared__ double sh[];
    fp64_group<false, KICK_TP>(RT, ntp, npl, 0, rtp, rpl, Gm, nullptr, lmask, acc, acc_is_zero, blockIdx.x * RT, sh, kv);
}

// Batched (ensemble) forms: block b takes item b = (system s, first receiver r0) of a
// table sorted by cost; system s's pl occupy [poff[s], poff[s] + npl[s]) and its tp
// [toff[s], toff[s] + ntp[s]).  nplm (optional): per system the count of fully
// interacting bodies (GMTINY, SyMBA), which selects the reference's loop shape as the single
// system does (KICK_SPLIT when the semi-interacting bodies outnumber the others); without
// it every system is fully interacting (KICK_DIRECT).  With sys_flag, the pl-pl form kicks
// only systems whose flag equals `phase`.
template <bool RAD>
__global__ void __launch_bounds__(fp64_threads(FP64_RT), FP64_BLOCKS)
    k_kick_plpl_fp64_batched(const int4 *__restrict__ items, const int32_t *__restrict__ poff,
                             const int32_t *__restrict__ npl, const double *__restrict__ r,
                             const double *__restrict__ Gm, const double *__restrict__ R, double *__restrict__ acc,
                             int acc_is_zero, const int32_t *__restrict__ sys_flag, int phase,
                             const int32_t *__restrict__ nplm) {
    extern __shared__ double sh[];
    const int4 w = items[blockIdx.x];
    if (sys_flag && sys_flag[w.x] != phase) return;  // another launch's system
    const int o = poff[w.x], n = npl[w.x], m = nplm ? nplm[w.x] : n;
    const double *rs = r + 3 * (size_t)o, *Rs = RAD ? R + o : nullptr;
    double *as = acc + 3 * (size_t)o;
    if (n - m > m)  // block-uniform
        fp64_group<RAD, KICK_SPLIT>(FP64_RT, n, n, m, rs, rs, Gm + o, Rs, nullptr, as, acc_is_zero, w.y, sh);
    else
        fp64_group<RAD, KICK_DIRECT>(FP64_RT, n, n, m, rs, rs, Gm + o, Rs, nullptr, as, acc_is_zero, w.y, sh);
}

__global__ void __launch_bounds__(fp64_threads(FP64_RT_TP), FP64_BLOCKS_TP)
    k_kick_tp_fp64_batched(const int4 *__restrict__ items, const int32_t *__restrict__ toff,
                           const int32_t *__restrict__ ntp, const int32_t *__restrict__ poff,
                           const int32_t *__restrict__ npl, const double *__restrict__ rtp,
                           const double *__restrict__ rpl, const double *__restrict__ Gm,
                           const int32_t *__restrict__ lmask, double *__restrict__ acc, int acc_is_zero) {
    extern __shared__ double sh[];
    const int4 w = items[blockIdx.x];
    const int ot = toff[w.x], op = poff[w.x];
    fp64_group<false, KICK_TP>(FP64_RT_TP, ntp[w.x], npl[w.x], 0, rtp + 3 * (size_t)ot, rpl + 3 * (size_t)op, Gm + op,
                               nullptr, lmask + ot, acc + 3 * (size_t)ot, acc_is_zero, w.y, sh);
}

constexpr size_t fp64_shared(int rt) { return sizeof(double) * ST * PT * term_stride(rt); }

static inline int div_up_i(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }

// Receivers per block of a single system's kick.  An SM's time per round of 32 partners is the
// work of its blocks (TERM_C cycles per receiver, FOLD_C per fold warp), at least the
// fold's chain of 32 dependent additions (~2100 cycles); the fullest SM sets the time, and the
// smallest blocks that reach it leave the least to wait for.
static int fp64_rt(int num_sms, int n, int most) {
    constexpr int TERM_C = 130, FOLD_C = 512, CHAIN_C = 2100;
    int best = 1;
    int64_t cost = INT64_MAX;
    for (int rt = 1; rt <= most; rt++) {
        const int64_t per_sm = div_up_i(div_up_i(n, rt), num_sms > 0 ? num_sms : 152);
        const int64_t c = per_sm * (rt * TERM_C + FOLD_C), t = c > CHAIN_C ? c : CHAIN_C;
        if (t < cost) {
            cost = t;
            best = rt;
        }
    }
    return best;
}

int kick_plpl_fp64(swg_ctx *c, int32_t npl, int32_t nplm, const double *r, const double *Gm, const double *R,
                   double *acc, int mode, int acc_is_zero, const KickVel &kv) {
    if (npl <= 0) return SWG_OK;
    const int rt = fp64_rt(c->num_sms, npl, FP64_RT), grid = div_up_i(npl, rt), th = fp64_threads(rt);
    const cudaStream_t st = c->stream;
    if (mode == KICK_DIRECT) {
        if (R)
            k_kick_plpl_fp64<true, KICK_DIRECT><<<grid, th, fp64_shared(rt), st>>>(rt, npl, nplm, r, Gm, R, acc, acc_is_zero, kv);
        else
            k_kick_plpl_fp64<false, KICK_DIRECT><<<grid, th, fp64_shared(rt), st>>>(rt, npl, nplm, r, Gm, R, acc, acc_is_zero, kv);
    } else {
        if (R)
            k_kick_plpl_fp64<true, KICK_SPLIT><<<grid, th, fp64_shared(rt), st>>>(rt, npl, nplm, r, Gm, R, acc, acc_is_zero, kv);
        else
            k_kick_plpl_fp64<false, KICK_SPLIT><<<grid, th, fp64_shared(rt), st>>>(rt, npl, nplm, r, Gm, R, acc, acc_is_zero, kv);
    }
    c->launches++;
    return launch_status(c, "kick_plpl_fp64");
}

int kick_tp_fp64(swg_ctx *c, int32_t ntp, int32_t npl, const double *rtp, const double *rpl, const double *Gm,
                 const int32_t *lmask, double *acc, int acc_is_zero, const KickVel &kv) {
    if (ntp <= 0) return SWG_OK;
    const int rt = fp64_rt(c->num_sms, ntp, FP64_RT_TP);
    k_kick_tp_fp64<<<div_up_i(ntp, rt), fp64_threads(rt), fp64_shared(rt), c->stream>>>(rt, ntp, npl, rtp, rpl, Gm, lmask, acc,
                                                                          acc_is_zero, kv);
    c->launches++;
    return launch_status(c, "kick_tp_fp64");
}

int kick_plpl_fp64_batched(swg_ctx *c, bool rad, int nitems, const int4 *items, const int32_t *poff,
                           const int32_t *npl, const double *r, const double *Gm, const double *R, double *acc,
                           int acc_is_zero, const int32_t *sys_flag, int phase, const int32_t *nplm) {
    if (nitems <= 0) return SWG_OK;
    constexpr int th = fp64_threads(FP64_RT);
    if (rad)
        k_kick_plpl_fp64_batched<true><<<nitems, th, fp64_shared(FP64_RT), c->stream>>>(items, poff, npl, r, Gm, R, acc, acc_is_zero,
                                                                     sys_flag, phase, nplm);
    else
        k_kick_plpl_fp64_batched<false><<<nitems, th, fp64_shared(FP64_RT), c->stream>>>(items, poff, npl, r, Gm, nullptr, acc,
                                                                      acc_is_zero, sys_flag, phase, nplm);
    c->launches++;
    return launch_status(c, "kick_plpl_fp64_batched");
}

int kick_tp_fp64_batched(swg_ctx *c, int nitems, const int4 *items, const int32_t *toff, const int32_t *ntp,
                         const int32_t *poff, const int32_t *npl, const double *rtp, const double *rpl,
                         const double *Gm, const int32_t *lmask, double *acc, int acc_is_zero) {
    if (nitems <= 0) return SWG_OK;
    k_kick_tp_fp64_batched<<<nitems, fp64_threads(FP64_RT_TP), fp64_shared(FP64_RT_TP), c->stream>>>(items, toff, ntp, poff, npl, rtp, rpl, Gm,
                                                                            lmask, acc, acc_is_zero);
    c->launches++;
    return launch_status(c, "kick_tp_fp64_batched");
}

}  // namespace swg
