// engine.cu -- device-resident refinement loop of the adaptive cubature.
//
// The reference's loop (rulecubature with parallel=1, src/hcubature.cpp:938-989)
// pops regions from a max-heap keyed on the error until the error left in the
// heap is within tolerance or the evaluation budget is spent, bisects them,
// evaluates the children and pushes them back.  Here each round is
//   k_select : one CTA per integral.  Sums the live regions' values and errors,
//              applies the reference's stopping tests (numEval >= maxEval,
//              converged(): err <= |val| rtol, src/converged.h:10-14) and picks
//              the regions the heap would pop: the largest errors, in order,
//              until the remaining error is <= rtol |val| (Gladwell), capped by
//              the evaluation budget.  Both cut-offs are found with histograms of
//              the IEEE bit patterns of the errors; the running error sums use
//              64-bit fixed point, so the choice is deterministic and independent
//              of thread scheduling.
//   k_scan   : prefix sum of the per-integral pop counts -> flat work list; sets
//              the graph's WHILE condition (no host round trip).
//   k_eval*  : cut + rule evaluation (eval_fp64.cu / evalmx_impl.cuh).
// Compiled with -fmad=false.
#include <cuda_runtime.h>

#include "g3l_device.cuh"
#include "idiv64.cuh"
#include "sel_bound.cuh"

namespace g3l {

constexpr int SEL_WARPS = SEL_BS / 32;
constexpr int SEL_BUCKETS = 1024;  // histogram of one selection pass (a multiple of SEL_BS)
constexpr int SEL_PER = SEL_BUCKETS / SEL_BS;

__device__ __forceinline__ unsigned long long ekey(const double *err, long long s)
{
    return (unsigned long long)__double_as_longlong(err[s]);
}

// deterministic block reduction (fixed pairing)
template <typename T>
__device__ T block_sum(T v, T *sh)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    T r = 0;
    if (threadIdx.x == 0) {
        for (int w = 0; w < SEL_WARPS; ++w) r += sh[w];
        sh[0] = r;
    }
    __syncthreads();
    r = sh[0];
    __syncthreads();
    return r;
}

// floor(t) of t >= 0, all ones from 1.8e19 on, by integer operations (an FP64 compare and
// conversion occupy the FP64 pipe for 64 cycles each)
__device__ __forceinline__ unsigned long long floor_u64(double t)
{
    const unsigned long long u = (unsigned long long)__double_as_longlong(t);
    if (u >= 0x43EF399B1438A100ull) return 0xFFFFFFFFFFFFFFFFull;  // 1.8e19
    const int e = (int)(u >> 52) - 1075;
    const unsigned long long m = (u & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
    return e >= 0 ? m << e : (e > -64 ? m >> -e : 0ull);
}

struct SelShared {
    unsigned int cnt[SEL_BUCKETS];
    unsigned long long sum[SEL_BUCKETS];
    unsigned long long ck[32], cq[32];  // candidates of the boundary bucket
    unsigned long long wk[2][SEL_WARPS];
    unsigned int wc[SEL_WARPS];
    unsigned long long bkey, qb, sum_above;
    unsigned int cnt_above, chosen, chosen_cnt, ncand;
    double dred[2 * SEL_WARPS];
    unsigned long long ured[SEL_WARPS];
    float fred[2 * SEL_WARPS];
    int ired[2][SEL_WARPS];
    int ubits;
    // set between the totals and the selection, each by one thread
    double scale;                    // 2^60 / E
    unsigned long long qthr, kcap;   // rtol |V| in units of 1 / scale; budget's region count
    double tau_thr, tau_sel;         // the two tolerances times |V|
};

// Block sums of two doubles (in block_sum's order) and of two FP32 values, over R regions
// (zeros from the threads without one); returns any odd.  The two doubles are added in one
// instruction, one in each half of the warp, and the warps without a region add nothing:
// on a pipe that issues one FP64 instruction per 64 cycles the additions are the time.
__device__ bool block_totals(double sv, double se, float fue, float fuv, bool odd, int R, SelShared &sh,
                             double &V, double &E, float &UE, float &UV)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = min(SEL_WARPS, (R + 31) >> 5);
    if (warp < nw) {
        double x = lane < 16 ? sv : se;
        x += __shfl_xor_sync(0xffffffffu, lane < 16 ? se : sv, 16);
        for (int o = 8; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o, 16);
        for (int o = 16; o > 0; o >>= 1) {
            fue += __shfl_down_sync(0xffffffffu, fue, o);
            fuv += __shfl_down_sync(0xffffffffu, fuv, o);
        }
        if ((lane & 15) == 0) sh.dred[(lane >> 4) * SEL_WARPS + warp] = x;
        if (lane == 0) {
            sh.fred[warp] = fue;
            sh.fred[SEL_WARPS + warp] = fuv;
        }
    }
    odd = __syncthreads_or(odd);
    UE = sh.fred[0];
    UV = sh.fred[SEL_WARPS];
    for (int w = 1; w < nw; ++w) {
        UE += sh.fred[w];
        UV += sh.fred[SEL_WARPS + w];
    }
    if (nw > 1) {
        double r = 0;
        if (threadIdx.x < 2)
            for (int w = 0; w < nw; ++w) r += sh.dred[threadIdx.x * SEL_WARPS + w];
        __syncthreads();
        if (threadIdx.x < 2) sh.dred[threadIdx.x * SEL_WARPS] = r;
        __syncthreads();
    }
    V = sh.dred[0];
    E = sh.dred[SEL_WARPS];
    return odd;
}

// One warp finds the boundary among n <= 32 candidates (sh.ck, sh.cq); sa, ca: sum and count
// of the keys above them all.
__device__ void rank_candidates(SelShared &sh, int n, bool by_sum, unsigned long long need,
                                unsigned long long sa, unsigned int ca)
{
    const int lane = threadIdx.x & 31;
    const unsigned long long k = lane < n ? sh.ck[lane] : 0, v = lane < n ? sh.cq[lane] : 0;
    unsigned long long gt = 0, ge = 0;
    unsigned int ngt = 0, nge = 0;
    for (int j = 0; j < n; ++j) {
        const unsigned long long kj = sh.ck[j], vj = sh.cq[j];
        if (kj > k) {
            gt += vj;
            ++ngt;
        }
        if (kj >= k) {
            ge += vj;
            ++nge;
        }
    }
    const unsigned long long from = by_sum ? sa : ca;
    // (the largest or smallest key where `need` lies outside the total)
    if (lane < n && (from + gt < need || ngt == 0) && (from + ge >= need || nge == (unsigned)n)) {
        sh.bkey = k;
        sh.qb = v;
        sh.cnt_above = ca + ngt;
        sh.sum_above = sa + (by_sum ? gt : 0);
    }
}

// Boundary of a selection of the largest keys of one integral (err: keys as doubles >= 0,
// descending by bit pattern).  by_sum: the key at which the cumulative q first reaches
// `need`; otherwise at which the cumulative count does.  Returns that key, the count and sum
// of the strictly larger keys and (by_sum) the q of the key.
//
// One pass histograms the keys' bit patterns linearly between the smallest and the largest
// (a logarithmic scale), which spreads them over the 1024 buckets: digits of the pattern
// itself start with bytes of sign and exponent that nearly all keys share, and the 64-bit
// atomics of a whole integral then queue at one or two addresses (8 such passes were most
// of k_select's time).  The boundary bucket is narrowed the same way until it holds at most
// 32 keys, which one warp ranks; an integral of at most 32 regions needs only that (every
// round of a small look, and the first ones of any).  All sums are integers: the result does not depend on the
// order of the threads.
__device__ void boundary_select(const double *err, const unsigned long long *q, long long base, int R,
                                bool by_sum, unsigned long long need, SelShared &sh,
                                unsigned long long &bkey, unsigned int &cnt_above,
                                unsigned long long &sum_above, unsigned long long &qb)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (R <= 32) {
        if (tid < 32) {
            if (lane < R) {
                sh.ck[lane] = ekey(err, base + lane);
                sh.cq[lane] = by_sum ? q[base + lane] : 1ull;
            }
            __syncwarp();
            rank_candidates(sh, R, by_sum, need, 0, 0);
        }
        __syncthreads();
        bkey = sh.bkey;
        qb = sh.qb;
        cnt_above = sh.cnt_above;
        sum_above = sh.sum_above;
        __syncthreads();
        return;
    }
    unsigned long long kmn = ~0ull, kmx = 0;
    for (int j = tid; j < R; j += SEL_BS) {
        const unsigned long long k = ekey(err, base + j);
        kmn = k < kmn ? k : kmn;
        kmx = k > kmx ? k : kmx;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long a = __shfl_xor_sync(0xffffffffu, kmn, o);
        const unsigned long long b = __shfl_xor_sync(0xffffffffu, kmx, o);
        kmn = a < kmn ? a : kmn;
        kmx = b > kmx ? b : kmx;
    }
    if (lane == 0) {
        sh.wk[0][warp] = kmn;
        sh.wk[1][warp] = kmx;
    }
    for (int b = 0; b < SEL_PER; ++b) {
        sh.cnt[b * SEL_BS + tid] = 0;
        sh.sum[b * SEL_BS + tid] = 0;
    }
    __syncthreads();
    kmn = sh.wk[0][0];
    kmx = sh.wk[1][0];
    for (int w = 1; w < SEL_WARPS; ++w) {
        kmn = sh.wk[0][w] < kmn ? sh.wk[0][w] : kmn;
        kmx = sh.wk[1][w] > kmx ? sh.wk[1][w] : kmx;
    }
    unsigned long long lo = kmn, span = kmx - kmn, sa = 0;
    unsigned int ca = 0;
    for (;;) {
        const int bits = 64 - __clzll((long long)span);
        const int shift = bits > 10 ? bits - 10 : 0;
        for (int j = tid; j < R; j += SEL_BS) {
            const unsigned long long d = ekey(err, base + j) - lo;  // wraps below lo
            if (d <= span) {
                const unsigned dg = (unsigned)(d >> shift);
                atomicAdd(&sh.cnt[dg], 1u);
                if (by_sum) atomicAdd(&sh.sum[dg], q[base + j]);
            }
        }
        __syncthreads();
        // thread t owns buckets 1023 - 4 t .. 1020 - 4 t (descending)
        const int top = SEL_BUCKETS - 1 - SEL_PER * tid;
        unsigned long long s = 0;
        unsigned int c = 0;
        for (int b = 0; b < SEL_PER; ++b) {
            s += sh.sum[top - b];
            c += sh.cnt[top - b];
        }
        unsigned long long si = s;
        unsigned int ci = c;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long ts = __shfl_up_sync(0xffffffffu, si, o);
            const unsigned int tc = __shfl_up_sync(0xffffffffu, ci, o);
            if (lane >= o) {
                si += ts;
                ci += tc;
            }
        }
        if (lane == 31) {
            sh.wk[0][warp] = si;
            sh.wc[warp] = ci;
        }
        __syncthreads();
        unsigned long long se = sa + si - s;  // larger keys' sum and count before this thread's
        unsigned int ce = ca + ci - c;
        for (int w = 0; w < warp; ++w) {
            se += sh.wk[0][w];
            ce += sh.wc[w];
        }
        const unsigned long long before = by_sum ? se : ce, here = by_sum ? s : c;
        // exactly one thread (the first or last where `need` lies outside the total)
        if ((before < need || tid == 0) && (before + here >= need || tid == SEL_BS - 1)) {
            int chosen = top;
            for (int b = 0; b < SEL_PER; ++b) {
                chosen = top - b;
                const unsigned long long v = by_sum ? se + sh.sum[chosen] : ce + sh.cnt[chosen];
                if (v >= need || b == SEL_PER - 1) break;
                se += sh.sum[chosen];
                ce += sh.cnt[chosen];
            }
            sh.chosen = (unsigned)chosen;
            sh.chosen_cnt = sh.cnt[chosen];
            sh.sum_above = se;
            sh.cnt_above = ce;
            sh.ncand = 0;
        }
        __syncthreads();
        lo += (unsigned long long)sh.chosen << shift;
        span = (1ull << shift) - 1;
        sa = sh.sum_above;
        ca = sh.cnt_above;
        if (shift == 0) {  // one key (and its equals) left
            if (by_sum)
                for (int j = tid; j < R; j += SEL_BS)
                    if (ekey(err, base + j) == lo) sh.qb = q[base + j];  // the same for all equals
            if (tid == 0) sh.bkey = lo;
            __syncthreads();
            break;
        }
        if (sh.chosen_cnt <= 32) {
            for (int j = tid; j < R; j += SEL_BS) {
                const unsigned long long k = ekey(err, base + j);
                if (k - lo <= span) {
                    const unsigned at = atomicAdd(&sh.ncand, 1u);
                    if (at < 32) {
                        sh.ck[at] = k;
                        sh.cq[at] = by_sum ? q[base + j] : 1ull;
                    }
                }
            }
            __syncthreads();
            if (tid < 32) rank_candidates(sh, min((int)sh.ncand, 32), by_sum, need, sa, ca);
            __syncthreads();
            sa = sh.sum_above;
            ca = sh.cnt_above;
            break;
        }
        for (int b = 0; b < SEL_PER; ++b) {
            sh.cnt[b * SEL_BS + tid] = 0;
            sh.sum[b * SEL_BS + tid] = 0;
        }
        __syncthreads();
    }
    bkey = sh.bkey;
    qb = sh.qb;
    cnt_above = ca;
    sum_above = sa;
    __syncthreads();
}

// Mixed precision: queue for FP64 re-evaluation the regions of integral i with the
// largest uncertainty keys (P.key, filled by the caller; U their sum), until the keys
// left sum to at most `keep`, and let the integral's selection wait for them.  Used
// when a threshold decision (convergence, the Gladwell count) lies within the FP32
// uncertainty of the sums it compares.
__device__ void escalate_keys(const IntDesc &d, IntState *S, const Pool &P, BatchHdr *H, int i,
                              long long base, int R, double U, double keep, int pass,
                              SelShared &sh)
{
    const double sc = 1152921504606846976.0 / U;  // 2^60 / U
    unsigned long long ql = 0;
    for (int j = threadIdx.x; j < R; j += SEL_BS) {
        const unsigned long long qq = floor_u64(P.key[base + j] * sc);
        P.q[base + j] = qq;
        ql += qq;
    }
    const unsigned long long Qk = block_sum(ql, sh.ured);
    const double kq = keep * sc;
    const unsigned long long qk = kq >= 1.8e19 ? 0xFFFFFFFFFFFFFFFFull : (unsigned long long)kq;
    const unsigned long long needp = Qk > qk ? Qk - qk : 1;
    unsigned long long pb, ps, pq;
    unsigned int pc;
    boundary_select(P.key, P.q, base, R, true, needp, sh, pb, pc, ps, pq);
    for (int j = threadIdx.x; j < R; j += SEL_BS) {
        const unsigned long long kb = (unsigned long long)__double_as_longlong(P.key[base + j]);
        if (kb >= pb && P.key[base + j] > 0.0) push_esc(H, P, pass, d.kind * 3 + d.term - 1, i, j | (1 << 30));
    }
    if (threadIdx.x == 0) {
        S[i].K = 0;
        S[i].defer = 1;
        atomicAdd(&H->deferred, 1ull);
        atomicAdd(&H->thr_checks, 1ull);
    }
    __syncthreads();
}

// pass 0 selects for every live integral; pass 1 (mixed precision) selects again, in
// the same round, for the integrals pass 0 deferred, once the FP64 re-evaluation of
// their ambiguous boundary regions has run.
//
// An integral of few regions is latency: the reads, the FP64 scalars (each formed by one
// warp), ~20 barriers.  One triplet at 30000 evaluations spends 14 us in a selection where it
// spent 24 with all warps forming the scalars and every block, also those without an
// integral, reading the host's cancel word first (call 2.05 -> 1.66 ms).  Blocks of 1024
// threads for the large integrals of such calls are slower (1.66 -> 1.83 ms: their barriers),
// and so are batched loads (more registers, fewer blocks).
__global__ void __launch_bounds__(SEL_BS, 3) k_select(const IntDesc *__restrict__ D,
                                                   IntState *__restrict__ S, Pool P, BatchHdr *H,
                                                   double tau_sel, double tau_val, int pass)
{
    __shared__ SelShared sh;
    __shared__ int s_flag[4];  // fin, status, polish passes
    __shared__ double s_tot[2];
    // threshold guard (mixed precision): bound multiplier (gthr) and the value bounds' basis
    const bool mixed = H->mixed;
    const float gthr32 = mixed ? H->thr_ratio : 0.f, vr32 = H->val_ratio;
    const bool guard = gthr32 > 0.f;
    const double gthr = (double)gthr32, vr = (double)vr32;
    const int end = H->gbeg[NGROUPS];
    if (H->gbeg[0] + (int)blockIdx.x >= end) return;  // (before the read of host memory)
    // a stop request: k_scan's (cancel or deadline), or a host cancel that arrived since (one
    // read of the host-mapped word per block, not waited for before thread 0 needs it)
    int stop = 0, host_stop = 0;
    if (threadIdx.x == 0) {
        stop = H->cancel;
        if (H->cancel_word) host_stop = *H->cancel_word;
    }
    for (int i = H->gbeg[0] + blockIdx.x; i < end; i += gridDim.x) {
        if (pass == 1 && !S[i].defer) continue;  // block-uniform
        __syncthreads();
        if (threadIdx.x == 0) S[i].defer = 0;
        if (S[i].done) {
            if (threadIdx.x == 0) S[i].K = 0;
            continue;
        }
        const IntDesc &d = D[i];
        const long long base = d.base;
        const int R = S[i].nR;
        const double rtol = d.rtol, err0 = S[i].err;
        const unsigned long long neval = S[i].neval, max_eval = d.max_eval;
        const int npts = d.npts;
        if (R == 0) {
            // fresh integral: its root region is this round's single work item (every warp has
            // to have read nR before it changes)
            __syncthreads();
            if (threadIdx.x == 0) {
                P.cand[base] = -1;
                S[i].K = 1;
                S[i].nR = 1;
                S[i].neval = (unsigned long long)npts;
            }
            __syncthreads();
            continue;
        }
        // Totals over live regions.  Mixed: and the FP32 uncertainty of each total, which
        // only thresholds are compared with.  In FP64 each of its terms takes three
        // instructions of a pipe that issues one per 64 cycles, so it is first bounded in
        // FP32 from the operands' leading bits, relative to 2^-sref, and summed in FP64 only
        // where that does not settle the comparison.
        const double eref = __double_as_longlong(err0) > 0 ? err0 : P.err[base];
        const int sref = 1023 - (int)(((unsigned long long)__double_as_longlong(eref) >> 52) & 0x7ffu);
        double sv = 0, se = 0;
        float fue = 0.f, fuv = 0.f;
        bool odd = false;
        for (int j = threadIdx.x; j < R; j += SEL_BS) {
            const double v = P.val[base + j], e = P.err[base + j];
            sv += v;
            se += e;
            if (guard) {
                fue = fmaf(f32_scaled(e, sref, odd), P.unc[base + j], fue);
                fuv = fmaf(f32_scaled(fabs(v), sref, odd), P.uval[base + j], fuv);
            }
        }
        double V, E;
        float fue_all, fuv_all;
        odd = block_totals(sv, se, fue, fuv, odd, R, sh, V, E, fue_all, fuv_all);
        // The selection's scalars, each by one thread of a warp of its own (a warp's FP64
        // instruction costs the pipe the same for one lane as for 32, and all eight warps
        // forming them would queue for it), beside thread 0's convergence test.
        if (threadIdx.x == 32) {
            const double sc = ddiv(1152921504606846976.0, E);  // fixed-point errors: floor(err * scale)
            const double thr = fabs(V) * rtol * sc;
            sh.scale = sc;
            sh.qthr = thr >= 1.8e19 ? 0xFFFFFFFFFFFFFFFFull : (unsigned long long)thr;
        } else if (threadIdx.x == 64) {
            unsigned long long kc = (unsigned long long)R;
            const unsigned long long twoNp = 2ull * (unsigned long long)npts;
            if (max_eval > neval) {
                const unsigned long long k = (max_eval - neval + twoNp - 1) / twoNp;
                if (k < kc) kc = k;
            }
            sh.kcap = kc;
            sh.tau_thr = H->tau_thr * fabs(V);
            sh.tau_sel = tau_sel * fabs(V);
        }
        // the FP32 bound of the uncertainty each comparison below has, in units of 2^-sref:
        // one whose margin is clear of the FP32 bound's own rounding (f32_within) is settled by
        // it, the others (and operands FP32 does not hold) take the FP64 sums
        const float fV = (float)rtol * vr32 * fuv_all, fU = gthr32 * (fue_all + fV);
        // FP64 totals of the uncertainty, formed on demand
        auto exact_unc = [&](double &UE, double &UV) {
            double sue = 0, suv = 0;
            for (int j = threadIdx.x; j < R; j += SEL_BS) {
                sue += P.err[base + j] * (double)P.unc[base + j];
                suv += fabs(P.val[base + j]) * (double)P.uval[base + j];
            }
            UE = gthr * block_sum(sue, sh.dred);
            UV = gthr * vr * block_sum(suv, sh.dred);
        };
        if (threadIdx.x == 0) {
            const auto expo = [](double x) { return ((unsigned long long)__double_as_longlong(x) >> 52) & 0x7ffu; };
            const bool finite = expo(V) != 0x7ffu && expo(E) != 0x7ffu;
            const double gate = fabs(V) * rtol;
            const int rounds = S[i].rounds, cancel = stop ? stop : (host_stop ? 1 : 0);
            int fin = 0, status = ST_OK;
            if (cancel) {
                fin = 1;
                status = cancel == 2 ? ST_DEADLINE : ST_CANCELLED;
            } else if (!finite) {
                fin = 1;
                status = ST_NONFINITE;
            } else if (max_eval && neval >= max_eval) {
                fin = 1;
            } else if (!(E > 0 && E > gate)) {
                fin = 1;  // converged (src/converged.h:10-14 with reqAbsError = 0)
            } else if (rounds >= H->max_rounds) {
                fin = 1;
                status = ST_ROUNDS;
            }
            S[i].val = V;
            S[i].err = E;
            s_flag[0] = fin;
            s_flag[1] = status;
            s_flag[2] = S[i].pad;  // polish passes so far
            s_tot[0] = V;
            s_tot[1] = E;
            // the convergence test E <= rtol |V| decided within the FP32 uncertainty: 1 = yes,
            // 2 = the FP32 bound of the uncertainty does not tell
            s_flag[3] = 0;
            if (guard && !cancel && finite && !(max_eval && neval >= max_eval)) {
                bool od = odd;
                const float dist = f32_scaled(fabs(E - gate), sref, od);
                s_flag[3] = f32_within(dist, fU, R, od);
            }
        }
        __syncthreads();
        if (s_flag[3] == 2) {
            double UE, UV;
            exact_unc(UE, UV);
            if (threadIdx.x == 0)
                s_flag[3] = (UE + rtol * UV) > 0.0 &&
                            fabs(s_tot[1] - fabs(s_tot[0]) * rtol) <= UE + rtol * UV;
            __syncthreads();
        }
        if (s_flag[3]) {
            const double margin = fabs(s_tot[1] - fabs(s_tot[0]) * rtol);
            double ul = 0;
            for (int j = threadIdx.x; j < R; j += SEL_BS) {
                const double kj = gthr * (P.err[base + j] * (double)P.unc[base + j] +
                                         rtol * vr * fabs(P.val[base + j]) * (double)P.uval[base + j]);
                P.key[base + j] = kj;
                ul += kj;
            }
            const double U = block_sum(ul, sh.dred);
            escalate_keys(d, S, P, H, i, base, R, U, 0.9 * margin, pass, sh);
            continue;
        }
        if (s_flag[0]) {
            // Mixed precision: before reporting, bound the FP32 noise left in the value.
            // If the regions' value bounds sum to more than tau_val |V|, re-evaluate in
            // FP64 the regions with the largest bounds until the rest is below half of it.
            bool polish = false;
            if (mixed && tau_val > 0.0 && s_flag[1] == ST_OK && s_flag[2] < 2) {
                const double Vt = s_tot[0];
                double uloc = 0;
                for (int j = threadIdx.x; j < R; j += SEL_BS) {
                    const double kj = fabs(P.val[base + j]) * (double)P.uval[base + j];
                    P.key[base + j] = kj;
                    uloc += kj;
                }
                const double U = block_sum(uloc, sh.dred);
                if (U > tau_val * fabs(Vt) && U > 0) {
                    polish = true;
                    const double sc = 1152921504606846976.0 / U;
                    unsigned long long ql = 0;
                    for (int j = threadIdx.x; j < R; j += SEL_BS) {
                        const unsigned long long qq = floor_u64(P.key[base + j] * sc);
                        P.q[base + j] = qq;
                        ql += qq;
                    }
                    const unsigned long long Qk = block_sum(ql, sh.ured);
                    const double keep = 0.5 * tau_val * fabs(Vt) * sc;
                    const unsigned long long qk = keep >= 1.8e19 ? 0xFFFFFFFFFFFFFFFFull : (unsigned long long)keep;
                    const unsigned long long needp = Qk > qk ? Qk - qk : 1;
                    unsigned long long pb;
                    unsigned int pc;
                    unsigned long long ps, pq;
                    boundary_select(P.key, P.q, base, R, true, needp, sh, pb, pc, ps, pq);
                    for (int j = threadIdx.x; j < R; j += SEL_BS) {
                        const unsigned long long kb =
                            (unsigned long long)__double_as_longlong(P.key[base + j]);
                        if (kb >= pb && P.uval[base + j] > 0.f) {
                            push_esc(H, P, pass, d.kind * 3 + d.term - 1, i, j | (1 << 30));
                        }
                    }
                    if (threadIdx.x == 0) {
                        S[i].K = 0;
                        S[i].pad += 1;
                        S[i].defer = 1;  // finish (or polish again) after the re-evaluation
                        atomicAdd(&H->polished, 1ull);
                    }
                }
            }
            if (!polish && threadIdx.x == 0) {
                S[i].done = 1;
                S[i].status = s_flag[1];
                S[i].K = 0;
            }
            __syncthreads();
            continue;
        }
        const unsigned long long Kcap = sh.kcap;
        const double scale = sh.scale;
        unsigned long long qs = 0;
        for (int j = threadIdx.x; j < R; j += SEL_BS) {
            const unsigned long long qq = floor_u64(P.err[base + j] * scale);
            P.q[base + j] = qq;
            qs += qq;
        }
        const unsigned long long Q = block_sum(qs, sh.ured);
        const unsigned long long qthr = sh.qthr;
        const unsigned long long need = Q > qthr ? Q - qthr : 0;
        // K_conv: smallest k >= 1 whose popped error sum reaches `need`
        unsigned long long Kconv;
        unsigned long long bkey = 0, tneed = 0;
        unsigned int cnt_above = 0;
        unsigned long long sum_above = 0;
        if (need == 0) {
            Kconv = 1;
        } else {
            unsigned long long qb;
            boundary_select(P.err, P.q, base, R, true, need, sh, bkey, cnt_above, sum_above, qb);
            unsigned long long rest = need - sum_above;
            tneed = qb ? (rest + qb - 1) / qb : 1;
            Kconv = (unsigned long long)cnt_above + tneed;
            // Mixed precision: the Gladwell count is the first k whose popped errors reach
            // `need` (the error left is <= rtol |V|).  If either neighbouring count is within
            // the FP32 uncertainty of the sums this compares (the errors not popped before
            // the boundary, and rtol |V|), and the choice can matter (it moves a region of
            // error b, and neighbours only where the budget allows), re-evaluate the regions
            // carrying that uncertainty first.
            if (guard && qb && Kconv <= Kcap && (long long)bkey > __double_as_longlong(sh.tau_thr)) {
                const unsigned long long m_hi = sum_above + tneed * qb - need;  // < qb
                const unsigned long long m_lo = qb - m_hi;
                unsigned long long m = 0xFFFFFFFFFFFFFFFFull;
                if (Kconv < Kcap && Kconv < (unsigned long long)R) m = m_hi;
                if (Kconv > 1 && m_lo < m) m = m_lo;
                if (m != 0xFFFFFFFFFFFFFFFFull) {
                    float fur = 0.f;
                    bool od = odd;
                    for (int j = threadIdx.x; j < R; j += SEL_BS)
                        if (ekey(P.err, base + j) <= bkey)
                            fur = fmaf(f32_scaled(P.err[base + j], sref, od), P.unc[base + j], fur);
                    const float m32 = (float)m * 8.67361738e-19f * f32_scaled(E, sref, od);  // m / scale
                    od = __syncthreads_or(od);
                    fur = block_sum(fur, sh.fred);
                    int close = f32_within(m32, gthr32 * (fur + fV), R, od);
                    if (close == 2) {
                        double ur = 0, UE, UV;
                        for (int j = threadIdx.x; j < R; j += SEL_BS)
                            if (ekey(P.err, base + j) <= bkey)
                                ur += P.err[base + j] * (double)P.unc[base + j];
                        ur = block_sum(ur, sh.dred);
                        exact_unc(UE, UV);
                        const double dlt = gthr * ur + rtol * UV;
                        close = dlt > 0.0 && (double)m / scale <= dlt;
                    }
                    if (close) {
                        const double m_abs = (double)m / scale;
                        double ul = 0;
                        for (int j = threadIdx.x; j < R; j += SEL_BS) {
                            const double e = P.err[base + j];
                            const double kj =
                                (ekey(P.err, base + j) <= bkey ? gthr * e * (double)P.unc[base + j] : 0.0) +
                                rtol * gthr * vr * fabs(P.val[base + j]) * (double)P.uval[base + j];
                            P.key[base + j] = kj;
                            ul += kj;
                        }
                        const double U = block_sum(ul, sh.dred);
                        escalate_keys(d, S, P, H, i, base, R, U, 0.9 * m_abs, pass, sh);
                        continue;
                    }
                }
            }
        }
        unsigned long long K = Kconv < Kcap ? Kconv : Kcap;
        if (K < 1) K = 1;
        if (K > (unsigned long long)R) K = R;
        if (K != Kconv || need == 0) {
            if (K == (unsigned long long)R) {
                bkey = 0;
                cnt_above = 0;
                tneed = R;  // every key >= 0: take all
            } else {
                unsigned long long qb;
                boundary_select(P.err, P.q, base, R, false, K, sh, bkey, cnt_above, sum_above, qb);
                tneed = K - cnt_above;
            }
        }
        // Mixed precision: if the boundary of this round's selection sits among regions
        // whose FP32-derived errors are uncertain (overlapping bounds), re-evaluate those
        // regions in FP64 first and select again next round.
        if (mixed && K < (unsigned long long)R) {
            if ((long long)bkey > __double_as_longlong(sh.tau_sel)) {
                if (threadIdx.x == 0) sh.ubits = 0;
                __syncthreads();
                for (int j = threadIdx.x; j < R; j += SEL_BS)  // bounds are >= 0: order as integers
                    if (ekey(P.err, base + j) == bkey) atomicMax(&sh.ubits, __float_as_int(P.unc[base + j]));
                __syncthreads();
                const float ub = __int_as_float(sh.ubits);
                // do the bounds of region j overlap the boundary's?  |key difference| 2^-52 is
                // at most 2 |ln(e / b)|, and an overlap with bounds below 1/4 has |ln(e / b)| <=
                // 2 (u + ub): what differs by more is told apart without FP64
                auto overlaps = [&](unsigned long long k, double e, float u) {
                    const int dk = abs((int)((long long)(k >> 20) - (long long)(bkey >> 20)));
                    if (u < 0.25f && ub < 0.25f && (float)dk * 2.3283064e-10f > 4.1f * (u + ub) + 1e-6f)
                        return false;
                    const double b = __longlong_as_double((long long)bkey);
                    return e * (1.0 + u) >= b * (1.0 - ub) && e * (1.0 - u) <= b * (1.0 + ub);
                };
                bool some = false;
                for (int j = threadIdx.x; j < R && !some; j += SEL_BS) {
                    const unsigned long long k = ekey(P.err, base + j);
                    const float u = P.unc[base + j];
                    some = k != bkey && (u > 0.f || ub > 0.f) && overlaps(k, P.err[base + j], u);
                }
                const int amb = __syncthreads_or(some);
                if (amb > 0) {
                    for (int j = threadIdx.x; j < R; j += SEL_BS) {
                        const float u = P.unc[base + j];
                        if (u > 0.f && overlaps(ekey(P.err, base + j), P.err[base + j], u))
                            push_esc(H, P, pass, d.kind * 3 + d.term - 1, i, j | (1 << 30));
                    }
                    if (threadIdx.x == 0) {
                        S[i].K = 0;
                        S[i].defer = 1;
                        atomicAdd(&H->deferred, 1ull);
                    }
                    __syncthreads();
                    continue;
                }
            }
        }
        // pool capacity
        if ((long long)R + (long long)K > (long long)d.cap) {
            if (threadIdx.x == 0) {
                S[i].done = 1;
                S[i].status = ST_POOL;
                S[i].K = 0;
            }
            __syncthreads();
            continue;
        }
        // Compact the selection in slot order: each warp counts its part of the regions, then
        // writes it behind the other warps' counts.  Mixed precision: selected parents whose
        // split is flagged unsettled get it re-taken in FP64 before this round's cut.
        {
            const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
            const int part = ((R + SEL_WARPS - 1) / SEL_WARPS + 31) & ~31;
            const int j0 = warp * part, j1 = min(R, j0 + part);
            const bool all = K == (unsigned long long)R;
            int ngt = 0, neq = 0;
            for (int c0 = j0; c0 < j1; c0 += 32) {
                const int j = c0 + lane;
                const unsigned long long k = j < j1 ? ekey(P.err, base + j) : 0;
                ngt += __popc(__ballot_sync(0xffffffffu, j < j1 && (all || k > bkey)));
                neq += __popc(__ballot_sync(0xffffffffu, j < j1 && !all && k == bkey));
            }
            if (lane == 0) {
                sh.ired[0][warp] = ngt;
                sh.ired[1][warp] = neq;
            }
            __syncthreads();
            long long ties = 0;  // equal keys before this warp's part
            int pos = 0;
            for (int w = 0; w < warp; ++w) {
                const long long left = (long long)tneed - ties, ne = sh.ired[1][w];
                pos += sh.ired[0][w] + (int)(left < 0 ? 0 : (left < ne ? left : ne));
                ties += ne;
            }
            for (int c0 = j0; c0 < j1; c0 += 32) {
                const int j = c0 + lane;
                const unsigned long long k = j < j1 ? ekey(P.err, base + j) : 0;
                const bool gt = j < j1 && (all || k > bkey), eq = j < j1 && !all && k == bkey;
                const unsigned be = __ballot_sync(0xffffffffu, eq), lower = (1u << lane) - 1u;
                const bool sel = gt || (eq && ties + __popc(be & lower) < (long long)tneed);
                const unsigned bs = __ballot_sync(0xffffffffu, sel);
                if (sel) {
                    P.cand[base + pos + __popc(bs & lower)] = j;
                    if (mixed && (P.split[base + j] & 0x80)) push_esc(H, P, pass, d.kind * 3 + d.term - 1, i, j);
                }
                pos += __popc(bs);
                ties += __popc(be);
            }
        }
        if (threadIdx.x == 0) {
            S[i].K = (int)K;
            S[i].neval = neval + 2ull * (unsigned long long)npts * K;
            S[i].nR = R + (int)K;
            S[i].rounds += 1;
        }
        __syncthreads();
    }
}

// prefix sum of K over integrals; work list offsets; loop condition
__global__ void __launch_bounds__(1024) k_scan(IntState *__restrict__ S, long long *woff,
                                               BatchHdr *H, cudaGraphConditionalHandle handle,
                                               int use_cond)
{
    __shared__ long long part[32];
    const int beg = H->gbeg[0], n = H->gbeg[NGROUPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = (n - beg + blockDim.x - 1) / blockDim.x;
    const int b = beg + threadIdx.x * per, e = min(n, b + per);
    long long loc = 0;
    for (int i = b; i < e; ++i) loc += S[i].K;
    long long run = loc;  // inclusive sum over the threads
    for (int o = 1; o < 32; o <<= 1) {
        const long long t = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += t;
    }
    if (lane == 31) part[warp] = run;
    __syncthreads();
    if (warp == 0) {
        long long w = part[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const long long t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        part[lane] = w;
    }
    __syncthreads();
    if (warp > 0) run += part[warp - 1];
    run -= loc;
    for (int i = b; i < e; ++i) {
        woff[i] = run;
        run += S[i].K;
    }
    if (threadIdx.x == blockDim.x - 1) {
        const long long tot = part[31];
        woff[n] = tot;
        H->total_work = tot;
        // Keep looping while there is work or a deferred FP64 re-evaluation.  The first stage's
        // queues have been consumed: count the round's entries and clear them (the second
        // stage's are cleared by the next round's first stage, k_re_fill).
        int pending = 0;
        for (int g = 0; g < NGROUPS; ++g) {
            const int n0 = H->n_esc[0][g], n1 = H->n_esc[1][g], cap = H->esc_cap[g];
            pending |= n1;
            H->escalated += (unsigned long long)(min(n0, cap) + min(n1, cap));
            H->n_esc[0][g] = 0;
        }
        const int more = tot > 0 || pending > 0;
        H->any_active = more;
        H->regions += 2ull * (unsigned long long)tot;
        if (more) H->rounds_done += 1;
        // a cancel from the host, or the deadline, stops every unfinished integral at the
        // next round's selection (this round's work still runs, so the pools stay whole)
        if (!H->cancel) {
            if (H->cancel_word && *H->cancel_word) H->cancel = 1;
            else if (H->deadline_ns && global_timer_ns() - H->t0_ns > H->deadline_ns)
                H->cancel = 2;
        }
        // a serving launch ends after chunk_rounds rounds; this round's body still runs,
        // so the states are consistent for the host between launches
        int go = more;
        if (more && H->chunk_rounds > 0 && ++H->chunk_count >= H->chunk_rounds) go = 0;
        if (use_cond) cudaGraphSetConditional(handle, go ? 1u : 0u);
    }
}

// root regions and fresh state
__global__ void k_init(const IntDesc *__restrict__ D, IntState *__restrict__ S, Pool P,
                       BatchHdr *H)
{
    const int beg = H->gbeg[0], n = H->gbeg[NGROUPS];
    for (int i = beg + blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const IntDesc &d = D[i];
        for (int k = 0; k < MAX_DIM; ++k) {
            if (k < d.dim) {
                P.center[k * P.stride + d.base] = d.c0[k];
                P.level[k * P.stride + d.base] = 0;
            }
        }
        IntState st;
        st.val = 0;
        st.err = 0;
        st.neval = 0;
        st.nR = 0;
        st.K = 0;
        st.done = 0;
        st.status = ST_OK;
        st.rounds = 0;
        st.pad = 0;
        st.defer = 0;
        st.pad2 = 0;
        S[i] = st;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        H->any_active = 1;
        H->total_work = 0;
        H->regions = (unsigned long long)(n - beg);
        H->rounds_done = 0;
        H->chunk_count = 0;
        H->ties = 0;
        H->small_arg = 0;
        for (int g = 0; g < NGROUPS; ++g) H->n_esc[0][g] = H->n_esc[1][g] = 0;
        H->escalated = 0;
        H->deferred = 0;
        H->polished = 0;
        H->esc_full = 0;
        H->thr_checks = 0;
        H->cancel = 0;
        H->t0_ns = global_timer_ns();
    }
}

// Serving: place m integrals (packed descriptors Dn) into table slots idx[] and start
// each one at its root region.
__global__ void k_admit(const IntDesc *__restrict__ Dn, const int *__restrict__ idx, int m,
                        IntDesc *__restrict__ D, IntState *__restrict__ S, Pool P)
{
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < m; j += gridDim.x * blockDim.x) {
        const IntDesc d = Dn[j];
        const int i = idx[j];
        D[i] = d;
        for (int k = 0; k < d.dim; ++k) {
            P.center[k * P.stride + d.base] = d.c0[k];
            P.level[k * P.stride + d.base] = 0;
        }
        IntState st;
        st.val = 0;
        st.err = 0;
        st.neval = 0;
        st.nR = 0;
        st.K = 0;
        st.done = 0;
        st.status = ST_OK;
        st.rounds = 0;
        st.pad = 0;
        st.defer = 0;
        st.pad2 = 0;
        S[i] = st;
    }
}

// Serving: a group's loop is entered only if the host counted unfinished integrals in it
__global__ void k_gate(const BatchHdr *H, cudaGraphConditionalHandle handle)
{
    cudaGraphSetConditional(handle, H->n > 0 ? 1u : 0u);
}

void *gate_kernel() { return (void *)k_gate; }
void *admit_kernel() { return (void *)k_admit; }
void *select_kernel() { return (void *)k_select; }
void *scan_kernel() { return (void *)k_scan; }
void *init_kernel() { return (void *)k_init; }

}  // namespace g3l
