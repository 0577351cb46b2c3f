// Sync-free persistent triangular sweeps over the approximate-Cholesky factor
// (the preconditioner's forward and backward solves; the reference's
// dataflow_kernel, src/cuda_dataflow.cu:321-478, and its CPU counterpart
// omp_sptrsv::solve_levelset, include/apxchol/solver/sptrsv/omp.h:1094-1119).
//
// Design (B200):
//  * A sweep is a dataflow launch plus, for the run of narrow levels that the
//    elimination ends in, a cluster-tail launch (one thread-block cluster,
//    solved rows in distributed shared memory; forward: after the dataflow,
//    backward: before it). The dataflow grid's warps work off the plan
//    (host_prep.hpp, sweep_plan): work items of up to 32 rows
//    of one level and one lane-group width G, G lanes per row, with the rows'
//    entries re-laid in processing order. A warp claims items from an atomic
//    ticket in level order, so a row only waits on rows of earlier items; the
//    lowest unfinished item is always being run by its owner, so progress
//    never depends on scheduling.
//  * Latency pipeline: a warp runs item i while the entries and right-hand
//    sides of item i+1 and the row descriptors of item i+2 are in flight, and
//    the ticket for item i+3 is being claimed. A row's critical path is then
//    its dependency loads, the arithmetic and one store.
//  * No level barriers and no separate ready flags: the output vector starts
//    filled with a signalling-NaN marker and a solved value replaces it, so one
//    relaxed load both tests a dependency and fetches it. The kernel re-arms
//    the buffer the next sweep writes (reset), so no fill pass runs between
//    applications.
//  * Every wait has a time budget (globaltimer): a warp that makes no progress
//    for the budget records APXB_ERR_TIMEOUT in the engine's error word and
//    every warp drains; the host turns it into an error status.
//  * fp64 sweep: products and sums are individually rounded (__dmul_rn /
//    __dadd_rn, no contraction) in the reference's order -- rows of "thin"
//    levels use the 4-way split sum of dot_thin (omp.h:1343-1357), rows of
//    "fat" levels one serial sum (omp.h:1434-1439), finished by one correctly
//    rounded subtract and divide (omp.h:1440). With G lanes per row the
//    products are formed in parallel and the order is replayed from shared
//    memory: the result is the reference CPU sweep's bytes.
//  * fp32 sweep: fp32 values and fp32 fused multiply-add accumulation, each
//    lane adding its entries in order, oldest dependency first, lane partials
//    combined by a fixed butterfly (deterministic); k right-hand sides per row
//    interleaved [row][k]: each factor entry is read once for all k.
//  * Rows are consumed progressively in the fp64 sweep: the reference's sum
//    order is advanced as operands arrive, so most of a row's arithmetic is
//    done before its last dependency lands.
//  * fp16 factor storage (the reference's GPU default, cuda.h:131-163): the
//    fp32 sweep reads binary16 weights of the column-scaled factor, widened
//    exactly to fp32, a per-row fp32 diagonal, and (backward) its right-hand
//    side times the fp64 inv_scale^2 (cuda_dataflow.cu:395), 6 instead of 8
//    bytes per stored entry.
#include <algorithm>
#include <cuda_fp16.h>

#include "kernels.cuh"

namespace apxb {

namespace {

constexpr int kBatch = 8;               // entries in flight per lane
constexpr uint32_t kNoRowDev = 0xffffffffu;

__device__ __forceinline__ unsigned backoff_ns(int spins) {
    return spins < 4 ? 0u : min(16u << min((spins - 4) >> 1, 3), 128u);
}

// Warp-uniform look at the error word and the time budget: another warp has
// failed, the budget is over, or neither.
enum wait_state : int { kWait = 0, kFailed = 1, kOver = 2 };
__device__ __forceinline__ int look(dev_error* err, unsigned long long t0, unsigned long long budget) {
    int st = kWait;
    if ((threadIdx.x & 31) == 0)
        st = ld_relaxed_int(&err->code) != 0 ? kFailed : (globaltimer() - t0 > budget ? kOver : kWait);
    return __shfl_sync(kFull, st, 0);
}
__device__ __forceinline__ bool run_out(dev_error* err, int where, uint32_t row) {
    if ((threadIdx.x & 31) == 0) raise_error(err, -4 /* APXB_ERR_TIMEOUT */, where, row);
    return true;
}

// Idle bookkeeping of a warp-uniform polling loop; returns true to drain. The
// budget limits the time without progress. A loop clears spins when an operand
// has come in, or tells when the budget is over whether its lanes wait for other
// operands than the last time it was over (moved()): then the budget starts anew,
// so such a wait ends between one and two budgets after its last operand. What
// the lanes waited for lies in shared memory, since a register for it cost the
// loops 1 to 8 % (fp64, R-MAT-14 in dataflow launches alone, 961 : 1036 us).
__device__ __forceinline__ unsigned long long& last_pending() {
    __shared__ unsigned long long words[kSweepThreads];
    return words[threadIdx.x];
}

struct idle_clock {
    int spins = 0;
    unsigned long long t0 = 0;
    template <class Moved>
    __device__ __forceinline__ bool idle(dev_error* err, unsigned long long budget, int where, uint32_t row, Moved&& moved) {
        if (spins == 0 && (threadIdx.x & 31) == 0) t0 = globaltimer();
        ++spins;
        if ((spins & 15) == 0) {
            const int st = look(err, __shfl_sync(kFull, t0, 0), budget);
            if (st == kFailed) return true;
            if (st == kOver) {
                if (!moved(row)) return run_out(err, where, row);
                if ((threadIdx.x & 31) == 0) t0 = globaltimer();
            }
        }
        const unsigned ns = backoff_ns(spins);
        if (ns) __nanosleep(ns);
        return false;
    }
    __device__ __forceinline__ bool idle(dev_error* err, unsigned long long budget, int where, uint32_t row) {
        return idle(err, budget, where, row, [](uint32_t) { return false; });
    }
    // The batch sweeps' form: the look and the error in one branch of lane 0 (a
    // solve of 64 columns at 96^3 takes 110.6 ms so, 111.4 with the form above).
    __device__ __forceinline__ bool idle_wide(dev_error* err, unsigned long long budget, int where, uint32_t row) {
        if (spins == 0 && (threadIdx.x & 31) == 0) t0 = globaltimer();
        ++spins;
        if ((spins & 15) == 0) {
            const unsigned long long since = __shfl_sync(kFull, t0, 0);
            int stop = 0;
            if ((threadIdx.x & 31) == 0) {
                if (ld_relaxed_int(&err->code) != 0) {
                    stop = 1;
                } else if (globaltimer() - since > budget) {
                    raise_error(err, -4 /* APXB_ERR_TIMEOUT */, where, row);
                    stop = 1;
                }
            }
            if (__shfl_sync(kFull, stop, 0) != 0) return true;
        }
        const unsigned ns = backoff_ns(spins);
        if (ns) __nanosleep(ns);
        return false;
    }
};

// Warp-uniform: some lane waits for other operands than at the last call.
__device__ __forceinline__ bool pending_changed(uint32_t row, uint32_t batch, unsigned mask) {
    const unsigned long long now = static_cast<unsigned long long>(row) << 32 | batch << 8 | mask;
    const bool changed = __any_sync(kFull, now != last_pending());
    last_pending() = now;
    return changed;
}

__device__ __forceinline__ void leave(sweep_ctl* ctl) {
    if ((threadIdx.x & 31) == 0) {
        const unsigned total = gridDim.x * (blockDim.x >> 5);
        if (atomicAdd(&ctl->done, 1u) == total - 1) {
            ctl->ticket = 0;
            ctl->done = 0;
        }
    }
}

__device__ __forceinline__ double dadd4(double a, double b, double c, double d) {
    return __dadd_rn(__dadd_rn(a, b), __dadd_rn(c, d));
}

// a / d correctly rounded for a divisor known before a, in two dependent
// operations: with 1 / d = h + l (l the rounded remainder of h = RN(1 / d), so
// the pair is within 2^-104), RN(a h + RN(a l)) differs from a / d by less than
// 2^-103 of it, and by at most another 2^-1075 where a l is subnormal, before
// its one rounding. d is an fp32 value: a / d lies at least 2^-79 of itself away
// from every midpoint of two doubles (a - m d is a nonzero whole multiple of the
// unit of the 54-bit m times the 24-bit d; it is not zero since m d has more than
// 53 bits), so the rounding is that of a / d. The short way is taken for
// 2^-120 <= |d| < 2^120 and 2^-831 <= |a| < 2^850: the quotient lies in
// (2^-951, 2^970), where 2^-1075 is below 2^-123 of it (down to 2^-995 it is
// below the 2^-80 that the midpoints leave) and nothing overflows. Other
// operands divide. fp64 operations take about 40 cycles each on the row's
// critical path here (a divide about nine of them).
struct recip64 {
    double d, h, l;
    unsigned span;   // biased exponents of a that take the short way: [192, 192 + span)
    __device__ __forceinline__ double quotient(double a) const {
        double q = __fma_rn(a, h, __dmul_rn(a, l));
        if (((static_cast<unsigned>(__double2hiint(a)) >> 20) & 0x7ffu) - 192u >= span) q = __ddiv_rn(a, d);
        return q;
    }
};
__device__ __forceinline__ recip64 recip_of(double d) {
    const double h = __drcp_rn(d);
    const unsigned ed = (static_cast<unsigned>(__double2hiint(d)) >> 20) & 0x7ffu;
    return {d, h, __dmul_rn(__fma_rn(-d, h, 1.0), h), ed - (1023u - 120u) < 240u ? 1681u : 0u};
}

// ---------------------------------------------------------------------------
// Exact-order accumulation for a G-lane group (G = 2^LG = 4..32). The products
// of a batch of kBatch steps of G entries lie in shared memory (pr: entry t of
// the row's batch from step jb on at 32 * (t / G - jb) + t % G). thin: chain c
// (entries t = c mod 4, t < gend) accumulates in lane c in entry order; fat:
// lane 0 adds every entry in order. The leading entries that have arrived are
// consumed, so most of a row's arithmetic is done before its last dependency
// arrives. The chain of dependent additions bounds this, so the products come
// from shared memory, where the loads run ahead of the chain.
template <unsigned LG>
__device__ __forceinline__ unsigned prod_at(uint32_t t, uint32_t jb) {
    return 32u * ((t >> LG) - jb) + (t & ((1u << LG) - 1u));
}

// Lane u's entries u, u + W, ... (W chains) from `at` while at + W <= upto.
template <unsigned LG, unsigned W>
__device__ __forceinline__ void chain_to(const double* pr, uint32_t jb, unsigned u, uint32_t upto, uint32_t& at, double& sum) {
    while (at + 8u * W <= upto) {
        double v[8];
#pragma unroll
        for (unsigned i = 0; i < 8; ++i) v[i] = pr[prod_at<LG>(at + W * i + u, jb)];
#pragma unroll
        for (unsigned i = 0; i < 8; ++i) sum = __dadd_rn(sum, v[i]);
        at += 8u * W;
    }
    while (at + W <= upto) {
        sum = __dadd_rn(sum, pr[prod_at<LG>(at + u, jb)]);
        at += W;
    }
}

// ---------------------------------------------------------------------------
// Pipeline stages shared by both precisions.

// Stage D: the item's descriptor words, loaded by every lane for its own slot.
struct stage_desc {
    unsigned c;          // item (>= n_items: none)
    uint32_t info, row, q, e;
};

// Descriptor of item c (nothing for c >= end); args: sweep_args or tail_args.
template <class A>
__device__ __forceinline__ void load_desc(const A& a, unsigned c, unsigned end, stage_desc& d) {
    const unsigned lane = threadIdx.x & 31u;
    d.c = c;
    d.info = 0; d.row = kNoRowDev; d.q = 0; d.e = 0;
    if (c < end) {
        const size_t pos = static_cast<size_t>(c) * 32 + lane;
        d.info = __ldg(a.info + c);
        d.row = __ldg(a.ord + pos);
        d.q = __ldg(a.ptr + pos);
        d.e = __ldg(a.ptr + pos + 1);
    }
}

// Lane view of an item after stage D: the lane's group, its row, and its range.
struct lane_view {
    unsigned c, lg, G, u, gid;
    bool valid, thin;
    uint32_t row, q, len;   // off-diagonals at [q, q + len); diagonal at q + len
};

__device__ __forceinline__ lane_view view_of(const stage_desc& d) {
    const unsigned lane = threadIdx.x & 31u;
    lane_view v;
    v.c = d.c;
    v.lg = (d.info >> 8) & 0xffu;
    v.G = 1u << v.lg;
    v.u = lane & (v.G - 1u);
    v.gid = lane >> v.lg;
    v.thin = (d.info >> 16) & 1u;
    // slot gid's descriptor lives in lane gid
    v.row = __shfl_sync(kFull, d.row, static_cast<int>(v.gid));
    v.q = __shfl_sync(kFull, d.q, static_cast<int>(v.gid));
    const uint32_t e = __shfl_sync(kFull, d.e, static_cast<int>(v.gid));
    v.valid = v.row != kNoRowDev;
    v.len = v.valid ? e - v.q - 1u : 0u;
    return v;
}

// Warp-uniform chunked claim: the items of the current chunk, then those of
// the pending chunk, whose ticket was taken when the current one began and
// whose bounds are loaded when the current chunk hands out its last item.
// A contended same-address atomic takes about (claimers x 0.7 ns), so the
// ticket is only read a chunk later.
struct chunk_claim {
    template <class T>
    __device__ __forceinline__ void start(const sweep_args<T>& a) {
        unsigned t = 0;
        if ((threadIdx.x & 31u) == 0) t = atomicAdd(&a.ctl->ticket, 1u);
        pend = __shfl_sync(kFull, t, 0);
    }
    unsigned cur = 0, end = 0;
    unsigned pend = 0;            // ticket of the next chunk
    unsigned plo = 0, phi = 0;    // its bounds (valid when loaded)
    bool loaded = false;
    template <class T>
    __device__ __forceinline__ void load_pending(const sweep_args<T>& a) {
        if (!loaded && pend < a.n_chunks) {
            plo = __ldg(a.chunk + pend);
            phi = __ldg(a.chunk + pend + 1);
            loaded = true;
        }
    }
    template <class T>
    __device__ __forceinline__ unsigned next(const sweep_args<T>& a) {
        if (cur >= end) {
            if (pend >= a.n_chunks) return a.n_items;
            load_pending(a);
            cur = plo;
            end = phi;
            loaded = false;
            unsigned t = 0;
            if ((threadIdx.x & 31u) == 0) t = atomicAdd(&a.ctl->ticket, 1u);
            pend = __shfl_sync(kFull, t, 0);
            return cur++;
        }
        const unsigned c = cur++;
        if (cur >= end) load_pending(a);
        return c;
    }
};

// ---------------------------------------------------------------------------
// fp64 dataflow sweep.

// Stage L data of one item (fp64).
struct stage_data64 {
    lane_view v;
    double rhs, d;   // of the group's first lane
    uint32_t jj[kBatch];
    float ww[kBatch];
};

__device__ __forceinline__ void load_data64(const sweep_args<double>& a, const stage_desc& ds, stage_data64& s) {
    s.v = view_of(ds);
    const lane_view& v = s.v;
    s.rhs = 0.0; s.d = 1.0;
    if (v.c >= a.n_items) return;
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
        const uint32_t t = (static_cast<uint32_t>(k) << v.lg) + v.u;
        if (t < v.len) { s.jj[k] = __ldg(a.idx + v.q + t); s.ww[k] = __ldg(a.val + v.q + t); }
    }
    if (v.valid && v.u == 0) {
        s.rhs = a.in[v.row];
        s.d = static_cast<double>(__ldg(a.val + v.q + v.len));
    }
}

// A lane waits on its newest pending operand alone, kLight polls at a time
// between passes over all of them: what it waits for last arrives last, and
// every poll of every waiting warp is a load that the working warps' loads
// queue behind.
constexpr int kLight = 4;

// k of the newest pending operand (bit k of pend), and its row and weight.
__device__ __forceinline__ int newest_of(unsigned pend, bool back) {
    return back ? __ffs(pend) - 1 : 31 - __clz(pend);
}
template <class V, int B>
__device__ __forceinline__ V pick(const V (&v)[B], int k) {
    V r = v[0];
#pragma unroll
    for (int i = 1; i < B; ++i) r = k == i ? v[i] : r;
    return r;
}

// Group rows (G = 2^LG lanes per row): batches of kBatch steps. A lane puts the
// product of an operand that has arrived into shared memory (prod: 32 doubles a
// step, the warp's own), and every group consumes its leading entries.
template <unsigned LG>
__device__ __forceinline__ bool run_group64(const sweep_args<double>& a, int where, bool back, stage_data64& s, double* prod, double& total) {
    constexpr unsigned G = 1u << LG;
    const lane_view& v = s.v;
    const unsigned lane = threadIdx.x & 31u;
    const double* pr = prod + G * v.gid;
    const uint32_t Jmax = __reduce_max_sync(kFull, (v.len + G - 1u) >> LG);
    const uint32_t gend = v.thin ? (v.len & ~3u) : v.len;   // entries the chains take
    double sum = 0.0;
    uint32_t at = 0;
    idle_clock clk;
    for (uint32_t jb = 0; jb < Jmax; jb += kBatch) {
        if (jb > 0) {
#pragma unroll
            for (int k = 0; k < kBatch; ++k) {
                const uint32_t t = ((jb + k) << LG) + v.u;
                if (t < v.len) { s.jj[k] = __ldg(a.idx + v.q + t); s.ww[k] = __ldg(a.val + v.q + t); }
            }
            __syncwarp();   // the last batch's products have been read
        }
        unsigned pend = 0;   // bit k: the operand of step k is still to come
        double y[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            const bool on = ((jb + k) << LG) + v.u < v.len;
            y[k] = sent_of(0.0);
            ld_if(on, a.out + s.jj[k], y[k]);
            pend |= on ? 1u << k : 0u;
        }
        for (;;) {
#pragma unroll
            for (int k = 0; k < kBatch; ++k)
                if (((pend >> k) & 1u) && !is_sent(y[k])) {
                    prod[32 * k + lane] = __dmul_rn(static_cast<double>(s.ww[k]), y[k]);
                    pend &= ~(1u << k);
                }
            bool open;
            for (int light = 0;; ++light) {
                // consume the entries before the group's first pending one
                __syncwarp();
                const unsigned any = __reduce_or_sync(kFull, pend);
                open = any != 0;
                const uint32_t st = open ? static_cast<uint32_t>(__ffs(any)) - 1u : kBatch;   // leading complete steps
                const unsigned miss = __ballot_sync(kFull, open && ((pend >> st) & 1u));
                const unsigned mine = G == 32 ? miss : (miss >> (v.gid * G)) & ((1u << (G & 31u)) - 1u);
                const uint32_t upto = min(gend, ((jb + st) << LG) + (mine ? static_cast<uint32_t>(__ffs(mine)) - 1u
                                                                          : (open ? G : 0u)));
                const uint32_t from = at;
                if (v.thin) {
                    if (v.u < 4) chain_to<LG, 4>(pr, jb, v.u, upto, at, sum);
                } else if (v.u == 0) {
                    chain_to<LG, 1>(pr, jb, 0, upto, at, sum);
                }
                if (!open) break;
                if (__any_sync(kFull, at != from)) clk.spins = 0;
                else if (clk.idle(a.err, a.budget_ns, where, v.row)) return false;
                if (light == kLight) break;
                const int kn = newest_of(pend, back);
                double w = sent_of(0.0);
                ld_if(pend != 0, a.out + pick(s.jj, kn), w);
                if (pend && !is_sent(w)) {
                    prod[32 * kn + lane] = __dmul_rn(static_cast<double>(pick(s.ww, kn)), w);
                    pend &= ~(1u << kn);
                }
            }
            if (!open) break;
#pragma unroll
            for (int k = 0; k < kBatch; ++k) ld_if((pend >> k) & 1u, a.out + s.jj[k], y[k]);
        }
    }
    const double s1 = __shfl_sync(kFull, sum, 1, static_cast<int>(G));
    const double s2 = __shfl_sync(kFull, sum, 2, static_cast<int>(G));
    const double s3 = __shfl_sync(kFull, sum, 3, static_cast<int>(G));
    if (v.thin) {   // the chains, then the <= 3 entries after gend (a row's last batch is the warp's)
        sum = dadd4(sum, s1, s2, s3);
        const uint32_t jl = Jmax ? ((Jmax - 1u) / kBatch) * kBatch : 0u;
        if (v.u == 0)
            for (uint32_t t = gend; t < v.len; ++t) sum = __dadd_rn(sum, pr[prod_at<LG>(t, jl)]);
    }
    __syncwarp();   // the products have been read
    total = sum;
    return true;
}

// The sum of a row of n <= kBatch products in the reference's order: chains
// 0..3 over the entries before gend, the rest in order. nmax: the warp's
// longest row (fp64 additions cost their latency also where they are masked).
__device__ __forceinline__ double lane_sum64(const double (&p)[kBatch], uint32_t n, uint32_t nmax, uint32_t gend) {
    double sum = 0.0;
    if (__any_sync(kFull, gend != 0)) {
        double c[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            c[k] = __dadd_rn(0.0, p[k]);
            const double c8 = __dadd_rn(c[k], p[4 + k]);
            c[k] = gend == 8 ? c8 : c[k];
        }
        const double q = dadd4(c[0], c[1], c[2], c[3]);
        sum = gend ? q : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
        if (static_cast<uint32_t>(k) >= nmax) break;
        if (static_cast<uint32_t>(k) >= gend && static_cast<uint32_t>(k) < n) sum = __dadd_rn(sum, p[k]);
    }
    return sum;
}

// One lane per row (<= kBatch off-diagonals): all operands, then the sum in
// straight line.
__device__ __forceinline__ bool run_lane64(const sweep_args<double>& a, int where, stage_data64& s, double& total) {
    const lane_view& v = s.v;
    const uint32_t n = v.len;   // <= kBatch for these rows
    double y[kBatch];
    idle_clock clk;
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
        y[k] = sent_of(0.0);
        ld_if(static_cast<uint32_t>(k) < n, a.out + s.jj[k], y[k]);
    }
    for (;;) {
        bool open = false;
#pragma unroll
        for (int k = 0; k < kBatch; ++k) open |= static_cast<uint32_t>(k) < n && is_sent(y[k]);
        if (!__any_sync(kFull, open)) break;
        const auto moved = [&](uint32_t row) {
            unsigned p = 0;
#pragma unroll
            for (int k = 0; k < kBatch; ++k) p |= static_cast<uint32_t>(k) < n && is_sent(y[k]) ? 1u << k : 0u;
            return pending_changed(row, 0, p);
        };
        if (clk.idle(a.err, a.budget_ns, where, v.row, moved)) return false;
#pragma unroll
        for (int k = 0; k < kBatch; ++k) ld_if(static_cast<uint32_t>(k) < n && is_sent(y[k]), a.out + s.jj[k], y[k]);
    }
    double p[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) p[k] = __dmul_rn(static_cast<double>(s.ww[k]), y[k]);
    total = lane_sum64(p, n, __reduce_max_sync(kFull, n), v.thin ? (n & ~3u) : 0u);
    return true;
}

// The off-diagonal sums of one item's rows in the reference's order. Returns
// false when the warp must drain.
__device__ __forceinline__ bool run_rows64(const sweep_args<double>& a, int where, bool back, stage_data64& s, double* prod, double& total) {
    switch (s.v.lg) {
        case 0: return run_lane64(a, where, s, total);
        case 2: return run_group64<2>(a, where, back, s, prod, total);
        case 3: return run_group64<3>(a, where, back, s, prod, total);
        case 4: return run_group64<4>(a, where, back, s, prod, total);
        default: return run_group64<5>(a, where, back, s, prod, total);
    }
}

// Run one item: wait for its operands, replay the reference's sum order, store.
// Returns false when the warp must drain.
template <int DIR>
__device__ __forceinline__ bool run64(const sweep_args<double>& a, stage_data64& s, double* prod) {
    const lane_view& v = s.v;
    double total = 0.0;
    const recip64 inv = recip_of(s.d);
    if (!run_rows64(a, DIR == 0 ? kFwdSweep : kBckSweep, DIR == 1, s, prod, total)) return false;
    if (v.valid && v.u == 0) {
        double rhs = s.rhs;
        if (a.rhs_sub) rhs = __dsub_rn(rhs, *a.rhs_sub);
        const double y = inv.quotient(__dsub_rn(rhs, total));
        st_relaxed(a.out + v.row, y);
        if (a.copy_out) a.copy_out[v.row] = y;
        // re-arm after the right-hand side was consumed: the backward sweep
        // reads it from the buffer it re-arms (a store issued right behind the
        // load of the same address would wait for that load)
        if (a.reset) a.reset[v.row] = sent_of(0.0);
    }
    return true;
}

template <int DIR>
__global__ void __launch_bounds__(kSweepThreads, 2) k_df64(const sweep_args<double> a) {
    if (a.skip && *a.skip) return;
    last_pending() = 0;
    __shared__ __align__(16) double prods[kSweepThreads / 32][32 * kBatch];
    const unsigned lane = threadIdx.x & 31u;
    double* prod = prods[threadIdx.x >> 5];
    chunk_claim cc;
    cc.start(a);
    stage_desc dD;
    load_desc(a, cc.next(a), a.n_items, dD);
    stage_data64 sL;
    load_data64(a, dD, sL);
    load_desc(a, cc.next(a), a.n_items, dD);
    int bad = 0;   // the error word, read one item late so the load is never waited on
    while (sL.v.c < a.n_items) {
        // rotate: run L, data for D, descriptor of the next claimed item
        stage_data64 sR = sL;
        load_data64(a, dD, sL);
        load_desc(a, cc.next(a), a.n_items, dD);
        if (__shfl_sync(kFull, bad, 0)) break;
        if (lane == 0) bad = ld_relaxed_int(&a.err->code);
        if (!run64<DIR>(a, sR, prod)) break;
    }
    leave(a.ctl);
}

// ---------------------------------------------------------------------------
// fp32, K right-hand sides per row.

template <int K>
__device__ __forceinline__ void ld_row(const float* p, float (&y)[K]) {
    if constexpr (K == 1) {
        y[0] = ld_relaxed(p);
    } else if constexpr (K == 2) {
        unsigned a0, a1;
        asm volatile("ld.relaxed.gpu.global.v2.b32 {%0,%1}, [%2];" : "=r"(a0), "=r"(a1) : "l"(p) : "memory");
        y[0] = __uint_as_float(a0); y[1] = __uint_as_float(a1);
    } else {
#pragma unroll
        for (int h = 0; h < K; h += 4) {
            unsigned a0, a1, a2, a3;
            asm volatile("ld.relaxed.gpu.global.v4.b32 {%0,%1,%2,%3}, [%4];"
                         : "=r"(a0), "=r"(a1), "=r"(a2), "=r"(a3) : "l"(p + h) : "memory");
            y[h] = __uint_as_float(a0); y[h + 1] = __uint_as_float(a1);
            y[h + 2] = __uint_as_float(a2); y[h + 3] = __uint_as_float(a3);
        }
    }
}

// The same where `on` (elsewhere y stays as it is), by predicate and not by branch.
template <int K>
__device__ __forceinline__ void ld_row_if(bool on, const float* p, float (&y)[K]) {
    const unsigned f = on;
    if constexpr (K == 1) {
        asm volatile("{.reg .pred q; setp.ne.u32 q, %1, 0; @q ld.relaxed.gpu.global.b32 %0, [%2];}"
                     : "+f"(y[0]) : "r"(f), "l"(p) : "memory");
    } else if constexpr (K == 2) {
        asm volatile("{.reg .pred q; setp.ne.u32 q, %2, 0; @q ld.relaxed.gpu.global.v2.b32 {%0,%1}, [%3];}"
                     : "+f"(y[0]), "+f"(y[1]) : "r"(f), "l"(p) : "memory");
    } else {
#pragma unroll
        for (int h = 0; h < K; h += 4)
            asm volatile("{.reg .pred q; setp.ne.u32 q, %4, 0; @q ld.relaxed.gpu.global.v4.b32 {%0,%1,%2,%3}, [%5];}"
                         : "+f"(y[h]), "+f"(y[h + 1]), "+f"(y[h + 2]), "+f"(y[h + 3]) : "r"(f), "l"(p + h) : "memory");
    }
}

template <int K>
__device__ __forceinline__ void st_row(float* p, const float (&y)[K]) {
    if constexpr (K == 1) {
        st_relaxed(p, y[0]);
    } else if constexpr (K == 2) {
        asm volatile("st.relaxed.gpu.global.v2.b32 [%0], {%1,%2};"
                     :: "l"(p), "r"(__float_as_uint(y[0])), "r"(__float_as_uint(y[1])) : "memory");
    } else {
#pragma unroll
        for (int h = 0; h < K; h += 4)
            asm volatile("st.relaxed.gpu.global.v4.b32 [%0], {%1,%2,%3,%4};"
                         :: "l"(p + h), "r"(__float_as_uint(y[h])), "r"(__float_as_uint(y[h + 1])),
                            "r"(__float_as_uint(y[h + 2])), "r"(__float_as_uint(y[h + 3])) : "memory");
    }
}

template <int K>
__device__ __forceinline__ bool row_ready(const float (&y)[K]) {
    bool ok = true;
#pragma unroll
    for (int s = 0; s < K; ++s) ok &= !is_sent(y[s]);
    return ok;
}

template <int K>
struct batch_of { static constexpr int value = K >= 16 ? 2 : (K >= 8 ? 4 : 8); };

template <int K>
struct stage_data32 {
    lane_view v;
    float rhs[K];
    float d;
    uint32_t jj[batch_of<K>::value];
    float ww[batch_of<K>::value];
};

// Entry t of a row in processing order: plan order forward; backward the plan
// lists the newest dependency first, so it is walked from its end.
__device__ __forceinline__ uint32_t entry_at(const lane_view& v, uint32_t t, bool back) {
    return v.q + (back ? v.len - 1u - t : t);
}

// Weight of plan entry e: fp32, or the binary16 value widened (exact).
template <bool H>
__device__ __forceinline__ float weight32(const sweep_args<float>& a, uint32_t e) {
    if constexpr (H) return __half2float(__ushort_as_half(__ldg(a.val16 + e)));
    else return __ldg(a.val + e);
}

template <int DIR, int K, bool H>
__device__ __forceinline__ void load_data32(const sweep_args<float>& a, const double* in64, const stage_desc& ds,
                                            stage_data32<K>& s) {
    constexpr int B = batch_of<K>::value;
    s.v = view_of(ds);
    const lane_view& v = s.v;
    s.d = 1.0f;
#pragma unroll
    for (int r = 0; r < K; ++r) s.rhs[r] = 0.0f;
    if (v.c >= a.n_items) return;
#pragma unroll
    for (int k = 0; k < B; ++k) {
        const uint32_t t = (static_cast<uint32_t>(k) << v.lg) + v.u;
        if (t < v.len) {
            const uint32_t e = entry_at(v, t, DIR == 1);
            s.jj[k] = __ldg(a.idx + e);
            s.ww[k] = weight32<H>(a, e);
        }
    }
    if (v.valid && v.u == 0) {
        const size_t base = static_cast<size_t>(v.row) * K;
        if (in64) {
#pragma unroll
            for (int r = 0; r < K; ++r) {
                double x = in64[base + r];
                if (a.rhs_sub) x -= a.rhs_sub[r];
                s.rhs[r] = static_cast<float>(x);
            }
        } else if (H && a.in_scale2) {
            const double sc = a.in_scale2[v.row];
#pragma unroll
            for (int r = 0; r < K; ++r) s.rhs[r] = static_cast<float>(static_cast<double>(a.in[base + r]) * sc);
        } else {
#pragma unroll
            for (int r = 0; r < K; ++r) s.rhs[r] = a.in[base + r];
        }
        s.d = H ? __ldg(a.diag16 + v.row) : __ldg(a.val + v.q + v.len);
    }
}

// Sums a lane's nk operand rows (at most B, loaded once into yv) into acc in
// order, oldest dependency first, polling for those still to come. Returns false
// when the warp must drain. Which polls are cheapest depends on the row's width:
//  * one column, straight-line code with one vote a pass and the sums behind the
//    last pass: a pass over the pending rows is what stands between the last
//    operand's arrival and the row;
//  * from 2 columns on a lane consumes its rows as they arrive and polls only
//    those from the first missing one on (the wider polls cost what the vote
//    saves), by predicate up to 4 columns and by branch from 8 on.
// One pair of sweeps, all levels in the dataflow launches, us, straight line for
// all -> this rule, mean of seven placements of the factor: R-MAT-14 k = 4
// 773 -> 743, k = 8 1074 -> 894, k = 16 1740 -> 1486; 6-regular n = 100003
// 1635 -> 1549, 2283 -> 1889, 3747 -> 3089; 96^3 grid 670 -> 621, 924 -> 797,
// 1396 -> 1258; k = 2 the same within 1.5 % (96^3 grid 653 -> 629). At one column
// in order against straight line: 758 : 724, 2204 : 2125, 754 : 732.
template <int B, int K>
__device__ __forceinline__ bool gather32(const sweep_args<float>& a, int where, uint32_t row, uint32_t batch, idle_clock& clk, uint32_t nk,
                                         const uint32_t (&jj)[B], const float (&ww)[B], float (&yv)[B][K], float (&acc)[K]) {
    if constexpr (K == 1) {
        for (;;) {
            bool open = false;
#pragma unroll
            for (int k = 0; k < B; ++k) open |= static_cast<uint32_t>(k) < nk && !row_ready<K>(yv[k]);
            if (!__any_sync(kFull, open)) break;
            const auto moved = [&](uint32_t r) {
                unsigned p = 0;
#pragma unroll
                for (int k = 0; k < B; ++k) p |= static_cast<uint32_t>(k) < nk && !row_ready<K>(yv[k]) ? 1u << k : 0u;
                return pending_changed(r, batch, p);
            };
            if (clk.idle(a.err, a.budget_ns, where, row, moved)) return false;
#pragma unroll
            for (int k = 0; k < B; ++k)
                ld_row_if<K>(static_cast<uint32_t>(k) < nk && !row_ready<K>(yv[k]), a.out + static_cast<size_t>(jj[k]) * K, yv[k]);
        }
#pragma unroll
        for (int k = 0; k < B; ++k)
            if (static_cast<uint32_t>(k) < nk)
#pragma unroll
                for (int r = 0; r < K; ++r) acc[r] = __fmaf_rn(ww[k], yv[k][r], acc[r]);
    } else {
        uint32_t kpos = 0;
        for (;;) {
            const uint32_t before = kpos;
#pragma unroll
            for (int k = 0; k < B; ++k) {
                if (kpos == static_cast<uint32_t>(k) && kpos < nk && row_ready<K>(yv[k])) {
#pragma unroll
                    for (int r = 0; r < K; ++r) acc[r] = __fmaf_rn(ww[k], yv[k][r], acc[r]);
                    ++kpos;
                }
            }
            if (__all_sync(kFull, kpos >= nk)) break;
            if (__any_sync(kFull, kpos != before)) clk.spins = 0;
            else if (clk.idle(a.err, a.budget_ns, where, row)) return false;
#pragma unroll
            for (int k = 0; k < B; ++k) {
                const bool on = static_cast<uint32_t>(k) >= kpos && static_cast<uint32_t>(k) < nk && !row_ready<K>(yv[k]);
                const float* p = a.out + static_cast<size_t>(jj[k]) * K;
                if constexpr (K <= 4) ld_row_if<K>(on, p, yv[k]);
                else if (on) ld_row<K>(p, yv[k]);
            }
        }
    }
    return true;
}

template <int DIR, int K, bool H>
__device__ __forceinline__ bool run32(const sweep_args<float>& a, stage_data32<K>& s) {
    constexpr int B = batch_of<K>::value;
    const lane_view& v = s.v;
    const int where = DIR == 0 ? kFwdSweep32 : kBckSweep32;
    const uint32_t J = (v.len + v.G - 1u) >> v.lg;
    const uint32_t Jmax = __reduce_max_sync(kFull, J);
    float acc[K];
#pragma unroll
    for (int r = 0; r < K; ++r) acc[r] = 0.0f;
    idle_clock clk;
    for (uint32_t jb = 0; jb < Jmax; jb += B) {
        if (jb > 0) {
#pragma unroll
            for (int k = 0; k < B; ++k) {
                const uint32_t t = ((jb + k) << v.lg) + v.u;
                if (t < v.len) {
                    const uint32_t e = entry_at(v, t, DIR == 1);
                    s.jj[k] = __ldg(a.idx + e);
                    s.ww[k] = weight32<H>(a, e);
                }
            }
        }
        // this lane's entries in the batch: steps 0 .. nk-1
        const uint32_t t0 = (jb << v.lg) + v.u;
        const uint32_t nk = t0 < v.len ? min(static_cast<uint32_t>(B), ((v.len - t0 - 1u) >> v.lg) + 1u) : 0u;
        float yv[B][K];
#pragma unroll
        for (int k = 0; k < B; ++k) {
#pragma unroll
            for (int r = 0; r < K; ++r) yv[k][r] = 0.0f;
            ld_row_if<K>(static_cast<uint32_t>(k) < nk, a.out + static_cast<size_t>(s.jj[k]) * K, yv[k]);
        }
        if (!gather32<B, K>(a, where, v.row, jb / B, clk, nk, s.jj, s.ww, yv, acc)) return false;
        clk.spins = 0;
    }
    // fixed butterfly over the group's lanes
    for (unsigned o = v.G >> 1; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < K; ++r) acc[r] += __shfl_xor_sync(kFull, acc[r], static_cast<int>(o), static_cast<int>(v.G));
    if (v.valid && v.u == 0) {
        // a plain division: a reciprocal formed before the wait (recip32) was slower here, where other warps
        // hide it (k = 1, us: R-MAT-16 2184 : 2213, 96^3 grid 709 : 732)
        float y[K];
#pragma unroll
        for (int r = 0; r < K; ++r) y[r] = __fdiv_rn(s.rhs[r] - acc[r], s.d);
        st_row<K>(a.out + static_cast<size_t>(v.row) * K, y);
        if (a.reset) {   // re-arm after the right-hand side was consumed (see run64)
            float sent[K];
#pragma unroll
            for (int r = 0; r < K; ++r) sent[r] = sent_of(0.0f);
            st_row<K>(a.reset + static_cast<size_t>(v.row) * K, sent);
        }
    }
    return true;
}

template <int DIR, int K, bool H>
__global__ void __launch_bounds__(kSweepThreads, 2) k_df32(const sweep_args<float> a, const double* in64) {
    if (a.skip && *a.skip) return;
    last_pending() = 0;
    const unsigned lane = threadIdx.x & 31u;
    chunk_claim cc;
    cc.start(a);
    stage_desc dD;
    load_desc(a, cc.next(a), a.n_items, dD);
    stage_data32<K> sL;
    load_data32<DIR, K, H>(a, in64, dD, sL);
    load_desc(a, cc.next(a), a.n_items, dD);
    int bad = 0;   // the error word, read one item late
    while (sL.v.c < a.n_items) {
        stage_data32<K> sR = sL;
        load_data32<DIR, K, H>(a, in64, dD, sL);
        load_desc(a, cc.next(a), a.n_items, dD);
        if (__shfl_sync(kFull, bad, 0)) break;
        if (lane == 0) bad = ld_relaxed_int(&a.err->code);
        if (!run32<DIR, K, H>(a, sR)) break;
    }
    leave(a.ctl);
}


// ---------------------------------------------------------------------------
// Batched fp32 sweep over a batch plan (host_prep.hpp, build_batch_plan).
// A row's G lanes are C column lanes x ge entry lanes: lane u of the group
// handles columns [KC * (u % C), KC * (u % C) + KC) and entries t = u / C,
// u / C + ge, ... of the row (oldest dependency first), 8 at a time, so each
// gather is one 16-byte load (k >= 4) and a lane keeps 8 of them in flight.
// Partial sums are combined by a fixed butterfly over the entry lanes. Work is
// claimed in chunks (consecutive items of one level) from the ticket counter;
// the next chunk is claimed when the current one starts, so the atomic's
// latency is hidden behind a chunk of work.

template <int K>
struct wide_cfg {
    static constexpr int KC = K < 4 ? K : 4;   // columns per lane
    static constexpr int C = K / KC;           // column lanes per row
    static constexpr int LC = C == 32 ? 5 : (C == 16 ? 4 : (C == 8 ? 3 : (C == 4 ? 2 : (C == 2 ? 1 : 0))));
    static constexpr int B = 8;                // entries in flight per lane
};

template <int K>
struct stage_wide {
    lane_view v;
    unsigned cl, ue, glg;        // column lane, entry lane, log2(entry lanes)
    float rhs[wide_cfg<K>::KC];
    float d;
    uint32_t jj[wide_cfg<K>::B];
    float ww[wide_cfg<K>::B];
};

template <int K, bool H>
__device__ __forceinline__ void load_wide(const sweep_args<float>& a, const stage_desc& ds, stage_wide<K>& s) {
    using W = wide_cfg<K>;
    s.v = view_of(ds);
    const lane_view& v = s.v;
    s.cl = v.u & static_cast<unsigned>(W::C - 1);
    s.ue = v.u >> W::LC;
    s.glg = v.lg - W::LC;
    s.d = 1.0f;
#pragma unroll
    for (int r = 0; r < W::KC; ++r) s.rhs[r] = 0.0f;
    if (v.c >= a.n_items) return;
#pragma unroll
    for (int k = 0; k < W::B; ++k) {
        const uint32_t t = (static_cast<uint32_t>(k) << s.glg) + s.ue;
        if (t < v.len) { s.jj[k] = __ldg(a.idx + v.q + t); s.ww[k] = weight32<H>(a, v.q + t); }
    }
    if (v.valid && s.ue == 0) {
        const size_t base = static_cast<size_t>(v.row) * K + s.cl * W::KC;
        if (H && a.in_scale2) {   // fp16 storage, backward: the input times inv_scale^2, in fp64, rounded once
            const double sc = a.in_scale2[v.row];
#pragma unroll
            for (int r = 0; r < W::KC; ++r) s.rhs[r] = static_cast<float>(static_cast<double>(a.in[base + r]) * sc);
        } else {
#pragma unroll
            for (int r = 0; r < W::KC; ++r) s.rhs[r] = a.in[base + r];
        }
        s.d = H ? __ldg(a.diag16 + v.row) : __ldg(a.val + v.q + v.len);
    }
}

// L2 prefetch of the dependency rows the lane will gather for its next item
// (whose indices arrived while the current item ran). A prefetch holds no
// register and L2 is the point of coherence, so the later relaxed load still
// sees whatever the row holds then, solved or not.
template <int K>
__device__ __forceinline__ void prefetch_wide(const sweep_args<float>& a, const stage_wide<K>& s) {
    using W = wide_cfg<K>;
    const lane_view& v = s.v;
    if (v.c >= a.n_items) return;
    const size_t col = static_cast<size_t>(s.cl) * W::KC;
#pragma unroll
    for (int k = 0; k < W::B; ++k) {
        const uint32_t t = (static_cast<uint32_t>(k) << s.glg) + s.ue;
        if (t < v.len) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.out + static_cast<size_t>(s.jj[k]) * K + col));
    }
}

template <int DIR, int K, bool H>
__device__ __forceinline__ bool run_wide(const sweep_args<float>& a, stage_wide<K>& s, const stage_wide<K>& next) {
    using W = wide_cfg<K>;
    constexpr int B = W::B, KC = W::KC;
    const lane_view& v = s.v;
    const int where = DIR == 0 ? kFwdSweep32 : kBckSweep32;
    const uint32_t ge = 1u << s.glg;
    const uint32_t J = (v.len + ge - 1u) >> s.glg;
    const uint32_t Jmax = __reduce_max_sync(kFull, J);
    const size_t col = static_cast<size_t>(s.cl) * KC;
    float acc[KC];
#pragma unroll
    for (int r = 0; r < KC; ++r) acc[r] = 0.0f;
    idle_clock clk;
    for (uint32_t jb = 0; jb < Jmax; jb += B) {
        if (jb > 0) {
#pragma unroll
            for (int k = 0; k < B; ++k) {
                const uint32_t t = ((jb + k) << s.glg) + s.ue;
                if (t < v.len) { s.jj[k] = __ldg(a.idx + v.q + t); s.ww[k] = weight32<H>(a, v.q + t); }
            }
        }
        const uint32_t t0 = (jb << s.glg) + s.ue;
        const uint32_t nk = t0 < v.len ? min(static_cast<uint32_t>(B), ((v.len - t0 - 1u) >> s.glg) + 1u) : 0u;
        float yv[B][KC];
#pragma unroll
        for (int k = 0; k < B; ++k)
            if (static_cast<uint32_t>(k) < nk) ld_row<KC>(a.out + static_cast<size_t>(s.jj[k]) * K + col, yv[k]);
        if (jb == 0) prefetch_wide<K>(a, next);   // the next item's gathers start while these are in flight
        uint32_t kpos = 0;
        for (;;) {
            const uint32_t before = kpos;
#pragma unroll
            for (int k = 0; k < B; ++k) {
                if (kpos == static_cast<uint32_t>(k) && kpos < nk && row_ready<KC>(yv[k])) {
#pragma unroll
                    for (int r = 0; r < KC; ++r) acc[r] = __fmaf_rn(s.ww[k], yv[k][r], acc[r]);
                    ++kpos;
                }
            }
            if (__all_sync(kFull, kpos >= nk)) break;
            if (__any_sync(kFull, kpos != before)) clk.spins = 0;
            else if (clk.idle_wide(a.err, a.budget_ns, where, v.row)) return false;
            // re-poll only the entry this lane is blocked on and the ones after it
#pragma unroll
            for (int k = 0; k < B; ++k)
                if (static_cast<uint32_t>(k) >= kpos && static_cast<uint32_t>(k) < nk && !row_ready<KC>(yv[k]))
                    ld_row<KC>(a.out + static_cast<size_t>(s.jj[k]) * K + col, yv[k]);
        }
    }
    // fixed butterfly over the entry lanes (same column lane)
    for (unsigned o = v.G >> 1; o >= static_cast<unsigned>(W::C); o >>= 1)
#pragma unroll
        for (int r = 0; r < KC; ++r) acc[r] += __shfl_xor_sync(kFull, acc[r], static_cast<int>(o), static_cast<int>(v.G));
    if (v.valid && s.ue == 0) {
        float y[KC];
#pragma unroll
        for (int r = 0; r < KC; ++r) y[r] = __fdiv_rn(s.rhs[r] - acc[r], s.d);
        st_row<KC>(a.out + static_cast<size_t>(v.row) * K + col, y);
        // re-arm the row in the buffer the other direction writes next; done
        // here, after the row's right-hand side has been consumed, since the
        // backward sweep reads its right-hand side from that same buffer
        if (a.reset) {
            float sent[KC];
#pragma unroll
            for (int r = 0; r < KC; ++r) sent[r] = sent_of(0.0f);
            st_row<KC>(a.reset + static_cast<size_t>(v.row) * K + col, sent);
        }
    }
    return true;
}

template <int DIR, int K, bool H>
__global__ void __launch_bounds__(kSweepThreads, 2) k_dw32(const sweep_args<float> a) {
    if (a.skip && *a.skip) return;
    const unsigned lane = threadIdx.x & 31u;
    chunk_claim cc;
    cc.start(a);
    stage_desc dD;
    load_desc(a, cc.next(a), a.n_items, dD);
    stage_wide<K> sL;
    load_wide<K, H>(a, dD, sL);
    load_desc(a, cc.next(a), a.n_items, dD);
    int bad = 0;   // the error word, read one item late so the load is never waited on
    while (sL.v.c < a.n_items) {
        stage_wide<K> sR = sL;
        load_wide<K, H>(a, dD, sL);
        load_desc(a, cc.next(a), a.n_items, dD);
        if (__shfl_sync(kFull, bad, 0)) break;
        if (lane == 0) bad = ld_relaxed_int(&a.err->code);
        if (!run_wide<DIR, K, H>(a, sR, sL)) break;
    }
    leave(a.ctl);
}

// ---------------------------------------------------------------------------
// Cluster tail: the run of narrow levels at the end of the elimination
// (forward: after the dataflow launch; backward: before it), one thread-block
// cluster per column slice (KC columns). Every CTA of the cluster
// holds a copy of the tail's solution in shared memory; the warp that solves a
// row stores it into all the copies (distributed shared memory) and into the
// output vector, and a row waits by polling its own SM's copy.
// What bounds it: the chain of levels. In the dataflow kernels a narrow level
// costs a store, an L2 round trip and the polls of every warp that waits
// further down (0.7 us alone, 1.1 us and more with the whole grid polling);
// here a hop is a DSM store and a shared-memory poll, and no other SM sees it.
// What is left of a hop (chains of one-row levels: 0.45 us in fp32, 0.61 in fp64,
// against 0.68 and 0.83 in the dataflow kernels; levels of some hundred rows,
// 6-regular n = 100003: 0.56 in fp32) is the instructions between the operand's
// arrival and the store, so those paths are short: a row's lanes all
// hold its sum, right-hand side and divisor, the batches of a row are compiled
// for 1, 2, 4 and 8 steps, the divisor's reciprocal, the store addresses and
// everything else that does not depend on the operands are ready before.
// Measured, one sweep pair (us), all levels in the dataflow launch before ->
// with the tail: fp64 6-regular n = 100003 2849 -> 1230, 61^3 grid 653 -> 346,
// 128^3 grid 1524 -> 870, 256^2 grid 180 -> 117; fp32 6-regular 2131 -> 571,
// 61^3 412 -> 214, 128^3 1019 -> 622; k = 16 6-regular 4866 -> 905.
// Items go to the cluster's warps round robin in level order (no claims), so
// the lowest unfinished item is always its warp's next one and, all CTAs of a
// cluster being resident together, progress never depends on scheduling. A warp
// has the operands from outside the tail, entries, right-hand sides and
// descriptors of its next items in flight while it waits for the current one.

constexpr int kTailThreads = 256;

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_size() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ unsigned peer_addr(unsigned local, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
__device__ __forceinline__ void near_ld_if(bool on, unsigned p, double& y) {
    unsigned long long v = static_cast<unsigned long long>(__double_as_longlong(y));
    asm volatile("{.reg .pred q; setp.ne.u32 q, %1, 0; @q ld.relaxed.cluster.shared::cta.b64 %0, [%2];}"
                 : "+l"(v) : "r"(static_cast<unsigned>(on)), "r"(p) : "memory");
    y = __longlong_as_double(static_cast<long long>(v));
}
__device__ __forceinline__ void peer_st(unsigned p, double y) {
    asm volatile("st.relaxed.cluster.shared::cluster.b64 [%0], %1;" ::"r"(p), "l"(__double_as_longlong(y)) : "memory");
}
template <int KC>
__device__ __forceinline__ void near_ld_row_if(bool on, unsigned p, float (&y)[KC]) {
    const unsigned f = on;
    if constexpr (KC == 1)
        asm volatile("{.reg .pred q; setp.ne.u32 q, %1, 0; @q ld.relaxed.cluster.shared::cta.b32 %0, [%2];}"
                     : "+f"(y[0]) : "r"(f), "r"(p) : "memory");
    else if constexpr (KC == 2)
        asm volatile("{.reg .pred q; setp.ne.u32 q, %2, 0; @q ld.relaxed.cluster.shared::cta.v2.b32 {%0,%1}, [%3];}"
                     : "+f"(y[0]), "+f"(y[1]) : "r"(f), "r"(p) : "memory");
    else
        asm volatile("{.reg .pred q; setp.ne.u32 q, %4, 0; @q ld.relaxed.cluster.shared::cta.v4.b32 {%0,%1,%2,%3}, [%5];}"
                     : "+f"(y[0]), "+f"(y[1]), "+f"(y[2]), "+f"(y[3]) : "r"(f), "r"(p) : "memory");
}
template <int KC>
__device__ __forceinline__ void peer_st_row(unsigned p, const float (&y)[KC]) {
    if constexpr (KC == 1)
        asm volatile("st.relaxed.cluster.shared::cluster.b32 [%0], %1;" ::"r"(p), "r"(__float_as_uint(y[0])) : "memory");
    else if constexpr (KC == 2)
        asm volatile("st.relaxed.cluster.shared::cluster.v2.b32 [%0], {%1,%2};"
                     ::"r"(p), "r"(__float_as_uint(y[0])), "r"(__float_as_uint(y[1])) : "memory");
    else
        asm volatile("st.relaxed.cluster.shared::cluster.v4.b32 [%0], {%1,%2,%3,%4};"
                     ::"r"(p), "r"(__float_as_uint(y[0])), "r"(__float_as_uint(y[1])), "r"(__float_as_uint(y[2])),
                       "r"(__float_as_uint(y[3])) : "memory");
}

// Polls of shared memory disturb no other SM and the loop around them has to be
// short: the error word and the time budget are looked at every 4096th poll, as
// in idle_clock.
struct near_clock {
    unsigned spins = 0, seen = 0;
    unsigned long long t0 = 0;
    template <class Pending>
    __device__ __forceinline__ bool idle(dev_error* err, unsigned long long budget, int where, uint32_t row, Pending&& pending) {
        if ((++spins & 4095u) != 0) return false;
        if (t0 == 0) t0 = globaltimer();
        const int st = look(err, __shfl_sync(kFull, t0, 0), budget);
        if (st == kWait) return false;
        const unsigned now = pending();
        if (st == kFailed || !__any_sync(kFull, now != seen)) return st == kFailed || run_out(err, where, row);
        seen = now;
        t0 = globaltimer();
        return false;
    }
    __device__ __forceinline__ bool idle(dev_error* err, unsigned long long budget, int where, uint32_t row) {
        return idle(err, budget, where, row, [this] { return seen; });
    }
};

__device__ __forceinline__ double quiet_nan(double) { return __longlong_as_double(0x7ff8000000000000ll); }
__device__ __forceinline__ float quiet_nan(float) { return __uint_as_float(0x7fc00000u); }

// The cluster's column slice and the warp's place among the cluster's warps.
struct tail_seat {
    unsigned col0, warp, warps, base;   // base: shared address of the CTA's copy
};

__device__ __forceinline__ tail_seat take_seat(int kc, unsigned base) {
    const unsigned cs = cluster_size();
    tail_seat t;
    t.col0 = (blockIdx.x / cs) * kc;
    t.warp = (threadIdx.x >> 5) * cs + cluster_rank();   // consecutive items on different SMs
    t.warps = cs * (kTailThreads / 32);
    t.base = base;
    return t;
}

// Lane view of a tail item: a factor plan's rows take all 32 lanes (its lane
// groups are sized for throughput; here few rows mean few entries per lane).
__device__ __forceinline__ lane_view spread_view(stage_desc d) {
    const unsigned rows = d.info & 0xffu;
    if (rows) {
        const unsigned lg = 5u - (32u - __clz(rows - 1u));   // 32 >> lg >= rows
        d.info = (d.info & ~0xff00u) | (lg << 8);
    }
    return view_of(d);
}

// Stores a solved row's value into every copy: lane u of the row's group into
// copies u, u + G, ...; at: the row's shared address, to: its address in copy u.
template <class St>
__device__ __forceinline__ void push_row(const lane_view& v, unsigned cs, unsigned at, unsigned to, St&& st) {
    if (v.valid && v.u < cs) st(to);
    for (unsigned q = v.u + v.G; q < cs; q += v.G)
        if (v.valid) st(peer_addr(at, q));
}

// ---- fp64: the reference's sum order, as run64

struct near_row64 {
    lane_view v;
    double rhs, d;               // every lane of the group
    uint32_t jj[kBatch];
    float ww[kBatch];
};

__device__ __forceinline__ void near_entries64(const tail_args<double>& p, const lane_view& v, uint32_t jb, near_row64& s) {
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
        const uint32_t t = ((jb + k) << v.lg) + v.u;
        s.jj[k] = 0xffffffffu;
        s.ww[k] = 0.0f;
        if (t < v.len) { s.jj[k] = __ldg(p.idx + v.q + t); s.ww[k] = __ldg(p.val + v.q + t); }
    }
}

__device__ __forceinline__ void near_data64(const tail_args<double>& a, const stage_desc& ds, near_row64& s) {
    // rows of one lane each in the plan keep it when there are more than eight (the 4-way sum needs 4 lanes a row)
    s.v = (ds.info & 0xff00u) == 0 && (ds.info & 0xffu) > 8u ? view_of(ds) : spread_view(ds);
    s.rhs = 0.0; s.d = 1.0;
    near_entries64(a, s.v, 0, s);
    if (s.v.valid) {
        s.rhs = a.in[s.v.row];
        s.d = static_cast<double>(__ldg(a.val + s.v.q + s.v.len));
    }
}

// Operands of a batch from outside the tail (complete before the launch); the
// tail's own are marked as to come.
__device__ __forceinline__ void near_outside64(const tail_args<double>& a, const near_row64& s, double (&y)[kBatch]) {
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
        y[k] = s.jj[k] == 0xffffffffu ? 0.0 : sent_of(0.0);
        if (s.jj[k] < a.first) {
            y[k] = a.out[s.jj[k]];
            if (is_sent(y[k])) y[k] = quiet_nan(0.0);   // the launch before this one failed
        }
    }
}

// One batch of NB steps (NB >= the warp's steps in it) of group rows: products
// into shared memory as the operands arrive; while some are missing the leading
// ones are consumed, and the rest when the last is in. Every lane runs the
// chain u mod 4 of its row (thin) or the serial sum (fat): the same values, no
// divergence.
template <int NB>
__device__ __forceinline__ bool near_batch64(const tail_args<double>& a, const tail_seat& t, const near_row64& s,
                                             double (&y)[kBatch], uint32_t jb, uint32_t gend, int where, double* prod,
                                             uint32_t& at, double& sum) {
    const lane_view& v = s.v;
    near_clock clk;
    const unsigned lane = threadIdx.x & 31u;
    const double* pr = prod + v.G * v.gid;
    const unsigned W = v.thin ? 4u : 1u, c = v.thin ? (v.u & 3u) : 0u;
    const auto prod_of = [&](uint32_t e) { return pr[32u * ((e >> v.lg) - jb) + (e & (v.G - 1u))]; };
    const auto take = [&](uint32_t upto) {
        while (at + 4u * W <= upto) {
            const double q0 = prod_of(at + c), q1 = prod_of(at + W + c), q2 = prod_of(at + 2u * W + c), q3 = prod_of(at + 3u * W + c);
            sum = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(sum, q0), q1), q2), q3);
            at += 4u * W;
        }
        while (at + W <= upto) {
            sum = __dadd_rn(sum, prod_of(at + c));
            at += W;
        }
    };
    bool w[NB];
#pragma unroll
    for (int k = 0; k < NB; ++k) w[k] = true;
    for (;;) {
        bool open = false, got = false;
#pragma unroll
        for (int k = 0; k < NB; ++k) near_ld_if(w[k] && is_sent(y[k]), t.base + (s.jj[k] - a.first) * 8u, y[k]);
#pragma unroll
        for (int k = 0; k < NB; ++k) {
            if (w[k] && !is_sent(y[k])) {
                prod[32 * k + lane] = __dmul_rn(static_cast<double>(s.ww[k]), y[k]);
                w[k] = false;
                got = true;
            }
            open |= w[k];
        }
        const bool more = __any_sync(kFull, open);
        if (!more) break;
        if (__any_sync(kFull, got)) {
            // the entries before the group's first missing one
            unsigned pend = 0;
#pragma unroll
            for (int k = 0; k < NB; ++k) pend |= w[k] ? 1u << k : 0u;
            __syncwarp();
            const uint32_t st = static_cast<uint32_t>(__ffs(__reduce_or_sync(kFull, pend))) - 1u;
            const unsigned miss = __ballot_sync(kFull, (pend >> st) & 1u) >> (v.gid << v.lg);
            const unsigned mine = v.lg == 5 ? miss : miss & ((1u << v.G) - 1u);
            take(min(gend, ((jb + st) << v.lg) + (mine ? static_cast<uint32_t>(__ffs(mine)) - 1u : v.G)));
            clk = near_clock{};
        }
        if (clk.idle(a.err, a.budget_ns, where, v.row)) return false;
    }
    __syncwarp();
    take(min(gend, (jb + NB) << v.lg));
    return true;
}

__device__ __forceinline__ bool near_group64(const tail_args<double>& a, const tail_seat& t, near_row64& s,
                                             double (&y)[kBatch], int where, double* prod, double& total) {
    const lane_view& v = s.v;
    const uint32_t Jmax = __reduce_max_sync(kFull, (v.len + v.G - 1u) >> v.lg);
    const uint32_t gend = v.thin ? (v.len & ~3u) : v.len;   // entries the chains take
    double sum = 0.0;
    uint32_t at = 0, jb = 0;
    for (; jb + kBatch < Jmax; jb += kBatch) {
        if (!near_batch64<kBatch>(a, t, s, y, jb, gend, where, prod, at, sum)) return false;
        near_entries64(a, v, jb + kBatch, s);
        near_outside64(a, s, y);
        __syncwarp();   // the batch's products have been read
    }
    const uint32_t nb = Jmax - jb;
    const bool ok = nb <= 1 ? near_batch64<1>(a, t, s, y, jb, gend, where, prod, at, sum)
                  : nb <= 2 ? near_batch64<2>(a, t, s, y, jb, gend, where, prod, at, sum)
                  : nb <= 4 ? near_batch64<4>(a, t, s, y, jb, gend, where, prod, at, sum)
                            : near_batch64<kBatch>(a, t, s, y, jb, gend, where, prod, at, sum);
    if (!ok) return false;
    if (v.thin) {   // (s0 + s1) + (s2 + s3), then the <= 3 entries left (in the row's last batch)
        sum = __dadd_rn(sum, __shfl_xor_sync(kFull, sum, 1));
        sum = __dadd_rn(sum, __shfl_xor_sync(kFull, sum, 2));
        const double* pr = prod + v.G * v.gid;
        for (uint32_t e = gend; e < v.len; ++e) sum = __dadd_rn(sum, pr[32u * ((e >> v.lg) - jb) + (e & (v.G - 1u))]);
    }
    __syncwarp();   // the products have been read
    total = sum;
    return true;
}

// More than eight rows of <= kBatch entries: a lane each.
__device__ __forceinline__ bool near_lane64(const tail_args<double>& a, const tail_seat& t, const near_row64& s,
                                            double (&y)[kBatch], int where, double& total) {
    const lane_view& v = s.v;
    near_clock clk;
    for (;;) {
        bool open = false;
#pragma unroll
        for (int k = 0; k < kBatch; ++k) near_ld_if(is_sent(y[k]), t.base + (s.jj[k] - a.first) * 8u, y[k]);
#pragma unroll
        for (int k = 0; k < kBatch; ++k) open |= is_sent(y[k]);
        if (!__any_sync(kFull, open)) break;
        const auto pending = [&] {
            unsigned p = 0;
#pragma unroll
            for (int k = 0; k < kBatch; ++k) p |= is_sent(y[k]) ? 1u << k : 0u;
            return p;
        };
        if (clk.idle(a.err, a.budget_ns, where, v.row, pending)) return false;
    }
    double p[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) p[k] = __dmul_rn(static_cast<double>(s.ww[k]), y[k]);
    total = lane_sum64(p, v.len, __reduce_max_sync(kFull, v.len), v.thin ? (v.len & ~3u) : 0u);
    return true;
}

__global__ void __launch_bounds__(kTailThreads, 1) k_tail64(const tail_args<double> a, int where) {
    if (a.skip && *a.skip) return;
    extern __shared__ __align__(16) double near_y[];
    __shared__ __align__(16) double prods[kTailThreads / 32][32 * kBatch];
    double* prod = prods[threadIdx.x >> 5];
    const tail_seat t = take_seat(1, static_cast<unsigned>(__cvta_generic_to_shared(near_y)));
    for (uint32_t i = threadIdx.x; i < a.rows; i += kTailThreads) near_y[i] = sent_of(0.0);
    cluster_barrier();
    const unsigned cs = cluster_size();
    uint32_t c = a.item0 + t.warp;
    stage_desc ds;
    near_row64 s0, s1;
    double y0[kBatch], y1[kBatch];
    load_desc(a, c, a.item1, ds);
    near_data64(a, ds, s0);
    load_desc(a, c + t.warps, a.item1, ds);
    near_data64(a, ds, s1);
    load_desc(a, c + 2 * t.warps, a.item1, ds);
    near_outside64(a, s0, y0);
    while (s0.v.c < a.item1) {
        near_outside64(a, s1, y1);   // the next item's indices came in with the last one
        const lane_view& v = s0.v;
        const recip64 inv = recip_of(s0.d);
        const unsigned at = t.base + (v.valid ? v.row - a.first : 0u) * 8u, to = peer_addr(at, v.u & (cs - 1u));
        double rhs = s0.rhs, total = 0.0;
        if (a.rhs_sub) rhs = __dsub_rn(rhs, *a.rhs_sub);
        if (!(v.lg == 0 ? near_lane64(a, t, s0, y0, where, total) : near_group64(a, t, s0, y0, where, prod, total))) break;
        const double y = inv.quotient(__dsub_rn(rhs, total));
        push_row(v, cs, at, to, [&](unsigned p) { peer_st(p, y); });
        if (v.valid && v.u == 0) {
            a.out[v.row] = y;
            if (a.copy_out) a.copy_out[v.row] = y;
            if (a.reset) a.reset[v.row] = sent_of(0.0);
        }
        s0 = s1;
#pragma unroll
        for (int k = 0; k < kBatch; ++k) y0[k] = y1[k];
        near_data64(a, ds, s1);
        c += t.warps;
        load_desc(a, c + 2 * t.warps, a.item1, ds);
    }
    cluster_barrier();   // no CTA leaves while another may still store into its copy
}

// ---- fp32: KC columns of the k per cluster, every lane adding its entries in
// order (oldest dependency first), the lanes' sums by a fixed butterfly

// a / d in fp32, correctly rounded, for a divisor known before the dividend: a
// Newton step on a r, r = RN(1 / d), makes the quotient faithful, and a faithful
// quotient corrected by its exact remainder times r is the rounded one
// (Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", 1990). Divisors and dividends whose reciprocal, quotient or
// remainder leaves the normal range divide.
struct recip32 {
    float d, r;
    unsigned span;   // exponents of a that take the short way: [67, 67 + span)
    __device__ __forceinline__ float quotient(float a) const {
        float q = __fmul_rn(a, r);
        q = __fmaf_rn(__fmaf_rn(-d, q, a), r, q);
        q = __fmaf_rn(__fmaf_rn(-d, q, a), r, q);
        if (((__float_as_uint(a) >> 23) & 0xffu) - 67u >= span) q = __fdiv_rn(a, d);
        return q;
    }
};
__device__ __forceinline__ recip32 recip_of(float d) {
    return {d, __frcp_rn(d), ((__float_as_uint(d) >> 23) & 0xffu) - (127u - 40u) < 80u ? 120u : 0u};
}

template <int KC>
struct near_row32 {
    lane_view v;
    float rhs[KC], d;            // every lane of the group
    uint32_t jj[kBatch];
    float ww[kBatch];
};

template <bool H>
__device__ __forceinline__ float tail_weight(const tail_args<float>& p, uint32_t e) {
    if constexpr (H) return __half2float(__ushort_as_half(__ldg(p.val16 + e)));
    else return __ldg(p.val + e);
}

template <int KC, bool H>
__device__ __forceinline__ void near_entries32(const tail_args<float>& p, const lane_view& v, uint32_t jb, bool back,
                                               near_row32<KC>& s) {
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
        const uint32_t t = ((jb + k) << v.lg) + v.u;
        s.jj[k] = 0xffffffffu;
        s.ww[k] = 0.0f;
        if (t < v.len) {
            const uint32_t e = entry_at(v, t, back);
            s.jj[k] = __ldg(p.idx + e);
            s.ww[k] = tail_weight<H>(p, e);
        }
    }
}

template <int KC, bool H>
__device__ __forceinline__ void near_data32(const tail_args<float>& a, const tail_seat& t, const stage_desc& ds, bool back,
                                            near_row32<KC>& s) {
    if (a.wide) {   // a batch plan's row keeps its entry lanes, and with them the dataflow launch's sums
        s.v = view_of(ds);   // (k <= 4: one column lane)
    } else {
        s.v = spread_view(ds);
    }
    const lane_view& v = s.v;
    s.d = 1.0f;
#pragma unroll
    for (int r = 0; r < KC; ++r) s.rhs[r] = 0.0f;
    near_entries32<KC, H>(a, v, 0, back && !a.wide, s);   // batch plans list the oldest dependency first both ways
    if (v.valid) {
        const size_t base = static_cast<size_t>(v.row) * a.k + t.col0;
        if (a.in64) {
#pragma unroll
            for (int r = 0; r < KC; ++r) {
                double x = a.in64[base + r];
                if (a.rhs_sub) x -= a.rhs_sub[t.col0 + r];
                s.rhs[r] = static_cast<float>(x);
            }
        } else if (H && back) {   // fp16 storage: the backward input times inv_scale^2, in fp64, rounded once
            const double sc = a.scale2[v.row];
#pragma unroll
            for (int r = 0; r < KC; ++r) s.rhs[r] = static_cast<float>(static_cast<double>(a.in[base + r]) * sc);
        } else {
#pragma unroll
            for (int r = 0; r < KC; ++r) s.rhs[r] = a.in[base + r];
        }
        s.d = H ? __ldg(a.diag16 + v.row) : __ldg(a.val + v.q + v.len);
    }
}

// Operand rows of a batch from outside the tail (complete before the launch);
// the tail's own are marked as to come, absent ones are 0 (with weight 0).
template <int KC>
__device__ __forceinline__ void near_outside32(const tail_args<float>& a, const tail_seat& t, const near_row32<KC>& s,
                                               float (&yv)[kBatch][KC]) {
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
        const uint32_t j = s.jj[k];
#pragma unroll
        for (int r = 0; r < KC; ++r) yv[k][r] = j == 0xffffffffu ? 0.0f : sent_of(0.0f);
        if (j >= a.first) continue;
        const float* src = a.out + static_cast<size_t>(j) * a.k + t.col0;
        if constexpr (KC == 4) {
            const float4 q = *reinterpret_cast<const float4*>(src);
            yv[k][0] = q.x; yv[k][1] = q.y; yv[k][2] = q.z; yv[k][3] = q.w;
        } else if constexpr (KC == 2) {
            const float2 q = *reinterpret_cast<const float2*>(src);
            yv[k][0] = q.x; yv[k][1] = q.y;
        } else {
            yv[k][0] = src[0];
        }
#pragma unroll
        for (int r = 0; r < KC; ++r)
            if (is_sent(yv[k][r])) yv[k][r] = quiet_nan(0.0f);   // the launch before this one failed
    }
}

// One batch of NB steps (NB >= the warp's steps in it): polls until every
// operand is in, then the sums in straight line.
template <int KC, int NB>
__device__ __forceinline__ bool near_batch32(const tail_args<float>& a, const tail_seat& t, const near_row32<KC>& s,
                                             float (&yv)[kBatch][KC], int where, float (&acc)[KC]) {
    near_clock clk;
    for (;;) {
        bool open = false;
#pragma unroll
        for (int k = 0; k < NB; ++k)
            near_ld_row_if<KC>(!row_ready<KC>(yv[k]), t.base + (s.jj[k] - a.first) * (4u * KC), yv[k]);
#pragma unroll
        for (int k = 0; k < NB; ++k) open |= !row_ready<KC>(yv[k]);
        if (!__any_sync(kFull, open)) break;
        const auto pending = [&] {
            unsigned p = 0;
#pragma unroll
            for (int k = 0; k < NB; ++k) p |= !row_ready<KC>(yv[k]) ? 1u << k : 0u;
            return p;
        };
        if (clk.idle(a.err, a.budget_ns, where, s.v.row, pending)) return false;
    }
#pragma unroll
    for (int k = 0; k < NB; ++k)
#pragma unroll
        for (int r = 0; r < KC; ++r) acc[r] = __fmaf_rn(s.ww[k], yv[k][r], acc[r]);
    return true;
}

template <int KC, bool H>
__device__ __forceinline__ bool near_run32(const tail_args<float>& a, const tail_seat& t, near_row32<KC>& s, bool back,
                                           int where, float (&yv)[kBatch][KC], float (&acc)[KC]) {
    const lane_view& v = s.v;
    const uint32_t Jmax = __reduce_max_sync(kFull, (v.len + v.G - 1u) >> v.lg);
#pragma unroll
    for (int r = 0; r < KC; ++r) acc[r] = 0.0f;
    uint32_t jb = 0;
    for (; jb + kBatch < Jmax; jb += kBatch) {
        if (!near_batch32<KC, kBatch>(a, t, s, yv, where, acc)) return false;
        near_entries32<KC, H>(a, v, jb + kBatch, back && !a.wide, s);
        near_outside32<KC>(a, t, s, yv);
    }
    const uint32_t nb = Jmax - jb;
    const bool ok = nb <= 1 ? near_batch32<KC, 1>(a, t, s, yv, where, acc)
                  : nb <= 2 ? near_batch32<KC, 2>(a, t, s, yv, where, acc)
                  : nb <= 4 ? near_batch32<KC, 4>(a, t, s, yv, where, acc)
                            : near_batch32<KC, kBatch>(a, t, s, yv, where, acc);
    if (!ok) return false;
#pragma unroll
    for (unsigned i = 5; i-- > 0;)
        if (v.lg > i)
#pragma unroll
            for (int r = 0; r < KC; ++r) acc[r] += __shfl_xor_sync(kFull, acc[r], 1 << i);
    return true;
}

template <int KC, bool H>
__global__ void __launch_bounds__(kTailThreads, 1) k_tail32(const tail_args<float> a, int back) {
    if (a.skip && *a.skip) return;
    extern __shared__ __align__(16) float near_f[];
    const tail_seat t = take_seat(KC, static_cast<unsigned>(__cvta_generic_to_shared(near_f)));
    for (uint32_t i = threadIdx.x; i < a.rows * KC; i += kTailThreads) near_f[i] = sent_of(0.0f);
    cluster_barrier();
    const unsigned cs = cluster_size();
    const int where = back ? kBckSweep32 : kFwdSweep32;
    uint32_t c = a.item0 + t.warp;
    stage_desc ds;
    near_row32<KC> s0, s1;
    float y0[kBatch][KC], y1[kBatch][KC];
    load_desc(a, c, a.item1, ds);
    near_data32<KC, H>(a, t, ds, back, s0);
    load_desc(a, c + t.warps, a.item1, ds);
    near_data32<KC, H>(a, t, ds, back, s1);
    load_desc(a, c + 2 * t.warps, a.item1, ds);
    near_outside32<KC>(a, t, s0, y0);
    while (s0.v.c < a.item1) {
        near_outside32<KC>(a, t, s1, y1);   // the next item's indices came in with the last one
        const lane_view& v = s0.v;
        const recip32 inv = recip_of(s0.d);
        const unsigned at = t.base + (v.valid ? v.row - a.first : 0u) * (4u * KC), to = peer_addr(at, v.u & (cs - 1u));
        float acc[KC], y[KC];
        if (!near_run32<KC, H>(a, t, s0, back, where, y0, acc)) break;
#pragma unroll
        for (int r = 0; r < KC; ++r) y[r] = inv.quotient(s0.rhs[r] - acc[r]);
        push_row(v, cs, at, to, [&](unsigned p) { peer_st_row<KC>(p, y); });
        if (v.valid && v.u == 0) {
            const size_t base = static_cast<size_t>(v.row) * a.k + t.col0;
            st_row<KC>(a.out + base, y);
            if (a.reset) {
                float sent[KC];
#pragma unroll
                for (int r = 0; r < KC; ++r) sent[r] = sent_of(0.0f);
                st_row<KC>(a.reset + base, sent);
            }
        }
        s0 = s1;
#pragma unroll
        for (int k = 0; k < kBatch; ++k)
#pragma unroll
            for (int r = 0; r < KC; ++r) y0[k][r] = y1[k][r];
        near_data32<KC, H>(a, t, ds, back, s1);
        c += t.warps;
        load_desc(a, c + 2 * t.warps, a.item1, ds);
    }
    cluster_barrier();   // no CTA leaves while another may still store into its copy
}

__global__ void k_fill64(double* p, size_t n, double v) {
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x)
        p[i] = v;
}
__global__ void k_fill32(float* p, size_t n, float v) {
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x)
        p[i] = v;
}

int fill_grid(size_t n) {
    const size_t b = (n + 255) / 256;
    return static_cast<int>(b < 4096 ? (b ? b : 1) : 4096);
}

template <int K>
int occ32() {
    int b0 = 0, b1 = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b0, k_df32<0, K, false>, kSweepThreads, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b1, k_df32<1, K, false>, kSweepThreads, 0);
    return b0 < b1 ? b0 : b1;
}

// One cluster per column slice (kc columns), of the tail's CTAs or of the largest
// power of two below that keeps all clusters within the sweep's grid (one CTA a
// slice at least). A row's sum does not depend on the cluster's size.
template <class F, class A>
void tail_launch(F* kernel, const tail_args<A>& a, int kc, int cluster, int grid, int flag, cudaStream_t s) {
    while (cluster > 1 && cluster * (a.k / kc) > grid) cluster /= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(a.k / kc) * static_cast<unsigned>(cluster));
    cfg.blockDim = dim3(kTailThreads);
    cfg.dynamicSmemBytes = static_cast<size_t>(a.rows) * kc * sizeof(A);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = static_cast<unsigned>(cluster);
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, a, flag);
}

template <int KC>
void tail32_kc(int dir, const tail_args<float>& a, bool fp16, int cluster, int grid, cudaStream_t s) {
    if (fp16) tail_launch(k_tail32<KC, true>, a, KC, cluster, grid, dir, s);
    else tail_launch(k_tail32<KC, false>, a, KC, cluster, grid, dir, s);
}

// The tail launch's arguments of a sweep (w.tail set).
template <class T>
tail_args<T> tail_args_of(const sweep_args<T>& w) {
    tail_args<T> a{};
    a.info = w.info; a.ord = w.ord; a.ptr = w.ptr; a.idx = w.idx; a.val = w.val;
    a.val16 = w.val16; a.diag16 = w.diag16; a.scale2 = w.in_scale2;
    a.item0 = w.tail->item0; a.item1 = w.tail->item1; a.first = w.tail->first; a.rows = w.tail->rows;
    a.in = w.in; a.rhs_sub = w.rhs_sub; a.out = w.out; a.reset = w.reset; a.copy_out = w.copy_out;
    a.err = w.err; a.skip = w.skip; a.budget_ns = w.budget_ns;
    return a;
}

void tail64(int dir, const sweep_args<double>& w, int grid, cudaStream_t s) {
    tail_args<double> a = tail_args_of(w);
    a.k = 1;
    tail_launch(k_tail64, a, 1, w.tail->cluster, grid, dir == 0 ? kFwdSweep : kBckSweep, s);
}

// wide: the plan is a batch plan.
void tail32(int dir, const sweep_args<float>& w, const double* in64, bool wide, int grid, cudaStream_t s) {
    tail_args<float> a = tail_args_of(w);
    a.k = w.k; a.in64 = in64;
    a.wide = wide;
    const bool fp16 = w.val16 != nullptr;
    // Up to four clusters: a row's sums and its store are on the chain of levels, so fewer columns a
    // cluster are faster (batch of k = 4, 6-regular n = 100003, forward / backward: 394 / 414 us with
    // one cluster of 4 columns, 294 / 299 with four).
    if (w.k >= 16) tail32_kc<4>(dir, a, fp16, w.tail->cluster, grid, s);
    else if (w.k == 8) tail32_kc<2>(dir, a, fp16, w.tail->cluster, grid, s);
    else tail32_kc<1>(dir, a, fp16, w.tail->cluster, grid, s);
}

// The claim units a dataflow launch works off: all, or the part outside the tail.
template <class T>
sweep_args<T> outside_tail(int dir, const sweep_args<T>& w) {
    sweep_args<T> a = w;
    if (w.tail) {
        if (dir == 0) {
            a.n_chunks = w.tail->chunk;
        } else {
            a.chunk = w.chunk + w.tail->chunk;
            a.n_chunks = w.n_chunks - w.tail->chunk;
        }
    }
    return a;
}

template <class F>
int clusters_of(F* kernel, int size) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kTailSmem)) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(size));
    cfg.blockDim = dim3(kTailThreads);
    cfg.dynamicSmemBytes = kTailSmem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = static_cast<unsigned>(size);
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

template <int K>
void sweep32_dir(int dir, const sweep_args<float>& w, const double* in64, int grid, cudaStream_t s) {
    const sweep_args<float> a = outside_tail(dir, w);
    if (dir == 1 && w.tail) tail32(dir, w, in64, false, grid, s);
    if (a.n_items && a.n_chunks) {
        if (a.val16) {
            if (dir == 0) k_df32<0, K, true><<<grid, kSweepThreads, 0, s>>>(a, in64);
            else          k_df32<1, K, true><<<grid, kSweepThreads, 0, s>>>(a, in64);
        } else {
            if (dir == 0) k_df32<0, K, false><<<grid, kSweepThreads, 0, s>>>(a, in64);
            else          k_df32<1, K, false><<<grid, kSweepThreads, 0, s>>>(a, in64);
        }
    }
    if (dir == 0 && w.tail) tail32(dir, w, in64, false, grid, s);
}

}  // namespace

int tail_cluster_size() {
    for (int size : {16, 8}) {
        const int n = std::min({clusters_of(k_tail64, size), clusters_of(k_tail32<1, false>, size), clusters_of(k_tail32<1, true>, size),
                                clusters_of(k_tail32<2, false>, size), clusters_of(k_tail32<2, true>, size),
                                clusters_of(k_tail32<4, false>, size), clusters_of(k_tail32<4, true>, size)});
        if (n > 0) return size;
    }
    return 0;
}

void launch_sweep64(int dir, const sweep_args<double>& w, int grid, cudaStream_t s) {
    const sweep_args<double> a = outside_tail(dir, w);
    if (dir == 1 && w.tail) tail64(dir, w, grid, s);
    if (a.n_items && a.n_chunks) {
        if (dir == 0) k_df64<0><<<grid, kSweepThreads, 0, s>>>(a);
        else          k_df64<1><<<grid, kSweepThreads, 0, s>>>(a);
    }
    if (dir == 0 && w.tail) tail64(dir, w, grid, s);
}

void launch_sweep32(int dir, const sweep_args<float>& a, int grid, cudaStream_t s) {
    launch_sweep32_from64(dir, a, nullptr, grid, s);
}

void launch_sweep32_from64(int dir, const sweep_args<float>& a, const double* in64, int grid, cudaStream_t s) {
    switch (a.k) {
        case 1:  sweep32_dir<1>(dir, a, in64, grid, s); break;
        case 2:  sweep32_dir<2>(dir, a, in64, grid, s); break;
        case 4:  sweep32_dir<4>(dir, a, in64, grid, s); break;
        case 8:  sweep32_dir<8>(dir, a, in64, grid, s); break;
        default: sweep32_dir<16>(dir, a, in64, grid, s); break;
    }
}

int sweep_grid64(int num_sms) {
    int b0 = 0, b1 = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b0, k_df64<0>, kSweepThreads, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b1, k_df64<1>, kSweepThreads, 0);
    const int b = b0 < b1 ? b0 : b1;
    return (b > 0 ? b : 1) * num_sms;
}

template <int K>
void sweep32_batch_dir(int dir, const sweep_args<float>& w, int grid, cudaStream_t s) {
    const sweep_args<float> a = outside_tail(dir, w);
    if (dir == 1 && w.tail) tail32(dir, w, nullptr, true, grid, s);
    if (a.n_items && a.n_chunks) {
        if (a.val16) {
            if (dir == 0) k_dw32<0, K, true><<<grid, kSweepThreads, 0, s>>>(a);
            else          k_dw32<1, K, true><<<grid, kSweepThreads, 0, s>>>(a);
        } else {
            if (dir == 0) k_dw32<0, K, false><<<grid, kSweepThreads, 0, s>>>(a);
            else          k_dw32<1, K, false><<<grid, kSweepThreads, 0, s>>>(a);
        }
    }
    if (dir == 0 && w.tail) tail32(dir, w, nullptr, true, grid, s);
}

void launch_sweep32_batch(int dir, const sweep_args<float>& a, int grid, cudaStream_t s) {
    switch (a.k) {
        case 1:  sweep32_batch_dir<1>(dir, a, grid, s); break;
        case 2:  sweep32_batch_dir<2>(dir, a, grid, s); break;
        case 4:  sweep32_batch_dir<4>(dir, a, grid, s); break;
        case 8:  sweep32_batch_dir<8>(dir, a, grid, s); break;
        case 16: sweep32_batch_dir<16>(dir, a, grid, s); break;
        case 32: sweep32_batch_dir<32>(dir, a, grid, s); break;
        case 64: sweep32_batch_dir<64>(dir, a, grid, s); break;
        default: sweep32_batch_dir<128>(dir, a, grid, s); break;
    }
}

template <int K>
int occ32_batch() {
    int b = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_dw32<1, K, false>, kSweepThreads, 0);
    return b;
}

int sweep_grid32_batch(int k, int num_sms) {
    int b = 1;
    switch (k) {
        case 1: b = occ32_batch<1>(); break;
        case 2: b = occ32_batch<2>(); break;
        case 4: b = occ32_batch<4>(); break;
        case 8: b = occ32_batch<8>(); break;
        case 16: b = occ32_batch<16>(); break;
        case 32: b = occ32_batch<32>(); break;
        case 64: b = occ32_batch<64>(); break;
        default: b = occ32_batch<128>(); break;
    }
    return (b > 0 ? b : 1) * num_sms;
}

int sweep_grid32(int k, int num_sms) {
    int b = 1;
    switch (k) {
        case 1: b = occ32<1>(); break;
        case 2: b = occ32<2>(); break;
        case 4: b = occ32<4>(); break;
        case 8: b = occ32<8>(); break;
        default: b = occ32<16>(); break;
    }
    return (b > 0 ? b : 1) * num_sms;
}

void launch_fill64(double* p, size_t n, double v, cudaStream_t s) {
    if (n) k_fill64<<<fill_grid(n), 256, 0, s>>>(p, n, v);
}
void launch_fill32(float* p, size_t n, float v, cudaStream_t s) {
    if (n) k_fill32<<<fill_grid(n), 256, 0, s>>>(p, n, v);
}
void launch_fill_sent64(double* p, size_t n, cudaStream_t s) {
    double v;
    const uint64_t bits = kSent64;
    __builtin_memcpy(&v, &bits, sizeof(v));
    launch_fill64(p, n, v, s);
}
void launch_fill_sent32(float* p, size_t n, cudaStream_t s) {
    float v;
    const uint32_t bits = kSent32;
    __builtin_memcpy(&v, &bits, sizeof(v));
    launch_fill32(p, n, v, s);
}

}  // namespace apxb
