// Complex128 LU of a block of columns by one thread-block cluster (sm_100a).
//
// A partial-pivoting factorisation is a chain of n pivot searches, each of
// which every row below the diagonal takes part in.  What bounds it at the
// orders of an antenna solve is the time of one link of that chain, so this
// kernel keeps the chain inside one cluster of at most 16 CTAs:
//   panel   W = 16 columns at a time, each row of the panel in the registers
//           of one thread (rows never move while the panel is factored: a
//           thread tracks the position its row would hold after LAPACK's
//           interchanges).  For every column each CTA sends its candidate's
//           key and row to all CTAs with st.async, which signals
//           the receiver's mbarrier: one one-way trip through distributed
//           shared memory per column and no barrier round trip (a cluster
//           barrier behind plain remote stores took 1,200 cycles of a
//           4,500-cycle column).  The next column's search and send
//           come before the bulk of the row update.  Up to 32 rows per CTA one
//           warp does it all.
//   rest    the panel's row interchanges and the W x W triangular solve of
//           the columns to its right, four lanes per column (all gathered
//           values in flight at once; every CTA already holds L11 and the
//           row order from the exchange), then the rank-W update on FP64
//           tensor instructions, 16 x 32 entries a warp.
//   B       right-hand sides ride along as further columns; with `back` the
//           kernel also substitutes backwards, each CTA its own right-hand
//           sides, so a small system is factored and solved by one launch.
// The batch is on the grid: cluster b works on matrix b.
//
// Once 256 rows or fewer are left, one CTA factors the panel alone
// (panel_solo): two CTA barriers a column beat the exchange.
//
// Measured on B200 (order 306, one right-hand side): 2.0 ms as a sequence of
// cooperative panels, swaps, leaves and products, 0.52 ms as one launch; 64
// such systems 125 ms one after the other, 0.80 ms as one batch.  A column
// of the exchange costs about 2,000 cycles, latencies all: the pivot's pick
// and reciprocal 600, the next search 200, sending the row 400, the flight
// (the other columns' update runs under it) 650.  512 threads a CTA with one
// row each measured slower (635 against 522 us at order 300: the update's
// registers spill), and so did two rows a thread in one CTA (646).
//
// The panel slots rotate: column 0 of the register row is always the current
// pivot column, a step shifts the row left by one and appends the multiplier
// on the right, so the column loop is one copy of code (an unrolled panel
// overflows the instruction cache).
//
// Pivot choice is LAPACK's izamax: largest |re| + |im|, smallest row on ties.
#include "common.cuh"
#include "lu_cluster.cuh"

#include <cooperative_groups.h>

namespace mw {
namespace cg = cooperative_groups;

mw_status zgemm_launch(bool ta, bool tb, int64_t m, int64_t n, int64_t k, cd alpha, const cd* A, int64_t lda,
                       const cd* B, int64_t ldb, cd beta, cd* C, int64_t ldc, cudaStream_t st, int max_ctas,
                       void* split_ws, size_t split_ws_bytes);
constexpr int kCtaPerTile = -1;  // max_ctas: a CTA per tile instead of persistent ones

namespace {

constexpr int kW = 16;          // panel width
constexpr int kCT = 256;        // threads per CTA
constexpr int kCWarps = kCT / 32;
constexpr int kMaxC = 16;       // CTAs per cluster
constexpr int kTM = 16, kTN = 32;  // a warp's update task
constexpr int kBackRows = 1696;  // order times right-hand sides a CTA substitutes at once
constexpr unsigned kNone = 0xffffffffu;
constexpr int kXchBytes = (kW + 1) * 16;  // one CTA's share of a column's exchange
constexpr int kSpinLimit = 1 << 21;       // polls of an exchange wait before it gives up (about two seconds)

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void group_barrier(int threads) {
    asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned map_rank(unsigned addr, int rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// 16 bytes to another CTA's shared memory, counted on that CTA's mbarrier
// (predicated, not branched around: a branch per destination costs more than
// the store)
__device__ __forceinline__ void st_async16(bool on, unsigned dst, cd v, unsigned mbar) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
        " @p st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];\n}" ::"r"(dst),
        "d"(v.re), "d"(v.im), "r"(mbar), "r"((unsigned)on)
        : "memory");
}
__device__ __forceinline__ void mbar_init(unsigned mbar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect(bool on, unsigned mbar, unsigned bytes) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n @p mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n}" ::"r"(
            mbar),
        "r"(bytes), "r"((unsigned)on)
        : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned mbar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(mbar), "r"(parity), "r"(1000u)  // suspended at most a microsecond a poll
        : "memory");
    return ok != 0;
}

// Waits for the phase of an mbarrier, all lanes of a warp together.  True when
// it gave up, after `limit` polls of at most a microsecond, and recorded
// MW_ERR_TIMEOUT.
__device__ __forceinline__ bool exchange_wait(unsigned mbar, unsigned parity, int limit, int32_t* err) {
    int spins = 0;
    bool dead = false;
    while (!mbar_try(mbar, parity))
        if (++spins > limit) {
            dead = true;
            *err = MW_ERR_TIMEOUT;
            break;
        }
    return __any_sync(0xffffffffu, dead);
}

// L2 loads: another CTA of the cluster may have written the line
__device__ __forceinline__ cd ld2(const cd* p) {
    const double2 v = __ldcg(reinterpret_cast<const double2*>(p));
    return cd{v.x, v.y};
}
__device__ __forceinline__ void st2(cd* p, cd v) { __stcg(reinterpret_cast<double2*>(p), make_double2(v.re, v.im)); }

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}
__device__ __forceinline__ cd csub_mul(cd c, cd a, cd b) {  // c - a b
    c.re = fma(-a.re, b.re, c.re);
    c.im = fma(-a.re, b.im, c.im);
    c.re = fma(a.im, b.im, c.re);
    c.im = fma(-a.im, b.re, c.im);
    return c;
}

// Warp-wide best of (value bits hi:lo, larger wins; then smaller pos); lanes
// without a candidate have pos = kNone.  Returns the lane that holds it (a
// lane without a candidate if all do).  Values are non-negative doubles,
// whose bits order like the values.  One reduction settles it unless two
// lanes share the high word.
// (The warp index of the kernels comes from a shuffle: that makes it the same
// in every lane as far as the compiler can see, and the votes and shuffles
// behind branches on it need no code that gathers the warp first.  47.7 -> 42.2
// us at order 21 on B200, 326 -> 306 at 200, 521 -> 495 at 300.)
__device__ __forceinline__ int warp_pick(unsigned mh, unsigned hi, unsigned lo, unsigned pos) {
    const bool h = pos != kNone && hi == mh;
    unsigned eq = __ballot_sync(0xffffffffu, h);
    if (__popc(eq) != 1) {
        const unsigned ml = __reduce_max_sync(0xffffffffu, h ? lo : 0u);
        const bool l = h && lo == ml;
        const unsigned mp = __reduce_min_sync(0xffffffffu, l ? pos : kNone);
        eq = __ballot_sync(0xffffffffu, l && pos == mp);
    }
    return eq ? __ffs(eq) - 1 : 0;
}
__device__ __forceinline__ int warp_best(unsigned hi, unsigned lo, unsigned pos) {
    return warp_pick(__reduce_max_sync(0xffffffffu, pos == kNone ? 0u : hi), hi, lo, pos);
}

struct Shared {
    // every CTA's candidate row, by column mod 4: a warp may still apply the
    // row of column t while the candidates of t + 1 and t + 2 arrive
    cd rows[4][kMaxC][kW];
    uint4 key[4][kMaxC];  // its key: value bits lo, hi, position, row
    unsigned long long mbar[4];
    cd pub[kW + 1];  // this CTA's candidate row and key on their way out
    uint4 wkey[2][kCWarps];  // the warps' candidates, by column parity
    int src[kW];             // row that ends in position c0 + i
    int disp[kW];            // where row c0 + i went (-1: it stays within the top W)
    cd tri[kW][kW + 1];      // W x W triangle of the solves
    cd dinv[kW];
    cd X[kW][4];  // a solved block of the back substitution
    cd inv[2];    // one-CTA panel: the pivot's reciprocal
    cd zero;
    cd y[kBackRows];  // the back substitution's right-hand sides
};

// The panel rows [c0, n) x columns [c0, c0 + w) by one CTA (n - c0 <= kCT):
// ipiv, the factored panel in A at its final positions, S.src, S.disp and
// S.tri.  As in the exchange below, rows stay in their threads and the
// register slots rotate.
__device__ __forceinline__ void panel_solo(Shared& S, cd* A, int64_t lda, int32_t* ipiv, int32_t* info, int n, int c0,
                                           int w) {
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int cnt = n - c0, nw = min(kCWarps, (cnt + 31) / 32);  // warps that hold rows
    if (warp >= nw) return;
    cd a[kW];
    unsigned pos = tid < cnt ? (unsigned)(c0 + tid) : kNone;  // the row's position; kNone: none, or a pivot already
#pragma unroll
    for (int x = 0; x < kW; ++x)
        a[x] = tid < cnt && x < w ? ld2(A + (c0 + tid) + (int64_t)(c0 + x) * lda) : cd{0.0, 0.0};
    unsigned tpos = (unsigned)(c0 + lane);  // lane i: position of row c0 + i
    for (int jj = 0; jj < w; ++jj) {
        const int par = jj & 1;
        const unsigned c = (unsigned)(c0 + jj);
        // the lane that holds the warp's candidate, then the pivot
        const cd z = a[0];
        const unsigned long long bb = (unsigned long long)__double_as_longlong(cabs1(z));
        const unsigned bhi = (unsigned)(bb >> 32), blo = (unsigned)bb;
        const unsigned mh = __reduce_max_sync(0xffffffffu, pos == kNone ? 0u : bhi);
        const cd binv = recip_fast(z);  // (in the shadow of the reduction)
        const int wsrc = warp_pick(mh, bhi, blo, pos);
        int g = wsrc;
        uint4 k = make_uint4(bhi, blo, pos, (unsigned)(c0 + tid));
        bool mine = lane == wsrc;
        if (nw > 1) {
            if (mine) S.wkey[par][warp] = k;
            group_barrier(nw * 32);
            k = S.wkey[par][lane & (kCWarps - 1)];
            g = warp_best(k.x, k.y, lane < nw ? k.z : kNone);
            mine = mine && warp == g;
        }
        const unsigned p = __shfl_sync(0xffffffffu, k.z, g), orig = __shfl_sync(0xffffffffu, k.w, g);
        // LAPACK: an exact zero pivot is neither divided by nor applied
        const bool apply = __shfl_sync(0xffffffffu, k.x | k.y, g) != 0;
        if (mine) {
            cd* row = S.rows[par][0];
#pragma unroll
            for (int x = 0; x < kW; ++x) row[x] = a[x];
            S.inv[par] = !apply ? cd{1.0, 0.0} : (recip_special(z) ? cdiv(cd{1.0, 0.0}, z) : binv);
        }
        if (nw > 1) group_barrier(nw * 32);
        else __syncwarp();
        const cd* piv = S.rows[par][0];
        const cd l = a[0] * S.inv[par];
        const int wj = apply ? kW - jj : 0;  // slots the pivot row updates; multipliers meet a zero
        tpos = tpos == p ? c : (tpos == c ? p : tpos);
        pos = pos == p ? kNone : (pos == c ? p : pos);
#pragma unroll
        for (int x = 0; x + 1 < kW; ++x) a[x] = csub_mul(a[x + 1], l, *(x + 1 < wj ? piv + x + 1 : &S.zero));
        a[kW - 1] = l;
        if (warp == nw - 1) {
            // the pivot row out: slot s < W - jj holds column jj + s, then
            // the multipliers
            if (lane < w) st2(A + c + (int64_t)(c0 + lane) * lda, piv[lane >= jj ? lane - jj : kW - jj + lane]);
            if (lane < jj) S.tri[jj][lane] = piv[kW - jj + lane];
            if (lane == 0) {
                S.src[jj] = (int)orig;
                ipiv[c] = (int32_t)(p + 1);
                if (!apply && info[0] == 0) info[0] = (int32_t)(c + 1);
            }
        }
    }
    // the rows below to their positions: the last w slots hold their multipliers
    if (pos != kNone) {
        cd* row = A + pos + (int64_t)c0 * lda;
#pragma unroll
        for (int s = 0; s < kW; ++s)
            if (s >= kW - w) st2(row + (int64_t)(s - (kW - w)) * lda, a[s]);
    }
    if (warp == 0 && lane < kW) S.disp[lane] = lane < w && tpos >= (unsigned)(c0 + w) ? (int)tpos : -1;
}

template <int RPT>
__global__ void __launch_bounds__(kCT, 1) zlu_cluster_kernel(ZluArgs P) {
    extern __shared__ __align__(16) unsigned char zlu_smem[];
    Shared& S = *reinterpret_cast<Shared*>(zlu_smem);
    cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int64_t mat = blockIdx.x / C;
    cd* const A = P.A + mat * P.a_stride;
    cd* const B = P.B + mat * P.b_stride;
    int32_t* const ipiv = P.ipiv + mat * P.ipiv_stride;
    int32_t* const info = P.info + mat * P.info_stride;
    const int64_t lda = P.lda, ldb = P.ldb;
    const int n = P.n, jend = P.j0 + P.jb;

    if (tid == 0) {
        S.zero = cd{0.0, 0.0};
        for (int i = 0; i < 4; ++i) mbar_init(smem_u32(&S.mbar[i]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (P.rid != nullptr)
        for (int r = P.j0 + rank * kCT + tid; r < n; r += C * kCT) P.rid[r] = r;
    __syncthreads();
    cluster_barrier();
    int step = 0;       // columns done: exchange buffer and mbarrier phase
    bool dead = false;  // an exchange wait gave up: no further waits

    for (int c0 = P.j0; c0 < jend; c0 += kW) {
        const int w = min(kW, jend - c0);
        // ---------------------------------------------------------- panel
        const bool solo = RPT == 1 && n - c0 <= kCT;
        if (solo) {
            // The rows fit one CTA: rank 0 factors the panel alone, two CTA
            // barriers a column instead of an exchange, and the others take
            // the row order and L11 from its shared memory: 104 against 118
            // us at order 64, 355 against 372 at 200.  (Two rows a thread are
            // the slower choice: 646 against 543 us at 300.)
            if (rank == 0) panel_solo(S, A, lda, ipiv, info, n, c0, w);
            __syncwarp();
            cluster_barrier();
            if (rank != 0) {
                if (tid < kW) {
                    S.src[tid] = *cl.map_shared_rank(&S.src[tid], 0);
                    S.disp[tid] = *cl.map_shared_rank(&S.disp[tid], 0);
                }
                if (tid < kW * kW) S.tri[tid / kW][tid % kW] = *cl.map_shared_rank(&S.tri[tid / kW][tid % kW], 0);
            }
        } else {
        const int per = (n - c0 + C - 1) / C;
        const int base = c0 + rank * per;
        const int cnt = max(0, min(per, n - base));
        const int nw = min(kCWarps, (per + 31) / 32);  // warps that hold rows
        if (warp < nw) {
            cd a[RPT][kW];
            unsigned pos[RPT];  // the row's current position; kNone: no row, or a pivot already
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                const int lr = tid + kCT * i;
                const bool ok = lr < cnt;
                pos[i] = ok ? (unsigned)(base + lr) : kNone;
#pragma unroll
                for (int x = 0; x < kW; ++x)
                    a[i][x] = ok && x < w ? ld2(A + (base + lr) + (int64_t)(c0 + x) * lda) : cd{0.0, 0.0};
            }
            unsigned tpos = (unsigned)(c0 + lane);  // lane i: position of row c0 + i
            // this thread's candidate of the next column, and the lane that
            // holds the warp's
            unsigned bhi = 0, blo = 0, bp = kNone;
            int bi = 0, wsrc = 0;
            cd next[RPT], l[RPT];  // next: the rows' entries of the next pivot column
            auto search = [&]() {
                unsigned long long bb = 0;
                bp = kNone;
                bi = 0;
#pragma unroll
                for (int i = 0; i < RPT; ++i)
                    if (pos[i] != kNone) {
                        const unsigned long long v = (unsigned long long)__double_as_longlong(cabs1(next[i]));
                        if (bp == kNone || v > bb || (v == bb && pos[i] < bp)) {
                            bb = v;
                            bp = pos[i];
                            bi = i;
                        }
                    }
                bhi = (unsigned)(bb >> 32);
                blo = (unsigned)bb;
                wsrc = warp_best(bhi, blo, bp);
            };
            // the other CTAs' shared memory: lanes 0-15 send to even, lanes
            // 16-31 to odd ranks
            const unsigned self = smem_u32(&S);
            unsigned peer[kMaxC / 2];
#pragma unroll
            for (int u = 0; u < kMaxC / 2; ++u) peer[u] = map_rank(self, min(2 * u + (lane >> 4), C - 1));
            const unsigned kpeer = map_rank(self, min(lane, C - 1));
            // Sends this CTA's candidate for panel column jj.  Its row is
            // raw (shifted by one slot from slot 1 on, the last pivot row
            // `piv` not yet applied; first column: as it is): the sending
            // lanes apply it, an element each.
            auto publish = [&](int jj, int st, const cd* piv, bool apply) {
                const int buf = st & 3;
                const unsigned mbar = smem_u32(&S.mbar[buf]), omb = mbar - self;
                bool mine = true;  // this warp holds the CTA's candidate
                if (nw > 1) {
                    if (lane == wsrc) S.wkey[st & 1][warp] = make_uint4(bhi, blo, bp, 0);
                    group_barrier(nw * 32);
                    const uint4 k = S.wkey[st & 1][lane & (kCWarps - 1)];
                    mine = warp == warp_best(k.x, k.y, lane < nw ? k.z : kNone);
                }
                mbar_expect(tid == 0, mbar, (unsigned)(C * kXchBytes));
                if (!mine) return;
                if (lane == wsrc) {
#pragma unroll
                    for (int i = 0; i < RPT; ++i)
                        if (RPT == 1 || i == bi) {
                            if (jj == 0) {
#pragma unroll
                                for (int x = 0; x < kW; ++x) S.pub[x] = a[i][x];
                            } else {
#pragma unroll
                                for (int x = 0; x + 1 < kW; ++x) S.pub[x] = a[i][x + 1];
                                S.pub[kW - 1] = l[i];
                            }
                        }
                    // key: value, position, row
                    S.pub[kW] =
                        cd{__longlong_as_double((long long)(((unsigned long long)bhi << 32) | blo)),
                           __longlong_as_double(
                               (long long)(((unsigned long long)(unsigned)(base + tid + kCT * bi) << 32) | bp))};
                }
                __syncwarp();
                const int x = lane & 15;
                cd v = S.pub[x];
                const cd kv = S.pub[kW];
                if (jj > 0 && apply && x < kW - jj) v = csub_mul(v, S.pub[kW - 1], piv[x + 1]);
                const unsigned orow = smem_u32(&S.rows[buf][rank][x]) - self;
                const unsigned okey = smem_u32(&S.key[buf][rank]) - self;
#pragma unroll
                for (int u = 0; u < kMaxC / 2; ++u)
                    st_async16(2 * u + (lane >> 4) < C, peer[u] + orow, v, peer[u] + omb);
                st_async16(lane < C, kpeer + okey, kv, kpeer + omb);
                __syncwarp();
            };
#pragma unroll
            for (int i = 0; i < RPT; ++i) next[i] = a[i][0];
            search();
            publish(0, step, nullptr, false);
            for (int jj = 0; jj < w; ++jj, ++step) {
                const int buf = step & 3;
                const unsigned c = (unsigned)(c0 + jj);
                if (!dead)
                    dead = exchange_wait(smem_u32(&S.mbar[buf]), (unsigned)((step >> 2) & 1), kSpinLimit, info + 1);
                // the winner, from this CTA's own copies; each lane takes the
                // reciprocal of one candidate in the reduction's shadow
                const uint4 k = S.key[buf][lane & (kMaxC - 1)];
                const unsigned kp = lane < C ? k.z : kNone;
                const unsigned mh = __reduce_max_sync(0xffffffffu, kp == kNone ? 0u : k.y);
                const cd z = S.rows[buf][lane & (kMaxC - 1)][0];
                const cd iv = recip_fast(z);
                const unsigned fl = ((k.x | k.y) != 0 ? 1u : 0u) | (recip_special(z) ? 2u : 0u);
                const int g = warp_pick(mh, k.y, k.x, kp) & (kMaxC - 1);
                const unsigned p = __shfl_sync(0xffffffffu, k.z, g), orig = __shfl_sync(0xffffffffu, k.w, g);
                // LAPACK: an exact zero pivot is neither divided by nor applied
                const unsigned flags = __shfl_sync(0xffffffffu, fl, g);
                const bool apply = (flags & 1u) != 0;
                const cd* piv = S.rows[buf][g];
                cd inv{__shfl_sync(0xffffffffu, iv.re, g), __shfl_sync(0xffffffffu, iv.im, g)};
                if (flags & 2u) inv = apply ? cdiv(cd{1.0, 0.0}, piv[0]) : cd{1.0, 0.0};
                const int wj = apply ? kW - jj : 0;  // slots the pivot row updates
                const cd p1 = *(1 < wj ? piv + 1 : &S.zero);
                tpos = tpos == p ? c : (tpos == c ? p : tpos);
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    pos[i] = pos[i] == p ? kNone : (pos[i] == c ? p : pos[i]);
                    l[i] = a[i][0] * inv;
                    next[i] = csub_mul(a[i][1], l[i], p1);
                }
                if (jj + 1 < w) {
                    search();
                    publish(jj + 1, step + 1, piv, apply);
                }
                // while the exchange is under way: the pivot row out, and the
                // other columns (slots that hold multipliers meet a zero; a
                // retired row's registers no longer matter)
                if (warp == nw - 1) {
                    if (rank == (jj & (C - 1)) && lane < w) {
                        // slot s < W - jj holds column jj + s, then the multipliers
                        const int sl = lane >= jj ? lane - jj : kW - jj + lane;
                        st2(A + c + (int64_t)(c0 + lane) * lda, piv[sl]);
                    }
                    if (lane < jj) S.tri[jj][lane] = piv[kW - jj + lane];
                    if (lane == 0) {
                        // (clamped: after a wait that gave up the word is not a row)
                        S.src[jj] = (int)min(max(orig, (unsigned)c0), (unsigned)(n - 1));
                        if (rank == 0) {
                            ipiv[c] = (int32_t)(p + 1);
                            if (!apply && info[0] == 0) info[0] = (int32_t)(c + 1);
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < RPT; ++i) a[i][0] = next[i];
#pragma unroll
                for (int x = 1; x + 1 < kW; ++x) {
                    const cd px = *(x + 1 < wj ? piv + x + 1 : &S.zero);
#pragma unroll
                    for (int i = 0; i < RPT; ++i) a[i][x] = csub_mul(a[i][x + 1], l[i], px);
                }
#pragma unroll
                for (int i = 0; i < RPT; ++i) a[i][kW - 1] = l[i];
            }
            // the rows below to their positions: the last w slots hold their
            // multipliers
#pragma unroll
            for (int i = 0; i < RPT; ++i)
                if (pos[i] != kNone) {
                    cd* row = A + min(pos[i], (unsigned)(n - 1)) + (int64_t)c0 * lda;
#pragma unroll
                    for (int s = 0; s < kW; ++s)
                        if (s >= kW - w) st2(row + (int64_t)(s - (kW - w)) * lda, a[i][s]);
                }
            if (warp == 0 && lane < kW)
                S.disp[lane] = lane < w && tpos >= (unsigned)(c0 + w) ? (int)min(tpos, (unsigned)(n - 1)) : -1;
        } else {
            step += w;
        }
        }
        __syncthreads();
        // ------------------------------------- interchanges, triangular solve
        const int left = c0 - P.j0, right = jend - c0 - w;
        const int ncols = left + right + P.nrhs;
        // four lanes a column (lane f of them holds rows f, f + 4, ...: a
        // single thread's substitution is one long chain), eight columns a
        // warp, to the warps of all CTAs in turn
        const int f = lane & 3;
        for (int qb = (warp * C + rank) * 8; qb < ncols; qb += kCWarps * C * 8) {
            const int q = qb + (lane >> 2);
            const bool ok = q < ncols;
            cd* col = q < left ? A + (int64_t)(P.j0 + q) * lda
                               : (q < left + right ? A + (int64_t)(c0 + w + q - left) * lda
                                                   : B + (int64_t)(q - left - right) * ldb);
            cd t[kW / 4], d[kW / 4];
#pragma unroll
            for (int u = 0; u < kW / 4; ++u) {
                const int i = 4 * u + f;
                t[u] = ok && i < w ? ld2(col + S.src[i]) : cd{0.0, 0.0};
                d[u] = ok && S.disp[i] >= 0 ? ld2(col + c0 + i) : cd{0.0, 0.0};
            }
            __syncwarp();  // the column is read before it is written
#pragma unroll
            for (int u = 0; u < kW / 4; ++u)
                if (ok && S.disp[4 * u + f] >= 0) st2(col + S.disp[4 * u + f], d[u]);
            if (qb + 7 >= left) {
#pragma unroll
                for (int k = 0; k + 1 < kW; ++k) {
                    const cd x{__shfl_sync(0xffffffffu, t[k / 4].re, (lane & ~3) | (k & 3)),
                               __shfl_sync(0xffffffffu, t[k / 4].im, (lane & ~3) | (k & 3))};
#pragma unroll
                    for (int u = k / 4; u < kW / 4; ++u) {
                        const int i = 4 * u + f;
                        if (i > k && i < w && q >= left) t[u] = csub_mul(t[u], S.tri[i][k], x);
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < kW / 4; ++u)
                if (ok && 4 * u + f < w) st2(col + c0 + 4 * u + f, t[u]);
        }
        if (P.rid != nullptr && rank == C - 1 && warp == kCWarps - 1) {
            // the rows' origins move like a column
            const int t = lane < w ? __ldcg(P.rid + S.src[lane]) : 0;
            const int dd = lane < w && S.disp[lane] >= 0 ? __ldcg(P.rid + c0 + lane) : 0;
            __syncwarp();
            if (lane < w) {
                __stcg(P.rid + c0 + lane, t);
                if (S.disp[lane] >= 0) __stcg(P.rid + S.disp[lane], dd);
            }
            __syncwarp();
        }
        __syncwarp();
        cluster_barrier();
        // ---------------------------------------------------- rank-w update
        // A warp takes 16 x 32 entries: 2 x 4 blocks of 8 x 8 for the FP64
        // tensor instruction, in the four-product complex form.  C, L and U
        // come straight from L2 in the instruction's fragment layout -- whole
        // 64- and 128-byte runs -- all loads in flight at once; no staging and
        // no barrier (64 x 32 tiles through shared memory took 4,600 cycles
        // for what 2,050 of products need).
        const int r0 = c0 + w, m2 = n - r0, n2 = right + P.nrhs;
        const int tm = (m2 + kTM - 1) / kTM, tn = (n2 + kTN - 1) / kTN;
        const int gid = lane >> 2, tig = lane & 3;
        for (int task = warp * C + rank; task < tm * tn; task += kCWarps * C) {
            const int i0 = (task % tm) * kTM, q0 = (task / tm) * kTN;
            auto colptr = [&](int q) {
                return q < right ? A + (int64_t)(r0 + q) * lda : B + (int64_t)(q - right) * ldb;
            };
            double cr[2][4][2], ci[2][4][2];
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int q = q0 + 8 * j + 2 * tig + h;
                    const cd* col = colptr(q) + r0 + i0 + gid;
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const cd v = q < n2 && i0 + gid + 8 * i < m2 ? ld2(col + 8 * i) : cd{0.0, 0.0};
                        cr[i][j][h] = v.re;
                        ci[i][j][h] = v.im;
                    }
                }
            cd la[kW / 4][2], ub[kW / 4][4];
#pragma unroll
            for (int k4 = 0; k4 < kW / 4; ++k4) {
                const int k = 4 * k4 + tig;
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    la[k4][i] = k < w && i0 + gid + 8 * i < m2
                                    ? ld2(A + (r0 + i0 + gid + 8 * i) + (int64_t)(c0 + k) * lda)
                                    : cd{0.0, 0.0};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int q = q0 + 8 * j + gid;
                    ub[k4][j] = k < w && q < n2 ? ld2(colptr(q) + c0 + k) : cd{0.0, 0.0};
                }
            }
#pragma unroll
            for (int k4 = 0; k4 < kW / 4; ++k4) {
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        dmma(cr[i][j][0], cr[i][j][1], -la[k4][i].re, ub[k4][j].re);
                        dmma(ci[i][j][0], ci[i][j][1], -la[k4][i].re, ub[k4][j].im);
                    }
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        dmma(cr[i][j][0], cr[i][j][1], la[k4][i].im, ub[k4][j].im);
                        dmma(ci[i][j][0], ci[i][j][1], -la[k4][i].im, ub[k4][j].re);
                    }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int q = q0 + 8 * j + 2 * tig + h;
                    if (q < n2) {
                        cd* col = colptr(q) + r0 + i0 + gid;
#pragma unroll
                        for (int i = 0; i < 2; ++i)
                            if (i0 + gid + 8 * i < m2) st2(col + 8 * i, cd{cr[i][j][h], ci[i][j][h]});
                    }
                }
        }
        __syncwarp();
        cluster_barrier();
    }
    if (P.rid != nullptr) {
        // the block's row order: src[i] the row that ends in position j0 + i,
        // disp[i] where row j0 + i went (-1: it stays within the block)
        int32_t* const src = P.order;
        int32_t* const disp = src + P.jb;
        for (int r = P.j0 + rank * kCT + tid; r < n; r += C * kCT) {
            const int o = __ldcg(P.rid + r);
            if (r < jend) src[r - P.j0] = o;
            if (o < jend) disp[o - P.j0] = r < jend ? -1 : r;
        }
    }
    if (!P.back) return;
    // ------------------------------------------------------ U X = L^-1 P B
    // The right-hand sides are independent: CTA r takes columns r, r + C, ...
    // up to four at a time, in shared memory, and needs no other CTA.  Per
    // block of 16 rows: sixteen lanes a right-hand side substitute (lane i
    // row i), then every thread updates its rows above; triangle, reciprocal
    // diagonal and the rows' U entries are fetched a block ahead.
    const int mine = P.nrhs > rank ? (P.nrhs - rank + C - 1) / C : 0;
    const int at_once = min(4, kBackRows / n);
    for (int q0 = 0; q0 < mine; q0 += at_once) {
        const int nq = min(at_once, mine - q0);
        cd* Bq = B + (int64_t)(rank + q0 * C) * ldb;
        const int64_t bstep = (int64_t)C * ldb;
        cd ft, fd, fu[kW];
        auto fetch = [&](int b0) {
            const int w = min(kW, n - b0), r = tid % kW, k = tid / kW;
            ft = r < k && k < w ? ld2(A + (b0 + r) + (int64_t)(b0 + k) * lda) : cd{0.0, 0.0};
            fd = tid < w ? ld2(A + (b0 + tid) + (int64_t)(b0 + tid) * lda) : cd{1.0, 0.0};
#pragma unroll
            for (int c = 0; c < kW; ++c)
                fu[c] = tid < b0 && c < w ? ld2(A + tid + (int64_t)(b0 + c) * lda) : cd{0.0, 0.0};
        };
        static_assert(kCT == kW * kW, "one triangle entry per thread");
        cd* y = S.y;  // [n][at_once]
        for (int e = tid; e < n * nq; e += kCT) y[(e % n) * at_once + e / n] = ld2(Bq + e % n + (e / n) * bstep);
        const int last = ((n - 1) / kW) * kW;
        fetch(last);
        for (int b0 = last; b0 >= 0; b0 -= kW) {
            const int w = min(kW, n - b0);
            S.tri[tid % kW][tid / kW] = ft;
            if (tid < kW) S.dinv[tid] = crecip(fd);
            cd u[kW];
#pragma unroll
            for (int c = 0; c < kW; ++c) u[c] = fu[c];
            if (b0 > 0) fetch(b0 - kW);
            __syncthreads();
            const int q = tid >> 4, i = tid & 15;
            if (warp < 2) {
                const bool ok = q < nq && i < w;
                cd t = ok ? y[(b0 + i) * at_once + q] : cd{0.0, 0.0};
                const cd di = S.dinv[i];
#pragma unroll
                for (int k = kW - 1; k >= 0; --k) {
                    if (i == k) t = t * di;
                    const cd x{__shfl_sync(0xffffffffu, t.re, (lane & 16) | k),
                               __shfl_sync(0xffffffffu, t.im, (lane & 16) | k)};
                    if (i < k) t = csub_mul(t, S.tri[i][k], x);
                }
                S.X[i][q] = t;
                if (ok) st2(Bq + b0 + i + q * bstep, t);
            }
            __syncthreads();
            for (int r = tid; r < b0; r += kCT) {
                if (r != tid)
#pragma unroll
                    for (int c = 0; c < kW; ++c)
                        u[c] = c < w ? ld2(A + r + (int64_t)(b0 + c) * lda) : cd{0.0, 0.0};
                for (int p = 0; p < nq; ++p) {
                    cd v = y[r * at_once + p], v2{0.0, 0.0};
#pragma unroll
                    for (int c = 0; c < kW; c += 2) {
                        v = csub_mul(v, u[c], S.X[c][p]);
                        v2 = csub_mul(v2, u[c + 1], S.X[c + 1][p]);
                    }
                    y[r * at_once + p] = v + v2;
                }
            }
            __syncthreads();
        }
    }
}

// The exchange's wait on rows that are expected and never sent.
__global__ void __launch_bounds__(32) exchange_wait_selftest_kernel(int32_t* err, int limit) {
    __shared__ __align__(8) unsigned long long mbar;
    const unsigned m = smem_u32(&mbar);
    if (threadIdx.x == 0) {
        mbar_init(m, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    cluster_barrier();
    mbar_expect(threadIdx.x == 0, m, 2 * kXchBytes);
    exchange_wait(m, 0, limit, err);
    __syncwarp();
    cluster_barrier();
}

// ------------------------------------------------------------ block solves
// X <- T^-1 P X for the jb <= 128 rows [j0, j0 + jb) of many columns, T the
// unit lower (or, UPPER, the upper) triangle of the diagonal block and P the
// block's row order (src / disp of the panel; null: the rows stay).  A CTA
// holds 32 columns of X in shared memory and takes the triangle in strips of
// 16 columns, fetched a strip ahead: four warps solve the strip's 16 rows
// (four lanes a column), all warps apply it to the rest.  The columns left of the block
// only take the interchanges: `left` of them from Aleft on, in CTAs of their
// own.  A gather of all rows at once replaces LAPACK's sequential swaps.
constexpr int kSN = 32, kSMax = 128;
constexpr int kSPitch = kSN + 1;
constexpr size_t kSolveSmem = sizeof(cd) * (kSMax * kSPitch + kW * kSMax + kW) + sizeof(int) * 2 * kSMax;

struct SolveArgs {
    const cd* T;  // the diagonal block
    int64_t ldt;
    int j0, jb;
    const int32_t *src, *disp;
    cd* Aleft;
    int64_t ldleft;
    int left;
    cd* X;  // column 0, row 0 of the right columns
    int64_t ldx;
    int ncols;
    cd* B;  // further right columns
    int64_t ldb;
    int nrhs;
};

template <bool UPPER>
__global__ void __launch_bounds__(kCT) zblock_solve_kernel(SolveArgs P) {
    extern __shared__ __align__(16) unsigned char zs_smem[];
    cd* X = reinterpret_cast<cd*>(zs_smem);  // [kSMax][kSPitch]
    cd* Ls = X + kSMax * kSPitch;            // [kW][kSMax]
    cd* dinv = Ls + kW * kSMax;
    int* src = reinterpret_cast<int*>(dinv + kW);
    int* disp = src + kSMax;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int nleft = (P.left + kSN - 1) / kSN;
    const bool isleft = (int)blockIdx.x < nleft;
    const int q0 = ((int)blockIdx.x - (isleft ? 0 : nleft)) * kSN;
    const int total = isleft ? P.left : P.ncols + P.nrhs;
    const int j0 = P.j0, jb = P.jb;
    auto colptr = [&](int q) {
        return isleft ? P.Aleft + (int64_t)q * P.ldleft
                      : (q < P.ncols ? P.X + (int64_t)q * P.ldx : P.B + (int64_t)(q - P.ncols) * P.ldb);
    };
    for (int i = tid; i < jb; i += kCT) {
        src[i] = P.src ? P.src[i] : j0 + i;
        disp[i] = P.src ? P.disp[i] : -1;
    }
    __syncthreads();
    constexpr int U = kSMax * kSN / kCT;
    {
        cd d[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = tid + u * kCT, r = e % kSMax, c = e / kSMax;
            const bool ok = r < jb && q0 + c < total;
            const cd* col = colptr(q0 + c);
            X[r * kSPitch + c] = ok ? ld2(col + src[r]) : cd{0.0, 0.0};
            d[u] = ok && disp[r] >= 0 ? ld2(col + j0 + r) : cd{0.0, 0.0};
        }
        __syncthreads();  // every row read before any is overwritten
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = tid + u * kCT, r = e % kSMax, c = e / kSMax;
            if (r < jb && q0 + c < total && disp[r] >= 0) st2(colptr(q0 + c) + disp[r], d[u]);
        }
    }
    const int nstrip = isleft ? 0 : (jb + kW - 1) / kW;
    // strip s: columns k0 .. k0 + w of the triangle, its rows from k0 down
    // (lower) or down to k0 + w (upper); fetched a strip ahead
    constexpr int F = kW * kSMax / kCT;
    cd fs[F], fd{1.0, 0.0};
    auto fetch = [&](int st) {
        const int k0 = (UPPER ? nstrip - 1 - st : st) * kW, w = min(kW, jb - k0);
        const int f0 = UPPER ? 0 : k0, f1 = UPPER ? k0 + w : jb;
#pragma unroll
        for (int u = 0; u < F; ++u) {
            const int e = tid + u * kCT, r = e % kSMax, k = e / kSMax;
            fs[u] = r >= f0 && r < f1 && k < w ? ld2(P.T + r + (int64_t)(k0 + k) * P.ldt) : cd{0.0, 0.0};
        }
        if (UPPER) fd = tid < w ? ld2(P.T + (k0 + tid) + (int64_t)(k0 + tid) * P.ldt) : cd{1.0, 0.0};
    };
    if (nstrip > 0) fetch(0);
    for (int s = 0; s < nstrip; ++s) {
        const int k0 = (UPPER ? nstrip - 1 - s : s) * kW, w = min(kW, jb - k0);
#pragma unroll
        for (int u = 0; u < F; ++u) {
            const int e = tid + u * kCT;
            Ls[(e / kSMax) * kSMax + e % kSMax] = fs[u];
        }
        if (UPPER && tid < kW) dinv[tid] = crecip(fd);
        __syncthreads();
        if (s + 1 < nstrip) fetch(s + 1);
        if (warp < kSN / 8) {
            // the strip's rows: four lanes a column (lane f of them rows f,
            // f + 4, ...), eight columns a warp
            const int f = lane & 3, c = warp * 8 + (lane >> 2);
            cd t[kW / 4];
#pragma unroll
            for (int u = 0; u < kW / 4; ++u)
                t[u] = 4 * u + f < w ? X[(k0 + 4 * u + f) * kSPitch + c] : cd{0.0, 0.0};
#pragma unroll
            for (int kk = 0; kk < kW; ++kk) {
                const int k = UPPER ? kW - 1 - kk : kk;
                if (UPPER && f == (k & 3)) t[k / 4] = t[k / 4] * dinv[k];
                const cd x{__shfl_sync(0xffffffffu, t[k / 4].re, (lane & ~3) | (k & 3)),
                           __shfl_sync(0xffffffffu, t[k / 4].im, (lane & ~3) | (k & 3))};
#pragma unroll
                for (int u = 0; u < kW / 4; ++u) {
                    const int i = 4 * u + f;
                    if ((UPPER ? i < k : i > k) && i < w) t[u] = csub_mul(t[u], Ls[k * kSMax + k0 + i], x);
                }
            }
#pragma unroll
            for (int u = 0; u < kW / 4; ++u)
                if (4 * u + f < w) X[(k0 + 4 * u + f) * kSPitch + c] = t[u];
        }
        __syncthreads();
        const int g0 = UPPER ? 0 : k0 + w, g1 = UPPER ? k0 : jb;
        if (g0 < g1) {
            cd xk[kW];
#pragma unroll
            for (int k = 0; k < kW; ++k) xk[k] = k < w ? X[(k0 + k) * kSPitch + lane] : cd{0.0, 0.0};
            for (int r = g0 + warp; r < g1; r += kCWarps) {
                cd y = X[r * kSPitch + lane], z{0.0, 0.0};
#pragma unroll
                for (int k = 0; k < kW; k += 2) {  // two chains
                    y = csub_mul(y, Ls[k * kSMax + r], xk[k]);
                    z = csub_mul(z, Ls[(k + 1) * kSMax + r], xk[k + 1]);
                }
                X[r * kSPitch + lane] = y + z;
            }
        }
        __syncthreads();
    }
#pragma unroll 4
    for (int u = 0; u < U; ++u) {
        const int e = tid + u * kCT, r = e % kSMax, c = e / kSMax;
        if (r < jb && q0 + c < total) st2(colptr(q0 + c) + j0 + r, X[r * kSPitch + c]);
    }
}

template <bool UPPER>
mw_status block_solve(const SolveArgs& P, cudaStream_t st) {
    static const cudaError_t attr = cudaFuncSetAttribute(
        zblock_solve_kernel<UPPER>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSolveSmem);
    MW_CHECK_CUDA(attr);
    const int ctas = (P.left + kSN - 1) / kSN + (P.ncols + P.nrhs + kSN - 1) / kSN;
    if (ctas == 0) return MW_OK;
    ProfileScope ps(PC_TRSM, st, 4.0 * (double)P.jb * P.jb * (P.ncols + P.nrhs),
                    32.0 * (double)P.jb * (P.left + P.ncols + P.nrhs));
    zblock_solve_kernel<UPPER><<<(unsigned)ctas, kCT, kSolveSmem, st>>>(P);
    MW_CHECK_CUDA(cudaGetLastError());
    count_launch();
    return MW_OK;
}

// Largest cluster this device can hold of the kernel: 16 CTAs (a
// non-portable size) where it fits, else 8.
template <int RPT>
int max_cluster() {
    static const int v = [] {
        auto kern = zlu_cluster_kernel<RPT>;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Shared)) !=
                cudaSuccess ||
            cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
            cudaGetLastError();
            return 8;
        }
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(kMaxC);
        cfg.blockDim = dim3(kCT);
        cfg.dynamicSmemBytes = sizeof(Shared);
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = kMaxC;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int num = 0;
        if (cudaOccupancyMaxActiveClusters(&num, kern, &cfg) != cudaSuccess) {
            cudaGetLastError();
            return 8;
        }
        return num >= 1 ? kMaxC : 8;
    }();
    return v;
}

template <int RPT>
mw_status launch(const ZluArgs& P, int C, int batch, cudaStream_t st) {
    MW_REQUIRE(C <= max_cluster<RPT>(), "cluster too large");  // (sets the kernel's attributes)
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(batch * C));
    cfg.blockDim = dim3(kCT);
    cfg.dynamicSmemBytes = sizeof(Shared);
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)C;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    ProfileScope ps(PC_PANEL, st, 4.0 * (double)(P.n - P.j0) * P.jb * P.jb * batch,
                    32.0 * (double)(P.n - P.j0) * P.jb * batch);
    MW_CHECK_CUDA(cudaLaunchKernelEx(&cfg, zlu_cluster_kernel<RPT>, P));
    count_launch();
    return MW_OK;
}

}  // namespace

int zlu_cluster_max_rows() { return max_cluster<3>() * kCT * 3; }

int zlu_cluster_ctas(int m, int max_ctas) {
    const int cap = max_ctas > 0 && max_ctas < kMaxC ? max_ctas : kMaxC;
    // CTAs per cluster: one up to a single panel, eight up to 256 rows (the
    // panel is one CTA's, the rest of the work still spreads: 49 us at order
    // 21 against 66 with one CTA, 355 at 200 against 408 with four and 362
    // with sixteen), sixteen beyond (549 against 601 us at 300); the panels have
    // become quicker for all of them since: 43, 306 and 495 us
    const int want = m <= kW ? 1 : (m <= kCT ? 8 : kMaxC);
    int C = 1;
    while (2 * C <= cap && C < want && C < max_cluster<1>()) C *= 2;
    // enough rows per thread for the panel
    while (C < kMaxC && (m + C - 1) / C > 3 * kCT) C *= 2;
    return C;
}

mw_status zlu_cluster(const ZluArgs& P, int batch, cudaStream_t st, int max_ctas) {
    MW_REQUIRE(batch >= 1 && P.jb >= 1 && P.j0 >= 0 && P.j0 + P.jb <= P.n, "bad block");
    MW_REQUIRE(!P.back || (P.j0 == 0 && P.jb == P.n && P.n <= kBackRows), "back substitution needs the whole matrix");
    const int m = P.n - P.j0, C = zlu_cluster_ctas(m, max_ctas);
    const int per = (m + C - 1) / C;
    if (per <= kCT) return launch<1>(P, C, batch, st);
    if (per <= 2 * kCT) return launch<2>(P, C, batch, st);
    MW_REQUIRE(per <= 3 * kCT, "block of %d rows too large for one cluster", m);
    return launch<3>(P, C, batch, st);
}

mw_status zlu_exchange_wait_selftest(int32_t* err, int limit, cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2);
    cfg.blockDim = dim3(32);
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 2;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    MW_CHECK_CUDA(cudaLaunchKernelEx(&cfg, exchange_wait_selftest_kernel, err, limit));
    return MW_OK;
}

// ------------------------------------------------------------------ driver
// Blocked factorisation of the whole matrix with nrhs carried columns (B <-
// L^-1 P B).  `rid`: n + 4 kZluBlock ints of workspace.  A look-ahead of one
// block on two streams: the critical one (highest priority) updates the next
// block's columns and factors them while the other applies the block to the
// rest of the matrix.  Panel j waits for that stream's step j - 2 only.  The
// rest's product is one block per tile, so that SMs free up in between and
// the next panel's cluster finds its sixteen together.  Measured on B200,
// factorisation and solve with 64 right-hand sides, one stream against two:
// 11.2 -> 9.5 ms at order 2,624, 32.9 -> 25.2 at 5,000, 162 -> 133 at 10,496 (8.2, 20.8 and 121 since, with
// quicker updates and block solves).
mw_status zlu_blocked(int64_t n, cd* A, int64_t lda, int32_t* ipiv, int32_t* info, cd* B, int64_t ldb, int64_t nrhs,
                      int32_t* rid, const volatile int32_t* cancel, cudaStream_t caller) {
    const int nb = kZluBlock;
    ZluStreams zs;
    if (mw_status s = zlu_streams(&zs); s != MW_OK) return s;
    const cudaStream_t st = zs.critical, tr = zs.trail;
    MW_CHECK_CUDA(cudaEventRecord(zs.ev_handover, caller));
    MW_CHECK_CUDA(cudaStreamWaitEvent(st, zs.ev_handover, 0));
    MW_CHECK_CUDA(cudaStreamWaitEvent(tr, zs.ev_handover, 0));
    Pace<4> pace;  // (the whole factorisation is enqueued in about two milliseconds)
    if (cancel) {
        mw_status s = pace.start(st);
        if (s != MW_OK) return s;
    }
    const cd m1{-1.0, 0.0}, p1{1.0, 0.0};
    for (int64_t j = 0, j0 = 0; j0 < n; ++j, j0 += nb) {
        if (cancel) {
            mw_status s = pace.step(j, st);
            if (s != MW_OK) return s;
        }
        if (cancel && *cancel) {
            // let both streams finish what they were given
            MW_CHECK_CUDA(cudaStreamSynchronize(tr));
            MW_CHECK_CUDA(cudaStreamSynchronize(st));
            set_error("factorisation cancelled");
            return MW_ERR_CANCELLED;
        }
        const int jb = (int)(n - j0 < nb ? n - j0 : nb);
        const int64_t c1 = j0 + jb, cn = n - c1 < nb ? n - c1 : nb, c2 = c1 + cn;
        ZluArgs P{};
        P.A = A;
        P.lda = lda;
        P.n = (int)n;
        P.j0 = (int)j0;
        P.jb = jb;
        P.ipiv = ipiv;
        P.info = info;
        P.rid = rid;
        P.order = rid + n + (j & 1) * 2 * kZluBlock;  // (the other stream may still read the last block's)
        mw_status s = zlu_cluster(P, 1, st);
        if (s != MW_OK) return s;
        SolveArgs Q{};
        Q.T = A + j0 + j0 * lda;
        Q.ldt = lda;
        Q.j0 = (int)j0;
        Q.jb = jb;
        Q.src = P.order;
        Q.disp = P.order + jb;
        MW_CHECK_CUDA(cudaEventRecord(zs.ev_main, st));
        MW_CHECK_CUDA(cudaStreamWaitEvent(tr, zs.ev_main, 0));
        if (cn > 0) {  // the next block's columns
            if (j > 0) MW_CHECK_CUDA(cudaStreamWaitEvent(st, zs.ev_trail[(j - 1) & 1], 0));
            SolveArgs N = Q;
            N.X = A + c1 * lda;
            N.ldx = lda;
            N.ncols = (int)cn;
            s = block_solve<false>(N, st);
            if (s == MW_OK)
                s = zgemm_launch(false, false, n - c1, cn, jb, m1, A + c1 + j0 * lda, lda, A + j0 + c1 * lda, lda, p1,
                                 A + c1 + c1 * lda, lda, st, 0, nullptr, 0);
            if (s != MW_OK) return s;
        }
        // everything else: the columns left of the block take its row order,
        // those right of the next block and the right-hand sides the rest too
        Q.Aleft = A;
        Q.ldleft = lda;
        Q.left = (int)j0;
        Q.X = A + c2 * lda;
        Q.ldx = lda;
        Q.ncols = (int)(n - c2);
        Q.B = B;
        Q.ldb = ldb;
        Q.nrhs = (int)nrhs;
        s = block_solve<false>(Q, tr);
        if (s == MW_OK && n - c2 > 0)
            s = zgemm_launch(false, false, n - c1, n - c2, jb, m1, A + c1 + j0 * lda, lda, A + j0 + c2 * lda, lda, p1,
                             A + c1 + c2 * lda, lda, tr, kCtaPerTile, nullptr, 0);
        if (s == MW_OK && nrhs > 0 && n - c1 > 0)
            s = zgemm_launch(false, false, n - c1, nrhs, jb, m1, A + c1 + j0 * lda, lda, B + j0, ldb, p1, B + c1, ldb,
                             tr, kCtaPerTile, nullptr, 0);
        if (s != MW_OK) return s;
        MW_CHECK_CUDA(cudaEventRecord(zs.ev_trail[j & 1], tr));
    }
    MW_CHECK_CUDA(cudaEventRecord(zs.ev_handover, st));
    MW_CHECK_CUDA(cudaStreamWaitEvent(caller, zs.ev_handover, 0));
    MW_CHECK_CUDA(cudaEventRecord(zs.ev_main, tr));
    MW_CHECK_CUDA(cudaStreamWaitEvent(caller, zs.ev_main, 0));
    return MW_OK;
}

// B <- U^-1 B, 128 rows at a time.
mw_status zlu_upper(int64_t n, const cd* LU, int64_t lda, cd* B, int64_t ldb, int64_t nrhs, cudaStream_t st) {
    for (int64_t j0 = (n - 1) / kSMax * kSMax; j0 >= 0; j0 -= kSMax) {
        SolveArgs Q{};
        Q.T = LU + j0 + j0 * lda;
        Q.ldt = lda;
        Q.j0 = (int)j0;
        Q.jb = (int)(n - j0 < kSMax ? n - j0 : kSMax);
        Q.X = B;
        Q.ldx = ldb;
        Q.ncols = (int)nrhs;
        mw_status s = block_solve<true>(Q, st);
        if (s == MW_OK && j0 > 0)
            s = zgemm_launch(false, false, j0, nrhs, Q.jb, cd{-1.0, 0.0}, LU + j0 * lda, lda, B + j0, ldb,
                             cd{1.0, 0.0}, B, ldb, st, 0, nullptr, 0);
        if (s != MW_OK) return s;
    }
    return MW_OK;
}

}  // namespace mw
