// Flooding normalized min-sum for batches that leave SMs idle: one codeword on
// a cluster of CTAs (sm_103a).
//
// decode_kernel walks a codeword's base rows in order on one SM, which is the
// better use of a full GPU but leaves most of it idle on a small batch.  Here
// the two halves of a flooding iteration are separate passes, each spread
// over every warp of the cluster:
//   * check-node pass: the CTA that owns a base row runs it for all Z
//     sub-rows from its own copy of the posteriors, keeps the row's 16-byte
//     state in shared memory and sends dt = R_new - R_old of each core edge to
//     the CTA that owns the edge's column (distributed shared memory);
//   * variable-node pass: the owner of a column adds its dt in ascending
//     base-row order and sends the sums to the CTAs whose rows read them.
// A suffix column has a single edge: its posterior stays in the row's state.
// The sums are those of decode_kernel term by term (L + dt_r0 + dt_r1 + ...,
// explicit round-to-nearest), so results are bit-identical to it.
//
// Everything is sent, nothing fetched: distributed shared memory moves about
// 17 B per clock and SM whichever way it is accessed (24 KB in 1,450 clocks of
// loads or stores, scalar or 128-bit; bulk copies slower), and a store of the
// check-node pass costs its warp no wait.  Fetching dt from the rows' owners
// instead took 5,700 of 12,300 clocks per iteration on 16 CTAs (BG1 Z=384).
//
// Early stop costs no pass of its own: the check-node pass of iteration t + 1
// reads every posterior of iteration t, so it collects the row parities of
// their hard decisions; when every row of the cluster is satisfied the
// codeword leaves with iteration t's posteriors, which the passes so far have
// not touched (the suffix hard decisions are kept in the state word).
//
// Shared memory per CTA: all core posteriors, the states of its rows and the
// dt of its columns.  When the dt do not fit, the rows run in phases
// (contiguous row ranges, both passes per phase) with the partial sums kept
// by their owners; the chain of adds is the same.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "nrldpc_internal.h"

namespace nrldpc {
namespace {

constexpr int kSplitThreads = kSplitMaxWarps * 32;
// How a pass hands over to the next: kOne, a cluster of one CTA (small codes):
// CTA barriers.  kCounted (one phase, no early stop): every CTA knows how many
// bytes of dt, and of posteriors, will reach it, the stores count them on its
// mbarriers, and it goes on when they are there.  kBarriers: cluster barriers,
// which early stop needs for its failures (sent and counted beside the dt they
// made BG2 Z=40 16 codewords 7% slower, 20.7 -> 22.2 us).  A cluster barrier
// takes 400-650 clocks of which 300-500 are the fence, more with stores on the
// way; counting instead, 10 iterations: BG1 Z=384 49.4 -> 42.4 us on 16 CTAs,
// 57.6 -> 52.3 on 10, 100.6 -> 95.7 on 4, BG2 Z=208 60 codewords 74.1 -> 65.6.
// No count can run into the next phase's: a CTA sends a column's dt only after
// it has that column's posteriors, which the owner sends after its dt are
// complete, and those include dt that their readers sent after the posteriors
// before were complete; a thread opens each phase after all have seen the last.
// The waits are bounded (kSplitWaitLimit polls): where one runs out the
// cluster reports it, and leaves without writing its codeword or taking
// another.
enum Mode { kOne, kCounted, kBarriers };

constexpr uint32_t kHdBit = 0x80000000u;  // state info: hard decision of the suffix posterior read

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ float lds(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts(uint32_t a, float v) {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
// Address of this CTA's shared address `a` in the CTA of rank `rank`.
__device__ __forceinline__ uint32_t mapa(uint32_t a, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ uint32_t ldc_u32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void stc(uint32_t a, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void stc_u32(uint32_t a, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
// This thread's asynchronous copy of 16 bytes from global to shared memory.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {  // this thread's copies have landed
    asm volatile("cp.async.wait_all;" ::: "memory");
}
__device__ __forceinline__ void stc_v4(uint32_t a, float4 v) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}
// Remote store that counts its bytes on an mbarrier of the CTA it writes to.
__device__ __forceinline__ void st_async(uint32_t a, uint32_t v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(a), "r"(v), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void mbar_init(uint32_t bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
// Opens a phase that ends when `bytes` have arrived.
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_poll(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait for the phase of this parity; false when the limit ran out.
// (The first poll stands outside the loop: 1.3 us less in 10 iterations of one
// BG1 Z=384 codeword than all of them inside.)
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int limit) {
    if (mbar_poll(bar, parity)) return true;
    for (int i = 1; i < limit; i++)
        if (mbar_poll(bar, parity)) return true;
    return false;
}
// Barrier over every thread of the cluster; shared-memory writes before it
// (local and remote) are seen after it.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

__device__ __forceinline__ float min3(float a, float b, float c) {  // NaN operands ignored
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// One lifted row: the arithmetic of decode.cu's row_update (flooding), with
// dt of each core edge sent to its column's owner instead of added here.
//   edge: the row's first {column, 4V, distance from a posterior to its edge's
//   dt at the owner}; l: shared address of the posteriors; s4: 4*s; st: the
//   row's state, st_out: where it goes; par: hard-decision parity of the
//   posteriors read (bit 0).
// Rows of up to kSplitKeep edges keep Q and the dt addresses in registers (the
// argmin is then found in the second half and the minima are taken in pairs,
// as in row_update); longer rows track the argmin and form the address again.
template <int D, bool WEIGHTED, int MODE>
__device__ __forceinline__ void cn_row(const uint4* edge, bool sfx, uint32_t s4, uint32_t l, uint32_t z4, uint4 st,
                                       uint4* st_out, const float* wprev, const float* wcur, float alpha, bool check,
                                       uint32_t& par) {
    constexpr int LAST = D - 1;
    constexpr bool kKeep = D <= kSplitKeep;
    uint32_t to[D];
    float lv[D];
#pragma unroll
    for (int i = 0; i < D; i++) {
        if (i == LAST && sfx) {
            to[i] = 0;
            lv[i] = __uint_as_float(st.w);
        } else {
            const uint4 ea = edge[i];
            const uint32_t t = s4 + ea.y, a = __viaddmin_u32(t, 0u - z4, t) + ea.x + l;
            lv[i] = lds(a);
            if (kKeep) to[i] = a + ea.z;
        }
    }
    if (check) {
#pragma unroll
        for (int i = 0; i < D; i++) par ^= lv[i] > 0.0f ? 0u : 1u;
    }
    const float om1 = __uint_as_float(st.x), om2 = __uint_as_float(st.y);
    const uint32_t oinfo = st.z;
    const int oidx = static_cast<int>(oinfo & 31u);
    float oa1 = 0.0f, oa2 = 0.0f;
    if (!WEIGHTED) {
        oa1 = __fmul_rn(alpha, om1);
        oa2 = __fmul_rn(alpha, om2);
    }
    float keep[D], qk[D];
    float m1 = 1000.0f, m2 = 1000.0f, first = 0.0f;
    int idx = 0;
    uint32_t qmask = 0;
#pragma unroll
    for (int i = 0; i < D; i++) {
        float mag;
        if (WEIGHTED)
            mag = __fmul_rn(wprev[i], i == oidx ? om2 : om1);
        else
            mag = i == oidx ? oa2 : oa1;
        const float ro = __uint_as_float(__float_as_uint(mag) ^ ((oinfo << (24 - D + i)) & 0x80000000u));
        const float q = __fsub_rn(lv[i], ro);
        keep[i] = ro;
        if (kKeep) qk[i] = q;
        const float qa = fabsf(q);
        qmask = __funnelshift_l(__float_as_uint(__fadd_rn(q, 0.0f)), qmask, 1);  // edge i at bit D-1-i, -0 as +0
        if (i == 0) {
            m1 = fminf(m1, qa);
        } else if (kKeep && (i & 1) && i + 1 < D) {
            first = qa;  // of a pair
        } else if (kKeep && !(i & 1)) {
            const float lo = fminf(first, qa), hi = max_nan(first, qa);
            m2 = min3(m2, hi, max_nan(m1, lo));
            m1 = fminf(m1, lo);
        } else {
            if (!kKeep && qa < m1) idx = i;
            const float mx = max_nan(m1, qa);  // NaN |Q| leaves min1/min2 untouched
            m1 = fminf(m1, qa);
            m2 = fminf(m2, mx);
        }
    }
    const uint32_t rsign = qmask ^ (0u - static_cast<uint32_t>(__popc(qmask) & 1));
    float a1 = 0.0f, a2 = 0.0f;
    if (!WEIGHTED) {
        a1 = __fmul_rn(alpha, m1);
        a2 = __fmul_rn(alpha, m2);
    }
    float sfx_new = 0.0f;
#pragma unroll
    for (int i = 0; i < D; i++) {
        const bool at_min = kKeep ? fabsf(qk[i]) == m1 : i == idx;
        if (kKeep && at_min) idx = i;
        float mag;
        if (WEIGHTED)
            mag = __fmul_rn(wcur[i], at_min ? m2 : m1);
        else
            mag = at_min ? a2 : a1;
        const float rn = __uint_as_float(__float_as_uint(mag) ^ ((rsign << (32 - D + i)) & 0x80000000u));
        const float d = __fsub_rn(rn, keep[i]);
        if (i == LAST && sfx) {
            sfx_new = __fadd_rn(__uint_as_float(st.w), d);
        } else {
            uint32_t a = to[i];
            if (!kKeep) {
                const uint4 ea = edge[i];
                const uint32_t t = s4 + ea.y;
                a = __viaddmin_u32(t, 0u - z4, t) + ea.x + l + ea.z;
            }
            if (MODE == kOne)
                sts(a, d);
            else if (MODE == kCounted)
                st_async(a, __float_as_uint(d), edge[i].w);
            else
                stc(a, d);
        }
    }
    uint32_t info = static_cast<uint32_t>(idx) | ((rsign & ((1u << D) - 1u)) << 8);
    if (!(__uint_as_float(st.w) > 0.0f)) info |= kHdBit;
    *st_out = make_uint4(__float_as_uint(m1), __float_as_uint(m2), info, __float_as_uint(sfx_new));
}

// Position of a suffix row's last column at sub-row s (rw.z: first position
// of the column << 9 | shift).
__device__ __forceinline__ int sfx_pos(const uint4& rw, uint32_t s, int z) {
    int p = static_cast<int>(s + (rw.z & 511u));
    if (p >= z) p -= z;
    return static_cast<int>(rw.z >> 9) + p;
}

template <bool W>
struct SplitWeights {
    using type = NoWeights;
};
template <>
struct SplitWeights<true> {
    using type = WeightTable;
};

// Bound by SM issue in the check-node pass and, on large clusters, by the
// distributed-shared-memory stores and the hand-overs; 24 warps per CTA hide
// more of it than 16, and the 80 registers that leaves hold a degree-19 row.
template <bool WEIGHTED, int MODE>
__global__ void __launch_bounds__(kSplitThreads, 1)
    split_decode_kernel(const __grid_constant__ SplitArgs a, const __grid_constant__ typename SplitWeights<WEIGHTED>::type wt) {
    constexpr bool ONE = MODE == kOne;
    extern __shared__ __align__(128) unsigned char smem[];
    const int rank = ONE ? 0 : static_cast<int>(cluster_rank()), C = ONE ? 1 : static_cast<int>(cluster_size());
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = blockDim.x, W = nt >> 5;
    auto sync = [] {
        if (ONE)
            __syncthreads();
        else
            cluster_sync();
    };
    const uint32_t bar_dt = smem_u32(smem), bar_l = bar_dt + 8;  // mbarriers of the dt and the posteriors
    // [2] an unsatisfied row, by iteration parity; [2] a wait of some thread of the cluster ran out
    uint32_t* s_fail = reinterpret_cast<uint32_t*>(smem + 16);
    uint32_t ph_dt = 0, ph_l = 0;                                // parities waited for next
    if (MODE == kCounted && tid == 0) {
        mbar_init(bar_dt);
        mbar_init(bar_l);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // Warps with task lists (a mixed batch's CTA may have more); 0 in a thread
    // of which a wait ran out: it waits and sends no more, and thread 0 opens no
    // further phase (an arrival on one that has not ended is undefined).  What
    // others still send to the CTA is counted on the open phases, two passes'
    // bytes at most: then they lack what it owes them.
    int lists = 1;
    auto wait = [&](uint32_t bar, uint32_t& parity) {
        if (lists && !mbar_wait(bar, parity, a.wait_limit)) lists = 0;
        parity ^= 1u;
        __syncthreads();  // all threads have seen it before the next phase opens
    };
    // the plan's head and this rank's tables; read where they are used, so
    // that the row bodies have the registers
    SplitHead* s_head = reinterpret_cast<SplitHead*>(smem + 32);
    const volatile SplitHead& h = *s_head;
    unsigned char* image = smem + kSplitHeader;
    if (tid < 3) s_fail[tid] = 0;
    const unsigned char* loaded = nullptr;
    for (int item = blockIdx.x / C; item < a.n_cw; item += gridDim.x / C) {
        const unsigned char* plan = a.plan;
        int cw = item;
        const float* llr = a.llr;
        uint8_t* packed = a.packed;
        if (a.jobs) {
            const SplitJob j = a.jobs[item];
            plan += j.plan;
            cw = j.job;
            llr += j.llr_offset;
            packed += j.out_offset;
        }
        if (plan != loaded) {  // head and this rank's tables
            if (a.jobs) {
                if (tid < static_cast<int>(sizeof(SplitHead) / 4))
                    reinterpret_cast<int*>(s_head)[tid] = reinterpret_cast<const int*>(plan)[tid];
            } else if (tid == 0) {
                *s_head = a.head;
            }
            __syncthreads();
            const unsigned char* src = plan + sizeof(SplitHead) + static_cast<size_t>(rank) * h.image_bytes;
            for (int k = tid; k < h.image_bytes / 16; k += nt) cp_async16(smem_u32(image) + 16u * k, src + 16 * k);
        }
        const int z = h.z, P = h.phases;
        lists = h.warps;
        const uint32_t z4 = 4u * static_cast<uint32_t>(z);
        if (!a.jobs) {
            llr += static_cast<size_t>(cw) * h.n_bp;
            packed += static_cast<size_t>(cw) * h.packed_bytes;
        }
        const uint32_t l_addr = smem_u32(smem) + h.off_l, dt_addr = smem_u32(smem) + h.off_dt;
        float* app = a.app ? a.app + static_cast<size_t>(cw) * h.n_bp : nullptr;
        // core LLRs: the whole copy by each CTA, or (host memory) its share, sent to all
        if (ONE || !a.llr_from_host) {
            for (int m = tid; m < h.core_floats / 4; m += nt) cp_async16(l_addr + 16u * m, llr + 4 * m);
        } else {
            const int total = h.core_floats / 4, per = (total + C - 1) / C;
            sync();  // every CTA runs
            for (int m = rank * per + tid; m < min(total, (rank + 1) * per); m += nt) {
                const float4 v = __ldcs(reinterpret_cast<const float4*>(llr) + m);
                for (int q = 0; q < C; q++) stc_v4(mapa(l_addr + 16u * m, q), v);
            }
        }
        cp_async_wait_all();
        if (plan != loaded) {  // dt place at the owner -> distance from the posterior to it
            __syncthreads();
            uint4* edge = reinterpret_cast<uint4*>(image + h.o_edge);
            for (int k = tid; k < h.n_edges; k += nt) {
                const uint32_t to = edge[k].z, base = ONE ? dt_addr : mapa(dt_addr, to >> 24);
                edge[k].z = base + (to & 0xffffffu) * z4 - (l_addr + edge[k].x);
                if (MODE == kCounted) edge[k].w = mapa(bar_dt, to >> 24);
            }
            loaded = plan;
        }
        sync();
        int it = a.n_iter;
        bool conv = false;
        for (int t = 0; t < a.n_iter && !conv; t++) {
            const bool check = MODE != kCounted && a.early_stop && t > 0;
            const float* wprev = nullptr;
            const float* wcur = nullptr;
            if constexpr (WEIGHTED) {
                wprev = wt.w[t == 0 ? kMaxWIters : min(t - 1, a.n_w_iters - 1)];
                wcur = wt.w[min(t, a.n_w_iters - 1)];
            }
            if (MODE == kCounted) {
                if (t > 0) wait(bar_l, ph_l);  // the posteriors of the last iteration
                if (tid == 0 && lists)
                    mbar_expect(bar_dt, reinterpret_cast<const uint32_t*>(image + h.o_bytes)[0]);
            }
            for (int p = 0; p < (MODE == kCounted ? 1 : P); p++) {
                const uint16_t* cnptr = reinterpret_cast<const uint16_t*>(image + h.o_cnptr) + p * lists + warp;
                const uint16_t* cn = reinterpret_cast<const uint16_t*>(image + h.o_cn);
                uint4* states = reinterpret_cast<uint4*>(smem + h.off_state);
                const int k1 = warp < lists ? cnptr[1] : 0;
                for (int k = warp < lists ? cnptr[0] : 0; k < k1; k++) {
                    const int task = cn[k];
                    const uint32_t s = static_cast<uint32_t>((task & 15) * 32 + lane);
                    const uint4 rw = reinterpret_cast<const uint4*>(image + h.o_row)[task >> 4];
                    uint32_t bad = 0;
                    if (s < static_cast<uint32_t>(z)) {
                        const bool sfx = (rw.w >> 8) != 0;
                        uint4* state = states + rw.y + s;
                        // first iteration: zero state (R_old = +0), the suffix LLR
                        uint4 st = make_uint4(0u, 0u, 0u, 0u);
                        if (t > 0)
                            st = *state;
                        else if (sfx)
                            st.w = __float_as_uint(__ldcs(llr + sfx_pos(rw, s, z)));
                        const uint4* edge = reinterpret_cast<const uint4*>(image + h.o_edge) + (rw.x & 0xffffu);
                        const uint32_t we = WEIGHTED ? rw.x >> 16 : 0u;
                        switch (rw.w & 255u) {
#define NRLDPC_CN_CASE(D)                                                                                             \
    case D:                                                                                                           \
        cn_row<D, WEIGHTED, MODE>(edge, sfx, 4u * s, l_addr, z4, st, state, WEIGHTED ? wprev + we : nullptr,           \
                                 WEIGHTED ? wcur + we : nullptr, a.alpha, check, bad);                                \
        break;
                            NRLDPC_CN_CASE(1) NRLDPC_CN_CASE(2) NRLDPC_CN_CASE(3) NRLDPC_CN_CASE(4)
                            NRLDPC_CN_CASE(5) NRLDPC_CN_CASE(6) NRLDPC_CN_CASE(7) NRLDPC_CN_CASE(8)
                            NRLDPC_CN_CASE(9) NRLDPC_CN_CASE(10) NRLDPC_CN_CASE(11) NRLDPC_CN_CASE(12)
                            NRLDPC_CN_CASE(13) NRLDPC_CN_CASE(14) NRLDPC_CN_CASE(15) NRLDPC_CN_CASE(16)
                            NRLDPC_CN_CASE(17) NRLDPC_CN_CASE(18) NRLDPC_CN_CASE(19)
#undef NRLDPC_CN_CASE
                            default:
                                break;
                        }
                        // the posterior the codeword leaves with if it stops here
                        if (check && app && sfx) app[sfx_pos(rw, s, z)] = __uint_as_float(st.w);
                    }
                    if (check && __any_sync(0xffffffffu, bad & 1u) && lane < C) {
                        const uint32_t f = smem_u32(&s_fail[t & 1]);
                        if (ONE)
                            s_fail[t & 1] = 1u;
                        else
                            stc_u32(mapa(f, lane), 1u);
                    }
                }
                // the dt of this phase, and (last phase) the failures, are in place
                if (MODE == kCounted) {
                    wait(bar_dt, ph_dt);
                } else {
                    sync();
                }
                if (check && p == P - 1 && s_fail[t & 1] == 0) {
                    conv = true;  // iteration t - 1 left a codeword: t iterations ran
                    it = t;
                    break;
                }
                if (MODE == kCounted && tid == 0 && lists)
                    mbar_expect(bar_l, reinterpret_cast<const uint32_t*>(image + h.o_bytes)[1]);
                const uint16_t* vnptr = reinterpret_cast<const uint16_t*>(image + h.o_vnptr) + warp;
                const uint16_t* vn = reinterpret_cast<const uint16_t*>(image + h.o_vn);
                const int v1 = warp < lists ? vnptr[1] : 0;
                for (int k = warp < lists ? vnptr[0] : 0; k < v1; k++) {
                    const int task = vn[k];
                    const uint32_t pos = static_cast<uint32_t>((task & 15) * 32 + lane);
                    const uint4 cm = reinterpret_cast<const uint4*>(image + h.o_col)[task >> 4];  // L offset, readers
                    const uint32_t be = reinterpret_cast<const uint32_t*>(image + h.o_beg)[(task >> 4) * P + p];
                    if (pos >= static_cast<uint32_t>(z)) continue;
                    const uint32_t la = l_addr + cm.x + 4u * pos;
                    uint32_t d = dt_addr + (be & 0xffffu) * z4 + 4u * pos;
                    float* acc = reinterpret_cast<float*>(smem + h.off_acc) + k * 32 + lane;
                    float v = p == 0 ? lds(la) : *acc;
                    for (int m = static_cast<int>(be >> 16); m > 0; m -= kSplitVnAhead) {
                        float x[kSplitVnAhead];
#pragma unroll
                        for (int i = 0; i < kSplitVnAhead; i++) {
                            if (i < m) x[i] = lds(d);
                            d += z4;
                        }
#pragma unroll
                        for (int i = 0; i < kSplitVnAhead; i++)
                            if (i < m) v = __fadd_rn(v, x[i]);
                    }
                    if (MODE == kCounted) {
                        for (uint32_t m = cm.y; m; m &= m - 1) {
                            const uint32_t q = __ffs(m) - 1;
                            st_async(mapa(la, q), __float_as_uint(v), mapa(bar_l, q));
                        }
                    } else if (p < P - 1) {
                        *acc = v;
                    } else if (ONE) {
                        sts(la, v);
                    } else {
                        for (uint32_t m = cm.y; m; m &= m - 1) stc(mapa(la, __ffs(m) - 1), v);
                    }
                }
                if (MODE != kCounted) sync();  // posteriors (last phase) or dt buffers free for the next pass
                if (tid == 0 && p == P - 1) s_fail[t & 1] = 0;  // written again two iterations on
            }
        }
        if (MODE == kCounted) {
            wait(bar_l, ph_l);
            if (!lists)
                for (int q = 0; q < C; q++) stc_u32(mapa(smem_u32(&s_fail[2]), q), 1u);
            sync();  // every CTA's posteriors and states are final, and none sends any more
            if (s_fail[2]) {
                // what was sent to a CTA whose wait ran out may be under way: as
                // many polls again before any leaves
                if (!lists) {
                    atomicExch(a.error_flag, kErrSplitTimeout);
                    for (int i = 0; i < a.wait_limit; i++) {
                        mbar_poll(bar_dt, 0);
                        mbar_poll(bar_l, 0);
                    }
                }
                sync();
                return;
            }
        }
        // Packed hard decisions (and posteriors): 32 positions per warp.
        const int n = h.n_bp, packed_bytes = h.packed_bytes, nc = h.n_core;
        const uint32_t* owners = reinterpret_cast<const uint32_t*>(image + h.o_own);
        const bool word_store = (reinterpret_cast<uintptr_t>(packed) & 3u) == 0;
        for (int w = rank * W + warp; w * 32 < n; w += C * W) {
            const int pos = w * 32 + lane;
            uint32_t one = 0;
            if (pos < n) {
                const int c = pos / z;
                const uint32_t own = owners[c];  // rank << 28 | state offset or 0 | shift
                uint32_t sa = l_addr + 4u * pos, word = 0;
                if (c >= nc) {
                    int s = pos - c * z - static_cast<int>(own & 511u);
                    if (s < 0) s += z;
                    sa = smem_u32(smem) + h.off_state + 16u * (((own >> 9) & 0x7ffffu) + s) + (conv ? 8u : 12u);
                }
                word = ONE ? __float_as_uint(lds(sa)) : ldc_u32(mapa(sa, own >> 28));
                if (c >= nc && conv) {
                    one = word >> 31;
                } else {
                    one = __uint_as_float(word) > 0.0f ? 0u : 1u;
                    if (app) app[pos] = __uint_as_float(word);
                }
            }
            const uint32_t word = __ballot_sync(0xffffffffu, one);
            const int b = 4 * w;
            if (word_store && b + 4 <= packed_bytes) {
                if (lane == 0) *reinterpret_cast<uint32_t*>(packed + b) = word;
            } else if (lane < 4 && b + lane < packed_bytes) {
                packed[b + lane] = static_cast<uint8_t>(word >> (8 * lane));
            }
        }
        if (a.iters && rank == 0 && tid == 0) a.iters[cw] = it;
        sync();  // no CTA reuses its shared memory, or leaves, while another reads it
    }
}

// Task lists of n_bins warps: items in the order given (largest cost first),
// each `chunks` tasks of its cost, every task to the least loaded warp (the
// first of several).  ptr[0..n_bins] and the tasks (item << 4 | chunk) bin by
// bin, from out[from] on; returns the end.
int spread(const uint8_t* items, const int* cost, int n, int chunks, int n_bins, int from, uint16_t* ptr,
           uint16_t* out) {
    constexpr int kLoads = 2048;  // above any load: an even share and one task (asserted below)
    uint32_t at_load[kLoads] = {0};  // the warps that have this load
    int count[kSplitMaxWarps + 1] = {0}, least = 0;
    uint8_t bin[kMaxCols * 12];
    at_load[0] = (1u << n_bins) - 1u;
    for (int i = 0, task = 0; i < n; i++)
        for (int c = 0; c < chunks; c++, task++) {
            while (!at_load[least]) least++;
            const int b = __builtin_ctz(at_load[least]);
            at_load[least] &= at_load[least] - 1;
            at_load[least + cost[i]] |= 1u << b;
            bin[task] = static_cast<uint8_t>(b);
            count[b + 1]++;
        }
    static_assert(kMaxCols * 12 * (kMaxRows + kSplitColCost) / kSplitMaxWarps + kMaxRows + kSplitColCost < kLoads,
                  "the columns' tasks; the rows' are fewer and cost less");
    for (int b = 0; b < n_bins; b++) {
        count[b + 1] += count[b];
        ptr[b] = static_cast<uint16_t>(from + count[b]);
    }
    ptr[n_bins] = static_cast<uint16_t>(from + count[n_bins]);
    for (int i = 0, task = 0; i < n; i++)
        for (int c = 0; c < chunks; c++, task++)
            out[from + count[bin[task]]++] = static_cast<uint16_t>(items[i] << 4 | c);
    return from + n * chunks;
}
static_assert(kSplitMaxWarps < 32 && kMaxRows <= kMaxCols && kMaxDeg + kSplitRowCost <= kMaxRows + kSplitColCost,
              "a bit per warp; rows' tasks within the bounds of columns'");

}  // namespace

// Rows and columns to CTAs and the shared-memory layout, first half of a plan:
// enough to compare cluster sizes by.  False when the code does not fit
// clusters of `ranks` CTAs.
bool deal_split(const CodeTable& t, int ranks, size_t smem_limit, SplitDeal* deal) {
    SplitDeal& d = *deal;
    const int chunks = (t.z + 31) / 32, rows = t.rows, nc = t.n_core;
    auto share = [ranks](int n) { return static_cast<size_t>((n + ranks - 1) / ranks); };
    // the posteriors and an even share of the states have to fit whatever the phases
    const size_t least = kSplitHeader + 4 * static_cast<size_t>(t.core_floats) + 16 * share(rows) * t.z;
    if (least > smem_limit) return false;
    int core[kMaxRows], total = 0, row_order[kMaxRows];
    uint8_t col_order[kMaxCols];
    std::memset(d.col_deg, 0, sizeof(d.col_deg));
    for (int r = 0; r < rows; r++) {  // rows and edges of each column, ascending
        core[r] = t.row_deg[r] - (t.row_sfx[r] ? 1 : 0);
        total += core[r];
        row_order[r] = r;
        for (int e = t.row_ptr[r]; e < t.row_ptr[r + 1]; e++) {
            const int c = t.edge_col[e];
            d.col_row[c][d.col_deg[c]] = static_cast<uint8_t>(r);
            d.col_edge[c][d.col_deg[c]++] = static_cast<uint16_t>(e);
        }
    }
    for (int c = 0; c < nc; c++) col_order[c] = static_cast<uint8_t>(c);
    std::stable_sort(col_order, col_order + nc, [&](int x, int y) { return d.col_deg[x] > d.col_deg[y]; });
    std::stable_sort(row_order, row_order + rows, [&](int x, int y) { return t.row_deg[x] > t.row_deg[y]; });
    for (int P = 1; P <= kSplitMaxPhases && P <= rows; P++) {
        // nor can even shares of the dt, the edges and (phases) the sums that do not fit
        if (least + 4 * share((total + P - 1) / P) * t.z + 16 * share(t.n_edges) + (P > 1 ? 128 * share(nc) * chunks : 0) >
            smem_limit)
            continue;
        // phases: contiguous rows, about the same edges each
        int phase_of[kMaxRows], sum = 0;
        for (int r = 0; r < rows; r++) {
            phase_of[r] = std::min(P - 1, static_cast<int>(static_cast<long>(sum + core[r] / 2) * P / std::max(1, total)));
            sum += core[r];
        }
        // columns to ranks, largest degree first, to the rank with the least
        // dt; dt places of a column's edges, ascending rows, per phase
        int deg_sum[kSplitMaxRanks] = {0}, max_dt = 0;
        std::memset(d.n_dt, 0, sizeof(d.n_dt));
        std::memset(d.n_cols, 0, sizeof(d.n_cols));
        for (int i = 0; i < nc; i++) {
            const int c = col_order[i];
            int k = 0;
            for (int j = 1; j < ranks; j++)
                if (deg_sum[j] < deg_sum[k]) k = j;
            d.col_rank[c] = static_cast<uint8_t>(k);
            deg_sum[k] += d.col_deg[c] + kSplitColCost;
            d.cols[k][d.n_cols[k]++] = static_cast<uint8_t>(c);
            for (int p = 0; p < P; p++) d.col_beg[c][p] = d.n_dt[k][p];
            for (int j = 0; j < d.col_deg[c]; j++) d.dt_of[d.col_edge[c][j]] = d.n_dt[k][phase_of[d.col_row[c][j]]]++;
            for (int p = 0; p < P; p++) {
                d.col_cnt[c][p] = d.n_dt[k][p] - d.col_beg[c][p];
                max_dt = std::max(max_dt, d.n_dt[k][p]);
            }
        }
        // rows of a phase to ranks, largest degree first, to the rank with
        // the least work in the phase (then the fewest rows so far)
        std::memset(d.n_rows, 0, sizeof(d.n_rows));
        int busiest = 0, most = 0;  // work summed over the phases, rows of a rank's phase
        for (int p = 0; p < P; p++) {
            int load[kSplitMaxRanks] = {0};
            for (int k = 0; k < ranks; k++) d.row_beg[k][p] = d.n_rows[k];
            for (int i = 0; i < rows; i++) {
                const int r = row_order[i];
                if (phase_of[r] != p) continue;
                int k = 0;
                for (int j = 1; j < ranks; j++)
                    if (load[j] < load[k] || (load[j] == load[k] && d.n_rows[j] < d.n_rows[k])) k = j;
                d.row_rank[r] = static_cast<uint8_t>(k);
                d.row_at[r] = static_cast<uint8_t>(d.n_rows[k]);
                d.rows[k][d.n_rows[k]++] = static_cast<uint8_t>(r);
                load[k] += t.row_deg[r] + kSplitRowCost;
            }
            for (int k = 0; k < ranks; k++) most = std::max(most, d.n_rows[k] - d.row_beg[k][p]);
            busiest += chunks * *std::max_element(load, load + ranks);
        }
        size_t n_rows = 0, n_cols = 0, n_edges = 0;
        for (int k = 0; k < ranks; k++) {
            size_t e = 0;
            for (int i = 0; i < d.n_rows[k]; i++) e += t.row_deg[d.rows[k][i]];
            d.row_beg[k][P] = d.n_rows[k];
            n_edges = std::max(n_edges, e);
            n_rows = std::max(n_rows, static_cast<size_t>(d.n_rows[k]));
            n_cols = std::max(n_cols, static_cast<size_t>(d.n_cols[k]));
        }
        const int W = std::max(4, std::min(kSplitMaxWarps, std::max(most, static_cast<int>(n_cols)) * chunks));
        // image layout (the same for every rank) and shared memory
        size_t at = 0;
        auto take = [&](size_t bytes) {
            const size_t here = at;
            at += (bytes + 15) / 16 * 16;
            return static_cast<int>(here);
        };
        SplitHead h{};
        h.z = t.z;
        h.n_bp = t.n_bp;
        h.packed_bytes = t.packed_bytes;
        h.n_core = nc;
        h.core_floats = t.core_floats;
        h.ranks = ranks;
        h.phases = P;
        h.warps = W;
        h.n_edges = static_cast<int>(n_edges);
        h.load = busiest;
        h.o_edge = take(16 * n_edges);
        h.o_row = take(16 * n_rows);
        h.o_col = take(16 * n_cols);
        h.o_beg = take(4 * n_cols * P);
        h.o_own = take(4 * static_cast<size_t>(t.cols));
        h.o_cnptr = take(2 * (static_cast<size_t>(P) * W + 1));
        h.o_cn = take(2 * n_rows * chunks);
        h.o_vnptr = take(2 * (static_cast<size_t>(W) + 1));
        h.o_vn = take(2 * n_cols * chunks);
        h.o_bytes = take(8);
        h.image_bytes = static_cast<int>(at);
        auto up = [](size_t x) { return (x + 127) / 128 * 128; };
        const size_t l = up(kSplitHeader + at), st = up(l + 4 * static_cast<size_t>(t.core_floats)),
                     dt = up(st + 16 * n_rows * t.z), acc = up(dt + 4 * static_cast<size_t>(max_dt) * t.z),
                     end = acc + (P > 1 ? 128 * n_cols * chunks : 0);
        if (end > smem_limit) continue;
        h.off_l = static_cast<int>(l);
        h.off_state = static_cast<int>(st);
        h.off_dt = static_cast<int>(dt);
        h.off_acc = static_cast<int>(acc);
        h.smem = static_cast<int>(end);
        d.head = h;
        return true;
    }
    return false;
}

// Second half: the head and one table image per rank, appended to `out`.
void make_split_plan(const CodeTable& t, const SplitDeal& d, std::vector<unsigned char>* out) {
    const SplitHead& h = d.head;
    const int chunks = (t.z + 31) / 32, nc = t.n_core, ranks = h.ranks, P = h.phases, W = h.warps;
    const size_t base = out->size(), at = static_cast<size_t>(h.image_bytes);
    out->resize(base + sizeof(SplitHead) + ranks * at, 0);
    std::memcpy(out->data() + base, &h, sizeof(h));
    int row_cost[kMaxRows], col_cost[kMaxCols];
    uint8_t index[kMaxCols];
    uint32_t need[kMaxCols];  // every rank that reads a column: its owner, for the output, and those with a row on it
    for (int c = 0; c < nc; c++) {
        need[c] = 1u << d.col_rank[c];
        for (int j = 0; j < d.col_deg[c]; j++) need[c] |= 1u << d.row_rank[d.col_row[c][j]];
    }
    for (int c = 0; c < kMaxCols; c++) index[c] = static_cast<uint8_t>(c);
    for (int k = 0; k < ranks; k++) {
        unsigned char* im = out->data() + base + sizeof(SplitHead) + k * at;
        auto* edge = reinterpret_cast<uint4*>(im + h.o_edge);
        auto* row = reinterpret_cast<uint4*>(im + h.o_row);
        auto* col = reinterpret_cast<uint4*>(im + h.o_col);
        auto* beg = reinterpret_cast<uint32_t*>(im + h.o_beg);
        auto* own = reinterpret_cast<uint32_t*>(im + h.o_own);
        auto* cnptr = reinterpret_cast<uint16_t*>(im + h.o_cnptr);
        auto* cn = reinterpret_cast<uint16_t*>(im + h.o_cn);
        auto* vnptr = reinterpret_cast<uint16_t*>(im + h.o_vnptr);
        auto* vn = reinterpret_cast<uint16_t*>(im + h.o_vn);
        uint32_t m = 0;
        for (int i = 0; i < d.n_rows[k]; i++) {
            const int r = d.rows[k][i], last = t.row_ptr[r + 1] - 1;
            row_cost[i] = t.row_deg[r] + kSplitRowCost;
            row[i] = make_uint4(m | (static_cast<uint32_t>(t.row_ptr[r]) << 16), static_cast<uint32_t>(i) * t.z,
                                ((static_cast<uint32_t>(t.edge_col[last]) * t.z) << 9) | t.edge_shift[last],
                                t.row_deg[r] | (t.row_sfx[r] ? 256u : 0u));
            for (int e = t.row_ptr[r]; e <= last; e++, m++) {
                const int c = t.edge_col[e];
                edge[m] = make_uint4(t.eaddr[e].x, t.eaddr[e].y, 0u, 0u);
                if (c < nc) edge[m].z = (static_cast<uint32_t>(d.col_rank[c]) << 24) | static_cast<uint32_t>(d.dt_of[e]);
            }
        }
        for (int i = 0; i < d.n_cols[k]; i++) {
            const int c = d.cols[k][i];
            col_cost[i] = d.col_deg[c] + kSplitColCost;
            col[i] = make_uint4(4u * static_cast<uint32_t>(c) * t.z, need[c], 0u, 0u);
            for (int p = 0; p < P; p++)
                beg[i * P + p] = static_cast<uint32_t>(d.col_beg[c][p]) | (static_cast<uint32_t>(d.col_cnt[c][p]) << 16);
        }
        for (int c = 0; c < nc; c++) own[c] = static_cast<uint32_t>(d.col_rank[c]) << 28;
        for (int c = nc; c < t.cols; c++) {
            const int r = t.sfx_row[c];
            own[c] = (static_cast<uint32_t>(d.row_rank[r]) << 28) | (static_cast<uint32_t>(d.row_at[r] * t.z) << 9) |
                     t.edge_shift[t.row_ptr[r + 1] - 1];
        }
        for (int p = 0, n = 0; p < P; p++) {
            const int from = d.row_beg[k][p];
            n = spread(index + from, row_cost + from, d.row_beg[k][p + 1] - from, chunks, W, n, cnptr + p * W, cn);
        }
        spread(index, col_cost, d.n_cols[k], chunks, W, 0, vnptr, vn);
        // bytes that reach the rank in a one-phase iteration: dt of its
        // columns, posteriors that its rows or its output read
        auto* bytes = reinterpret_cast<uint32_t*>(im + h.o_bytes);
        bytes[0] = 4u * static_cast<uint32_t>(t.z) * static_cast<uint32_t>(d.n_dt[k][0]);
        uint32_t n_read = 0;
        for (int c = 0; c < nc; c++) n_read += need[c] >> k & 1u;
        bytes[1] = 4u * static_cast<uint32_t>(t.z) * n_read;
    }
}

namespace {
template <int MODE>
const void* split_kernel_of(bool weighted) {
    return weighted ? reinterpret_cast<const void*>(&split_decode_kernel<true, MODE>)
                    : reinterpret_cast<const void*>(&split_decode_kernel<false, MODE>);
}
int mode_of(const SplitHead& h, int early_stop) {
    return h.ranks == 1 ? kOne : h.phases == 1 && !early_stop ? kCounted : kBarriers;
}
const void* split_kernel(bool weighted, int mode) {
    return mode == kOne       ? split_kernel_of<kOne>(weighted)
           : mode == kCounted ? split_kernel_of<kCounted>(weighted)
                              : split_kernel_of<kBarriers>(weighted);
}
void split_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, const SplitHead& h, int n_clusters,
                  cudaStream_t stream) {
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = static_cast<unsigned>(h.ranks);
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cfg->gridDim = dim3(static_cast<unsigned>(h.ranks * n_clusters));
    cfg->blockDim = dim3(static_cast<unsigned>(h.warps * 32));
    cfg->dynamicSmemBytes = static_cast<size_t>(h.smem);
    cfg->stream = stream;
    cfg->attrs = attr;
    cfg->numAttrs = 1;
}
}  // namespace

cudaError_t split_kernel_attributes(size_t smem) {
    for (int w = 0; w < 6; w++) {
        const void* k = split_kernel((w & 1) != 0, w / 2);
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

int split_max_clusters(const SplitHead& h) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    split_config(&cfg, &attr, h, 1, nullptr);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, split_kernel(false, mode_of(h, 1)), &cfg) != cudaSuccess) {
        cudaGetLastError();  // clusters of this size are not available
        return 0;
    }
    return n;
}

bool split_counts(const SplitHead& h, int early_stop) { return mode_of(h, early_stop) == kCounted; }

cudaError_t launch_split(const SplitHead& h, const SplitArgs& args, const WeightTable* weights, int n_clusters,
                         cudaStream_t stream) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    split_config(&cfg, &attr, h, n_clusters, stream);
    NoWeights none{};
    void* params[2] = {const_cast<SplitArgs*>(&args),
                       weights ? const_cast<WeightTable*>(weights) : static_cast<void*>(&none)};
    return cudaLaunchKernelExC(&cfg, split_kernel(weights != nullptr, mode_of(h, args.early_stop)), params);
}

cudaError_t launch_split_timeout(const SplitHead& h, SplitArgs args, void* expected, int n_clusters,
                                 cudaStream_t stream) {
    uint32_t bytes = 0;
    cudaError_t e = cudaMemcpyAsync(&bytes, expected, sizeof(bytes), cudaMemcpyDeviceToHost, stream);
    if (e != cudaSuccess || (e = cudaStreamSynchronize(stream)) != cudaSuccess) return e;
    const uint32_t more = bytes + 16;
    args.wait_limit = 1024;
    e = cudaMemcpyAsync(expected, &more, sizeof(more), cudaMemcpyHostToDevice, stream);
    if (e == cudaSuccess) e = launch_split(h, args, nullptr, n_clusters, stream);
    const cudaError_t back = cudaMemcpyAsync(expected, &bytes, sizeof(bytes), cudaMemcpyHostToDevice, stream);
    const cudaError_t done = cudaStreamSynchronize(stream);
    return e != cudaSuccess ? e : back != cudaSuccess ? back : done;
}

}  // namespace nrldpc
