// Internal types shared by the CUDA sources and the C-ABI layer.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <algorithm>
#include <cstdint>
#include <vector>

#include "../../include/nr_gpu_ldpc_gb300.h"

namespace nrldpc {

constexpr int kMaxRows = 46;    // BG1
constexpr int kMaxCols = 68;    // BG1
constexpr int kMaxEdges = 320;  // BG1 has 316
constexpr int kMaxDeg = 19;     // BG1 rows 0..3
constexpr int kMaxZ = 384;
constexpr int kMaxThreads = 384;  // decode CTA size bound (cw_per_cta * Z)

// Lifted-code description passed to kernels by value (__grid_constant__).
struct alignas(16) CodeTable {
    int rows, cols, z, n_edges, n_bp, packed_bytes;
    int kb;                        // systematic base columns (encoder)
    // Base columns [n_core, cols) are suffix columns: each has degree 1 and is
    // the last edge of its row, and no row has two.  (5G NR: the extension
    // parity columns, 42 of 68 in BG1, 38 of 52 in BG2.)  The decoder keeps
    // their posteriors in the owning row's check-node state instead of in
    // shared memory.
    int n_core;
    int core_floats;               // n_core * Z rounded up to a multiple of 4
    uint16_t row_ptr[kMaxRows + 1];
    uint8_t row_deg[kMaxRows];
    uint8_t sync_after[kMaxRows];  // 1: CTA barrier after this row (row groups
                                   // between barriers share no base column)
    uint8_t row_sfx[kMaxRows];     // 1: the row's last edge is a suffix column
    uint8_t sfx_row[kMaxCols];     // suffix column -> its row
    // per edge, row-major ascending (row, then column) = the reference's
    // h_compact1 order: low 16 bits blk_col*Z + V, high 16 bits Z - V
    uint32_t edge[kMaxEdges];
    uint16_t ethr[kMaxEdges];      // Z - V: sub-rows from here on wrap
    uint8_t edge_col[kMaxEdges];
    uint16_t edge_shift[kMaxEdges];  // V mod Z
    // byte offset of the edge's column in a posterior buffer and 4V, one 64-bit
    // read per edge: sub-row s's position is at 4 ((s + V) mod Z) from it
    uint2 eaddr[kMaxEdges];
};

// Check-node state of one lifted row, kept between iterations (16 B, one
// uint4 per (row, sub-row), [slot][rows][Z]): min1 (raw |Q|), min2,
// info = idx (bits 0..4) | R sign of edge i at bit 8+i, and the posterior of
// the row's suffix column at this sub-row (unused in rows without one).
constexpr size_t kStateBytesPerRow = 16;
// Learned weights of the weighted decoder, passed by value as a kernel
// parameter (constant bank: every lane of a warp reads the same edge's
// weight).  Rows t < n_w_iters hold w[t][e]; row kMaxWIters stays zero (no
// previous message in the first iteration).
constexpr int kMaxWIters = 16;
struct alignas(16) WeightTable {
    float w[kMaxWIters + 1][kMaxEdges];
};
struct NoWeights {
    int unused;
};
struct DecodeArgs {
    const float* llr;
    uint8_t* packed;
    float* app;
    int32_t* iters;
    uint32_t* state;        // [grid * cpb][rows * Z][4]
    int* work_counter;      // dynamic codeword-group scheduler, zeroed per launch
    int* error_flag;        // bounded-wait failures
    int n_cw, n_iter, cpb, n_groups, n_w_iters, early_stop;
    int llr_from_host;      // 1: llr is pinned host memory read over the host link
    float alpha;
    // bounded-wait self-test only (0 in every decode): iterations of the LLR
    // copy wait (0: the default limit), and bytes the copy barrier expects
    // beyond what the copies deliver, so that wait runs out
    int wait_limit;
    uint32_t extra_tx;
};

// What the row loops are compiled for: any code, or one whose rows are like
// BG1's or BG2's (row_traits); kBg2Mixed: BG2's in a kernel that also holds
// BG1's
enum class RowClass { kAny, kBg1, kBg2, kBg2Mixed };
// kAny1, kAny2: any code, one or two CTAs per SM in the register budget
enum class DecodeKind { kAny1, kAny2, kBg1, kBg2 };
enum DeviceError : int { kErrNone = 0, kErrLlrLoadTimeout = 1, kErrSplitTimeout = 2 };

// Mixed-code batches (batch.cu): a work item is up to `count` codewords of
// one code, listed at order[start .. start+count).
constexpr int kNumZ = 51;  // lifting sizes of each base graph
struct WorkItem {
    int32_t code;   // index into the table array: BG1 from 0, BG2 from kNumZ
    int32_t start;
    int32_t count;
    int32_t spt;    // sub-rows per thread: Z / spt threads per codeword (1 or 2)
};
constexpr size_t kHeaderBytesBatch = 1024;  // mbarrier, item id, per-slot flags
constexpr size_t kBatchTableCopy = (sizeof(CodeTable) + 15) / 16 * 16;
constexpr size_t kBatchTableBytes = (kBatchTableCopy + 127) / 128 * 128;
struct BatchDecodeArgs {
    const CodeTable* tables;
    const WorkItem* items;
    const int32_t* order;       // job indices sorted by code
    const nrldpc_job* jobs;
    const float* llr;
    uint8_t* packed;
    int32_t* iters;
    uint32_t* state;            // [grid][slot_words]
    int* work_counter;
    int* error_flag;
    size_t slot_words;          // state words per CTA (largest cpb * 4 * rows * Z)
    int n_items, n_iter, early_stop;
    float alpha;
};
// Shared memory of one decode group of cpb codewords: Lold and Lnew over the
// core columns, plus one hard-decision byte per lifted row for the suffix
// columns.  Lnew is `far` bytes after Lold, the decisions in the gap when they
// fit; far = 0: right after it, the decisions last.  At a distance that the
// compiler knows, an edge's Lnew accesses are its Lold address and an
// immediate offset.
constexpr uint32_t kFarLong = kMaxThreads * 26 * 4;   // BG1's core columns at the most sub-rows per CTA
constexpr uint32_t kFarShort = kMaxThreads * 14 * 4;  // BG2's
// What is known of a class: decode_kernel's distance from Lold to Lnew, the
// degrees that occur (bit d), which of them end in a suffix column (those up
// to most_sfx), the longest row whose Q stay in registers in unweighted
// flooding, and how many edges ahead of the store Lnew is read.  In both NR
// base graphs a row's degree tells whether it has a suffix column, so the
// classes' row bodies have no test for one.  BG2's kernels have the registers
// to read a whole row of Lnew first (2.9% over 15 sizes, BG2 Z=208 1,001
// codewords 563 -> 549 us, Z=256 with early stop 1% slower); the job lists'
// kernel, whose registers BG1's rows take, is 1.4% slower with it.
struct RowTraits {
    uint32_t far, degrees;
    int most_sfx, keep_q, ahead;
};
__host__ __device__ constexpr RowTraits row_traits(RowClass c) {
    return c == RowClass::kBg1        ? RowTraits{kFarLong, 0x807f8u, 10, 10, 4}
           : c == RowClass::kBg2      ? RowTraits{kFarShort, 0x578u, 6, 10, 10}
           : c == RowClass::kBg2Mixed ? RowTraits{kFarShort, 0x578u, 6, 8, 4}
                                      : RowTraits{0u, 0xffffeu, -1, 10, 4};
}
inline RowClass row_class(const CodeTable& t) {
    for (RowClass c : {RowClass::kBg1, RowClass::kBg2}) {
        const RowTraits k = row_traits(c);
        bool fits = true;
        for (int r = 0; r < t.rows; r++)
            fits &= (k.degrees >> t.row_deg[r] & 1) && (t.row_sfx[r] != 0) == (t.row_deg[r] <= k.most_sfx);
        if (fits) return c;
    }
    return RowClass::kAny;
}
__host__ __device__ inline uint32_t group_hd_offset(uint32_t half, uint32_t hd, uint32_t far) {
    return far == 0 ? 2 * half : half + hd <= far ? half : far + half;
}
inline size_t group_smem_bytes(const CodeTable& t, int cpb, uint32_t far) {
    const size_t hd = (static_cast<size_t>(cpb) * t.rows * t.z + 15) / 16 * 16;
    const size_t half = static_cast<size_t>(cpb) * t.core_floats * sizeof(float);
    return far == 0 ? 2 * half + hd : far + half + (half + hd <= far ? 0 : hd);
}
// CTAs per SM by registers (80 a thread) and shared memory
inline int decode_ctas(int threads, size_t smem, size_t smem_sm) {
    return static_cast<int>(std::min<size_t>(65536 / (80 * threads), smem_sm / (smem + 1024)));
}
// classes: one sub-row per thread, and the layout of each base graph's class
const void* batch_decode_kernel_ptr(bool classes);

// One codeword on a cluster of CTAs (split.cu).  A plan is a head and one
// table image per rank, contiguous in device memory: which CTA owns which base
// row and core column, the check-node and variable-node tasks of each warp
// (32 sub-rows or positions each), and the shared-memory layout.
constexpr int kSplitMaxRanks = 16;   // CTAs per cluster
constexpr int kSplitMaxPhases = 8;   // row ranges of an iteration
constexpr int kSplitMaxWarps = 24;   // per CTA
constexpr size_t kSplitHeader = 144;  // mbarriers, failure flags, head
constexpr int kSplitWaitLimit = 1 << 20;  // polls, as decode_kernel's
constexpr int kSplitKeep = 10;       // longest row whose Q and dt addresses stay in registers
constexpr int kSplitVnAhead = 8;     // dt requested before the first add
constexpr int kSplitRowCost = 4;     // a row's fixed work, in edges
constexpr int kSplitColCost = 6;     // a column's fixed work, in edges
struct alignas(16) SplitHead {
    int z, n_bp, packed_bytes, n_core, core_floats, ranks, phases, warps, n_edges;
    int load;  // edges (and fixed work) of the busiest rank's tasks, per warp of sub-rows
    // image: edges {column, 4V, owner << 24 | dt place} of the
    // rank's rows; rows {first edge | edge in the code << 16, state, suffix
    // column << 9 | shift, degree | suffix << 8}; columns {offset, ranks that
    // read it}; their dt {first | count << 16} per phase; every column's
    // owner; task lists per (phase,) warp; bytes of dt and of posteriors that
    // reach the rank per iteration
    int o_edge, o_row, o_col, o_beg, o_own, o_cnptr, o_cn, o_vnptr, o_vn, o_bytes, image_bytes;
    int off_l, off_state, off_dt, off_acc, smem;  // shared memory
};
struct SplitJob {            // one codeword of a mixed batch
    int64_t llr_offset, out_offset;
    int32_t plan, job;       // byte offset of its code's plan; iteration-count index
};
struct SplitArgs {
    SplitHead head;          // of the plan (without jobs)
    const unsigned char* plan;
    const SplitJob* jobs;    // null: n_cw codewords of one code, back to back
    const float* llr;
    uint8_t* packed;
    float* app;
    int32_t* iters;
    int* error_flag;         // bounded-wait failures
    int n_cw, n_iter, n_w_iters, early_stop, llr_from_host;
    float alpha;
    int32_t wait_limit = kSplitWaitLimit;  // polls before a wait gives up
};
static_assert(kSplitHeader >= 32 + sizeof(SplitHead) && kSplitHeader % 16 == 0, "flags, then the head");
// Cluster sizes tried: each holds more codewords at once than the one before
// (GB300 at one CTA per SM: 7, 13, 23, 28, 36, 46, 76 and 152 clusters; a
// GPC's SMs do not divide evenly by the other sizes).
constexpr int kSplitRanks[] = {16, 10, 6, 5, 4, 3, 2, 1};
constexpr int kSplitSizes = 8;
constexpr int kSplitMinTasks = 12;  // 32-sub-row tasks per CTA worth a larger cluster
// Time estimates of the two decoders, in edges of one warp (45 ns per 10
// iterations on GB300): one wave of clusters takes 667 per phase (barriers,
// the passes' latency) plus the busiest CTA's edges; decode_kernel's walk down
// the rows costs per row and edge, more with more warps in the CTA.
inline long split_cost(const SplitHead& h) { return 667L * h.phases + h.load; }
inline long fused_row_walk(const CodeTable& t, long warps) {
    return t.rows * (29 + 21 * warps / 10) + t.n_edges * (81 + 4 * warps) / 10;
}
// Which CTA owns which base row and core column.
struct SplitDeal {
    SplitHead head;
    uint8_t col_deg[kMaxCols], col_row[kMaxCols][kMaxRows];  // each column's rows and edges, ascending
    uint16_t col_edge[kMaxCols][kMaxRows];
    uint8_t col_rank[kMaxCols], row_rank[kMaxRows], row_at[kMaxRows];  // owners; a row's place there
    uint8_t cols[kSplitMaxRanks][kMaxCols], rows[kSplitMaxRanks][kMaxRows];  // of each rank, in order
    int n_cols[kSplitMaxRanks], n_rows[kSplitMaxRanks];
    int row_beg[kSplitMaxRanks][kSplitMaxPhases + 1];  // first row of each phase
    int col_beg[kMaxCols][kSplitMaxPhases], col_cnt[kMaxCols][kSplitMaxPhases];  // a column's dt places per phase
    int dt_of[kMaxEdges], n_dt[kSplitMaxRanks][kSplitMaxPhases];
};
bool deal_split(const CodeTable& tab, int ranks, size_t smem_limit, SplitDeal* deal);
void make_split_plan(const CodeTable& tab, const SplitDeal& deal, std::vector<unsigned char>* out);
cudaError_t split_kernel_attributes(size_t smem);
int split_max_clusters(const SplitHead& head);  // resident at once
bool split_counts(const SplitHead& head, int early_stop);  // whether its passes wait for counted bytes
// launch_split with a short wait limit and, for its time, 16 bytes more in the
// count at `expected`, of the bytes that reach a plan's first CTA.
cudaError_t launch_split_timeout(const SplitHead& head, SplitArgs args, void* expected, int n_clusters,
                                 cudaStream_t stream);
cudaError_t launch_split(const SplitHead& head, const SplitArgs& args, const WeightTable* weights, int n_clusters,
                         cudaStream_t stream);

// Live decoders of the process and whether their last call is still running.
// A small batch spread over the whole GPU is the fastest alone but takes about
// twice the SM time of decode_kernel, so the choice counts the other decoders
// of the device that are busy on other streams as as many batches like its
// own.  The first call of a round sees the others idle, so the count falls by
// one a call at most, unless one decoder calls twice in a row beside idle ones
// (a hint: either choice gives the same bits).
struct InFlight {
    int device = -1;
    cudaEvent_t done = nullptr;  // after the last call
    cudaStream_t stream = nullptr;
    bool recorded = false;
    int neighbours = -1;  // what the caller says instead of the count
};
// Whether work on the stream is being captured; true also where that cannot be
// told.  pending: an error of the caller's that it has not read yet, left alone.
bool is_captured(cudaStream_t stream, bool pending);
bool in_flight_join(InFlight* me, int device);
void in_flight_leave(InFlight* me);
// Busy ones beside `me`; 0 where as many calls of `sms` SMs as there are
// decoders fit the GPU's.  While the stream is captured, all others: what runs
// beside a replay is not known then.  Six graphs of 40 BG1 Z=384 codewords, 5
// iterations, replayed on six streams: 0.400 ms a round spread, 0.208 on
// decode_kernel; one of them alone 0.081 and 0.148.
int in_flight_others(const InFlight* me, cudaStream_t stream, long sms, int sm_count);
void in_flight_note(InFlight* me, cudaStream_t stream);  // after a call's launches

// A copy from pageable memory and a memset may return before the device has the
// data, and work on other streams than the legacy one is not ordered after
// them: waited for before a handle is given out.
inline cudaError_t uploads_landed() { return cudaStreamSynchronize(cudaStreamLegacy); }

// Host-side launchers (decode.cu / channel.cu).
// kind: which kernels serve a code and geometry (decode_shape).
// weights: null for the plain decoder; layered: row-sequential schedule (no
// reference counterpart) instead of flooding.
cudaError_t launch_decode(const CodeTable& tab, const DecodeArgs& args, const WeightTable* weights, int grid,
                          int threads, size_t smem, bool layered, DecodeKind kind, cudaStream_t stream);
size_t decode_smem_bytes(const CodeTable& tab, int cpb, uint32_t far = 0);
// CTA geometry of cpb codewords per CTA
struct DecodeShape {
    int cpb = 1, threads = 32;
    size_t smem = 0;
    DecodeKind kind = DecodeKind::kAny1;
};
DecodeShape decode_shape(const CodeTable& tab, int cpb, size_t smem_block, size_t smem_sm);
cudaError_t decode_kernel_attributes(DecodeKind kind, size_t smem);
int decode_max_ctas_per_sm(DecodeKind kind, bool weighted, int threads, size_t smem);

// Learned weighted min-sum training kernels (wms.cu).
size_t wms_smem_bytes(const CodeTable& tab, int cpb, bool layered);
cudaError_t wms_kernel_attributes(const CodeTable& tab, int cpb);
int wms_ctas_per_sm(const CodeTable& tab, int cpb, int threads);  // the fewest of the code's four kernels
cudaError_t launch_wms(bool backward, bool layered, const CodeTable& tab, const float* llr, const uint8_t* cw,
                       const float* weights, uint4* states, float* gseed, uint4* gq, float* gh, double* loss,
                       double* grad, float* app, int* counters, int n_cw, int T, int cpb, int grid,
                       int threads, float scale, cudaStream_t stream);
cudaError_t launch_adam(int n, float* w, const double* grad, float* m, float* v, int step, float lr,
                        float b1, float b2, float eps, float w_min, cudaStream_t stream);

// 5G NR (bg, z) code table, built on the caller's storage (no allocation).
bool make_nr_table(int bg, int z, CodeTable* t);

struct EncodePlan {
    int n_core_steps;              // rows solved one parity column at a time
    int core_row[kMaxRows];
    int core_col[kMaxRows];
    int p0_col, p0_shift;          // first parity column = P^{-v} * sum(lambda)
    int n_stair;                   // staircase rows summed for p0
};
bool make_encode_plan(const CodeTable& tab, EncodePlan* plan);
cudaError_t launch_gen_llr(const CodeTable& tab, const EncodePlan& plan, uint64_t seed,
                           uint64_t cw_base, int n_cw, const float* sigma, int n_punct_cols,
                           float* llr, uint8_t* cw_packed, cudaStream_t stream);
cudaError_t launch_dequant(const void* in, int qtype, float scale, size_t n, float* out,
                           cudaStream_t stream);
cudaError_t launch_crc(const uint8_t* packed, int n_cw, int stride, int n_bits, uint32_t poly, int len,
                       uint32_t* rem, cudaStream_t stream);
// Code-block segmentation (channel.cu): between a transport block and C code
// blocks of k_prime bits (data_bits of it data), with a CRC of len bits
// attached to or checked over each block (len 0: none).
cudaError_t launch_cb_segment(const uint8_t* tb, int C, int data_bits, int k_prime, uint8_t* blocks, int stride,
                              uint32_t poly, int len, cudaStream_t stream);
cudaError_t launch_cb_desegment(const uint8_t* blocks, int stride, int C, int data_bits, int k_prime, uint8_t* tb,
                                uint32_t poly, int len, uint32_t* rem, cudaStream_t stream);
cudaError_t launch_count_errors(const uint8_t* packed, const uint8_t* cw_packed, int n_cw,
                                int packed_bytes, int n_info, unsigned long long* counts,
                                cudaStream_t stream);

}  // namespace nrldpc
