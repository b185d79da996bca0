// Mixed-code batches: every 5G NR (BG, Z) in one handle, a device work queue
// of codeword groups, one persistent decode launch replayed from a CUDA graph,
// and job-based rate matching (3GPP TS 38.212 5.4.2.1 bit selection with
// filler bits, full circular buffer, BPSK so no interleaver) on the GPU.
// No reference counterpart: the reference compiles in one base graph and one
// Z per process (src/globals.h:15, constant memory in src/ldpc_kernels.cu:18-27)
// and has no rate matching (src/main.cpp:64-65).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <new>
#include <vector>

#include "../../include/nr_gpu_ldpc_gb300.h"
#include "channel_dev.cuh"
#include "nrldpc_internal.h"

namespace nrldpc {
bool make_nr_table(int bg, int z, CodeTable* t);
}

using namespace nrldpc;

namespace {

constexpr int kNumCodes = 2 * kNumZ;
constexpr int kBaseZ[8] = {2, 3, 5, 7, 9, 11, 13, 15};

struct PlanDev {
    int32_t n_stair, p0_col, p0_shift, n_steps;
    uint8_t step_row[kMaxRows];
    uint8_t step_col[kMaxRows];
};

static_assert(sizeof(nrldpc_job) == 56, "nrldpc_job layout (mirrored by the Python binding)");

// Rate-matching geometry of one job, resolved on the host.
struct JobDev {
    int32_t code;
    int32_t k_prime;   // info bits (filler from k_prime to kb*Z)
    int32_t e;         // transmitted bits
    int32_t k0;        // start in the circular buffer
    float sigma;
    int32_t qm;        // modulation order of the bit interleaver (1: none)
    int64_t llr_offset, e_offset, out_offset;
};

int z_list[kNumZ];
int z_index(int z) {
    for (int i = 0; i < kNumZ; i++)
        if (z_list[i] == z) return i;
    return -1;
}
void init_z_list() {
    if (z_list[0]) return;
    int n = 0;
    for (int zz = 2; zz <= 384; zz++)
        for (int i = 0; i < 8; i++) {
            bool hit = false;
            for (int v = kBaseZ[i]; v <= 384; v *= 2) hit |= v == zz;
            if (hit) {
                z_list[n++] = zz;
                break;
            }
        }
}

int rm_k0(int bg, int z, int rv) {
    static const int a1[4] = {0, 17, 33, 56}, a2[4] = {0, 13, 25, 43};
    if (rv < 0 || rv > 3 || (bg != 1 && bg != 2)) return -1;
    const long n = bg == 1 ? 66 : 50, ncb = n * z;  // full buffer
    return static_cast<int>(((bg == 1 ? a1[rv] : a2[rv]) * ncb) / (n * z)) * z;
}

// d index of transmitted bit k (filler run [f0, f1) of d removed, wrap at Ncb).
__device__ __forceinline__ int rm_index(int z, int ncb, int kbz, int kp, int k0, int k) {
    const int f0 = kp - 2 * z, f1 = kbz - 2 * z, nf = f1 - f0, nc = ncb - nf;
    const int c0 = k0 < f0 ? k0 : (k0 < f1 ? f0 : k0 - nf);
    const int c = static_cast<int>((static_cast<long long>(c0) + k) % nc);
    return c < f0 ? c : c + nf;
}

struct GenBatchArgs {
    const CodeTable* tables;
    const PlanDev* plans;
    const JobDev* jobs;
    float* llr_e;
    uint8_t* cw;
    uint64_t seed, cw_base;
    int n_jobs;
};

// Bit interleaver of TS 38.212 5.4.2.2, f[i + j*Qm] = e[i*E/Qm + j]: the e
// index of the bit sent at position p, and the position of e index k.
__device__ __forceinline__ int il_src(int e, int qm, int p) {
    return qm == 1 ? p : (p % qm) * (e / qm) + p / qm;
}
__device__ __forceinline__ int il_pos(int e, int qm, int k) {
    if (qm == 1) return k;
    const int rows = e / qm;
    return k / rows + (k % rows) * qm;
}

// One CTA per job: info bits, encode, select e bits from k0, interleave,
// BPSK + AWGN per transmitted position.
__global__ void __launch_bounds__(256) batch_gen_kernel(const __grid_constant__ GenBatchArgs g) {
    extern __shared__ uint8_t x[];  // [n_bp] codeword bits, then [z] scratch
    const uint32_t k0s = static_cast<uint32_t>(g.seed), k1s = static_cast<uint32_t>(g.seed >> 32);
    for (int i = blockIdx.x; i < g.n_jobs; i += gridDim.x) {
        const JobDev jb = g.jobs[i];
        const CodeTable& tab = g.tables[jb.code];
        const PlanDev& pl = g.plans[jb.code];
        const int z = tab.z, n = tab.n_bp, K = tab.kb * z, ncb = n - 2 * z;
        uint8_t* acc = x + n;
        const uint64_t id = g.cw_base + static_cast<uint64_t>(i);
        const uint32_t id0 = static_cast<uint32_t>(id), id1 = static_cast<uint32_t>(id >> 32);
        for (int b = threadIdx.x; b * 128 < K; b += blockDim.x) {
            uint32_t o[4];
            dev::philox4x32(static_cast<uint32_t>(b), id0, id1, 1u, k0s, k1s, o);
            for (int j = 0; j < 128 && b * 128 + j < K; j++) {
                const int pos = b * 128 + j;
                x[pos] = pos < jb.k_prime ? (o[j >> 5] >> (j & 31)) & 1u : 0u;
            }
        }
        __syncthreads();
        dev::encode_in_smem(tab, pl.n_stair, pl.p0_col, pl.p0_shift, pl.n_steps, pl.step_row,
                            pl.step_col, x, acc);
        if (g.cw) {
            uint8_t* out = g.cw + jb.out_offset;
            for (int b = threadIdx.x; b < tab.packed_bytes; b += blockDim.x) {
                uint32_t v = 0;
                for (int j = 0; j < 8; j++)
                    if (8 * b + j < n) v |= static_cast<uint32_t>(x[8 * b + j]) << j;
                out[b] = static_cast<uint8_t>(v);
            }
        }
        const float sg = jb.sigma, s2 = __fmul_rn(sg, sg);
        float* out = g.llr_e + jb.e_offset;
        for (int t = threadIdx.x; t * 4 < jb.e; t += blockDim.x) {
            uint32_t o[4];
            dev::philox4x32(static_cast<uint32_t>(t), id0, id1, 3u, k0s, k1s, o);
            float gs[4];
            dev::gauss4(o, gs);
            for (int q = 0; q < 4 && 4 * t + q < jb.e; q++) {
                const int p = 4 * t + q;
                const int j = 2 * z + rm_index(z, ncb, K, jb.k_prime, jb.k0, il_src(jb.e, jb.qm, p));
                out[p] = dev::bpsk_llr(x[j], gs[q], sg, s2);
            }
        }
        __syncthreads();
    }
}

struct DerateArgs {
    const CodeTable* tables;
    const JobDev* jobs;
    const int32_t* order;  // largest codes first
    const float* llr_e;
    float* llr;
    int n_jobs, parts, part;
};

// Each job's output in `parts` parts of `part` positions or interleaver rows,
// one CTA per (job, part) at a time: as many parts as it takes for a few jobs
// to fill the GPU, one where the jobs do (nrldpc_batch_set_jobs); the largest
// jobs first and every other round of CTAs backwards, so that the CTAs' shares
// differ little.  Not interleaved and without repetition (e <= Nc): the output
// in order, four positions a store, each position's LLR, zero or filler looked
// up.  Interleaved: a thread takes one interleaver row, reads its qm
// neighbouring LLRs (bits i, i + E/qm, ...) and writes each beside its
// neighbours' -- no division per bit.  With repetition each position c
// collects bits k = k_first, k_first + Nc, ... in order, the first copy taken
// as is, later ones added.  Bound by the writes: the 8,192-codeword mix (0.40
// GB written, 0.23 read) takes 154 us without its reads, 190 with them; in
// input order, four bytes a store, it took 257, 1,000 codewords 73 (now 24).

__global__ void __launch_bounds__(256) batch_derate_kernel(const __grid_constant__ DerateArgs a) {
    const float inf = __int_as_float(0x7f800000);
    const long n_work = static_cast<long>(a.n_jobs) * a.parts;
    for (long base = 0, back = 0; base < n_work; base += gridDim.x, back ^= 1) {
        const long w = base + (back ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
        if (w >= n_work) continue;
        const int at = static_cast<int>(w / a.parts), from = static_cast<int>(w - static_cast<long>(at) * a.parts) * a.part;
        const JobDev jb = a.jobs[a.order[at]];
        const int z = a.tables[jb.code].z, n = a.tables[jb.code].n_bp, K = a.tables[jb.code].kb * z, ncb = n - 2 * z;
        const int f0 = jb.k_prime - 2 * z, nf = K - jb.k_prime, nc = ncb - nf;
        const int c0 = jb.k0 < f0 ? jb.k0 : (jb.k0 < f0 + nf ? f0 : jb.k0 - nf);
        float* out = a.llr + jb.llr_offset;
        const float* in = a.llr_e + jb.e_offset;
        if (jb.qm == 1 && jb.e <= nc && reinterpret_cast<uintptr_t>(out) % 16 == 0) {
            auto value = [&](int j) {  // of position j of the mother codeword
                if (j < 2 * z) return 0.0f;
                if (j >= jb.k_prime && j < K) return inf;
                int k = j - 2 * z - (j < K ? 0 : nf) - c0;
                if (k < 0) k += nc;
                return k < jb.e ? __ldcs(in + k) : 0.0f;
            };
            const int to = min(n, from + a.part);  // a multiple of 4, as 52 Z and 68 Z are
            for (int j = from + 4 * threadIdx.x; j < to; j += 4 * blockDim.x)
                *reinterpret_cast<float4*>(out + j) = make_float4(value(j), value(j + 1), value(j + 2), value(j + 3));
            continue;
        }
        if (from == 0) {
            for (int j = threadIdx.x; j < 2 * z; j += blockDim.x) out[j] = 0.0f;
            for (int j = jb.k_prime + threadIdx.x; j < K; j += blockDim.x) out[j] = inf;
        }
        // position of bit k: c = (c0 + k) mod Nc, past the filler run
        auto put = [&](int k, float v) {
            int c = c0 + k;
            if (c >= nc) c -= nc;
            out[2 * z + (c < f0 ? c : c + nf)] = v;
        };
        if (jb.e <= nc) {
            const int rows = jb.qm == 1 ? jb.e : jb.e / jb.qm;
            if (jb.qm == 1) {
#pragma unroll 4
                for (int k = from + threadIdx.x; k < min(rows, from + a.part); k += blockDim.x) put(k, __ldcs(in + k));
            } else {
                for (int i = from + threadIdx.x; i < min(rows, from + a.part); i += blockDim.x) {
                    const float* row = in + static_cast<long>(i) * jb.qm;
                    for (int j = 0, k = i; j < jb.qm; j++, k += rows) put(k, row[j]);
                }
            }
#pragma unroll 4
            for (int k = jb.e + from + threadIdx.x; k < min(nc, jb.e + from + a.part); k += blockDim.x) put(k, 0.0f);
        } else {
            for (int k = from + threadIdx.x; k < min(nc, from + a.part); k += blockDim.x) {
                float v = in[il_pos(jb.e, jb.qm, k)];
                for (int m = k + nc; m < jb.e; m += nc) v = __fadd_rn(v, in[il_pos(jb.e, jb.qm, m)]);
                put(k, v);
            }
        }
    }
}

struct CountArgs {
    const CodeTable* tables;
    const JobDev* jobs;
    const uint8_t* packed;
    const uint8_t* cw;
    unsigned long long* counts;
    int n_jobs;
};

__global__ void __launch_bounds__(256) batch_count_kernel(const __grid_constant__ CountArgs a) {
    __shared__ unsigned int warp_sum[8];
    for (int i = blockIdx.x; i < a.n_jobs; i += gridDim.x) {
        const JobDev jb = a.jobs[i];
        const uint8_t* p = a.packed + jb.out_offset;
        const uint8_t* q = a.cw + jb.out_offset;
        const int full = jb.k_prime / 8, rem = jb.k_prime % 8;
        unsigned int errs = 0;
        for (int k = threadIdx.x; k < full; k += blockDim.x) errs += __popc(p[k] ^ q[k]);
        if (rem && threadIdx.x == 0) errs += __popc((p[full] ^ q[full]) & ((1u << rem) - 1u));
        for (int off = 16; off > 0; off >>= 1) errs += __shfl_down_sync(0xffffffffu, errs, off);
        if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = errs;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned int tot = 0;
            for (int w = 0; w < (blockDim.x + 31) / 32; w++) tot += warp_sum[w];
            if (tot) {
                atomicAdd(&a.counts[0], static_cast<unsigned long long>(tot));
                atomicAdd(&a.counts[1], 1ull);
            }
        }
        __syncthreads();
    }
}

struct Batch {
    InFlight in_flight;
    int device = 0;
    float alpha = 0.75f;
    int max_jobs = 0;
    int sm_count = 1;
    size_t smem_optin = 0, smem_sm = 0;
    CodeTable h_tables[kNumCodes];
    bool code_ok[kNumCodes];
    int cpb[kNumCodes];
    int spt[kNumCodes];  // sub-rows per thread (threads per codeword = Z / spt)
    CodeTable* d_tables = nullptr;
    PlanDev* d_plans = nullptr;
    // job list
    int n_jobs = 0, n_items = 0;
    std::vector<JobDev> h_jobs;
    // the job list on the device: one allocation, one copy per set_jobs
    unsigned char* d_lists = nullptr;
    cudaEvent_t lists_sent = nullptr;  // after that copy, on the legacy stream
    bool lists_landed = true;
    std::vector<unsigned char> h_lists;
    JobDev* d_jobs_rm = nullptr;
    nrldpc_job* d_jobs = nullptr;
    int32_t* d_order = nullptr;
    WorkItem* d_items = nullptr;
    int derate_parts = 1, derate_part = 256;
    // few jobs: one codeword on a cluster of CTAs (split.cu).  A plan's tables
    // are made when a job list first runs on it, and kept; split: the current
    // list's launch, ranks 0: none
    struct Plan {
        int state = 0;  // 1: head known, -1: the code does not fit such clusters
        int32_t at = -1;  // its place in d_plans_split
        SplitHead head;
    };
    std::vector<Plan> plans;  // [code][cluster size]
    unsigned char* d_plans_split = nullptr;
    size_t plans_bytes = 0;
    SplitJob* d_split = nullptr;
    SplitHead split{};
    int split_clusters = 0;
    size_t split_count_at = 0;  // of the bytes that the first CTA of the list's first code expects (self-test)
    size_t slot_words = 0, smem = 0;
    bool classes = false;  // of rows and layouts (batch_decode_kernel)
    int grid = 0, threads = kMaxThreads;
    uint32_t* d_state = nullptr;
    size_t state_words = 0;
    int* d_scratch = nullptr;
    // decode graph
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaGraphNode_t knode = nullptr;
    BatchDecodeArgs kargs{};
};

// Room for the plans of every code and cluster size (6.6 MB), so that no list
// allocates or frees device memory for them.
constexpr size_t kPlansRoom = 8u << 20;

constexpr size_t kListBytes =
    sizeof(JobDev) + sizeof(nrldpc_job) + sizeof(int32_t) + sizeof(WorkItem) + sizeof(SplitJob);

int map_cuda(cudaError_t e) { return e == cudaSuccess ? NRLDPC_OK : NRLDPC_ERR_CUDA; }

// Most codewords per CTA of code id with spt sub-rows per thread: Z / spt
// threads each within kMaxThreads, and their shared memory within the
// device's opt-in limit.
int max_cpb(const Batch* b, int id, int spt) {
    const CodeTable& t = b->h_tables[id];
    const int tpc = t.z / spt;
    const size_t room = b->smem_optin - kHeaderBytesBatch - kBatchTableBytes;
    int c = std::max(1, kMaxThreads / tpc);
    while (c > 1 && group_smem_bytes(t, c, 0) > room) c--;
    return std::min(c, 48);
}

int code_id(int bg, int z) {
    const int zi = z_index(z);
    if ((bg != 1 && bg != 2) || zi < 0) return -1;
    return (bg - 1) * kNumZ + zi;
}

void drop_graph(Batch* b) {
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    b->exec = nullptr;
    b->graph = nullptr;
    b->knode = nullptr;
}

void free_batch(Batch* b) {
    if (!b) return;
    in_flight_leave(&b->in_flight);
    drop_graph(b);
    cudaFree(b->d_tables);
    cudaFree(b->d_plans);
    cudaFree(b->d_lists);
    if (b->lists_sent) cudaEventDestroy(b->lists_sent);
    cudaFree(b->d_plans_split);
    cudaFree(b->d_state);
    cudaFree(b->d_scratch);
    delete b;
}

SplitArgs split_args(const Batch* b, const float* llr, uint8_t* packed, int n_iter) {
    SplitArgs a{};
    a.plan = b->d_plans_split;
    a.jobs = b->d_split;
    a.llr = llr;
    a.packed = packed;
    a.error_flag = b->d_scratch + 1;
    a.n_cw = b->n_jobs;
    a.n_iter = n_iter;
    a.alpha = b->alpha;
    return a;
}

// Before work on `stream` reads the lists and plans: their copies come from
// pageable memory, so they may still be under way when set_jobs returns, and
// only the legacy stream is ordered after them.  Waiting in set_jobs instead
// took 8 us of every slot (26 BG1 Z=384 blocks 125.5 -> 133.2 us).
cudaError_t wait_lists(Batch* b, cudaStream_t stream) {
    if (b->lists_landed || stream == nullptr || stream == cudaStreamLegacy) return cudaSuccess;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;  // a capture is not disturbed
    cudaThreadExchangeStreamCaptureMode(&mode);
    const cudaError_t e = cudaEventSynchronize(b->lists_sent);
    cudaThreadExchangeStreamCaptureMode(&mode);
    b->lists_landed = e == cudaSuccess;
    return e;
}

// The clusters for this job list (b->split, b->split_clusters and the jobs'
// plans), or none where the time estimate favours the persistent kernel.
// Cluster sizes from the largest that holds at least half the jobs at once
// down to the first that holds all; the jobs are in order of falling work.
int choose_split(Batch* b, const std::vector<int32_t>& order, const std::vector<WorkItem>& items,
                 std::vector<SplitJob>* jobs) {
    static const int kRoom[kSplitSizes] = {7, 13, 23, 28, 36, 46, 76, 152};  // at one CTA per SM of 152
    const int n = static_cast<int>(order.size());
    SplitDeal deal;
    if (n > 2L * kRoom[kSplitSizes - 1] * b->sm_count / 152) return NRLDPC_OK;
    long fused_sum = 0, least = 0;
    for (const WorkItem& it : items) {
        const long c = fused_row_walk(b->h_tables[it.code], b->threads / 32);
        fused_sum += c;
        least = std::max(least, c);  // the longest item
    }
    least = std::max(least, fused_sum * 33 / 40 / b->sm_count);  // two CTAs per SM: 1.65 times one's time
    int tasks = 0;
    for (const int32_t j : order) {
        const CodeTable& t = b->h_tables[b->h_jobs[j].code];
        tasks = std::max(tasks, t.rows * ((t.z + 31) / 32));
    }
    b->plans.resize(kNumCodes * kSplitSizes);
    int best = -1;
    for (int s = 0; s < kSplitSizes; s++) {
        const int ranks = kSplitRanks[s];
        if (n > 2L * kRoom[s] * b->sm_count / 152 || (ranks > 1 && tasks < ranks * kSplitMinTasks)) continue;
        SplitHead launch{};
        launch.ranks = ranks;
        bool fits = true;
        for (size_t i = 0; fits && i < order.size(); i++) {
            const int code = b->h_jobs[order[i]].code;
            Batch::Plan& p = b->plans[code * kSplitSizes + s];
            if (p.state == 0) {
                p.state = deal_split(b->h_tables[code], ranks, b->smem_optin, &deal) ? 1 : -1;
                if (p.state > 0) p.head = deal.head;
            }
            fits = p.state > 0;
            launch.warps = std::max(launch.warps, p.head.warps);
            launch.phases = std::max(launch.phases, p.head.phases);
            launch.smem = std::max(launch.smem, p.head.smem);
        }
        if (!fits) continue;
        const int room = split_max_clusters(launch);
        if (room < 1) continue;
        long cost = 0;
        for (int i = 0; i < n; i += room) cost += split_cost(b->plans[b->h_jobs[order[i]].code * kSplitSizes + s].head);
        if (cost < least) {
            least = cost;
            best = s;
            b->split = launch;
            b->split_clusters = std::min(n, room);
        }
        if (room >= n) break;
    }
    if (best < 0) return NRLDPC_OK;
    std::vector<unsigned char> fresh;  // tables that no list has run on yet
    std::vector<Batch::Plan*> placed;
    for (const int32_t j : order) {
        const CodeTable& t = b->h_tables[b->h_jobs[j].code];
        Batch::Plan& p = b->plans[b->h_jobs[j].code * kSplitSizes + best];
        if (p.at >= 0) continue;
        p.at = static_cast<int32_t>(b->plans_bytes + fresh.size());
        placed.push_back(&p);
        if (deal_split(t, kSplitRanks[best], b->smem_optin, &deal)) make_split_plan(t, deal, &fresh);
    }
    if (!fresh.empty()) {
        const bool room = b->plans_bytes + fresh.size() <= kPlansRoom;
        if (!room || cudaMemcpy(b->d_plans_split + b->plans_bytes, fresh.data(), fresh.size(),
                                cudaMemcpyHostToDevice) != cudaSuccess) {
            for (Batch::Plan* p : placed) p->at = -1;
            b->split.ranks = 0;  // the persistent kernel needs none
            return room ? NRLDPC_ERR_CUDA : NRLDPC_OK;
        }
        b->plans_bytes += fresh.size();
    }
    const Batch::Plan& first = b->plans[b->h_jobs[order[0]].code * kSplitSizes + best];
    b->split_count_at = first.at + sizeof(SplitHead) + first.head.o_bytes;
    jobs->resize(n);
    for (int i = 0; i < n; i++) {
        const JobDev& d = b->h_jobs[order[i]];
        (*jobs)[i] = {d.llr_offset, d.out_offset, b->plans[d.code * kSplitSizes + best].at, order[i]};
    }
    return NRLDPC_OK;
}

}  // namespace

extern "C" {

int nrldpc_rm_k0(int bg, int z, int rv) {
    init_z_list();
    if (z_index(z) < 0) return NRLDPC_ERR_BAD_CONFIG;
    const int k = rm_k0(bg, z, rv);
    return k < 0 ? NRLDPC_ERR_INVALID_ARG : k;
}

int nrldpc_batch_create(int device, int max_jobs, float alpha, nrldpc_batch** out) {
    if (!out || max_jobs < 1 || !(alpha > 0.0f)) return NRLDPC_ERR_INVALID_ARG;
    *out = nullptr;
    init_z_list();
    int n_dev = 0;
    if (cudaGetDeviceCount(&n_dev) != cudaSuccess || device < 0 || device >= n_dev) return NRLDPC_ERR_NO_DEVICE;
    cudaSetDevice(device);
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return NRLDPC_ERR_NO_DEVICE;
    Batch* b = new (std::nothrow) Batch();
    if (!b) return NRLDPC_ERR_NO_MEMORY;
    b->device = device;
    b->alpha = alpha;
    b->max_jobs = max_jobs;
    b->sm_count = prop.multiProcessorCount;
    b->smem_optin = prop.sharedMemPerBlockOptin;
    b->smem_sm = prop.sharedMemPerMultiprocessor;
    std::vector<PlanDev> plans(kNumCodes);
    for (int bg = 1; bg <= 2; bg++)
        for (int zi = 0; zi < kNumZ; zi++) {
            const int id = (bg - 1) * kNumZ + zi, z = z_list[zi];
            CodeTable& t = b->h_tables[id];
            EncodePlan ep{};
            b->code_ok[id] = make_nr_table(bg, z, &t) && make_encode_plan(t, &ep);
            PlanDev& pd = plans[id];
            std::memset(&pd, 0, sizeof(pd));
            if (b->code_ok[id]) {
                pd.n_stair = ep.n_stair;
                pd.p0_col = ep.p0_col;
                pd.p0_shift = ep.p0_shift;
                pd.n_steps = ep.n_core_steps;
                for (int k = 0; k < ep.n_core_steps; k++) {
                    pd.step_row[k] = static_cast<uint8_t>(ep.core_row[k]);
                    pd.step_col[k] = static_cast<uint8_t>(ep.core_col[k]);
                }
            }
            // default: one sub-row per thread, as many codewords as 384
            // threads and shared memory allow
            b->spt[id] = 1;
            b->cpb[id] = max_cpb(b, id, 1);
        }
    if (cudaMalloc(&b->d_tables, sizeof(CodeTable) * kNumCodes) != cudaSuccess ||
        cudaMalloc(&b->d_plans, sizeof(PlanDev) * kNumCodes) != cudaSuccess ||
        cudaMalloc(&b->d_lists, kListBytes * max_jobs + 5 * 256) != cudaSuccess ||
        cudaMalloc(&b->d_plans_split, kPlansRoom) != cudaSuccess ||
        cudaMalloc(&b->d_scratch, 256) != cudaSuccess) {
        free_batch(b);
        return NRLDPC_ERR_NO_MEMORY;
    }
    if (cudaMemcpy(b->d_tables, b->h_tables, sizeof(CodeTable) * kNumCodes, cudaMemcpyHostToDevice) ||
        cudaMemcpy(b->d_plans, plans.data(), sizeof(PlanDev) * kNumCodes, cudaMemcpyHostToDevice) ||
        cudaMemset(b->d_scratch, 0, 256) ||
        cudaFuncSetAttribute(batch_decode_kernel_ptr(false), cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(b->smem_optin)) ||
        cudaFuncSetAttribute(batch_decode_kernel_ptr(true), cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(b->smem_optin)) ||
        split_kernel_attributes(b->smem_optin) || uploads_landed()) {
        free_batch(b);
        return NRLDPC_ERR_CUDA;
    }
    if (cudaEventCreateWithFlags(&b->lists_sent, cudaEventDisableTiming) != cudaSuccess ||
        !in_flight_join(&b->in_flight, device)) {
        free_batch(b);
        return NRLDPC_ERR_CUDA;
    }
    *out = reinterpret_cast<nrldpc_batch*>(b);
    return NRLDPC_OK;
}

int nrldpc_batch_destroy(nrldpc_batch* batch) {
    free_batch(reinterpret_cast<Batch*>(batch));
    return NRLDPC_OK;
}

int nrldpc_batch_set_cw_per_cta(nrldpc_batch* batch, int bg, int z, int cpb) {
    Batch* b = reinterpret_cast<Batch*>(batch);
    const int id = b ? code_id(bg, z) : -1;
    if (!b || id < 0 || cpb < 0) return NRLDPC_ERR_INVALID_ARG;
    const int most = max_cpb(b, id, b->spt[id]);
    if (cpb == 0) cpb = most;
    if (cpb > most) return NRLDPC_ERR_BAD_CONFIG;  // threads or shared memory
    b->cpb[id] = cpb;
    return NRLDPC_OK;
}

int nrldpc_batch_set_sub_rows_per_thread(nrldpc_batch* batch, int bg, int z, int spt) {
    Batch* b = reinterpret_cast<Batch*>(batch);
    const int id = b ? code_id(bg, z) : -1;
    if (!b || id < 0 || spt < 0 || spt > 2) return NRLDPC_ERR_INVALID_ARG;
    if (spt == 0) spt = 1;
    if (z % spt != 0) return NRLDPC_ERR_BAD_CONFIG;  // sub-rows s and s + Z/2
    b->spt[id] = spt;
    b->cpb[id] = std::min(b->cpb[id], max_cpb(b, id, spt));
    return NRLDPC_OK;
}

int nrldpc_batch_get_sub_rows_per_thread(nrldpc_batch* batch, int bg, int z, int* spt) {
    Batch* b = reinterpret_cast<Batch*>(batch);
    const int id = b ? code_id(bg, z) : -1;
    if (!b || id < 0 || !spt) return NRLDPC_ERR_INVALID_ARG;
    *spt = b->spt[id];
    return NRLDPC_OK;
}

int nrldpc_batch_get_cw_per_cta(nrldpc_batch* batch, int bg, int z, int* cpb) {
    Batch* b = reinterpret_cast<Batch*>(batch);
    const int id = b ? code_id(bg, z) : -1;
    if (!b || id < 0 || !cpb) return NRLDPC_ERR_INVALID_ARG;
    *cpb = b->cpb[id];
    return NRLDPC_OK;
}

int nrldpc_batch_set_jobs(nrldpc_batch* batch, const nrldpc_job* jobs, int n_jobs) {
    Batch* b = reinterpret_cast<Batch*>(batch);
    if (!b || (n_jobs > 0 && !jobs) || n_jobs < 0) return NRLDPC_ERR_INVALID_ARG;
    if (n_jobs > b->max_jobs) return NRLDPC_ERR_TOO_LARGE;
    cudaSetDevice(b->device);
    b->h_jobs.assign(n_jobs, JobDev{});
    std::vector<int32_t> order(n_jobs);
    int longest = 0;
    for (int i = 0; i < n_jobs; i++) {
        const nrldpc_job& j = jobs[i];
        const int id = code_id(j.bg, j.z);
        if (id < 0 || !b->code_ok[id]) return NRLDPC_ERR_BAD_CONFIG;
        const CodeTable& t = b->h_tables[id];
        const int K = t.kb * t.z, ncb = t.n_bp - 2 * t.z;
        const int kp = j.k_prime ? j.k_prime : K;
        const int qm = j.qm ? j.qm : 1;
        const int e = j.e ? j.e : ncb - (K - kp);
        if (kp <= 2 * t.z || kp > K || j.e < 0 || j.rv < 0 || j.rv > 3 || j.llr_offset < 0 ||
            j.llr_offset % 4 != 0 || j.e_offset < 0 || j.out_offset < 0 ||
            (qm != 1 && qm != 2 && qm != 4 && qm != 6 && qm != 8 && qm != 10) || e % qm != 0)
            return NRLDPC_ERR_INVALID_ARG;
        JobDev& d = b->h_jobs[i];
        d.code = id;
        d.k_prime = kp;
        d.e = e;
        d.qm = qm;
        d.k0 = rm_k0(j.bg, t.z, j.rv);
        d.sigma = j.sigma;
        d.llr_offset = j.llr_offset;
        d.e_offset = j.e_offset;
        d.out_offset = j.out_offset;
        order[i] = i;
        const int nc = ncb - (K - kp);  // positions a bit can land on
        longest = std::max(longest, e > nc ? nc : qm == 1 ? t.n_bp : std::max(e / qm, nc - e));
    }
    // eight CTAs per SM, in parts of at least 256 positions
    b->derate_part = std::max(256, (longest * static_cast<int>(std::min(n_jobs, 8 * b->sm_count)) / (8 * b->sm_count) + 255) / 256 * 256);
    b->derate_parts = std::max(1, (longest + b->derate_part - 1) / b->derate_part);
    // group by code; largest codes first so the tail of the queue is short work
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
        const CodeTable& a = b->h_tables[b->h_jobs[x].code];
        const CodeTable& c = b->h_tables[b->h_jobs[y].code];
        const long wa = static_cast<long>(a.n_edges) * a.z, wc = static_cast<long>(c.n_edges) * c.z;
        if (wa != wc) return wa > wc;
        return b->h_jobs[x].code < b->h_jobs[y].code;
    });
    std::vector<WorkItem> items;
    size_t slot_words = 0, bufs = 0, class_bufs = 0;
    int threads = 32;
    bool classes = true;
    for (int i = 0; i < n_jobs;) {
        const int id = b->h_jobs[order[i]].code;
        int k = i;
        while (k < n_jobs && b->h_jobs[order[k]].code == id) k++;
        const int cpb = b->cpb[id], spt = b->spt[id];
        const CodeTable& t = b->h_tables[id];
        for (int s = i; s < k; s += cpb) {
            const int cnt = std::min(cpb, k - s);
            items.push_back(WorkItem{id, s, cnt, spt});
            threads = std::max(threads, (cnt * (t.z / spt) + 31) / 32 * 32);
            slot_words = std::max(slot_words, static_cast<size_t>(cnt) * 4 * t.rows * t.z);
            bufs = std::max(bufs, group_smem_bytes(t, cnt, 0));
            const uint32_t far = id < kNumZ ? kFarLong : kFarShort;
            class_bufs = std::max(class_bufs, group_smem_bytes(t, cnt, far));
            classes &= spt == 1 && 4l * cnt * t.core_floats <= far;
        }
        i = k;
    }
    b->n_jobs = 0;  // until everything is in place: the list before no longer is
    b->n_items = static_cast<int>(items.size());
    b->slot_words = slot_words;
    b->smem = kHeaderBytesBatch + kBatchTableBytes + bufs;
    b->threads = threads;  // the widest work item's threads
    // the classes' layouts when they cost no resident CTA (as decode_shape)
    const size_t class_smem = kHeaderBytesBatch + kBatchTableBytes + class_bufs;
    b->classes = classes && class_smem <= b->smem_optin &&
                 decode_ctas(threads, class_smem, b->smem_sm) >= decode_ctas(threads, b->smem, b->smem_sm);
    if (b->classes) b->smem = class_smem;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_decode_kernel_ptr(b->classes), b->threads, b->smem);
    b->grid = std::max(1, std::min(b->n_items, std::max(per_sm, 1) * b->sm_count));
    const size_t need = static_cast<size_t>(b->grid) * std::max<size_t>(slot_words, 1);
    if (need > b->state_words) {
        cudaFree(b->d_state);
        b->d_state = nullptr;
        b->state_words = 0;
        if (cudaMalloc(&b->d_state, need * sizeof(uint32_t)) != cudaSuccess) return NRLDPC_ERR_NO_MEMORY;
        b->state_words = need;
    }
    b->split.ranks = 0;
    if (n_jobs == 0) return NRLDPC_OK;
    std::vector<SplitJob> split;
    const int rc = choose_split(b, order, items, &split);
    if (rc) return rc;
    // one copy for all lists
    b->h_lists.clear();
    auto put = [&](const void* p, size_t bytes) {
        const size_t at = b->h_lists.size();
        b->h_lists.resize((at + bytes + 255) / 256 * 256);
        std::memcpy(b->h_lists.data() + at, p, bytes);
        return b->d_lists + at;
    };
    b->d_jobs_rm = reinterpret_cast<JobDev*>(put(b->h_jobs.data(), sizeof(JobDev) * n_jobs));
    b->d_jobs = reinterpret_cast<nrldpc_job*>(put(jobs, sizeof(nrldpc_job) * n_jobs));
    b->d_order = reinterpret_cast<int32_t*>(put(order.data(), sizeof(int32_t) * n_jobs));
    b->d_items = reinterpret_cast<WorkItem*>(put(items.data(), sizeof(WorkItem) * items.size()));
    if (!split.empty()) b->d_split = reinterpret_cast<SplitJob*>(put(split.data(), sizeof(SplitJob) * split.size()));
    if (cudaMemcpy(b->d_lists, b->h_lists.data(), b->h_lists.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaEventRecord(b->lists_sent, cudaStreamLegacy) != cudaSuccess)
        return NRLDPC_ERR_CUDA;
    b->lists_landed = false;
    b->n_jobs = n_jobs;
    return NRLDPC_OK;
}

int nrldpc_batch_gen(nrldpc_batch* batch, uint64_t seed, uint64_t cw_base, float* d_llr_e, uint8_t* d_cw,
                     nrldpc_stream_t stream) {
    Batch* b = reinterpret_cast<Batch*>(batch);
    if (!b || !d_llr_e) return NRLDPC_ERR_INVALID_ARG;
    if (b->n_jobs == 0) return NRLDPC_OK;
    if (wait_lists(b, reinterpret_cast<cudaStream_t>(stream)) != cudaSuccess) return NRLDPC_ERR_CUDA;
    GenBatchArgs g{b->d_tables, b->d_plans, b->d_jobs_rm, d_llr_e, d_cw, seed, cw_base, b->n_jobs};
    const int grid = std::min(b->n_jobs, 8 * b->sm_count);
    batch_gen_kernel<<<grid, 256, kMaxCols * kMaxZ + kMaxZ, reinterpret_cast<cudaStream_t>(stream)>>>(g);
    return map_cuda(cudaGetLastError());
}

int nrldpc_batch_derate(nrldpc_batch* batch, const float* d_llr_e, float* d_llr, nrldpc_stream_t stream) {
    Batch* b = reinterpret_cast<Batch*>(batch);
    if (!b || !d_llr_e || !d_llr) return NRLDPC_ERR_INVALID_ARG;
    if (b->n_jobs == 0) return NRLDPC_OK;
    if (wait_lists(b, reinterpret_cast<cudaStream_t>(stream)) != cudaSuccess) return NRLDPC_ERR_CUDA;
    DerateArgs a{b->d_tables, b->d_jobs_rm, b->d_order, d_llr_e, d_llr, b->n_jobs, b->derate_parts, b->derate_part};
    const int grid = static_cast<int>(std::min<long>(static_cast<long>(b->n_jobs) * b->derate_parts, 8L * b->sm_count));
    batch_derate_kernel<<<grid, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(a);
    return map_cuda(cudaGetLastError());
}

int nrldpc_batch_count_errors(nrldpc_batch* batch, const uint8_t* d_packed, const uint8_t* d_cw,
                              unsigned long long* d_counts, nrldpc_stream_t stream) {
    Batch* b = reinterpret_cast<Batch*>(batch);
    if (!b || !d_packed || !d_cw || !d_counts) return NRLDPC_ERR_INVALID_ARG;
    if (b->n_jobs == 0) return NRLDPC_OK;
    if (wait_lists(b, reinterpret_cast<cudaStream_t>(stream)) != cudaSuccess) return NRLDPC_ERR_CUDA;
    CountArgs a{b->d_tables, b->d_jobs_rm, d_packed, d_cw, d_counts, b->n_jobs};
    const int grid = std::min(b->n_jobs, 8 * b->sm_count);
    batch_count_kernel<<<grid, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(a);
    return map_cuda(cudaGetLastError());
}

int nrldpc_batch_decode(nrldpc_batch* batch, const float* d_llr, uint8_t* d_packed, int n_iter,
                        int early_stop, int32_t* d_iters, nrldpc_stream_t stream) {
    Batch* b = reinterpret_cast<Batch*>(batch);
    if (!b || n_iter < 1 || (early_stop != 0 && early_stop != 1)) return NRLDPC_ERR_INVALID_ARG;
    if (b->n_jobs == 0) return NRLDPC_OK;
    if (!d_llr || !d_packed) return NRLDPC_ERR_INVALID_ARG;
    if (reinterpret_cast<uintptr_t>(d_llr) % 16 != 0) return NRLDPC_ERR_ALIGNMENT;
    if (wait_lists(b, reinterpret_cast<cudaStream_t>(stream)) != cudaSuccess) return NRLDPC_ERR_CUDA;
    // clusters while they and those of as many lists like this one as other
    // decoders are busy have the GPU's SMs, the queue kernel else
    if (b->split.ranks &&
        static_cast<long>(b->n_jobs) * b->split.ranks *
                in_flight_others(&b->in_flight, reinterpret_cast<cudaStream_t>(stream),
                                 static_cast<long>(b->n_jobs) * b->split.ranks, b->sm_count) <= b->sm_count) {
        SplitArgs a = split_args(b, d_llr, d_packed, n_iter);
        a.iters = d_iters;
        a.early_stop = early_stop;
        const int rc =
            map_cuda(launch_split(b->split, a, nullptr, b->split_clusters, reinterpret_cast<cudaStream_t>(stream)));
        in_flight_note(&b->in_flight, reinterpret_cast<cudaStream_t>(stream));
        return rc;
    }
    BatchDecodeArgs& k = b->kargs;
    k.tables = b->d_tables;
    k.items = b->d_items;
    k.order = b->d_order;
    k.jobs = b->d_jobs;
    k.llr = d_llr;
    k.packed = d_packed;
    k.iters = d_iters;
    k.state = b->d_state;
    k.work_counter = b->d_scratch;
    k.error_flag = b->d_scratch + 1;
    k.slot_words = b->slot_words;
    k.n_items = b->n_items;
    k.n_iter = n_iter;
    k.early_stop = early_stop;
    k.alpha = b->alpha;
    void* params[1] = {&k};
    if (cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
        is_captured(st, cudaPeekAtLastError() != cudaSuccess)) {
        // a graph launch cannot be captured, what it does can
        if (cudaMemsetAsync(b->d_scratch, 0, sizeof(int), st) != cudaSuccess) return NRLDPC_ERR_CUDA;
        return map_cuda(cudaLaunchKernel(batch_decode_kernel_ptr(b->classes), dim3(b->grid), dim3(b->threads), params,
                                         b->smem, st));
    }
    cudaKernelNodeParams kp{};
    kp.func = const_cast<void*>(batch_decode_kernel_ptr(b->classes));
    kp.gridDim = dim3(b->grid);
    kp.blockDim = dim3(b->threads);
    kp.sharedMemBytes = static_cast<unsigned int>(b->smem);
    kp.kernelParams = params;
    if (!b->exec) {  // memset of the queue head, then the persistent kernel
        cudaMemsetParams mp{};
        mp.dst = b->d_scratch;
        mp.value = 0;
        mp.elementSize = 4;
        mp.width = 1;
        mp.height = 1;
        cudaGraphNode_t mnode;
        if (cudaGraphCreate(&b->graph, 0) || cudaGraphAddMemsetNode(&mnode, b->graph, nullptr, 0, &mp) ||
            cudaGraphAddKernelNode(&b->knode, b->graph, &mnode, 1, &kp) ||
            cudaGraphInstantiate(&b->exec, b->graph, 0)) {
            drop_graph(b);
            return NRLDPC_ERR_CUDA;
        }
    } else if (cudaGraphExecKernelNodeSetParams(b->exec, b->knode, &kp) != cudaSuccess) {
        return NRLDPC_ERR_CUDA;
    }
    const int rc = map_cuda(cudaGraphLaunch(b->exec, reinterpret_cast<cudaStream_t>(stream)));
    in_flight_note(&b->in_flight, reinterpret_cast<cudaStream_t>(stream));
    return rc;
}

int nrldpc_batch_set_neighbours(nrldpc_batch* batch, int n) {
    Batch* b = reinterpret_cast<Batch*>(batch);
    if (!b || n < -1) return NRLDPC_ERR_INVALID_ARG;
    b->in_flight.neighbours = n;
    return NRLDPC_OK;
}

int nrldpc_batch_device_error(nrldpc_batch* batch) {
    Batch* b = reinterpret_cast<Batch*>(batch);
    if (!b) return NRLDPC_ERR_INVALID_ARG;
    int v = 0;
    if (cudaMemcpy(&v, b->d_scratch + 1, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return NRLDPC_ERR_CUDA;
    if (v) cudaMemset(b->d_scratch + 1, 0, sizeof(int));
    return v ? NRLDPC_ERR_TIMEOUT : NRLDPC_OK;
}

int nrldpc_selftest_batch_timeout(nrldpc_batch* batch, const float* d_llr, uint8_t* d_packed,
                                  nrldpc_stream_t stream) {
    Batch* b = reinterpret_cast<Batch*>(batch);
    if (!b || !d_llr || !d_packed) return NRLDPC_ERR_INVALID_ARG;
    if (reinterpret_cast<uintptr_t>(d_llr) % 16 != 0) return NRLDPC_ERR_ALIGNMENT;
    if (b->n_jobs == 0 || !b->split.ranks || !split_counts(b->split, 0)) return NRLDPC_ERR_BAD_CONFIG;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (wait_lists(b, st) != cudaSuccess) return NRLDPC_ERR_CUDA;
    return map_cuda(launch_split_timeout(b->split, split_args(b, d_llr, d_packed, 2),
                                         b->d_plans_split + b->split_count_at, b->split_clusters, st));
}

}  // extern "C"
