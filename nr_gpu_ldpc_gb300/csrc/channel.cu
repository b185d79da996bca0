// Seeded channel simulation on the GPU: info bits, structural QC encoder,
// BPSK, AWGN and LLRs, plus an info-bit error counter.
//
// No reference counterpart on the GPU: the reference builds its inputs on the
// host (src/encoding_tools.cpp:13-99 with the OAI encoder).  This generator
// keeps the reference's signal model -- BPSK 0 -> +1, y = x + noise*sigma
// (src/encoding_tools.cpp:62), LLR = (2y)/(sigma*sigma) with the first 2Z
// columns punctured to 0 (src/encoding_tools.cpp:85-99) -- and draws its
// randomness from Philox4x32-10 (Salmon et al., SC'11) keyed by
// (seed, codeword id), with Gaussians by Box-Muller using log / sin / cos
// evaluated from +, -, *, / and sqrt only.  Every float operation is an
// explicit round-to-nearest intrinsic in the same order as the CPU oracle's
// C code, so both produce the same bits.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <vector>

#include "channel_dev.cuh"
#include "nrldpc_internal.h"

namespace nrldpc {
namespace {
using namespace dev;

struct GenArgs {
    uint64_t seed, cw_base;
    const float* sigma;
    float* llr;
    uint8_t* cw_packed;
    int n_cw, n_punct_cols;
    int n_stair, p0_col, p0_shift, n_core_steps;
    uint8_t step_row[kMaxRows];
    uint8_t step_col[kMaxRows];
};

// One CTA per codeword (grid-stride over codewords).
__global__ void __launch_bounds__(256) gen_llr_kernel(const __grid_constant__ CodeTable tab,
                                                      const __grid_constant__ GenArgs g) {
    extern __shared__ uint8_t x[];  // [n_bp] codeword bits, then [z] scratch
    const int z = tab.z, n = tab.n_bp, K = tab.kb * z;
    uint8_t* acc = x + n;
    const uint32_t k0 = static_cast<uint32_t>(g.seed), k1 = static_cast<uint32_t>(g.seed >> 32);
    for (int i = blockIdx.x; i < g.n_cw; i += gridDim.x) {
        const uint64_t id = g.cw_base + static_cast<uint64_t>(i);
        const uint32_t id0 = static_cast<uint32_t>(id), id1 = static_cast<uint32_t>(id >> 32);
        // info bits: block b holds bits 128b .. 128b+127
        for (int b = threadIdx.x; b * 128 < K; b += blockDim.x) {
            uint32_t o[4];
            philox4x32(static_cast<uint32_t>(b), id0, id1, 1u, k0, k1, o);
            for (int j = 0; j < 128 && b * 128 + j < K; j++) x[b * 128 + j] = (o[j >> 5] >> (j & 31)) & 1u;
        }
        __syncthreads();
        encode_in_smem(tab, g.n_stair, g.p0_col, g.p0_shift, g.n_core_steps, g.step_row, g.step_col, x,
                       acc);
        if (g.cw_packed) {
            uint8_t* out = g.cw_packed + static_cast<size_t>(i) * tab.packed_bytes;
            for (int b = threadIdx.x; b < tab.packed_bytes; b += blockDim.x) {
                uint32_t v = 0;
                for (int j = 0; j < 8; j++)
                    if (8 * b + j < n) v |= static_cast<uint32_t>(x[8 * b + j]) << j;
                out[b] = static_cast<uint8_t>(v);
            }
        }
        const float sg = g.sigma[i];
        const float s2 = __fmul_rn(sg, sg);
        const int p0 = g.n_punct_cols * z;
        float* out = g.llr + static_cast<size_t>(i) * n;
        for (int j = threadIdx.x; j < p0; j += blockDim.x) out[j] = 0.0f;
        const int n_blk = (n - p0 + 3) / 4;
        for (int t = threadIdx.x; t < n_blk; t += blockDim.x) {
            uint32_t o[4];
            philox4x32(static_cast<uint32_t>(t), id0, id1, 2u, k0, k1, o);
            float gs[4];
            gauss4(o, gs);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int j = p0 + 4 * t + k;
                if (j >= n) break;
                out[j] = bpsk_llr(x[j], gs[k], sg, s2);
            }
        }
        __syncthreads();  // x is rewritten for the next codeword
    }
}

__global__ void __launch_bounds__(256) count_errors_kernel(const uint8_t* __restrict__ packed,
                                                           const uint8_t* __restrict__ cw,
                                                           int n_cw, int packed_bytes, int n_info,
                                                           unsigned long long* counts) {
    __shared__ unsigned int warp_sum[8];
    for (int i = blockIdx.x; i < n_cw; i += gridDim.x) {
        const uint8_t* a = packed + static_cast<size_t>(i) * packed_bytes;
        const uint8_t* b = cw + static_cast<size_t>(i) * packed_bytes;
        unsigned int errs = 0;
        const int full = n_info / 8, rem = n_info % 8;
        for (int k = threadIdx.x; k < full; k += blockDim.x) errs += __popc(a[k] ^ b[k]);
        if (rem && threadIdx.x == 0) errs += __popc((a[full] ^ b[full]) & ((1u << rem) - 1u));
        for (int off = 16; off > 0; off >>= 1) errs += __shfl_down_sync(0xffffffffu, errs, off);
        if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = errs;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned int tot = 0;
            for (int w = 0; w < (blockDim.x + 31) / 32; w++) tot += warp_sum[w];
            if (tot) {
                atomicAdd(&counts[0], static_cast<unsigned long long>(tot));
                atomicAdd(&counts[1], 1ull);
            }
        }
        __syncthreads();
    }
}

// CRC of a bit string by one warp: each lane divides its own stretch of whole
// bytes (256-entry table in shared memory), and stretches of equal length,
// zeros in front of the first, are joined pairwise -- the left remainder
// times x^(bits of the right) -- with the factors of CrcArgs; lane 0 then
// takes the last n_bits % 8 bits.  MSB-first long division: bit i of the
// packed bytes is the coefficient of D^(n-1-i).  One thread per codeword
// instead (the serial division) took 43 us for 8,424 bits, and 138 us bit by
// bit in the CRC attachment, whatever the number of codewords.
struct CrcArgs {
    uint32_t poly, mask, top;
    int len, n_bits, per_lane;  // bytes per lane
    uint32_t join[5];           // x^(8 per_lane 2^k) mod the polynomial
};

__host__ __device__ inline uint32_t crc_times(uint32_t a, uint32_t b, uint32_t poly, uint32_t mask, uint32_t top) {
    uint32_t r = 0;
    for (uint32_t bit = top; bit; bit >>= 1) {  // Horner over b's coefficients
        r = ((r & top) ? ((r << 1) ^ poly) : (r << 1)) & mask;
        if (b & bit) r ^= a;
    }
    return r;
}

CrcArgs crc_args(uint32_t poly, int len, int n_bits) {
    CrcArgs c{};
    c.poly = poly;
    c.len = len;
    c.n_bits = n_bits;
    c.mask = len >= 32 ? 0xffffffffu : (1u << len) - 1u;
    c.top = 1u << (len - 1);
    c.per_lane = (n_bits / 8 + 31) / 32;
    uint32_t x8 = 1u << 8, f = 1u;  // lengths are above 8
    for (int k = c.per_lane; k; k >>= 1) {
        if (k & 1) f = crc_times(f, x8, poly, c.mask, c.top);
        x8 = crc_times(x8, x8, poly, c.mask, c.top);
    }
    for (uint32_t& j : c.join) {
        j = f;
        f = crc_times(f, f, poly, c.mask, c.top);
    }
    return c;
}

__device__ __forceinline__ void crc_table(const CrcArgs& c, uint32_t* table) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
        uint32_t r = static_cast<uint32_t>(i) << (c.len - 8);
        for (int k = 0; k < 8; k++) r = ((r & c.top) ? ((r << 1) ^ c.poly) : (r << 1)) & c.mask;
        table[i] = r;
    }
}

// Remainder in lane 0; every lane of the warp calls it.
__device__ __forceinline__ uint32_t warp_crc(const CrcArgs& c, const uint32_t* table, const uint8_t* p) {
    const int lane = static_cast<int>(threadIdx.x & 31u), nb = c.n_bits / 8;
    const int first = nb - (32 - lane) * c.per_lane;  // below 0: zeros
    uint32_t r = 0;
    for (int k = 0; k < c.per_lane; k += 8) {
        uint32_t v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int b = first + k + i;
            v[i] = (k + i < c.per_lane && b >= 0) ? __brev(static_cast<uint32_t>(p[b])) >> 24 : 0u;
        }
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (k + i < c.per_lane) r = ((r << 8) ^ table[((r >> (c.len - 8)) ^ v[i]) & 0xffu]) & c.mask;
    }
#pragma unroll
    for (int k = 0; k < 5; k++) {  // the lane's stretch is the left one of its pair
        const uint32_t right = __shfl_down_sync(0xffffffffu, r, 1 << k);
        r = crc_times(r, c.join[k], c.poly, c.mask, c.top) ^ right;
    }
    for (int i = nb * 8; i < c.n_bits; i++) {
        const uint32_t fb = ((r & c.top) != 0) ^ ((p[i >> 3] >> (i & 7)) & 1u);
        r = (r << 1) & c.mask;
        if (fb) r ^= c.poly;
    }
    return r;
}

// One warp per codeword.
__global__ void __launch_bounds__(256) crc_kernel(const uint8_t* __restrict__ packed, int n_cw, int stride,
                                                  const __grid_constant__ CrcArgs c, uint32_t* __restrict__ rem) {
    __shared__ uint32_t table[256];
    crc_table(c, table);
    __syncthreads();
    const int cw = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    if (cw >= n_cw) return;
    const uint32_t r = warp_crc(c, table, packed + static_cast<size_t>(cw) * stride);
    if ((threadIdx.x & 31u) == 0) rem[cw] = r;
}

// Widen transferred LLRs to fp32: qtype 1 = IEEE half (exact), 2 = int8
// times `scale` (one rounding, the product).
__global__ void __launch_bounds__(256) dequant_kernel(const void* __restrict__ in, int qtype,
                                                      float scale, size_t n, float* __restrict__ out) {
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        if (qtype == 1)
            out[i] = __half2float(__ushort_as_half(static_cast<const unsigned short*>(in)[i]));
        else
            out[i] = __fmul_rn(static_cast<float>(static_cast<const int8_t*>(in)[i]), scale);
    }
}

}  // namespace

cudaError_t launch_dequant(const void* in, int qtype, float scale, size_t n, float* out,
                           cudaStream_t stream) {
    const size_t blocks = (n + 255) / 256;
    dequant_kernel<<<static_cast<unsigned>(blocks < 4096 ? blocks : 4096), 256, 0, stream>>>(in, qtype, scale,
                                                                                             n, out);
    return cudaGetLastError();
}

// ---- code-block segmentation (TS 38.212 5.2.2) ------------------------------------
// One CTA per code block.  Its bytes: byte j holds transport-block bits
// r*data_bits + 8j .. + 7, zero at or past data_bits; then its first warp
// divides them and writes the remainder behind the data, MSB first (parity
// bit p_0 = remainder bit len-1), so that the remainder over all k_prime bits
// is 0.  One launch for both: the two kernels it replaces took 3 + 138 us for
// 26 blocks.
__global__ void __launch_bounds__(256) cb_segment_kernel(const uint8_t* __restrict__ tb, int C, int data_bits,
                                                         int k_prime, uint8_t* blocks, int stride, bool attach,
                                                         const __grid_constant__ CrcArgs c) {
    __shared__ uint32_t table[256];
    if (attach) crc_table(c, table);
    const int r = blockIdx.x;
    uint8_t* p = blocks + static_cast<size_t>(r) * stride;
    const long from = static_cast<long>(r) * data_bits, tb_bytes = (static_cast<long>(C) * data_bits + 7) / 8;
    const int nbytes = (k_prime + 7) / 8;
    for (int j = threadIdx.x; j < nbytes; j += blockDim.x) {
        const int left = data_bits - 8 * j;  // data bits from this byte on
        uint32_t v = 0;
        if (left > 0) {
            const long t = from + 8 * j;
            const int sh = static_cast<int>(t & 7);
            v = tb[t >> 3] >> sh;
            if (sh && (t >> 3) + 1 < tb_bytes) v |= static_cast<uint32_t>(tb[(t >> 3) + 1]) << (8 - sh);
            v &= left >= 8 ? 0xffu : (1u << left) - 1u;
        }
        p[j] = static_cast<uint8_t>(v);
    }
    if (!attach) return;
    __syncthreads();
    if (threadIdx.x >= 32) return;
    const uint32_t rem = __shfl_sync(0xffffffffu, warp_crc(c, table, p), 0);
    const int b = data_bits / 8 + static_cast<int>(threadIdx.x);
    if (b <= (data_bits + c.len - 1) / 8) {
        uint32_t v = threadIdx.x == 0 ? p[b] : 0u;  // data bits of the byte the CRC starts in
        for (int i = 0; i < 8; i++) {
            const int k = 8 * b + i - data_bits;  // place in the CRC
            if (k >= 0 && k < c.len) v |= ((rem >> (c.len - 1 - k)) & 1u) << i;
        }
        p[b] = static_cast<uint8_t>(v);
    }
}

// One thread per transport-block byte (bit t comes from block t / data_bits),
// and with check one warp per block for its remainder over all k_prime bits.
__global__ void __launch_bounds__(256) cb_desegment_kernel(const uint8_t* __restrict__ blocks, int stride, int C,
                                                           int data_bits, uint8_t* __restrict__ tb, bool check,
                                                           const __grid_constant__ CrcArgs c,
                                                           uint32_t* __restrict__ rem) {
    __shared__ uint32_t table[256];
    const int warps = blockDim.x / 32, cw = blockIdx.x * warps + static_cast<int>(threadIdx.x >> 5);
    if (check && static_cast<long>(blockIdx.x) * warps < C) {
        crc_table(c, table);
        __syncthreads();
        if (cw < C) {
            const uint32_t r = warp_crc(c, table, blocks + static_cast<size_t>(cw) * stride);
            if ((threadIdx.x & 31u) == 0) rem[cw] = r;
        }
    }
    const long total = static_cast<long>(C) * data_bits;
    const long j = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
    if (j >= (total + 7) / 8) return;
    const long t0 = 8 * j;
    const int r0 = static_cast<int>(t0 / data_bits);
    int k = static_cast<int>(t0 - static_cast<long>(r0) * data_bits);
    const uint8_t* p = blocks + static_cast<size_t>(r0) * stride;
    uint32_t v = 0;
    for (int i = 0; i < 8 && t0 + i < total; i++) {
        v |= ((p[k >> 3] >> (k & 7)) & 1u) << i;
        if (++k == data_bits) {
            k = 0;
            p += stride;
        }
    }
    tb[j] = static_cast<uint8_t>(v);
}

cudaError_t launch_crc(const uint8_t* packed, int n_cw, int stride, int n_bits, uint32_t poly, int len,
                       uint32_t* rem, cudaStream_t stream) {
    crc_kernel<<<(n_cw + 7) / 8, 256, 0, stream>>>(packed, n_cw, stride, crc_args(poly, len, n_bits), rem);
    return cudaGetLastError();
}

// Staircase encoding plan (host): see the oracle's structural encoder.
bool make_encode_plan(const CodeTable& tab, EncodePlan* plan) {
    const int z = tab.z, kb = tab.kb;
    std::vector<int> col_deg(tab.cols, 0);
    for (int e = 0; e < tab.n_edges; e++) col_deg[tab.edge_col[e]]++;
    int m = 0;
    for (int r = 0; r < tab.rows; r++) {
        const int last = tab.edge_col[tab.row_ptr[r + 1] - 1];
        if (col_deg[last] == 1 && r > 0) break;
        m = r + 1;
    }
    std::vector<int> cnt(z, 0);
    for (int r = 0; r < m; r++)
        for (int e = tab.row_ptr[r]; e < tab.row_ptr[r + 1]; e++)
            if (tab.edge_col[e] == kb) cnt[tab.edge_shift[e]]++;
    int v_odd = -1;
    for (int v = 0; v < z; v++)
        if (cnt[v] & 1) {
            if (v_odd >= 0) return false;
            v_odd = v;
        }
    if (v_odd < 0) return false;
    std::vector<int> solved(tab.cols, 0);
    for (int j = 0; j <= kb && j < tab.cols; j++) solved[j] = 1;
    int n = 0;
    for (int r = 0; r < tab.rows; r++) {
        if (r == m - 1) continue;
        int unknown = -1;
        for (int e = tab.row_ptr[r]; e < tab.row_ptr[r + 1]; e++) {
            const int j = tab.edge_col[e];
            if (solved[j]) continue;
            if (unknown < 0 && tab.edge_shift[e] == 0) unknown = j;
            else return false;
        }
        if (unknown < 0) continue;
        solved[unknown] = 1;
        plan->core_row[n] = r;
        plan->core_col[n] = unknown;
        n++;
    }
    for (int j = 0; j < tab.cols; j++)
        if (!solved[j]) return false;
    plan->n_core_steps = n;
    plan->p0_col = kb;
    plan->p0_shift = v_odd;
    plan->n_stair = m;
    return true;
}

cudaError_t launch_gen_llr(const CodeTable& tab, const EncodePlan& plan, uint64_t seed,
                           uint64_t cw_base, int n_cw, const float* sigma, int n_punct_cols,
                           float* llr, uint8_t* cw_packed, cudaStream_t stream) {
    GenArgs g{};
    g.seed = seed;
    g.cw_base = cw_base;
    g.sigma = sigma;
    g.llr = llr;
    g.cw_packed = cw_packed;
    g.n_cw = n_cw;
    g.n_punct_cols = n_punct_cols;
    g.n_stair = plan.n_stair;
    g.p0_col = plan.p0_col;
    g.p0_shift = plan.p0_shift;
    g.n_core_steps = plan.n_core_steps;
    for (int k = 0; k < plan.n_core_steps; k++) {
        g.step_row[k] = static_cast<uint8_t>(plan.core_row[k]);
        g.step_col[k] = static_cast<uint8_t>(plan.core_col[k]);
    }
    const int grid = n_cw < 4096 ? n_cw : 4096;
    const size_t smem = static_cast<size_t>(tab.n_bp) + tab.z;
    gen_llr_kernel<<<grid, 256, smem, stream>>>(tab, g);
    return cudaGetLastError();
}

cudaError_t launch_count_errors(const uint8_t* packed, const uint8_t* cw_packed, int n_cw,
                                int packed_bytes, int n_info, unsigned long long* counts,
                                cudaStream_t stream) {
    const int grid = n_cw < 4096 ? n_cw : 4096;
    count_errors_kernel<<<grid, 256, 0, stream>>>(packed, cw_packed, n_cw, packed_bytes, n_info,
                                                  counts);
    return cudaGetLastError();
}

}  // namespace nrldpc

namespace nrldpc {
cudaError_t launch_cb_segment(const uint8_t* tb, int C, int data_bits, int k_prime, uint8_t* blocks, int stride,
                              uint32_t poly, int len, cudaStream_t stream) {
    cb_segment_kernel<<<C, 256, 0, stream>>>(tb, C, data_bits, k_prime, blocks, stride, len > 0,
                                             len > 0 ? crc_args(poly, len, data_bits) : CrcArgs{});
    return cudaGetLastError();
}
cudaError_t launch_cb_desegment(const uint8_t* blocks, int stride, int C, int data_bits, int k_prime, uint8_t* tb,
                                uint32_t poly, int len, uint32_t* rem, cudaStream_t stream) {
    const long bytes = (static_cast<long>(C) * data_bits + 7) / 8;
    const long warps = len > 0 ? (C + 7) / 8 : 0;
    const long grid = (bytes + 255) / 256 > warps ? (bytes + 255) / 256 : warps;
    cb_desegment_kernel<<<static_cast<unsigned>(grid), 256, 0, stream>>>(blocks, stride, C, data_bits, tb, len > 0,
                                                                         len > 0 ? crc_args(poly, len, k_prime)
                                                                                 : CrcArgs{},
                                                                         rem);
    return cudaGetLastError();
}
}  // namespace nrldpc
