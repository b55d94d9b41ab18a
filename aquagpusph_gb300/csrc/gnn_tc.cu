// Dense-layer forward of the learned proposal on the 5th-generation tensor
// cores: Y = act(X W^T + b) with tcgen05.mma (kind::f16, BF16 x BF16 ->
// FP32) accumulating in tensor memory.  No counterpart in the reference.
//
// One CTA of 128 threads works on tiles of 128 rows:
//   - W (N x K) is staged once in shared memory, X tiles (128 x K) per tile,
//     both in the K-major layout without swizzle: 8-row x 16-byte core
//     matrices, consecutive along K (leading byte offset 128 B), row groups
//     K/8 core matrices apart (stride byte offset);
//   - thread 0 issues K/16 MMAs of 128 x N x 16 into an N-column TMEM
//     accumulator and commits them to an mbarrier;
//   - every warp reads its 32 TMEM lanes (rows) back with tcgen05.ld, adds
//     the bias, applies the activation and stores Z (f32) and / or Y (bf16).
// Every wait on the mbarrier is bounded: on time-out the kernel records
// an error, skips the tile's stores, frees its TMEM and returns.
#include <cuda_bf16.h>
#include <atomic>
#include <cstdint>

#include "aqua_learned.h"
#include "arith.cuh"

namespace aqua {
// test-only switch of aqua_debug_fake_timeouts() (api.cu)
extern int g_debug_fake_timeout;
}  // namespace aqua

namespace {

constexpr int kTcThreads = 128;
constexpr int kTcRows = 128;
constexpr uint32_t kWaitLimit = 1u << 22;

// bytes of a 128 x K operand tile that the epilogue reuses: 4 KB per warp
inline size_t
tc_operand_bytes(uint32_t K)
{
    const size_t tile = (size_t)kTcRows * K * 2, out = (size_t)kTcThreads / 32 * 4096;
    return tile > out ? tile : out;
}

__device__ __forceinline__ uint32_t
smem_addr(const void* p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

// shared-memory matrix descriptor: K-major, no swizzle
__device__ __forceinline__ uint64_t
make_desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo & 0x3FFFFu) >> 4) << 16;
    d |= (uint64_t)((sbo & 0x3FFFFu) >> 4) << 32;
    d |= (uint64_t)1 << 46;  // descriptor version of tcgen05
    return d;                // base offset 0, swizzle none
}

// instruction descriptor of kind::f16: D f32, A and B bf16, both K-major,
// M = 128, N = n
__host__ __device__ constexpr uint32_t
make_idesc(uint32_t n)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) |
           ((uint32_t)(kTcRows >> 4) << 24);
}

// SiLU of two bf16 values (a packed pair) in packed bf16 arithmetic:
// z * sigmoid(z), sigmoid(z) = (1 + tanh(z / 2)) / 2 on the hardware tanh
// (tanh.approx.bf16x2); four instructions for the pair, each result
// rounded to bf16
__device__ __forceinline__ uint32_t
silu_bf16x2(uint32_t z)
{
    const uint32_t half = 0x3f003f00u;  // 0.5 in both halves
    uint32_t h, t, s, y;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(h) : "r"(z), "r"(half));
    asm("tanh.approx.bf16x2 %0, %1;" : "=r"(t) : "r"(h));
    asm("fma.rn.bf16x2 %0, %1, %2, %2;" : "=r"(s) : "r"(t), "r"(half));
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(y) : "r"(z), "r"(s));
    return y;
}

// two floats rounded to bf16 (round to nearest even), lo in the low half
__device__ __forceinline__ uint32_t
pack2(float lo, float hi)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// Starts asynchronous copies of a rows x K bf16 block (row-major, ld elements,
// rows a multiple of 8, K of 16) into core matrices of 8 rows x 16 bytes:
// element (r, k) goes to (r / 8) * row_step + (k / 8) * col_step + (r % 8) * 16
// + (k % 8) * 2; rows past `valid` are filled with zeros.  Eight consecutive
// lanes fill one core matrix (128 contiguous bytes, no bank conflict) and
// sixteen read whole 32-byte sectors of eight rows.
__device__ __forceinline__ void
stage_async(uint8_t* dst, const uint16_t* src, uint32_t ld, uint32_t rows,
            uint32_t valid, uint32_t K, uint32_t row_step, uint32_t col_step)
{
    const uint32_t r8 = threadIdx.x & 7, h = (threadIdx.x >> 3) & 1;
    const uint32_t pairs = K / 16, tasks = rows / 8 * pairs;
    const uint32_t step = blockDim.x / 16;
    // (row block, pair of column groups) of this half-warp's next task
    uint32_t rb = (threadIdx.x >> 4) / pairs, pr = (threadIdx.x >> 4) % pairs;
    const uint32_t drb = step / pairs, dpr = step % pairs;
    for (uint32_t t = threadIdx.x >> 4; t < tasks; t += step) {
        const uint32_t g = pr * 2 + h;
        const uint32_t r = rb * 8 + r8;
        const bool ok = r < valid;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n"
                     :: "r"(smem_addr(dst + rb * row_step + g * col_step + r8 * 16)),
                        "l"(src + (size_t)(ok ? r : 0u) * ld + g * 8), "r"(ok ? 16u : 0u)
                     : "memory");
        rb += drb;
        pr += dpr;
        if (pr >= pairs) {
            pr -= pairs;
            rb++;
        }
    }
}

__device__ __forceinline__ void
stage_wait()
{
    asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// K-major operand: rows x K with consecutive core matrices along K
__device__ __forceinline__ void
stage(uint8_t* dst, const uint16_t* src, uint32_t ld, uint32_t rows,
      uint32_t valid, uint32_t K)
{
    stage_async(dst, src, ld, rows, valid, K, K / 8 * 128, 128);
    stage_wait();
}

// One warp's 32 rows x 128 bytes in shared memory, 16-byte chunk c of row r
// at chunk c ^ (r % 8): a lane writes or reads its own row, or a warp whole
// rows of global memory (4 per instruction), either way without bank
// conflicts.  Rows of 64 bytes (32 bf16) use chunks 0-3 in the same way.
__device__ __forceinline__ uint4*
warp_chunk(uint8_t* buf, uint32_t r, uint32_t c)
{
    return reinterpret_cast<uint4*>(buf + r * 128 + ((c ^ (r & 7)) * 16));
}

// Copies `chunks` (2, 4 or 8) 16-byte chunks of each of the warp's rows to
// global memory: row r at g + r * ld bytes, r < valid
__device__ __forceinline__ void
warp_store_rows(uint8_t* buf, uint8_t* g, size_t ld, uint32_t valid,
                uint32_t chunks)
{
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t per = 32 / chunks, c = lane % chunks;
    for (uint32_t r = lane / chunks; r < 32; r += per)
        if (r < valid)
            *reinterpret_cast<uint4*>(g + r * ld + c * 16) = *warp_chunk(buf, r, c);
}

// 32 columns of the warp's 32 tensor-memory lanes
__device__ __forceinline__ void
ld_tmem32(uint32_t addr, float (&z)[32])
{
    uint32_t v[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]),
          "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
          "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
          "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),
          "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]),
          "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]),
          "=r"(v[31])
        : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n");
#pragma unroll
    for (int j = 0; j < 32; j++)
        z[j] = __uint_as_float(v[j]);
}

// Bound by memory: a row of 64 inputs with both outputs moves 512 bytes.
// Rows leave through shared memory (stores of whole rows): with each lane
// storing 16 bytes of its own row the load / store unit was 72% busy and
// 10.3M rows took 1.82 ms; now 0.90.
template<int N>
__global__ void __launch_bounds__(kTcThreads, 1)
k_linear_fwd_tc(uint32_t M, uint32_t K, const uint16_t* __restrict__ X,
                uint32_t ldx, const uint16_t* __restrict__ W,
                const float* __restrict__ bias, float* Z, uint32_t ldz,
                uint16_t* Y, uint32_t ldy, int act, int* err, uint32_t fake)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_base;
    __shared__ __align__(16) float sbias[N];
    uint8_t* sB = smem;                                // N x K
    // 128 x K, and 4 KB per warp for the outputs
    uint8_t* sA = smem + ((N * K * 2 + 1023) / 1024) * 1024;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x < N)
        sbias[threadIdx.x] = bias ? bias[threadIdx.x] : 0.f;

    stage(sB, W, K, N, N, K);
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n"
                     :: "r"(smem_addr(&mbar)));
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 "
                     "[%0], %1;\n" :: "r"(smem_addr(&tmem_base)), "r"((uint32_t)N));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    const uint32_t tmem = tmem_base;
    const uint32_t idesc = make_idesc(N);
    const uint32_t kg = K / 8;
    const uint32_t sbo = kg * 128;  // next 8-row group
    uint32_t phase = 0;
    bool failed = false;
    const uint32_t tiles = (M + kTcRows - 1) / kTcRows;
    for (uint32_t tile = blockIdx.x; tile < tiles && !failed; tile += gridDim.x) {
        const uint32_t m0 = tile * kTcRows;
        const uint32_t valid = min((uint32_t)kTcRows, M - m0);
        stage(sA, X + (size_t)m0 * ldx, ldx, kTcRows, valid, K);
        // generic-proxy stores -> visible to the tensor core (async proxy)
        asm volatile("fence.proxy.async.shared::cta;\n");
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;\n");
            for (uint32_t ks = 0; ks < K / 16; ks++) {
                const uint64_t ad = make_desc(smem_addr(sA) + ks * 256, 128, sbo);
                const uint64_t bd = make_desc(smem_addr(sB) + ks * 256, 128, sbo);
                const uint32_t acc = ks > 0 ? 1u : 0u;
                asm volatile(
                    "{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\n"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                    :: "r"(tmem), "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one."
                         "shared::cluster.b64 [%0];\n" :: "r"(smem_addr(&mbar)));
        }
        // bounded wait for the MMAs of this tile
        uint32_t done = 0;
        for (uint32_t it = 0; it < kWaitLimit && !done; it++) {
            asm volatile("{\n.reg .pred p;\n"
                         "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                         "selp.u32 %0, 1, 0, p;\n}\n"
                         : "=r"(done) : "r"(smem_addr(&mbar)), "r"(phase));
        }
        // `fake` (test switch): a wait that completed counts as timed out
        if (!__all_sync(0xffffffffu, done) || fake) {
            failed = true;
            if (lane == 0)
                atomicExch(err, 1);
        }
        failed = __syncthreads_or(failed);
        if (failed)
            break;
        phase ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;\n");
        // epilogue: warp w owns rows 32w .. 32w + 31 (TMEM lanes)
        // 32 columns at a time, through the warp's rows of the operand buffer
        // (its MMAs have completed) so that they leave as whole rows
        const uint32_t row0 = m0 + warp * 32;
        const uint32_t wvalid = row0 < M ? min(32u, M - row0) : 0u;
        const uint32_t taddr = tmem + ((warp * 32u) << 16);
        uint8_t* wbuf = sA + warp * 4096;
#pragma unroll
        for (int c0 = 0; c0 < N; c0 += 32) {
            float z[32];
            ld_tmem32(taddr + (uint32_t)c0, z);
            if (bias)
                for (int j = 0; j < 32; j += 4) {
                    const float4 b4 = *reinterpret_cast<const float4*>(sbias + c0 + j);
                    z[j] += b4.x;
                    z[j + 1] += b4.y;
                    z[j + 2] += b4.z;
                    z[j + 3] += b4.w;
                }
            if (Z) {
                __syncwarp();
                for (int j = 0; j < 8; j++)
                    *reinterpret_cast<float4*>(warp_chunk(wbuf, lane, j)) =
                        make_float4(z[4 * j], z[4 * j + 1], z[4 * j + 2], z[4 * j + 3]);
                __syncwarp();
                warp_store_rows(wbuf, reinterpret_cast<uint8_t*>(Z + (size_t)row0 * ldz + c0),
                                (size_t)ldz * 4, wvalid, 8);
            }
            if (Y) {
                uint32_t p[16];
                for (int j = 0; j < 16; j++) {
                    p[j] = pack2(z[2 * j], z[2 * j + 1]);
                    if (act == AQUA_ACT_SILU)
                        p[j] = silu_bf16x2(p[j]);
                }
                __syncwarp();
                for (int j = 0; j < 4; j++)
                    *warp_chunk(wbuf, lane, j) =
                        make_uint4(p[4 * j], p[4 * j + 1], p[4 * j + 2], p[4 * j + 3]);
                __syncwarp();
                warp_store_rows(wbuf, reinterpret_cast<uint8_t*>(Y + (size_t)row0 * ldy + c0),
                                (size_t)ldy * 2, wvalid, 4);
            }
        }
        // the next tile's MMAs overwrite the accumulator and sA
        asm volatile("tcgen05.fence::before_thread_sync;\n");
        __syncthreads();
    }
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n"
                     :: "r"(tmem), "r"((uint32_t)N));
    }
}

// ---------------------------------------------------------------------------
// Fused three-layer edge MLP: Y = L3(act(L2(act(L1(X))))) on tiles of 128
// edges, every activation kept on chip.  The layer-1 input of each tile is
// gathered into shared memory by asynchronous copies: rows of X, or, in PAIR
// mode, the concatenation [H[recv[e]] (64), H[send[e]] (64), Ef[e] (16)] that
// aqua_gnn_gather_pair materialises.  The layers accumulate in 64 columns of
// tensor memory (layer 1 in its own, layers 2 and 3 in turn); each epilogue
// reads them back (tcgen05.ld), adds the bias, applies the activation, rounds
// to BF16 and writes the next layer's A operand into shared memory, exactly the
// values the unfused layers store to and reload from global memory, so the
// result is bit-identical to three aqua_gnn_linear_fwd_tc calls.  Only the BF16
// output of layer 3 is written.  A wait that times out sets *err; the group
// finishes that tile (its outputs are then not to be trusted) and stops.
//
// The tile's chain of layers, barriers and sums bounds it, not the tensor pipe
// (10%) nor memory: three groups a CTA run three chains, and a warp of each
// takes the gather and layer 1 of the next tile off the chain (eight warps that
// gathered themselves stood 3,000 cycles of 18,000 in the copies' queue).  40.4M
// edges: pair input 5.8 ms with three CTAs of 8 warps an SM, 5.1 with the
// gathering warp, 3.9 with swizzled rows; 16-wide input 3.5 and 3.6.
//
// With SUM the layer-3 output never leaves the chip either: it is summed
// into the receivers (aqua_gnn_segment_sum fused in).  Each group owns a
// contiguous range of receivers (about E / groups edges) and walks its edges
// in 128-edge tiles, in order.  The layer-3 tile is staged in shared memory
// (row-major, 16-byte groups XOR-swizzled by row), the receivers' runs of
// rows are summed by the warps (run k by warp k mod 8, lanes over column
// pairs), and a receiver whose edges continue in the next tile carries its
// partial sums there.  Every receiver's sum is thus the same sequence of
// FP32 additions, in edge order from zero, as aqua_gnn_segment_sum's: the
// output is bit-identical to the unfused kernels'.

__device__ __forceinline__ void
cp_async_16z(void* dst, const void* src, bool valid)
{
    // src-size 0 fills the 16 bytes with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n"
                 :: "r"(smem_addr(dst)), "l"(src), "r"(valid ? 16u : 0u)
                 : "memory");
}

// bytes of the layer-1 operand buffer, and of the activation buffer (128 x 64)
template<int K1>
__host__ __device__ constexpr uint32_t
edge_operand_bytes()
{
    return ((128u * K1 * 2u + 1023u) / 1024u) * 1024u;
}
constexpr uint32_t kEdgeAct = 128u * 64u * 2u;

// A CTA is kEdgeGroups groups that share the weights; each walks its own tiles
// and has its own barriers, accumulators and buffers.  Eight warps of a group
// read the accumulators (warps w and w + 4 the same 32 tensor-memory lanes, rows
// 32 (w % 4) .., each one half of the 64 columns); a ninth gathers the layer-1
// input of the next tile and issues its MMAs meanwhile.
constexpr int kEdgeThreads = 256;
constexpr int kEdgeWarps = kEdgeThreads / 32;
constexpr int kEdgeGroups = 3;
constexpr int kEdgeBlock = kEdgeGroups * (kEdgeThreads + 32);
constexpr uint32_t kEdgeTmem = 512;  // columns: 128 a group, a power of two

// shared memory after a group's two buffers: the receiver-sum bookkeeping
struct EdgeShared {
    uint32_t recv[kTcRows];   // receiver of each row of the tile (~0: none)
    uint32_t start[4];        // rows that start a receiver's run, per 32 rows
    float carry[2][64];       // partial sums carried into the next tile
    uint32_t carry_node[2];   // their receiver (~0: none)
    uint32_t nodes[2];        // this group's receivers [nodes[0], nodes[1])
    uint32_t next_recv;       // receiver of the edge after the tile (~0: none)
    uint32_t stop;            // the group gave up: no further tile is gathered
    uint32_t pad[2];
};
static_assert(sizeof(EdgeShared) % 16 == 0, "buffers stay aligned");

// barrier of one group, with the or of `v` over its threads
__device__ __forceinline__ void
group_sync(uint32_t group)
{
    asm volatile("barrier.sync %0, %1;\n" :: "r"(group + 1u), "r"((uint32_t)kEdgeThreads)
                 : "memory");
}
__device__ __forceinline__ bool
group_sync_or(uint32_t group, bool v)
{
    uint32_t any;
    asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %3, 0;\n"
                 "barrier.red.or.pred q, %1, %2, p;\nselp.u32 %0, 1, 0, q;\n}\n"
                 : "=r"(any)
                 : "r"(group + 1u), "r"((uint32_t)kEdgeThreads), "r"((uint32_t)v)
                 : "memory");
    return any != 0u;
}

template<int K1, bool PAIR, bool SUM>
__global__ void __launch_bounds__(kEdgeBlock, 1)
k_edge_mlp_tc(uint32_t E, const uint16_t* __restrict__ X, uint32_t ldx,
              const uint32_t* __restrict__ recv, const uint32_t* __restrict__ send,
              const uint16_t* __restrict__ H, uint32_t ldh,
              const uint16_t* __restrict__ Ef,
              const uint16_t* __restrict__ W1, const float* __restrict__ b1,
              const uint16_t* __restrict__ W2, const float* __restrict__ b2,
              const uint16_t* __restrict__ W3, const float* __restrict__ b3,
              int act1, int act2, int act3, uint16_t* Y, uint32_t ldy, int* err,
              uint32_t fake,
              uint32_t n_nodes, const uint32_t* __restrict__ off, float scale,
              uint32_t col)
{
    constexpr uint32_t kW1 = ((64u * K1 * 2u + 1023u) / 1024u) * 1024u;
    constexpr uint32_t kW = 64u * 64u * 2u;            // W2, W3
    constexpr uint32_t kOp = edge_operand_bytes<K1>();
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // the swizzled operand starts on a 1024-byte boundary
    uint8_t* smem = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);
    // layer 1 done, its accumulator read, layers 2 and 3 done
    __shared__ __align__(8) uint64_t mbars[kEdgeGroups][3];
    __shared__ uint32_t tmem_base;
    __shared__ __align__(16) float sbias[3][64];
    uint8_t* sW1 = smem;
    uint8_t* sW2 = sW1 + kW1;
    uint8_t* sW3 = sW2 + kW;
    // the last kEdgeGroups warps gather
    const bool producer = threadIdx.x >= kEdgeThreads * kEdgeGroups;
    const uint32_t tid = producer ? threadIdx.x % 32u : threadIdx.x % kEdgeThreads;
    const uint32_t group = producer ? (threadIdx.x - kEdgeThreads * kEdgeGroups) / 32u
                                    : threadIdx.x / kEdgeThreads;
    const uint32_t warp = tid >> 5, lane = tid & 31;
    // the group's buffers: the layer-1 input (128 x K1), free for the next
    // tile's rows once layer 1's MMAs have completed, and the 128 x 64
    // activations of layers 1 and 2 (and, with SUM, the layer-3 output tile)
    uint8_t* const sX = sW3 + kW + group * (kOp + kEdgeAct);
    uint8_t* const sA1 = sX + kOp;
    EdgeShared* ss = reinterpret_cast<EdgeShared*>(
                         sW3 + kW + kEdgeGroups * (kOp + kEdgeAct)) + group;

    for (uint32_t e = threadIdx.x; e < 64u * K1 / 8u; e += blockDim.x) {
        const uint32_t row = e / (K1 / 8), g = e % (K1 / 8);
        *reinterpret_cast<uint4*>(sW1 + ((row / 8) * (K1 / 8) + g) * 128 + (row % 8) * 16) =
            *reinterpret_cast<const uint4*>(W1 + (size_t)row * K1 + g * 8);
    }
    for (uint32_t e = threadIdx.x; e < 64u * 8u; e += blockDim.x) {
        const uint32_t row = e / 8, g = e % 8;
        const uint32_t o = ((row / 8) * 8 + g) * 128 + (row % 8) * 16;
        *reinterpret_cast<uint4*>(sW2 + o) =
            *reinterpret_cast<const uint4*>(W2 + (size_t)row * 64 + g * 8);
        *reinterpret_cast<uint4*>(sW3 + o) =
            *reinterpret_cast<const uint4*>(W3 + (size_t)row * 64 + g * 8);
    }
    if (threadIdx.x < 192) {
        const uint32_t t = threadIdx.x;
        sbias[t / 64][t % 64] = (t < 64 ? b1 : (t < 128 ? b2 : b3))[t % 64];
    }
    const uint32_t mbar1 = smem_addr(&mbars[group][0]);
    const uint32_t mread = smem_addr(&mbars[group][1]);
    const uint32_t mbar = smem_addr(&mbars[group][2]);
    if (tid == 0 && !producer) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" :: "r"(mbar1));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n"
                     :: "r"(mread), "r"((uint32_t)kEdgeWarps));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" :: "r"(mbar));
        ss->stop = 0;
    }
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 "
                     "[%0], %1;\n" :: "r"(smem_addr(&tmem_base)), "r"(kEdgeTmem));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    const uint32_t tmem1 = tmem_base + group * 128u;  // layer 1
    const uint32_t tmem = tmem1 + 64u;                // layers 2 and 3
    const uint32_t idesc = make_idesc(64);
    uint32_t phase = 0;
    bool failed = false;

    // one thread issues the MMAs of one layer
    auto mma = [&](uint32_t acc0, const uint8_t* sA, const uint8_t* sB, uint32_t K,
                   uint32_t bar) {
        asm volatile("tcgen05.fence::after_thread_sync;\n");
        const uint32_t sbo = (K / 8) * 128;
        for (uint32_t ks = 0; ks < K / 16; ks++) {
            // the pair input: 64 columns of the receiver and 64 of the sender,
            // swizzled rows of 128 bytes (K steps of 32 bytes in them), then
            // the features as core matrices
            const uint64_t ad =
                PAIR && K == K1
                    ? (ks < 8 ? make_desc(smem_addr(sA) + (ks / 4) * 16384u + (ks % 4) * 32u,
                                          16, 1024) | (2ull << 61)
                              : make_desc(smem_addr(sA) + 32768u, 128, 256))
                    : make_desc(smem_addr(sA) + ks * 256, 128, sbo);
            const uint64_t bd = make_desc(smem_addr(sB) + ks * 256, 128, sbo);
            const uint32_t acc = ks > 0 ? 1u : 0u;
            asm volatile(
                "{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\n"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                :: "r"(acc0), "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one."
                     "shared::cluster.b64 [%0];\n" :: "r"(bar));
    };
    auto arrived = [&](uint32_t bar, uint32_t parity) {
        uint32_t done;
        asm volatile("{\n.reg .pred p;\n"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                     "selp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(done) : "r"(bar), "r"(parity));
        return done != 0u;
    };
    bool tile_bad = false;
    auto wait = [&](uint32_t bar, uint32_t parity) {
        bool done = false;
        for (uint32_t it = 0; it < kWaitLimit && !done; it++)
            done = arrived(bar, parity);
        // a time-out is recorded and acted on at the end of the tile (one
        // group-wide vote per tile instead of one per layer)
        const bool bad = !__all_sync(0xffffffffu, done) || fake != 0u;
        if (bad && lane == 0)
            atomicExch(err, 1);
        tile_bad = tile_bad || bad;
        asm volatile("tcgen05.fence::after_thread_sync;\n");
    };
    // layers 2 and 3: thread 0 issues, everyone waits
    auto layer = [&](const uint8_t* sB) {
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;\n");
        group_sync(group);
        if (tid == 0)
            mma(tmem, sA1, sB, 64, mbar);
        wait(mbar, phase);
        phase ^= 1u;
    };
    // this thread's row of the accumulator and half of its columns
    const uint32_t row = (warp & 3u) * 32u + lane;
    const uint32_t half = warp >> 2;
    // read the accumulator (32 columns), add the bias, activate;
    // `emit(g, packed8)` receives the row's k-group g (8 bf16 as a uint4)
    auto epilogue = [&](int layer_index, int act, auto&& emit) {
        const uint32_t taddr = (layer_index == 0 ? tmem1 : tmem) +
                               (((warp & 3u) * 32u) << 16) + half * 32u;
        uint32_t v[32];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
            "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
            "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]),
              "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
              "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
              "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),
              "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
              "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]),
              "=r"(v[30]), "=r"(v[31])
            : "r"(taddr));
        asm volatile("tcgen05.wait::ld.sync.aligned;\n");
        if (layer_index == 0) {  // the next tile's layer 1 may overwrite it
            asm volatile("tcgen05.fence::before_thread_sync;\n");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" :: "r"(mread)
                             : "memory");
        }
        const float* bias = sbias[layer_index] + half * 32u;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            uint32_t p[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int c = q * 8 + 2 * j;
                const float z0 = __uint_as_float(v[c]) + bias[c];
                const float z1 = __uint_as_float(v[c + 1]) + bias[c + 1];
                p[j] = pack2(z0, z1);
                if (act == AQUA_ACT_SILU)
                    p[j] = silu_bf16x2(p[j]);
            }
            emit((int)(half * 4u) + q, make_uint4(p[0], p[1], p[2], p[3]));
        }
    };
    auto to_a1 = [&](int g, uint4 val) {
        *reinterpret_cast<uint4*>(sA1 + ((row / 8) * 8 + g) * 128 + (row % 8) * 16) = val;
    };

    // the edges of this group: every tile (grid-stride), or, with SUM, the
    // edges of its receivers; few tiles go to one group of each CTA first
    const uint32_t groups = gridDim.x * kEdgeGroups;
    const uint32_t me = group * gridDim.x + blockIdx.x;
    uint32_t e_begin = 0, e_end = E;
    if constexpr (SUM) {
        if (tid == 0 && !producer) {
            // first node s in [0, n_nodes] with off[s] >= v
            auto lower = [&](uint64_t v) -> uint32_t {
                uint32_t lo = 0, hi = n_nodes;
                while (lo < hi) {
                    const uint32_t mid = lo + (hi - lo) / 2;
                    if ((uint64_t)off[mid] < v)
                        lo = mid + 1;
                    else
                        hi = mid;
                }
                return lo;
            };
            const uint64_t G = groups;
            ss->nodes[0] = me == 0 ? 0u : lower((uint64_t)me * E / G);
            ss->nodes[1] = me + 1 == groups ? n_nodes
                                            : lower((uint64_t)(me + 1) * E / G);
            ss->carry_node[0] = ss->carry_node[1] = 0xffffffffu;
        }
        __syncthreads();
        const uint32_t n_lo = ss->nodes[0], n_hi = ss->nodes[1];
        // receivers without edges: a zero sum
        for (uint32_t s = n_lo + tid; s < n_hi && !producer; s += kEdgeThreads)
            if (off[s] == off[s + 1]) {
                uint4* dst = reinterpret_cast<uint4*>(Y + (size_t)s * ldy + col);
                for (int g = 0; g < 8; g++)
                    dst[g] = make_uint4(0u, 0u, 0u, 0u);
            }
        e_begin = off[n_lo];
        e_end = off[n_hi];
    }
    const uint32_t tiles = SUM ? (e_end - e_begin + kTcRows - 1) / kTcRows
                               : (E + kTcRows - 1) / kTcRows;
    const uint32_t stride = SUM ? 1u : groups;
    uint32_t tile = SUM ? 0u : me;
    if (producer) {
        // rows of 32 bytes and multiples (X, the features): a lane copies every
        // other k-group of 8 rows, so that a copy instruction of the warp reads
        // whole 32-byte sectors.  Node rows of 128 bytes: eight lanes a row,
        // and swizzled rows in shared memory, so that a line that arrives is
        // written at once: as core matrices its pieces fall into the same
        // banks, and the epilogues' own accesses waited for them (an epilogue
        // was 3,900 cycles instead of 1,400)
        constexpr uint32_t kg = PAIR ? 2 : K1 / 8;
        const uint32_t r0 = (lane & 7u) + ((lane >> 4) << 3), gh = (lane >> 3) & 1u;
        uint32_t ei[4], es[4];  // receivers and senders of rows lane, lane + 32, ..
        auto load_idx = [&](uint32_t t) {
#pragma unroll
            for (uint32_t q = 0; q < 4; q++) {
                const uint32_t e = e_begin + t * kTcRows + q * 32u + lane;
                const bool valid = PAIR && t < tiles && e < e_end;
                ei[q] = valid ? recv[e] : 0u;
                es[q] = valid ? send[e] : 0u;
            }
        };
        load_idx(tile);
        for (uint32_t n = 0; tile < tiles; n++, tile += stride) {
            const uint32_t e0 = e_begin + tile * kTcRows;
            if (PAIR) {
                const uint32_t c = lane & 7u, rl = lane >> 3;
#pragma unroll
                for (uint32_t j = 0; j < 32; j++) {
                    const uint32_t row = j * 4u + rl;
                    const bool valid = e0 + row < e_end;
                    const uint32_t from = (j & 7u) * 4u + rl;
                    const uint32_t vr = __shfl_sync(0xffffffffu, ei[j / 8], from);
                    const uint32_t vs = __shfl_sync(0xffffffffu, es[j / 8], from);
                    uint8_t* dst = sX + row * 128u + ((c ^ (row & 7u)) << 4);
                    cp_async_16z(dst, H + (size_t)vr * ldh + c * 8, valid);
                    cp_async_16z(dst + 16384, H + (size_t)vs * ldh + c * 8, valid);
                }
            }
            const uint16_t* src = PAIR ? Ef : X;
            const uint32_t ld = PAIR ? 16u : ldx;
#pragma unroll
            for (uint32_t j = 0; j < 8; j++) {
                const uint32_t row = j * 16u + r0;
                const bool valid = e0 + row < e_end;
                const size_t ev = valid ? e0 + row : 0u;
                uint8_t* dst = sX + (PAIR ? 32768u : 0u) + (row / 8) * kg * 128 +
                               (row % 8) * 16 + gh * 128;
#pragma unroll
                for (uint32_t g = 0; g < kg; g += 2)
                    cp_async_16z(dst + g * 128, src + ev * ld + (g + gh) * 8, valid);
            }
            load_idx(tile + stride);
            asm volatile("cp.async.wait_all;\n" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();  // every lane's copies, before lane 0's MMAs read them
            // the accumulator of the tile before has been read
            bool ok = n == 0;
            for (uint32_t it = 0; it < kWaitLimit && !ok; it++) {
                ok = arrived(mread, (n - 1u) & 1u);
                if (!ok && *(volatile uint32_t*)&ss->stop)
                    break;
            }
            if (!__all_sync(0xffffffffu, ok))
                break;
            if (lane == 0)
                mma(tmem1, sX, sW1, K1, mbar1);
            wait(mbar1, n & 1u);  // the operand buffer is free
            if (tile_bad)
                break;
        }
    }
    // the receiver of row tid of tile t, loaded one tile ahead (~0 past the
    // last edge)
    auto load_recv = [&](uint32_t t) {
        const uint32_t e = e_begin + t * kTcRows + tid;
        return SUM && tid < kTcRows && t < tiles && e < e_end ? recv[e] : 0xffffffffu;
    };
    uint32_t ei_cur = producer ? 0u : load_recv(tile);
    for (uint32_t n = 0; !producer && tile < tiles && !failed; n++, tile += stride) {
        const uint32_t ei_next = load_recv(tile + stride);
        const uint32_t eb = e_begin + tile * kTcRows;
        const uint32_t e = eb + row;
        const bool valid = e < e_end;
        if (SUM && tid < kTcRows)
            ss->recv[tid] = ei_cur;
        wait(mbar1, n & 1u);
        epilogue(0, act1, to_a1);
        layer(sW2);
        epilogue(1, act2, to_a1);
        layer(sW3);
        if constexpr (!SUM) {
            epilogue(2, act3, [&](int g, uint4 val) {
                if (valid)
                    *reinterpret_cast<uint4*>(Y + (size_t)e * ldy + g * 8) = val;
            });
        } else {
            // layer-3 tile into shared memory: row r at r * 128 bytes, its
            // 16-byte group g at position g ^ (r % 8)
            epilogue(2, act3, [&](int g, uint4 val) {
                *reinterpret_cast<uint4*>(sA1 + row * 128u + ((g ^ (row & 7u)) * 16u)) = val;
            });
            // the receiver of the edge after this tile's (~0 at the end of the
            // group's edges): it tells whether the tile's last run is complete
            if (tid == 0)
                ss->next_recv = ei_next;
            const uint32_t nvalid = min((uint32_t)kTcRows, e_end - eb);
            if (warp < 4) {
                const uint32_t rr = warp * 32u + lane;
                const bool st = rr < nvalid && (rr == 0 || ss->recv[rr] != ss->recv[rr - 1]);
                const uint32_t bal = __ballot_sync(0xffffffffu, st);
                if (lane == 0)
                    ss->start[warp] = bal;
            }
            group_sync(group);
            const uint32_t par = tile & 1u;
            // run k of the tile: warp k % 8, two columns a lane
            const uint32_t cg = (lane >> 2) << 4;
            const uint8_t* sc = sA1 + (lane & 3u) * 4u;
            uint32_t ord = 0;
            for (uint32_t wq = 0; wq < 4; wq++) {
                uint32_t m = ss->start[wq];
                while (m) {
                    const uint32_t a = wq * 32u + (uint32_t)(__ffs(m) - 1);
                    m &= m - 1;
                    if ((ord++ % kEdgeWarps) != warp)
                        continue;
                    // the run ends at the next start or at the last row
                    uint32_t b = nvalid;
                    if (m) {
                        b = wq * 32u + (uint32_t)(__ffs(m) - 1);
                    } else {
                        for (uint32_t w2 = wq + 1; w2 < 4; w2++) {
                            const uint32_t m2 = ss->start[w2];
                            if (m2) {
                                b = w2 * 32u + (uint32_t)(__ffs(m2) - 1);
                                break;
                            }
                        }
                    }
                    const uint32_t node = ss->recv[a];
                    float s0 = 0.f, s1 = 0.f;  // columns 2 lane, 2 lane + 1
                    if (a == 0 && ss->carry_node[par] == node) {
                        s0 = ss->carry[par][2 * lane];
                        s1 = ss->carry[par][2 * lane + 1];
                    }
                    // eight loads in flight, then the additions in row order;
                    // the swizzle is the same for rows eight apart
                    uint32_t o[8];
#pragma unroll
                    for (uint32_t u = 0; u < 8; u++)
                        o[u] = u * 128u + (cg ^ (((a + u) & 7u) << 4));
                    const uint8_t* q = sc + a * 128u;
                    uint32_t left = b - a, v[8];
                    for (; left >= 8u; left -= 8u, q += 1024) {
#pragma unroll
                        for (uint32_t u = 0; u < 8; u++)
                            v[u] = *reinterpret_cast<const uint32_t*>(q + o[u]);
#pragma unroll
                        for (uint32_t u = 0; u < 8; u++) {
                            s0 += __uint_as_float(v[u] << 16);
                            s1 += __uint_as_float(v[u] & 0xffff0000u);
                        }
                    }
#pragma unroll
                    for (uint32_t u = 0; u < 7; u++)
                        if (u < left)
                            v[u] = *reinterpret_cast<const uint32_t*>(q + o[u]);
#pragma unroll
                    for (uint32_t u = 0; u < 7; u++)
                        if (u < left) {
                            s0 += __uint_as_float(v[u] << 16);
                            s1 += __uint_as_float(v[u] & 0xffff0000u);
                        }
                    if (b < nvalid || ss->next_recv != node) {
                        *reinterpret_cast<uint32_t*>(Y + (size_t)node * ldy + col + 2 * lane) =
                            pack2(s0 * scale, s1 * scale);
                    } else {
                        // the last run: its receiver continues in the next tile
                        ss->carry[par ^ 1u][2 * lane] = s0;
                        ss->carry[par ^ 1u][2 * lane + 1] = s1;
                        if (lane == 0)
                            ss->carry_node[par ^ 1u] = node;
                    }
                }
            }
        }
        // the next tile reuses the activations and the accumulator; a
        // time-out in any layer ends the group
        asm volatile("tcgen05.fence::before_thread_sync;\n");
        failed = group_sync_or(group, tile_bad);
        ei_cur = ei_next;
        if (failed && tid == 0)
            *(volatile uint32_t*)&ss->stop = 1u;
    }
    // no copy may still be in flight when the CTA ends (after a time-out)
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.fence::after_thread_sync;\n");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n"
                     :: "r"(tmem_base), "r"(kEdgeTmem));
    }
}

template<int K1>
constexpr size_t
edge_mlp_smem()
{
    return ((64u * K1 * 2u + 1023u) / 1024u) * 1024u + 2u * 64u * 64u * 2u +
           kEdgeGroups * (edge_operand_bytes<K1>() + kEdgeAct + sizeof(EdgeShared)) + 1024u;
}
static_assert(edge_mlp_smem<144>() <= 226 * 1024, "one CTA per SM");

// ---------------------------------------------------------------------------
// Backward of a dense layer on the tensor cores (training).
//
// dgrad: dX = dY W, times silu'(Zprev) when the previous layer is SiLU.  It
// is the forward's product with dY (M x N) as A and W^T (K x N, the
// transposed weights kept by the model) as B: reduction over N (16 or 64),
// K output columns (up to 160) in a tensor-memory accumulator of `tcols`
// columns; the epilogue multiplies by silu'(Zprev) and rounds to BF16.
//
// wgrad: dW += dY^T X and db += column sums of dY.  The reduction runs over
// the M rows (edges or nodes), 128 per chunk: each chunk of dY (padded with
// zeros to the MMA's 128 outputs) and X is copied as its rows lie in memory,
// both operands MN-major, and the MMAs accumulate over all the CTA's chunks in
// tensor memory.  One extra output of ones in B makes the column K of the
// product the column sums of dY (db).  At the end each CTA adds its partial
// dW, db to the outputs with atomics.

// bounded wait for a commit on `mbar` (phase parity `phase`); every thread
// of the CTA returns the same verdict
__device__ __forceinline__ bool
tc_wait(uint64_t* mbar, uint32_t phase, uint32_t fake)
{
    uint32_t done = 0;
    for (uint32_t it = 0; it < kWaitLimit && !done; it++) {
        asm volatile("{\n.reg .pred p;\n"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                     "selp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(done) : "r"(smem_addr(mbar)), "r"(phase));
    }
    // `fake` (test switch): a wait that completed counts as timed out
    return !__syncthreads_or(!done || fake);
}

__global__ void __launch_bounds__(kTcThreads, 1)
k_linear_dgrad_tc(uint32_t M, uint32_t N, uint32_t K,
                  const uint16_t* __restrict__ dY, uint32_t ldy,
                  const uint16_t* __restrict__ Wt,
                  const float* __restrict__ Zp, uint32_t ldzp, int act_prev,
                  uint16_t* dX, uint32_t ldx, uint32_t tcols, int* err,
                  uint32_t fake)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_base;
    uint8_t* sB = smem;                                        // K x N
    // 128 x N, and 4 KB per warp for Zp and dX
    uint8_t* sA = smem + ((K * N * 2 + 1023) / 1024) * 1024;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    stage(sB, Wt, N, K, K, N);
    if (threadIdx.x == 0)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n"
                     :: "r"(smem_addr(&mbar)));
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 "
                     "[%0], %1;\n" :: "r"(smem_addr(&tmem_base)), "r"(tcols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    const uint32_t tmem = tmem_base;
    const uint32_t idesc = make_idesc(K);
    const uint32_t sbo = (N / 8) * 128;
    const bool grad = Zp && act_prev == AQUA_ACT_SILU;
    uint32_t phase = 0;
    const uint32_t tiles = (M + kTcRows - 1) / kTcRows;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint32_t m0 = tile * kTcRows;
        const uint32_t valid = min((uint32_t)kTcRows, M - m0);
        stage(sA, dY + (size_t)m0 * ldy, ldy, kTcRows, valid, N);
        asm volatile("fence.proxy.async.shared::cta;\n");
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;\n");
            for (uint32_t ks = 0; ks < N / 16; ks++) {
                const uint64_t ad = make_desc(smem_addr(sA) + ks * 256, 128, sbo);
                const uint64_t bd = make_desc(smem_addr(sB) + ks * 256, 128, sbo);
                const uint32_t acc = ks > 0 ? 1u : 0u;
                asm volatile(
                    "{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\n"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                    :: "r"(tmem), "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one."
                         "shared::cluster.b64 [%0];\n" :: "r"(smem_addr(&mbar)));
        }
        if (!tc_wait(&mbar, phase, fake)) {
            if (threadIdx.x == 0)
                atomicExch(err, 1);
            tc_wait(&mbar, phase, 0u);  // the MMAs in flight, again bounded
            break;
        }
        phase ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;\n");
        // epilogue: warp w owns rows 32w .. 32w + 31 (TMEM lanes), 32 columns
        // at a time (the last 16 alone); Zp and dX pass through the warp's
        // rows of the operand buffer so that whole rows move
        const uint32_t row0 = m0 + warp * 32;
        const uint32_t wvalid = row0 < M ? min(32u, M - row0) : 0u;
        const uint32_t taddr = tmem + ((warp * 32u) << 16);
        uint8_t* wbuf = sA + warp * 4096;
        for (uint32_t c0 = 0; c0 < K; c0 += 32) {
            const uint32_t w16 = min(32u, K - c0) / 16u;  // 16-column groups
            if (grad) {
                // rows of Zp -> shared memory (8 chunks of 4 floats, or 4)
                const uint32_t ch = 4u * w16, per = 32u / ch, cc = lane % ch;
                const float* zp = Zp + (size_t)row0 * ldzp + c0;
                float4 zz[8];
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const uint32_t r = lane / ch + q * per;
                    zz[q] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (r < wvalid && r < 32u)
                        zz[q] = *reinterpret_cast<const float4*>(zp + (size_t)r * ldzp + cc * 4);
                }
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const uint32_t r = lane / ch + q * per;
                    if (r < 32u)
                        *reinterpret_cast<float4*>(warp_chunk(wbuf, r, cc)) = zz[q];
                }
                __syncwarp();
            }
            uint32_t pk[16];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                if (h >= (int)w16)
                    break;
                uint32_t v[16];
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                    "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]),
                      "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
                      "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
                      "=r"(v[14]), "=r"(v[15])
                    : "r"(taddr + c0 + 16 * h));
                asm volatile("tcgen05.wait::ld.sync.aligned;\n");
                float d[16];
                for (int j = 0; j < 16; j++)
                    d[j] = __uint_as_float(v[j]);
                if (grad) {
                    for (int j = 0; j < 16; j += 4) {
                        const float4 zz = *reinterpret_cast<const float4*>(
                            warp_chunk(wbuf, lane, 4 * h + j / 4));
                        d[j] *= aqua::silu_grad_f(zz.x);
                        d[j + 1] *= aqua::silu_grad_f(zz.y);
                        d[j + 2] *= aqua::silu_grad_f(zz.z);
                        d[j + 3] *= aqua::silu_grad_f(zz.w);
                    }
                }
                for (int j = 0; j < 8; j++)
                    pk[8 * h + j] = pack2(d[2 * j], d[2 * j + 1]);
            }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (j < 2 * (int)w16)
                    *warp_chunk(wbuf, lane, j) =
                        make_uint4(pk[4 * j], pk[4 * j + 1], pk[4 * j + 2], pk[4 * j + 3]);
            __syncwarp();
            warp_store_rows(wbuf, reinterpret_cast<uint8_t*>(dX + (size_t)row0 * ldx + c0),
                            (size_t)ldx * 2, wvalid, 2u * w16);
            __syncwarp();
        }
        // the next tile's MMAs overwrite the accumulator and sA
        asm volatile("tcgen05.fence::before_thread_sync;\n");
        __syncthreads();
    }
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n"
                     :: "r"(tmem), "r"(tcols));
    }
}

constexpr int kWgThreads = 256;  // wgrad: 8 warps stage, warps 0-3 read TMEM

__global__ void __launch_bounds__(kWgThreads, 1)
k_linear_wgrad_tc(uint32_t M, uint32_t N, uint32_t K,
                  const uint16_t* __restrict__ dY, uint32_t ldy,
                  const uint16_t* __restrict__ X, uint32_t ldx, float* dW,
                  float* db, uint32_t KB, uint32_t nbuf, uint32_t tcols,
                  int* err, uint32_t fake)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t mbar[2];
    __shared__ uint32_t tmem_base;
    // nbuf (1 or 2) buffers, each A = dY^T (128 rows, N used) x 128 and
    // B = X^T (KB rows: X^T, then the row of ones for db, then zeros) x 128,
    // both MN-major: core matrices of 8 reduction rows x 16 bytes, as the
    // rows lie in memory (no transposition: 10.3M rows with the 4-byte loads
    // and stmatrix.trans of one took 1.08 ms, now 0.80); 16 core matrices
    // along the reduction per 8 outputs.  With two buffers a chunk is copied
    // while the MMAs of the one before run.
    const uint32_t bufb = 128 * 128 * 2 + KB * 128 * 2;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t chunks = (M + kTcRows - 1) / kTcRows;
    if ((uint32_t)blockIdx.x >= chunks)
        return;  // no chunk for this CTA (before any allocation)
    for (uint32_t b = 0; b < nbuf; b++) {
        uint8_t* sA = smem + b * bufb;
        uint8_t* sB = sA + 128 * 128 * 2;
        for (uint32_t e = threadIdx.x; e < 128u * 128u / 8u; e += kWgThreads)
            reinterpret_cast<uint4*>(sA)[e] = make_uint4(0, 0, 0, 0);
        for (uint32_t e = threadIdx.x; e < (KB - K) * 128u; e += kWgThreads) {
            const uint32_t r = K + e / 128u, m = e % 128u;
            const uint16_t one = (r == K && db) ? 0x3F80u : 0u;  // bf16 1.0
            *reinterpret_cast<uint16_t*>(
                sB + ((r / 8) * 16 + m / 8) * 128 + (m % 8) * 16 + (r % 8) * 2) = one;
        }
    }
    if (threadIdx.x == 0)
        for (int b = 0; b < 2; b++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n"
                         :: "r"(smem_addr(&mbar[b])));
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 "
                     "[%0], %1;\n" :: "r"(smem_addr(&tmem_base)), "r"(tcols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    const uint32_t tmem = tmem_base;
    // A and B MN-major (bits 15, 16)
    const uint32_t idesc = make_idesc(KB) | (1u << 15) | (1u << 16);
    constexpr uint32_t sbo = 16 * 128;  // next 8 outputs: 16 core matrices on
    uint32_t phase[2] = { 0u, 0u };
    uint32_t pending[2] = { 0u, 0u };  // a commit of the buffer not yet waited
    bool failed = false;
    uint32_t it = 0;
    // starts the copies of a chunk into buffer b, one group
    auto copy = [&](uint32_t ch, uint32_t b) {
        uint8_t* sA = smem + b * bufb;
        uint8_t* sB = sA + 128 * 128 * 2;
        const uint32_t m0 = ch * kTcRows;
        const uint32_t valid = min((uint32_t)kTcRows, M - m0);
        stage_async(sA, dY + (size_t)m0 * ldy, ldy, kTcRows, valid, N, 128, 16 * 128);
        stage_async(sB, X + (size_t)m0 * ldx, ldx, kTcRows, valid, K, 128, 16 * 128);
    };
    // waits for the MMAs that read buffer b
    auto drained = [&](uint32_t b) -> bool {
        if (!pending[b])
            return true;
        if (!tc_wait(&mbar[b], phase[b], fake))
            return false;
        phase[b] ^= 1u;
        pending[b] = 0u;
        return true;
    };
    if (nbuf == 2) {
        copy(blockIdx.x, 0);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    for (uint32_t ch = blockIdx.x; ch < chunks && !failed; ch += gridDim.x, it++) {
        const uint32_t b = it % nbuf;
        uint8_t* sA = smem + b * bufb;
        uint8_t* sB = sA + 128 * 128 * 2;
        if (nbuf == 2) {
            // the next chunk into the other buffer, then wait for this one's
            if (ch + gridDim.x < chunks) {
                if (!drained(b ^ 1u)) {
                    failed = true;
                    break;
                }
                copy(ch + gridDim.x, b ^ 1u);
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            if (!drained(b)) {
                failed = true;
                break;
            }
            copy(ch, b);
            stage_wait();
        }
        asm volatile("fence.proxy.async.shared::cta;\n");
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;\n");
            for (uint32_t ks = 0; ks < 8; ks++) {
                const uint64_t ad = make_desc(smem_addr(sA) + ks * 256, 128, sbo);
                const uint64_t bd = make_desc(smem_addr(sB) + ks * 256, 128, sbo);
                const uint32_t acc = (it == 0 && ks == 0) ? 0u : 1u;
                asm volatile(
                    "{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\n"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                    :: "r"(tmem), "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one."
                         "shared::cluster.b64 [%0];\n" :: "r"(smem_addr(&mbar[b])));
        }
        pending[b] = 1u;
    }
    stage_wait();  // none is left in flight
    // the last commits (the MMAs run in order: the later one covers both)
    for (int b = 0; b < 2; b++) {
        if (!pending[b])
            continue;
        if (!tc_wait(&mbar[b], phase[b], failed ? 0u : fake)) {
            failed = true;
            tc_wait(&mbar[b], phase[b], 0u);  // in flight, again bounded
        }
    }
    if (failed) {
        if (threadIdx.x == 0)
            atomicExch(err, 1);
    } else if (warp < 4) {
        asm volatile("tcgen05.fence::after_thread_sync;\n");
        // epilogue: rows n = 32w + lane < N add their partial sums
        const uint32_t n = warp * 32 + lane;
        const uint32_t taddr = tmem + ((warp * 32u) << 16);
        for (uint32_t c0 = 0; c0 < KB; c0 += 16) {
            uint32_t v[16];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]),
                  "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
                  "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
                  "=r"(v[14]), "=r"(v[15])
                : "r"(taddr + c0));
            asm volatile("tcgen05.wait::ld.sync.aligned;\n");
            if (n < N) {
                for (int j = 0; j < 16; j++) {
                    const uint32_t col = c0 + j;
                    if (col < K)
                        atomicAdd(&dW[(size_t)n * K + col], __uint_as_float(v[j]));
                    else if (col == K && db)
                        atomicAdd(&db[n], __uint_as_float(v[j]));
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n"
                     :: "r"(tmem), "r"(tcols));
    }
}
}  // namespace

namespace {

// sets the shared-memory limit of the four fused edge-MLP kernels once per
// device (the limit is a per-device attribute of each kernel)
aqua_status
edge_mlp_configure(int& sms)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) !=
            cudaSuccess)
        return AQUA_ERR_CUDA;
    static std::atomic<uint64_t> configured{ 0 };
    const uint64_t bit = dev < 64 ? (1ull << dev) : 0ull;
    if (!bit || !(configured.load() & bit)) {
        const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
        if (cudaFuncSetAttribute(k_edge_mlp_tc<16, false, false>, a,
                                 (int)edge_mlp_smem<16>()) != cudaSuccess ||
            cudaFuncSetAttribute(k_edge_mlp_tc<80, false, false>, a,
                                 (int)edge_mlp_smem<80>()) != cudaSuccess ||
            cudaFuncSetAttribute(k_edge_mlp_tc<144, true, false>, a,
                                 (int)edge_mlp_smem<144>()) != cudaSuccess ||
            cudaFuncSetAttribute(k_edge_mlp_tc<16, false, true>, a,
                                 (int)edge_mlp_smem<16>()) != cudaSuccess ||
            cudaFuncSetAttribute(k_edge_mlp_tc<144, true, true>, a,
                                 (int)edge_mlp_smem<144>()) != cudaSuccess)
            return AQUA_ERR_CUDA;
        configured.fetch_or(bit);
    }
    return AQUA_OK;
}

bool
a16(const void* p)
{
    return (reinterpret_cast<uintptr_t>(p) & 15) == 0;
}

// the arguments both fused forms share; row inputs are 16 wide (edge
// features), or 80 wide where `rows80` (the first node MLP, n1)
bool
edge_mlp_args_ok(uint32_t K1, bool rows80, const uint16_t* X, uint32_t ldx,
                 const uint32_t* recv, const uint32_t* send, const uint16_t* H,
                 uint32_t ldh, const uint16_t* Ef, const uint16_t* W1,
                 const float* b1, const uint16_t* W2, const float* b2,
                 const uint16_t* W3, const float* b3, const int32_t* err)
{
    if (!W1 || !b1 || !W2 || !b2 || !W3 || !b3 || !err || !a16(W1) ||
        !a16(W2) || !a16(W3))
        return false;
    if (X == nullptr)
        return K1 == 144 && recv && send && H && Ef && ldh >= 64 && ldh % 8 == 0 &&
               a16(H) && a16(Ef);
    return (K1 == AQUA_GNN_FEATURES || (rows80 && K1 == 80)) && ldx >= K1 &&
           ldx % 8 == 0 && a16(X);
}

}  // namespace

extern "C" aqua_status
aqua_gnn_edge_mlp_tc(uint32_t E, uint32_t K1, const uint16_t* X, uint32_t ldx,
                     const uint32_t* recv, const uint32_t* send,
                     const uint16_t* H, uint32_t ldh, const uint16_t* Ef,
                     const uint16_t* W1, const float* b1, const uint16_t* W2,
                     const float* b2, const uint16_t* W3, const float* b3,
                     int32_t act1, int32_t act2, int32_t act3, uint16_t* Y,
                     uint32_t ldy, int32_t* err, void* stream)
{
    const bool pair = (X == nullptr);
    if (!edge_mlp_args_ok(K1, true, X, ldx, recv, send, H, ldh, Ef, W1, b1, W2,
                          b2, W3, b3, err) ||
        !Y || ldy < 64 || ldy % 8 || !a16(Y))
        return AQUA_ERR_INVALID;
    if (E == 0)
        return AQUA_OK;
    int sms = 0;
    const aqua_status st = edge_mlp_configure(sms);
    if (st != AQUA_OK)
        return st;
    // one CTA per SM (shared memory; it holds all 512 tensor-memory columns)
    const uint32_t tiles = (E + kTcRows - 1) / kTcRows;
    const uint32_t grid = tiles < (uint32_t)sms ? tiles : (uint32_t)sms;
    cudaStream_t s = (cudaStream_t)stream;
    if (pair) {
        k_edge_mlp_tc<144, true, false>
            <<<grid, kEdgeBlock, edge_mlp_smem<144>(), s>>>(
                E, nullptr, 0, recv, send, H, ldh, Ef, W1, b1, W2, b2, W3, b3,
                act1, act2, act3, Y, ldy, err, (uint32_t)aqua::g_debug_fake_timeout, 0u, nullptr, 0.f, 0u);
    } else if (K1 == 80) {
        // the first node MLP, n1 (80-wide rows)
        k_edge_mlp_tc<80, false, false>
            <<<grid, kEdgeBlock, edge_mlp_smem<80>(), s>>>(
                E, X, ldx, nullptr, nullptr, nullptr, 0, nullptr, W1, b1, W2,
                b2, W3, b3, act1, act2, act3, Y, ldy, err, (uint32_t)aqua::g_debug_fake_timeout, 0u, nullptr, 0.f, 0u);
    } else {
        k_edge_mlp_tc<16, false, false>
            <<<grid, kEdgeBlock, edge_mlp_smem<16>(), s>>>(
                E, X, ldx, nullptr, nullptr, nullptr, 0, nullptr, W1, b1, W2,
                b2, W3, b3, act1, act2, act3, Y, ldy, err, (uint32_t)aqua::g_debug_fake_timeout, 0u, nullptr, 0.f, 0u);
    }
    return cudaGetLastError() == cudaSuccess ? AQUA_OK : AQUA_ERR_CUDA;
}

extern "C" aqua_status
aqua_gnn_edge_mlp_sum_tc(uint32_t n_nodes, uint32_t E, uint32_t K1,
                         const uint16_t* X, uint32_t ldx,
                         const uint32_t* offsets, const uint32_t* recv,
                         const uint32_t* send, const uint16_t* H, uint32_t ldh,
                         const uint16_t* Ef, const uint16_t* W1,
                         const float* b1, const uint16_t* W2, const float* b2,
                         const uint16_t* W3, const float* b3, int32_t act1,
                         int32_t act2, int32_t act3, float scale,
                         uint16_t* out, uint32_t ld, uint32_t col,
                         int32_t* err, void* stream)
{
    const bool pair = (X == nullptr);
    if (!edge_mlp_args_ok(K1, false, X, ldx, recv, send, H, ldh, Ef, W1, b1, W2, b2,
                          W3, b3, err) ||
        !offsets || !recv || !out || !a16(out) || ld % 8 || col % 8 ||
        col + 64 > ld || E >= 0x80000000u)
        return AQUA_ERR_INVALID;
    if (n_nodes == 0)
        return AQUA_OK;
    int sms = 0;
    const aqua_status st = edge_mlp_configure(sms);
    if (st != AQUA_OK)
        return st;
    // each group of a CTA owns the receivers of about E / groups edges; a
    // small graph gets fewer CTAs (at least one, for the receivers without
    // edges)
    const uint32_t tiles = (E + kTcRows - 1) / kTcRows;
    uint32_t grid = (uint32_t)sms;
    if (tiles < grid)
        grid = tiles > 0 ? tiles : 1u;
    cudaStream_t s = (cudaStream_t)stream;
    if (pair)
        k_edge_mlp_tc<144, true, true>
            <<<grid, kEdgeBlock, edge_mlp_smem<144>(), s>>>(
                E, nullptr, 0, recv, send, H, ldh, Ef, W1, b1, W2, b2, W3, b3,
                act1, act2, act3, out, ld, err, (uint32_t)aqua::g_debug_fake_timeout, n_nodes, offsets, scale, col);
    else
        k_edge_mlp_tc<16, false, true>
            <<<grid, kEdgeBlock, edge_mlp_smem<16>(), s>>>(
                E, X, ldx, recv, nullptr, nullptr, 0, nullptr, W1, b1, W2, b2,
                W3, b3, act1, act2, act3, out, ld, err, (uint32_t)aqua::g_debug_fake_timeout, n_nodes, offsets, scale,
                col);
    return cudaGetLastError() == cudaSuccess ? AQUA_OK : AQUA_ERR_CUDA;
}

extern "C" aqua_status
aqua_gnn_linear_fwd_tc(uint32_t M, uint32_t K, uint32_t N, const uint16_t* X,
                       uint32_t ldx, const uint16_t* W, const float* b,
                       float* Z, uint32_t ldz, uint16_t* Y, uint32_t ldy,
                       int32_t act, int32_t* err, void* stream)
{
    if (!X || !W || !err || (!Z && !Y) || K == 0 || K % 16 || K > 160 ||
        N != 64 || ldx < K || ldx % 8 || (Z && (ldz < N || ldz % 4)) ||
        (Y && (ldy < N || ldy % 8)) ||
        (reinterpret_cast<uintptr_t>(X) & 15) || (reinterpret_cast<uintptr_t>(W) & 15) ||
        (Z && (reinterpret_cast<uintptr_t>(Z) & 15)) ||
        (Y && (reinterpret_cast<uintptr_t>(Y) & 15)))
        return AQUA_ERR_INVALID;
    if (M == 0)
        return AQUA_OK;
    size_t bytes = ((size_t)N * K * 2 + 1023) / 1024 * 1024 + tc_operand_bytes(K);
    // at least 30 KB per CTA keeps <= 7 CTAs on an SM (7 x 64 of the 512
    // tensor-memory columns), so tcgen05.alloc never has to wait
    if (bytes < 30 * 1024)
        bytes = 30 * 1024;
    int sms = 0, dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) !=
            cudaSuccess)
        return AQUA_ERR_CUDA;
    static std::atomic<uint64_t> configured{ 0 };
    const uint64_t bit = dev < 64 ? (1ull << dev) : 0ull;
    if (!bit || !(configured.load() & bit)) {
        if (cudaFuncSetAttribute(k_linear_fwd_tc<64>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 64 * 1024) != cudaSuccess)
            return AQUA_ERR_CUDA;
        configured.fetch_or(bit);
    }
    const uint32_t tiles = (M + kTcRows - 1) / kTcRows;
    const uint32_t grid = tiles < (uint32_t)sms * 8u ? tiles : (uint32_t)sms * 8u;
    k_linear_fwd_tc<64><<<grid, kTcThreads, bytes, (cudaStream_t)stream>>>(
        M, K, X, ldx, W, b, Z, ldz, Y, ldy, act, err, (uint32_t)aqua::g_debug_fake_timeout);
    return cudaGetLastError() == cudaSuccess ? AQUA_OK : AQUA_ERR_CUDA;
}

namespace {

// tensor-memory columns for an accumulator of `cols` columns (a power of 2,
// at least 32), and the shared memory that keeps the CTAs of one SM within
// its 512 columns, so that tcgen05.alloc never waits
uint32_t
tc_cols(uint32_t cols)
{
    uint32_t t = 32;
    while (t < cols)
        t *= 2;
    return t;
}

size_t
tc_min_smem(uint32_t tcols)
{
    return (size_t)233472 / (512u / tcols + 1u);
}

cudaError_t
tc_sms(int* sms)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev);
    return e;
}

bool
al16(const void* p)
{
    return (reinterpret_cast<uintptr_t>(p) & 15) == 0;
}

}  // namespace

extern "C" aqua_status
aqua_gnn_linear_dgrad_tc(uint32_t M, uint32_t N, uint32_t K,
                         const uint16_t* dY, uint32_t ldy, const uint16_t* Wt,
                         const float* Zprev, uint32_t ldzp, int32_t act_prev,
                         uint16_t* dX, uint32_t ldx, int32_t* err, void* stream)
{
    if (!dY || !Wt || !dX || !err || (N != 16 && N != 64) || K == 0 ||
        K % 16 || K > 160 || ldy < N || ldy % 8 || ldx < K || ldx % 8 ||
        !al16(dY) || !al16(Wt) || !al16(dX) ||
        (Zprev && act_prev == AQUA_ACT_SILU &&
         (ldzp < K || ldzp % 4 || !al16(Zprev))))
        return AQUA_ERR_INVALID;
    if (M == 0)
        return AQUA_OK;
    const uint32_t tcols = tc_cols(K);
    size_t bytes = ((size_t)K * N * 2 + 1023) / 1024 * 1024 + tc_operand_bytes(N);
    if (bytes < tc_min_smem(tcols))
        bytes = tc_min_smem(tcols);
    int sms = 0;
    if (tc_sms(&sms) != cudaSuccess)
        return AQUA_ERR_CUDA;
    if (cudaFuncSetAttribute(k_linear_dgrad_tc,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)bytes) != cudaSuccess)
        return AQUA_ERR_CUDA;
    const uint32_t tiles = (M + kTcRows - 1) / kTcRows;
    const uint32_t cap = (uint32_t)sms * (512u / tcols);
    const uint32_t grid = tiles < cap ? tiles : cap;
    k_linear_dgrad_tc<<<grid, kTcThreads, bytes, (cudaStream_t)stream>>>(
        M, N, K, dY, ldy, Wt, Zprev, ldzp, act_prev, dX, ldx, tcols, err,
        (uint32_t)aqua::g_debug_fake_timeout);
    return cudaGetLastError() == cudaSuccess ? AQUA_OK : AQUA_ERR_CUDA;
}

extern "C" aqua_status
aqua_gnn_linear_wgrad_tc(uint32_t M, uint32_t N, uint32_t K,
                         const uint16_t* dY, uint32_t ldy, const uint16_t* X,
                         uint32_t ldx, float* dW, float* db, int32_t* err,
                         void* stream)
{
    if (!dY || !X || !dW || !err || (N != 16 && N != 64) || K == 0 ||
        K % 16 || K > 160 || ldy < N || ldy % 8 || ldx < K || ldx % 8 ||
        !al16(dY) || !al16(X))
        return AQUA_ERR_INVALID;
    if (M == 0)
        return AQUA_OK;
    const uint32_t KB = K + 16;  // + the row of ones (db) and zero padding
    const uint32_t tcols = tc_cols(KB);
    const size_t buf = (size_t)128 * 128 * 2 + (size_t)KB * 128 * 2;
    // two staging buffers where two CTAs per SM still fit, else one
    const uint32_t nbuf = 233472 / (2 * buf + 1024) >= 2 ? 2u : 1u;
    size_t bytes = nbuf * buf;
    if (bytes < tc_min_smem(tcols))
        bytes = tc_min_smem(tcols);
    int sms = 0;
    if (tc_sms(&sms) != cudaSuccess)
        return AQUA_ERR_CUDA;
    if (cudaFuncSetAttribute(k_linear_wgrad_tc,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)bytes) != cudaSuccess)
        return AQUA_ERR_CUDA;
    const uint32_t chunks = (M + kTcRows - 1) / kTcRows;
    // CTAs resident per SM: tensor-memory columns and shared memory
    uint32_t per_sm = 512u / tcols;
    const uint32_t by_smem = (uint32_t)(233472 / (bytes + 1024));
    if (by_smem < per_sm)
        per_sm = by_smem;
    const uint32_t cap = (uint32_t)sms * (per_sm > 0 ? per_sm : 1u);
    const uint32_t grid = chunks < cap ? chunks : cap;
    k_linear_wgrad_tc<<<grid, kWgThreads, bytes, (cudaStream_t)stream>>>(
        M, N, K, dY, ldy, X, ldx, dW, db, KB, nbuf, tcols, err,
        (uint32_t)aqua::g_debug_fake_timeout);
    return cudaGetLastError() == cudaSuccess ? AQUA_OK : AQUA_ERR_CUDA;
}
