// k_reduce.cu -- deterministic reductions over pitched fields (sm_100a).
//
// The reference finishes every reduction in f64 on the host from f32 workgroup partials
// (crates/qm-gpu/src/reduce.rs:1-3, :225-234). Here the whole reduction stays on the device: a
// kernel writes one f64 partial per CTA and value (fixed grid size, fixed per-thread order, fixed
// shuffle tree), and `finish` sums the partials of all CTAs in index order with Neumaier
// compensation. The same inputs therefore give the same bits on every run, and no host round
// trip is needed until a scalar is actually wanted on the host.
#include <cmath>
#include <cudaTypedefs.h>
#include "kernels.cuh"
#include "reduce_util.cuh"
#include "harmonics.cuh"

namespace ks {

namespace {

constexpr int TPB = 256;

// One warp per value: lane l sums the partials of CTAs l, l+32, ... (Neumaier), then the lanes are
// combined by a fixed shuffle tree -- the same order on every run.
__global__ void finish_kernel(const double* __restrict__ partials, int blocks, int nvals, double scale, double* __restrict__ out) {
    const int v = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (v >= nvals) return;
    double sum = 0.0, comp = 0.0;
    for (int b = lane; b < blocks; b += 32) {
        double x = partials[(size_t)b * nvals + v];
        double t = sum + x;
        if (fabs(sum) >= fabs(x)) comp += (sum - t) + x; else comp += (x - t) + sum;
        sum = t;
    }
    double total = warp_sum(sum + comp);
    if (lane == 0) out[v] = total * scale;
}

// The same sums for many values, up to two descriptors (values [0, a.nvals) finish a, the next b.nvals finish b): a CTA
// owns 32 consecutive values, lane = value, so every read is a whole coalesced line; warp w sums the partials of the CTAs
// w, w + 8, ... (Neumaier) and the warps' sums are combined in a fixed order. The warp-per-value form above reads one
// 8-byte value per line and was bound by that: 9.1 us for the 1160 values of a 24 x 48 Gram with its norms.
constexpr int FW = 8;
__global__ void __launch_bounds__(FW * 32) finish_many_kernel(FinishDesc a, FinishDesc b) {
    __shared__ double part[FW][32], pcomp[FW][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int v = (int)blockIdx.x * 32 + lane;
    const bool second = v >= a.nvals;
    const double* p = second ? b.partials : a.partials;
    const int nvals = second ? b.nvals : a.nvals, blocks = second ? b.blocks : a.blocks;
    if (second) v -= a.nvals;
    double sum = 0.0, comp = 0.0;
    if (v < nvals) {
#pragma unroll 4
        for (int blk = warp; blk < blocks; blk += FW) {
            const double x = p[(size_t)blk * nvals + v];
            const double t = sum + x;
            if (fabs(sum) >= fabs(x)) comp += (sum - t) + x; else comp += (x - t) + sum;
            sum = t;
        }
    }
    part[warp][lane] = sum;
    pcomp[warp][lane] = comp;
    __syncthreads();
    if (warp != 0 || v >= nvals) return;
    for (int w = 1; w < FW; ++w) {
        const double x = part[w][lane], t = sum + x;
        if (fabs(sum) >= fabs(x)) comp += (sum - t) + x; else comp += (x - t) + sum;
        comp += pcomp[w][lane];
        sum = t;
    }
    const int trows = second ? b.trows : a.trows, tcols = second ? b.tcols : a.tcols;
    const int o = trows > 0 ? (v % tcols) * trows + v / tcols : v;
    (second ? b.out : a.out)[o] = (sum + comp) * (second ? b.scale : a.scale);
}

__global__ void finish_max_kernel(const double* __restrict__ partials, int blocks, double* __restrict__ out) {
    double m = 0.0;
    for (int b = threadIdx.x; b < blocks; b += blockDim.x) m = fmax(m, partials[b]);
    m = block_max(m);
    if (threadIdx.x == 0) out[0] = m;
}

__global__ void dots_kernel(long long F4, Pairs p, double* __restrict__ partials) {
    double acc[Pairs::MAX];
#pragma unroll
    for (int q = 0; q < Pairs::MAX; ++q) acc[q] = 0.0;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < F4; e += (long long)gridDim.x * blockDim.x) {
#pragma unroll
        for (int q = 0; q < Pairs::MAX; ++q) {
            if (q < p.count) {
                float4 a = reinterpret_cast<const float4*>(p.a[q])[e];
                float4 b = reinterpret_cast<const float4*>(p.b[q])[e];
                acc[q] += (double)a.x * b.x + (double)a.y * b.y + (double)a.z * b.z + (double)a.w * b.w;
            }
        }
    }
    for (int q = 0; q < p.count; ++q) {
        double s = block_sum(acc[q]);
        if (threadIdx.x == 0) partials[(size_t)blockIdx.x * p.count + q] = s;
    }
}

// ---- the Gram block G = S^T [S | T] on CUDA cores.
// Thread-per-point, register-blocked warp tiles: lane l of a warp owns one grid point of the
// CTA's current 32-point chunk and an 8 x 8 tile of G (64 f32 accumulators); the warps of the CTA
// cover up to GW tiles of G and walk the same chunks, so each field value is fetched from HBM
// once and served to the other warps from L1. Lanes accumulate in f32 over their points (a few
// dozen per lane), the lanes of a warp are combined in f64.
constexpr int GT = 8;    // warp tile edge
constexpr int GW = 16;   // warps per CTA (tiles per CTA row of blockIdx.y)

__global__ void __launch_bounds__(GW * 32) gram_kernel(long long F, int m, const float* __restrict__ S, int mt,
                                                       const float* __restrict__ T, int tiles_c, int ntiles,
                                                       double* __restrict__ partials) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.y * GW + warp;
    const int mc = m + mt;
    const long long chunks = (F + 31) / 32;
    float acc[GT][GT];
#pragma unroll
    for (int a = 0; a < GT; ++a)
#pragma unroll
        for (int b = 0; b < GT; ++b) acc[a][b] = 0.f;
    int r0 = 0, c0 = 0;
    const float* rowp[GT];
    const float* colp[GT];
    if (tile < ntiles) {
        r0 = (tile / tiles_c) * GT;
        c0 = (tile % tiles_c) * GT;
#pragma unroll
        for (int a = 0; a < GT; ++a) {
            int r = min(r0 + a, m - 1);
            rowp[a] = S + (long long)r * F;
            int c = min(c0 + a, mc - 1);
            colp[a] = c < m ? S + (long long)c * F : T + (long long)(c - m) * F;
        }
        for (long long ch = blockIdx.x; ch < chunks; ch += gridDim.x) {
            long long e = ch * 32 + lane;
            if (e < F) {
                float rv[GT], cv[GT];
#pragma unroll
                for (int a = 0; a < GT; ++a) rv[a] = __ldg(rowp[a] + e);
#pragma unroll
                for (int b = 0; b < GT; ++b) cv[b] = __ldg(colp[b] + e);
#pragma unroll
                for (int a = 0; a < GT; ++a)
#pragma unroll
                    for (int b = 0; b < GT; ++b) acc[a][b] = fmaf(rv[a], cv[b], acc[a][b]);
            }
        }
    }
    if (tile >= ntiles) return;  // whole warp: no CTA-wide sync below
    const size_t base = (size_t)(blockIdx.x) * ((size_t)m * mc);
#pragma unroll
    for (int a = 0; a < GT; ++a)
#pragma unroll
        for (int b = 0; b < GT; ++b) {
            double v = warp_sum((double)acc[a][b]);
            if (lane == 0 && r0 + a < m && c0 + b < mc) partials[base + (size_t)(r0 + a) * mc + (c0 + b)] = v;
        }
}

// ---- the Gram block on CUDA cores, staged in shared memory.
// A warp computes a whole piece of G, up to 32 rows (fields of S) x 32 columns of S and 32 of T, over its own 32-point
// slabs: lane (a, b) = (lane / 8, lane % 8) owns the rows a + 4 i and the columns b + 8 j, so a pair (i, j) of a lane's tile
// is a 4 x 8 patch of G across the warp. A slab is two TMA boxes (the rows of S and of T, 128 bytes of points each) with the
// 128-byte swizzle: a lane reads four points of a row as one 16-byte quad, the 8 rows of a column group (or the 4 of a row
// group) come from distinct banks and are broadcast, so an operand costs one shared-memory wavefront; and the quad's two
// register pairs feed packed f32x2 FMAs directly (even and odd points in the two halves of an accumulator). At m = mt = 24
// that is 12 wavefronts and 60 FMA instructions per four points and warp; one warp per 8 x 8 tile with lanes on points (the
// form this replaces) took 64 wavefronts per 256, as much of the shared memory as of the FMA pipe. The warps are
// independent: each refills its own slots, and no barrier is shared until the end. Patches that the symmetry of S^T S makes
// redundant are skipped, and with LOWER also those of S^T T above the diagonal, which a Rayleigh-Ritz step never reads
// (24 patches instead of 30).
// Measured (with the finish): m = mt = 24 on 95^3 99.7 -> 57.3 us, 8 / 8 69 -> 24.6, 128^3 24 / 24 208 -> 114, 48^3 12 / 12 25.8 ->
// 16.4; in a solve, where LOWER applies, 96.7 -> 49.6 us. At 3.3 TB/s no unit is above 60 %: three or four warps per scheduler
// leave the FMA pipe (58 % active) throttled while they multiply in bursts and idle while the operands load. Scalar FMAs took the
// same time. Rows of 512 bytes by one bulk copy each, at a padded pitch, measured slower: 85 us copied by the consumers, 95 us
// by a producer warp.
// Sums: f32 over 16 points of a slab, f32 over a warp's slabs, f64 across the warps and (launch_finish) the CTAs.
// Larger blocks are several pieces: DIAG pieces (rows, the same columns of S and of T) and pieces of one foreign column block.
constexpr int GP = 32;             // points per slab (one 128-byte swizzle row)
constexpr int G_DEPTH = 8;         // slots per warp at most
constexpr int G_SMEM = 208 * 1024;
constexpr long long G_WAIT_LIMIT = 1LL << 22;
// a box's inner extent is 128 bytes and its x coordinate a multiple of 32 floats: both multiples of 16 bytes, as TMA
// requires (a violation faults the GPU instead of returning an error)
static_assert((GP * 4) % 16 == 0 && GP * 4 == 128, "TMA boxes of whole 128-byte swizzle rows");
__device__ __forceinline__ unsigned g_su32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool g_wait(uint64_t* bar, unsigned parity, long long limit) {
    for (long long n = 0;; ++n) {
        unsigned ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(g_su32(bar)), "r"(parity)
                     : "memory");
        if (ok) return true;
        if (n > limit) return false;
    }
}
__device__ __forceinline__ void g_tma(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(g_su32(dst)),
        "l"((unsigned long long)map), "r"(x), "r"(y), "r"(g_su32(bar))
        : "memory");
}
__device__ __forceinline__ unsigned long long g_fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// The patch (i, j) of a piece is computed: always for foreign columns; on a DIAG piece the S columns j < M8 below the
// diagonal (some row 4 i + 3 reaches the first column 8 j), the T columns likewise with LOWER.
template <int M8, bool DIAG, bool LOWER>
__host__ __device__ constexpr bool g_patch(int i, int j) {
    if (!DIAG) return true;
    if (j < M8) return 4 * i + 3 >= 8 * j;
    return LOWER ? 4 * i + 3 >= 8 * (j - M8) : true;
}
// warps of a CTA: a patch takes three registers (two halves of the slab's sum, the running sum)
template <int M8, int T8, bool DIAG, bool LOWER>
constexpr int g_warps() {
    int n = 0;
    for (int i = 0; i < 2 * M8; ++i)
        for (int j = 0; j < (DIAG ? M8 : 0) + T8; ++j) n += g_patch<M8, DIAG, LOWER>(i, j);
    // 128, 168 or 255 registers each; two slots of 7 KB (9 KB) and more do not fit for 16 (12) warps
    return n <= 24 && M8 + T8 <= 6 ? 16 : n <= 32 && M8 + T8 <= 8 ? 12 : 8;
}

// Rows: fields [32 rb, 32 rb + 8 M8) of S. DIAG: columns the same fields of S, then fields [32 rb, 32 rb + 8 T8) of T. Else
// the columns are the fields [CB cb, CB cb + 8 T8) of tm_t's block (nt fields), at column colT of G. mc: columns of G.
template <int M8, int T8, bool DIAG, bool LOWER, int DEPTH>
__global__ void __launch_bounds__(32 * g_warps<M8, T8, DIAG, LOWER>(), 1)
    gram_piece_kernel(const __grid_constant__ CUtensorMap tm_s, const __grid_constant__ CUtensorMap tm_t, int slabs, int m, int nt, int mc,
                      int rb, int cb, int colT, bool mirrorT, double* __restrict__ partials, int* err) {
    constexpr int W = g_warps<M8, T8, DIAG, LOWER>();
    constexpr int RI = 2 * M8, C = (DIAG ? M8 : 0) + T8, SLAB = (M8 + T8) * 1024;
    constexpr int CB = T8 > 4 ? 64 : 32;  // column blocks
    extern __shared__ unsigned char g_raw[];
    unsigned char* base = g_raw + ((1024 - (g_su32(g_raw) & 1023)) & 1023);
    __shared__ __align__(8) uint64_t full[W * DEPTH];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int a = lane >> 3, b = lane & 7;
    unsigned char* mine = base + (size_t)warp * DEPTH * SLAB;
    uint64_t* bars = full + warp * DEPTH;
    if (lane == 0) {
        for (int d = 0; d < DEPTH; ++d) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(g_su32(&bars[d])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    // slabs (k W + warp) gridDim.x + blockIdx.x: a small grid's slabs spread over the SMs first
    const int first = warp * (int)gridDim.x + (int)blockIdx.x, stride = W * (int)gridDim.x;
    const int nmine = first < slabs ? (slabs - first + stride - 1) / stride : 0;
    const int tb = DIAG ? rb : cb;
    auto issue = [&](int k, int d) {
        const int x = (first + k * stride) * GP;
        unsigned char* dst = mine + (size_t)d * SLAB;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(g_su32(&bars[d])), "r"((unsigned)SLAB) : "memory");
        g_tma(dst, &tm_s, x, 32 * rb, &bars[d]);  // whole boxes land, the zero fill past F and past the last field included
        if (T8 > 0) g_tma(dst + M8 * 1024, &tm_t, x, CB * tb, &bars[d]);
    };
    int issued = min(DEPTH, nmine);
    if (lane == 0)
        for (int k = 0; k < issued; ++k) issue(k, k);
    float sum[RI][C];
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int j = 0; j < C; ++j) sum[i][j] = 0.f;
    bool alive = true;
    int d = 0;
    unsigned ph = 0;
    for (int k = 0; k < nmine; ++k) {
        if (!g_wait(&bars[d], ph, G_WAIT_LIMIT)) {
            if (err) atomicExch(err, 1);  // the partials are undefined; the host's next readback reports the error
            alive = false;
            break;
        }
        const unsigned char* slot = mine + (size_t)d * SLAB;
        const unsigned char* rp = slot + a * 128;
        const unsigned char* cp = slot + (DIAG ? 0 : M8 * 1024) + b * 128;
        unsigned long long acc[RI][C];  // (even points, odd points)
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
            for (int j = 0; j < C; ++j) acc[i][j] = 0ull;
#pragma unroll 2
        for (int q = 0; q < GP / 4; ++q) {  // the 16-byte quad q of a row lies at chunk q ^ (row % 8)
            const int oc = (q ^ b) << 4, oe = (q ^ a) << 4, oo = oe ^ 64;
            ulonglong2 cv[C];
#pragma unroll
            for (int j = 0; j < C; ++j) cv[j] = *reinterpret_cast<const ulonglong2*>(cp + j * 1024 + oc);
#pragma unroll
            for (int i = 0; i < RI; ++i) {
                const ulonglong2 r = *reinterpret_cast<const ulonglong2*>(rp + i * 512 + ((i & 1) ? oo : oe));
#pragma unroll
                for (int j = 0; j < C; ++j)
                    if (g_patch<M8, DIAG, LOWER>(i, j)) acc[i][j] = g_fma2(r.x, cv[j].x, acc[i][j]);
#pragma unroll
                for (int j = 0; j < C; ++j)
                    if (g_patch<M8, DIAG, LOWER>(i, j)) acc[i][j] = g_fma2(r.y, cv[j].y, acc[i][j]);
            }
        }
        if (k + DEPTH < nmine) {
            // the warp's reads of the slot come before the writes of the copies that refill it, which are the async proxy's
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) issue(k + DEPTH, d);
        }
        if (k + DEPTH < nmine) issued = k + DEPTH + 1;
        if (++d == DEPTH) { d = 0; ph ^= 1u; }
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
            for (int j = 0; j < C; ++j)
                if (g_patch<M8, DIAG, LOWER>(i, j))
                    sum[i][j] += __uint_as_float((unsigned)acc[i][j]) + __uint_as_float((unsigned)(acc[i][j] >> 32));
    }
    // after a wait gave up: the copies in flight get a bounded time to land before the shared memory is reused
    if (!alive && lane == 0)
        for (int k = max(0, issued - DEPTH); k < issued; ++k) g_wait(&bars[k % DEPTH], (unsigned)((k / DEPTH) & 1), 1LL << 16);
    __syncthreads();
    // across the warps in f64, from the last warp to the first. Either direction is as exact; the direction was chosen because
    // solves that end at the f32 residual floor are sensitive to the last bit of these sums, and with it all of the tests'
    // tight warm solves converge in the steps that they allow.
    float* red = reinterpret_cast<float*>(base);  // [warp][patch][lane]
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int j = 0; j < C; ++j)
            if (g_patch<M8, DIAG, LOWER>(i, j)) red[(warp * RI * C + i * C + j) * 32 + lane] = sum[i][j];
    __syncthreads();
    double* out = partials + (size_t)blockIdx.x * m * mc;
    for (int p = warp; p < RI * C; p += W) {
        const int i = p / C, j = p % C;
        if (!g_patch<M8, DIAG, LOWER>(i, j)) continue;
        double v = 0.0;
        for (int w = W - 1; w >= 0; --w) v += (double)red[(w * RI * C + p) * 32 + lane];
        const int row = 32 * rb + a + 4 * i;
        if (row >= m) continue;
        if (DIAG && j < M8) {
            const int col = 32 * rb + b + 8 * j;
            if (col <= row) {  // row < m
                out[(size_t)row * mc + col] = v;
                if (col != row) out[(size_t)col * mc + row] = v;
            }
        } else {
            const int t = CB * (DIAG ? rb : cb) + b + 8 * (j - (DIAG ? M8 : 0));
            if (t < nt) {
                out[(size_t)row * mc + colT + t] = v;
                if (mirrorT) out[(size_t)t * mc + row] = v;  // a foreign block of S itself: both halves of S^T S
            }
        }
    }
}

PFN_cuTensorMapEncodeTiled_v12000 g_encode() {
    static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        cudaDriverEntryPointQueryResult q;
        void* ptr = nullptr;
        KS_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q));
        if (q != cudaDriverEntryPointSuccess || !ptr) throw DeviceError("cuTensorMapEncodeTiled is not available");
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
    }();
    return fn;
}

// fields of F floats (stride F) as a 2-D tensor map with boxes of 32 points x `box_rows` fields, 128-byte swizzle
void g_rows_map(CUtensorMap* map, const float* base, long long F, int fields, int box_rows) {
    cuuint64_t dims[2] = {(cuuint64_t)F, (cuuint64_t)fields};
    cuuint64_t strides[1] = {(cuuint64_t)F * 4};
    cuuint32_t box[2] = {(cuuint32_t)GP, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode()(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw DeviceError("cuTensorMapEncodeTiled (CUDA-core Gram) failed, code " + std::to_string((int)r));
}

struct GramMaps { CUtensorMap s, t; };

template <int M8, int T8, bool DIAG, bool LOWER>
void launch_gram_piece(int blocks, long long F, const CUtensorMap& ms, const CUtensorMap& mt, int m, int nt, int mc, int rb, int cb, int colT,
                       bool mirrorT, double* partials, cudaStream_t s) {
    constexpr int W = g_warps<M8, T8, DIAG, LOWER>(), SLAB = (M8 + T8) * 1024;
    constexpr int depth = G_SMEM / (W * SLAB) < G_DEPTH ? G_SMEM / (W * SLAB) : G_DEPTH;
    constexpr int red = W * 2 * M8 * ((DIAG ? M8 : 0) + T8) * 128;
    constexpr int smem = (W * depth * SLAB > red ? W * depth * SLAB : red) + 1024;
    static_assert(depth >= 2 && smem <= 227 * 1024 - 1024, "gram piece: shared memory");
    static std::atomic<unsigned long long> attr_set{0};
    once_per_device(attr_set, [] {
        KS_CUDA(cudaFuncSetAttribute(gram_piece_kernel<M8, T8, DIAG, LOWER, depth>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    });
    gram_piece_kernel<M8, T8, DIAG, LOWER, depth><<<blocks, W * 32, smem, s>>>(ms, mt, (int)((F + GP - 1) / GP), m, nt, mc, rb, cb, colT, mirrorT,
                                                                              partials, device_error_flag());
    KS_LAUNCH_CHECK();
}

// a DIAG piece of m8 row groups and t8 groups of T
void launch_gram_diag(int m8, int t8, bool lower, int blocks, long long F, const GramMaps& g, int m, int mt, int rb,
                      double* partials, cudaStream_t s) {
#define KS_GRAM_DIAG(M, N)                                                                                                     \
    if (m8 == M && t8 == N) {                                                                                                  \
        if (lower && M == N) launch_gram_piece<M, N, true, M == N>(blocks, F, g.s, g.t, m, mt, m + mt, rb, rb, m, false, partials, s); \
        else launch_gram_piece<M, N, true, false>(blocks, F, g.s, g.t, m, mt, m + mt, rb, rb, m, false, partials, s);              \
        return;                                                                                                                \
    }
#define KS_GRAM_DIAGS(M) KS_GRAM_DIAG(M, 0) KS_GRAM_DIAG(M, 1) KS_GRAM_DIAG(M, 2) KS_GRAM_DIAG(M, 3) KS_GRAM_DIAG(M, 4)
    KS_GRAM_DIAGS(1) KS_GRAM_DIAGS(2) KS_GRAM_DIAGS(3) KS_GRAM_DIAGS(4)
    KS_GRAM_DIAG(1, 5) KS_GRAM_DIAG(1, 6) KS_GRAM_DIAG(1, 7) KS_GRAM_DIAG(1, 8)
#undef KS_GRAM_DIAGS
#undef KS_GRAM_DIAG
    throw std::logic_error("gram: piece out of range");
}

// a piece of m8 row groups and column block cb of T: 64 fields for one row group, else 32
void launch_gram_foreign(int m8, int blocks, long long F, const GramMaps& g, int m, int mt, int rb, int cb, double* partials, cudaStream_t s) {
    if (m8 == 1) launch_gram_piece<1, 8, false, false>(blocks, F, g.s, g.t, m, mt, m + mt, rb, cb, m, false, partials, s);
    else if (m8 == 2) launch_gram_piece<2, 4, false, false>(blocks, F, g.s, g.t, m, mt, m + mt, rb, cb, m, false, partials, s);
    else if (m8 == 3) launch_gram_piece<3, 4, false, false>(blocks, F, g.s, g.t, m, mt, m + mt, rb, cb, m, false, partials, s);
    else launch_gram_piece<4, 4, false, false>(blocks, F, g.s, g.t, m, mt, m + mt, rb, cb, m, false, partials, s);
}

// ---- multipole moments with on-the-fly real solid harmonics: the recurrence of harmonics.cuh with its (l, m) constants
// read from a table (f_l = sqrt((2l - 1) / (2l)), b_lm = sqrt(max((l - 1)^2 - m^2, 0)) and 1 / sqrt(l^2 - m^2), computed once
// on the host), the two previous rows kept in registers and each R_lm added to its moment as it is formed: no square
// root or division per point, no per-point array in local memory. The only difference from solid_harmonics_dev is the
// product by 1 / d instead of the division by d (within an ulp per step).
__constant__ double c_hf[7];
__constant__ double c_hb[7][7];
__constant__ double c_hinvd[7][7];

__global__ void __launch_bounds__(TPB) moments_kernel(int n, int P, long long F, double h, double origin, const float* __restrict__ rho,
                                                      double* __restrict__ partials) {
    double acc[49];
#pragma unroll
    for (int q = 0; q < 49; ++q) acc[q] = 0.0;
    const double s2 = 1.4142135623730951;
    const long long N = (long long)n * n * n;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < N; p += (long long)gridDim.x * blockDim.x) {
        int i = (int)(p % n);
        long long rest = p / n;
        int j = (int)(rest % n), k = (int)(rest / n);
        const double r = (double)rho[((long long)k * n + j) * P + i];
        if (r == 0.0) continue;
        const double x = origin + i * h, y = origin + j * h, z = origin + k * h;
        const double r2 = x * x + y * y + z * z;
        double pr[7], pi[7], qr[7], qi[7];  // rows l - 1 and l - 2 of the recurrence
        pr[0] = 1.0;
        pi[0] = 0.0;
        acc[0] += r * 1.0;
#pragma unroll
        for (int l = 1; l <= 6; ++l) {
            double cr[7], ci[7];
            cr[l] = c_hf[l] * (x * pr[l - 1] - y * pi[l - 1]);
            ci[l] = c_hf[l] * (x * pi[l - 1] + y * pr[l - 1]);
            const double a = (2.0 * l - 1.0) * z;
#pragma unroll
            for (int m = 0; m < l; ++m) {
                const double r0 = (l >= 2 && m <= l - 2) ? qr[m] : 0.0, i0 = (l >= 2 && m <= l - 2) ? qi[m] : 0.0;
                const double b = c_hb[l][m] * r2;
                cr[m] = (a * pr[m] - b * r0) * c_hinvd[l][m];
                ci[m] = (a * pi[m] - b * i0) * c_hinvd[l][m];
            }
            acc[l * l + l] += r * cr[0];
#pragma unroll
            for (int m = 1; m <= l; ++m) {
                acc[l * l + l + m] += r * (s2 * cr[m]);
                acc[l * l + l - m] += r * (s2 * ci[m]);
            }
#pragma unroll
            for (int m = 0; m <= l; ++m) {
                qr[m] = pr[m];
                qi[m] = pi[m];
                pr[m] = cr[m];
                pi[m] = ci[m];
            }
        }
    }
    // unrolled, so that acc stays in registers (a runtime index would put it in local memory for the whole kernel)
#pragma unroll
    for (int q = 0; q < 49; ++q) {
        double s = block_sum(acc[q]);
        if (threadIdx.x == 0) partials[(size_t)blockIdx.x * 49 + q] = s;
    }
}

__global__ void face_max_kernel(int n, int P, const float* __restrict__ f, double* __restrict__ partials) {
    double m = 0.0;
    const long long per_face = (long long)n * n;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < 6 * per_face; t += (long long)gridDim.x * blockDim.x) {
        int face = (int)(t / per_face);
        long long uv = t % per_face;
        int u = (int)(uv % n), v = (int)(uv / n);
        int c = (face & 1) ? n - 1 : 0;
        int i, j, k;
        switch (face >> 1) {
            case 0: i = c; j = u; k = v; break;
            case 1: i = u; j = c; k = v; break;
            default: i = u; j = v; k = c; break;
        }
        m = fmax(m, fabs((double)f[((long long)k * n + j) * P + i]));
    }
    m = block_max(m);
    if (threadIdx.x == 0) partials[blockIdx.x] = m;
}

// forces.rs:167-172 g'(d) for g(d) = erf(d/(sigma sqrt2))/d; 0 below 1e-8
__device__ __forceinline__ double g_prime(double d, double sigma) {
    if (d < 1e-8) return 0.0;
    double u = d / (sigma * 1.4142135623730951);
    return ((2.0 / 1.7724538509055159) * u * exp(-u * u) - erf(u)) / (d * d);
}

constexpr int MAX_NUC = 32;
__global__ void __launch_bounds__(TPB) forces_kernel(int n, int P, double h, double origin, const float* __restrict__ rho,
                                                     const Nuc* __restrict__ nuc, int nn, double sigma, double* __restrict__ partials) {
    double acc[3 * MAX_NUC];
    for (int q = 0; q < 3 * nn; ++q) acc[q] = 0.0;
    const long long N = (long long)n * n * n;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < N; p += (long long)gridDim.x * blockDim.x) {
        int i = (int)(p % n);
        long long rest = p / n;
        int j = (int)(rest % n), k = (int)(rest / n);
        double r = (double)rho[((long long)k * n + j) * P + i];
        if (r == 0.0) continue;
        double x = origin + i * h, y = origin + j * h, z = origin + k * h;
        for (int a = 0; a < nn; ++a) {
            double dx = x - nuc[a].x, dy = y - nuc[a].y, dz = z - nuc[a].z;
            double d = sqrt(dx * dx + dy * dy + dz * dz);
            if (d < 1e-8) continue;
            double gp = -nuc[a].Z * g_prime(d, sigma) / d;
            double w = r * gp;
            acc[3 * a] += w * dx;
            acc[3 * a + 1] += w * dy;
            acc[3 * a + 2] += w * dz;
        }
    }
    for (int q = 0; q < 3 * nn; ++q) {
        double s = block_sum(acc[q]);
        if (threadIdx.x == 0) partials[(size_t)blockIdx.x * 3 * nn + q] = s;
    }
}

// The adjoint of the Kohn-Sham energy with respect to the nuclear positions and the smearing width.
// At self-consistency E is stationary in the density, so the response of the Hartree and XC terms
// (and of the kinetic energy) to a change of V_ext vanishes and the VJP reduces to
//     dE/dR_I     = integral rho(r) dV_I/dR_I = integral rho Z_I g'(d)/d (r - R_I),   g(d) = erf(d / (sigma sqrt 2)) / d
//     dE/dsigma   = integral rho(r) sum_I dV_I/dsigma = integral rho sum_I Z_I sqrt(2/pi) exp(-d^2 / (2 sigma^2)) / sigma^2
// (V_I = -Z_I g(d); crates/qm/src/nuclear.rs:258-272 and crates/qm/src/forces.rs:177-227 for the
// position term). rho is recomputed here from the occupied orbitals of both spins in f64, not read
// from a stored density. partials: [blocks][3 nn + 1], dV not applied.
__global__ void __launch_bounds__(TPB) vjp_kernel(int n, int P, long long F, double h, double origin, const float* __restrict__ up, int nup,
                                                  const double* __restrict__ wu, const float* __restrict__ dn, int ndn,
                                                  const double* __restrict__ wd, const Nuc* __restrict__ nuc, int nn, double sigma,
                                                  double* __restrict__ partials) {
    double acc[3 * MAX_NUC + 1];
    for (int q = 0; q < 3 * nn + 1; ++q) acc[q] = 0.0;
    const long long N = (long long)n * n * n;
    const double inv2s2 = 1.0 / (2.0 * sigma * sigma);
    const double csig = 0.79788456080286536 / (sigma * sigma);  // sqrt(2/pi) / sigma^2
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < N; p += (long long)gridDim.x * blockDim.x) {
        int i = (int)(p % n);
        long long rest = p / n;
        int j = (int)(rest % n), k = (int)(rest / n);
        const long long e = ((long long)k * n + j) * P + i;
        double r = 0.0;
        for (int v = 0; v < nup; ++v) {
            const double x = (double)up[(long long)v * F + e];
            r += (wu ? wu[v] : 1.0) * x * x;
        }
        for (int v = 0; v < ndn; ++v) {
            const double x = (double)dn[(long long)v * F + e];
            r += (wd ? wd[v] : 1.0) * x * x;
        }
        if (r == 0.0) continue;
        double x = origin + i * h, y = origin + j * h, z = origin + k * h;
        for (int a = 0; a < nn; ++a) {
            double dx = x - nuc[a].x, dy = y - nuc[a].y, dz = z - nuc[a].z;
            double d2 = dx * dx + dy * dy + dz * dz;
            acc[3 * nn] += r * nuc[a].Z * csig * exp(-d2 * inv2s2);
            double d = sqrt(d2);
            if (d < 1e-8) continue;
            double w = r * nuc[a].Z * g_prime(d, sigma) / d;
            acc[3 * a] += w * dx;
            acc[3 * a + 1] += w * dy;
            acc[3 * a + 2] += w * dz;
        }
    }
    for (int q = 0; q < 3 * nn + 1; ++q) {
        double s = block_sum(acc[q]);
        if (threadIdx.x == 0) partials[(size_t)blockIdx.x * (3 * nn + 1) + q] = s;
    }
}

}  // namespace

int reduce_blocks(long long F) {
    long long want = (F / 4 + TPB - 1) / TPB;
    long long cap = 2LL * sm_count();
    return (int)std::max(1LL, std::min(want, cap));
}

void launch_finish(const double* partials, int blocks, int nvals, double scale, double* out, cudaStream_t s) {
    if (nvals >= 32) {  // enough values to fill whole lines
        FinishDesc a;
        a.partials = partials;
        a.blocks = blocks;
        a.nvals = nvals;
        a.scale = scale;
        a.out = out;
        launch_finish_pair(a, FinishDesc(), s);
        return;
    }
    finish_kernel<<<ceil_div((long long)nvals * 32, 256), 256, 0, s>>>(partials, blocks, nvals, scale, out);
    KS_LAUNCH_CHECK();
}

void launch_finish_pair(const FinishDesc& a, const FinishDesc& b, cudaStream_t s) {
    finish_many_kernel<<<ceil_div(a.nvals + b.nvals, 32), FW * 32, 0, s>>>(a, b);
    KS_LAUNCH_CHECK();
}

void launch_finish_transposed(const double* partials, int blocks, int rows, int cols, double scale, double* out, cudaStream_t s) {
    FinishDesc a;
    a.partials = partials;
    a.blocks = blocks;
    a.nvals = rows * cols;
    a.scale = scale;
    a.out = out;
    a.trows = rows;
    a.tcols = cols;
    launch_finish_pair(a, FinishDesc(), s);
}

void launch_finish_max(const double* partials, int blocks, double* out, cudaStream_t s) {
    finish_max_kernel<<<1, TPB, 0, s>>>(partials, blocks, out);
    KS_LAUNCH_CHECK();
}

void launch_dots(long long F, const Pairs& p, double* partials, int blocks, cudaStream_t s) {
    if (p.count < 1 || p.count > Pairs::MAX) throw std::invalid_argument("dots: 1..16 pairs");
    dots_kernel<<<blocks, TPB, 0, s>>>(F / 4, p, partials);
    KS_LAUNCH_CHECK();
}

static bool gram_aligned(long long F, const float* S, int mt, const float* T) {
    return F % 4 == 0 && reinterpret_cast<uintptr_t>(S) % 16 == 0 && (mt == 0 || reinterpret_cast<uintptr_t>(T) % 16 == 0);
}

int gram_blocks(long long F) { return (int)std::min((long long)sm_count(), (F + GP - 1) / GP); }

int launch_gram(long long F, int m, const float* S, int mt, const float* T, double* partials, cudaStream_t s, bool lower) {
    lower = lower && m == mt;
    const int blocks = gram_blocks(F);
    if (!gram_aligned(F, S, mt, T)) {
        // TMA needs 16-byte aligned fields: blocks of 4-byte aligned ones beyond 16 tiles take the direct form
        const int tr = ceil_div(m, GT), tt = ceil_div(mt, GT);
        if (tr * (tr + 1) / 2 + tr * tt <= 16) throw std::invalid_argument("gram: fields must be 16-byte aligned with F a multiple of 4 floats");
        const int tiles_c = ceil_div(m + mt, GT), ntiles = tr * tiles_c;
        dim3 grid(blocks, ceil_div(ntiles, GW));
        // partials are indexed by blockIdx.x only: every tile of a CTA column writes its own entries
        gram_kernel<<<grid, GW * 32, 0, s>>>(F, m, S, mt, T, tiles_c, ntiles, partials);
        KS_LAUNCH_CHECK();
        return blocks;
    }
    // 32 x 32 pieces, the row groups of 8 exact where there is one row block, and 64 columns of T for one row group, whose
    // pieces repeat the most (m = 8, mt = 120 on 48^3 / 95^3: with 8 x 32 33 / 136 us, with 8 x 64 23 / 119 us): per row
    // block the DIAG piece with its own T block (if there is one), then the foreign blocks of S below the diagonal
    // (mirrored) and the other blocks of T
    const int cw = m <= 8 ? 64 : 32, nr = ceil_div(m, 32), nt = ceil_div(mt, cw);
    const int m8 = nr == 1 ? ceil_div(m, 8) : 4, t8 = nt > 1 ? cw / 8 : ceil_div(mt, 8);
    GramMaps g;
    g_rows_map(&g.s, S, F, m, 8 * m8);
    if (mt > 0) g_rows_map(&g.t, T, F, mt, 8 * (nr > 1 ? 4 : t8));
    else g.t = g.s;
    for (int rb = 0; rb < nr; ++rb) {
        launch_gram_diag(m8, rb >= nt ? 0 : nr > 1 ? 4 : t8, lower, blocks, F, g, m, mt, rb, partials, s);
        for (int cb = 0; cb < rb; ++cb) launch_gram_piece<4, 4, false, false>(blocks, F, g.s, g.s, m, m, m + mt, rb, cb, 0, true, partials, s);
        for (int cb = 0; cb < nt; ++cb)
            if (cb != rb && !(lower && cb > rb)) launch_gram_foreign(m8, blocks, F, g, m, mt, rb, cb, partials, s);
    }
    return blocks;
}

void launch_moments(const Layout& L, const float* rho, double* partials, int blocks, cudaStream_t s) {
    static std::atomic<unsigned long long> consts_set{0};
    once_per_device(consts_set, [] {
        double f[7] = {0}, b[7][7] = {{0}}, invd[7][7] = {{0}};
        for (int l = 1; l <= 6; ++l) {
            f[l] = std::sqrt((2.0 * l - 1.0) / (2.0 * l));
            for (int m = 0; m < l; ++m) {
                b[l][m] = std::sqrt(std::fmax((l - 1.0) * (l - 1.0) - (double)m * m, 0.0));
                invd[l][m] = 1.0 / std::sqrt((double)l * l - (double)m * m);
            }
        }
        KS_CUDA(cudaMemcpyToSymbol(c_hf, f, sizeof(f)));
        KS_CUDA(cudaMemcpyToSymbol(c_hb, b, sizeof(b)));
        KS_CUDA(cudaMemcpyToSymbol(c_hinvd, invd, sizeof(invd)));
    });
    moments_kernel<<<blocks, TPB, 0, s>>>(L.n, L.P, L.F, L.h, L.origin, rho, partials);
    KS_LAUNCH_CHECK();
}

void launch_face_max(const Layout& L, const float* f, double* partials, int blocks, cudaStream_t s) {
    face_max_kernel<<<blocks, TPB, 0, s>>>(L.n, L.P, f, partials);
    KS_LAUNCH_CHECK();
}

void launch_vjp(const Layout& L, const float* up, int nup, const double* wu, const float* dn, int ndn, const double* wd, const Nuc* nuc,
                int nn, double sigma, double* partials, int blocks, cudaStream_t s) {
    if (nn > MAX_NUC) throw std::invalid_argument("vjp: at most 32 nuclei");
    vjp_kernel<<<blocks, TPB, 0, s>>>(L.n, L.P, L.F, L.h, L.origin, up, nup, wu, dn, ndn, wd, nuc, nn, sigma, partials);
    KS_LAUNCH_CHECK();
}

void launch_forces(const Layout& L, const float* rho, const Nuc* nuc, int nn, double sigma, double* partials, int blocks,
                   cudaStream_t s) {
    if (nn > MAX_NUC) throw std::invalid_argument("forces: at most 32 nuclei");
    forces_kernel<<<blocks, TPB, 0, s>>>(L.n, L.P, L.h, L.origin, rho, nuc, nn, sigma, partials);
    KS_LAUNCH_CHECK();
}

}  // namespace ks
