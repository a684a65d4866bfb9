// k_stencil.cu -- the 8th-order finite-difference stencil family on sm_100a: Laplacian, H psi
// (-1/2 lap + V psi) and the fused damped-Jacobi sweep of the LOBPCG preconditioner.
//
// Reference operators: crates/qm/src/stencil.rs:21-51 (coefficients c = [-205/72, 8/5, -1/5,
// 8/315, -1/560], Dirichlet zero outside the box), crates/qm-gpu/src/shaders/stencil.wgsl:58-106
// (hamiltonian, jacobi_step). The centre is folded into differences of neighbours (below), exact in real arithmetic
// because c_0 = -2 sum c_m, and exact per difference in f32 for smooth f, which keeps the f32 residual floor of the
// reference's stop rules. The operator's scale (1/h^2, or -1/(2 h^2) for H) multiplies the sum.
//
// B200 design ("2.5-D" tiling): a CTA owns a BX x 16 (x, y) tile of one field and marches a z-chunk. Each z-plane
// of the tile plus its 4-point xy halo is staged in shared memory by one TMA load (cp.async.bulk.tensor.4d); the tensor
// map's extent is n on every axis, so the halo beyond the box arrives as the hardware's zero fill -- the Dirichlet
// boundary costs no branches and no ghost storage. A ring of 8 planes keeps up to four planes of prefetch in flight.
// Each thread owns four consecutive x-outputs of two adjacent rows: it reads its centre, x- and y-neighbours as 16-byte
// quads (16 shared loads per 8 outputs: the new plane's two, the centre's two, four x-neighbours and eight more y-rows, ten
// rows serving both output rows) and works on packed pairs with Blackwell's f32x2 arithmetic. The z-direction holds no queue
// of planes: a new plane's second difference is added to the seven outputs it belongs to (ZRow), so nothing moves between
// registers. The V / R reads (cp.async copies one plane ahead into a small shared ring) and the stores are coalesced 16-byte
// accesses; the quad's pad columns are stored as 0.
//
// What bounds it: instruction issue and the fixed latencies behind it at 12 warps per SM (58 % of the issue slots, FMA pipe
// 53 % active). With one row per thread, a nine-deep register queue in z and symmetric differences (the form this
// replaces) 128 outputs took 250 warp instructions, now 173. Measured per launch, before and after, H psi back to back: 95^3 x
// 16 vectors 43.0 -> 34.9 us, 128^3 x 40 216 -> 170 us, 48^3 x 8 8.3 -> 7.2 us, 33^3 x 3 5.4 -> 4.9 us of device time; a sweep on
// 128^3 x 20 in a solve 160 -> 125 us.
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <cudaTypedefs.h>
#include "kernels.cuh"
#include "reduce_util.cuh"

namespace ks {

namespace {

typedef unsigned long long u64;

constexpr int BY = 16;                              // tile rows
constexpr int HYW = BY + 8;
constexpr int ROWS = 2;                             // adjacent rows per thread
// A tile of BX columns: the staged plane with its halo, and one thread per x-quad and row pair. 12 warps per SM (registers
// capped at 168 per thread): 6 CTAs of 64 threads, 4 of 96 or 3 of 128; only the sweep at BX = 32 holds 10, since the shared
// memory of its larger side ring (39 KB per CTA) fits 5 times.
template <int BX>
struct Tile {
    static constexpr int HXW = BX + 8;
    static constexpr int QX = BX / 4;
    static constexpr int THREADS = QX * (BY / ROWS);
    static constexpr int PLANE_FLOATS = HXW * HYW;
    static constexpr unsigned PLANE_BYTES = PLANE_FLOATS * 4;
    static constexpr int CTAS_PER_SM = 12 * 32 / THREADS;
    // The TMA rules the plane loads rely on, checked here because a violation faults the GPU instead of returning an
    // error: the box's inner extent is a multiple of 16 bytes; a load's x coordinate, x0 - 4 with x0 a multiple of BX,
    // times 4 bytes is a multiple of 16 (negative x is allowed for loads and reads the zero fill); each ring plane starts
    // on a 128-byte boundary. The quads the threads read start on 16-byte boundaries: rows of HXW floats, quads at
    // 4 * tx + 4 (and +-4 for the x-neighbours).
    static_assert((HXW * 4) % 16 == 0, "TMA box inner extent must be a multiple of 16 bytes");
    static_assert((BX * 4) % 16 == 0 && (4 * 4) % 16 == 0, "TMA x coordinate x0 - 4 must be a multiple of 16 bytes");
    static_assert(PLANE_BYTES % 128 == 0, "ring planes must start on 128-byte boundaries");
    static_assert(THREADS % 32 == 0, "whole warps");
};
// ring depth in planes: a step reads planes s + 4 (the centre) and s + 8 (the newest), so five planes are live and the
// others in flight. The Jacobi mode's larger side ring leaves room for 7.
template <int MODE>
constexpr int ring_depth() { return MODE == ST_JACOBI ? 7 : 8; }
// The per-plane global reads of a step (V; r and the stored factor in the Jacobi mode) are staged one plane ahead by
// per-thread cp.async copies into a 2-deep shared "side" ring (at BX = 32, 48, 64: 12, 18, 24 KB per CTA in the Jacobi mode, 4,
// 6, 8 KB for H and the residual form), so their latency runs behind the previous plane's arithmetic without holding registers.
constexpr int SD = 2;
template <int MODE>
constexpr int n_side() { return MODE == ST_JACOBI ? 3 : (MODE == ST_LAPLACIAN ? 0 : 1); }
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
constexpr long long WAIT_LIMIT = 1LL << 22;         // bounded mbarrier waits (~seconds)
constexpr long long DRAIN_LIMIT = 1LL << 16;        // waits for copies in flight after a wait gave up

// The 8th-order second difference sum_m c_m (f_m - 2 f_0 + f_-m) on the first differences e_j = f_j+1 - f_j
//     sum_{j=0..3} b_j (e_j - e_-1-j),  b_j = sum_{m > j} c_m   (x and y)
// and on the second differences s_i = e_i - e_i-1
//     sum_{|i| <= 3} g_|i| s_i,         g_i = sum_{j >= i} b_j  (z).
// kappa is free in exact arithmetic: the coefficients are divided by it and the operator's scale multiplied. It is the
// f32 value in [1, 2) for which the rounded coefficients come closest to the exact ones in the operator's second moment
// (what a smooth field sees: sum_j (2j + 1) b_j and g_0 + 2 (g_1 + g_2 + g_3) are off by 4e-11) and in b_0, b_1, g_0, g_1; the
// plain c_m rounded to f32 are off by up to 8e-8. The scale is applied as an f32 pair hi + lo, so 1/h^2 is not rounded
// to f32 either. Against 64 bits the operator's error is 0.82 .. 1.06 of the direct difference form's
// sum_m c_m [(f_m - f_0) + (f_-m - f_0)] over h = 0.18 .. 0.30, smooth and rough fields (0.93 in the mean).
constexpr double KAPPA = 1.6073455810546875;
constexpr double C1 = 8.0 / 5.0, C2 = -1.0 / 5.0, C3 = 8.0 / 315.0, C4 = -1.0 / 560.0;
constexpr double B3D = C4, B2D = C3 + B3D, B1D = C2 + B2D, B0D = C1 + B1D;
constexpr double G2D = B2D + B3D, G1D = B1D + G2D, G0D = B0D + G1D;
constexpr float CB0 = (float)(B0D / KAPPA), CB1 = (float)(B1D / KAPPA), CB2 = (float)(B2D / KAPPA), CB3 = (float)(B3D / KAPPA);
constexpr float CG0 = (float)(G0D / KAPPA), CG1 = (float)(G1D / KAPPA), CG2 = (float)(G2D / KAPPA);

struct Params {
    int n, P;
    long long F;
    int tiles_x, tiles_y, zc;
    float scale_hi, scale_lo, omega, diag_t;
    const float* V;
    const float* R;
    const double* lambda;
    double* dot_partials;
    int* err;
    int vec0;
    const double* theta;
    float* out2;
    float* dinv;
};

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: false (and the error flag raised) when the copy did not complete within `limit` polls.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity, int* err, long long limit = WAIT_LIMIT) {
    long long spins = 0;
    while (!mbar_try_wait(bar, parity)) {
        if (++spins > limit) {
            if (err) atomicExch(err, 1);
            return false;
        }
    }
    return true;
}
__device__ __forceinline__ void tma_load_plane(float* dst, const CUtensorMap* map, int x, int y, int z, int v, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(
            smem_u32(dst)),
        "l"((unsigned long long)map), "r"(x), "r"(y), "r"(z), "r"(v), "r"(smem_u32(bar))
        : "memory");
}

// Before a TMA load refills a ring slot: the barrier orders the CTA's reads of the slot before this thread, the fence
// orders them before the load's writes, which are the async proxy's. What counts is one proxy fence on the path from the
// reads to the load: here the barrier makes the issuing thread's enough; where the readers signal an mbarrier instead (the
// block update, the CUDA-core Gram) they fence before they signal. Without it reads that were still in flight when
// the barrier released thread 0 could see the new plane: with kernels of three streams on the chip, solves stopped
// being bit for bit reproducible.
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ---- packed f32x2 arithmetic (sm_100): one instruction for two x-neighbours
__device__ __forceinline__ u64 add2(u64 a, u64 b) { u64 d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ u64 sub2(u64 a, u64 b) { u64 d; asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ u64 mul2(u64 a, u64 b) { u64 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
    u64 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ u64 pk(float lo, float hi) {
    u64 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float lo_of(u64 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi_of(u64 v) { return __uint_as_float((unsigned)(v >> 32)); }
// four x-consecutive values as two packed pairs
struct Quad { u64 a, b; };
__device__ __forceinline__ Quad ldq(const float* p) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    return {v.x, v.y};
}
__device__ __forceinline__ Quad ldq(const float4* p) { return ldq(reinterpret_cast<const float*>(p)); }
__device__ __forceinline__ Quad operator-(const Quad& x, const Quad& y) { return {sub2(x.a, y.a), sub2(x.b, y.b)}; }
__device__ __forceinline__ Quad operator+(const Quad& x, const Quad& y) { return {add2(x.a, y.a), add2(x.b, y.b)}; }
__device__ __forceinline__ Quad fmaq(u64 k, const Quad& x, const Quad& y) { return {fma2(k, x.a, y.a), fma2(k, x.b, y.b)}; }
__device__ __forceinline__ Quad mulq(u64 k, const Quad& x) { return {mul2(k, x.a), mul2(k, x.b)}; }
__device__ __forceinline__ Quad fmaq(const Quad& x, const Quad& y, const Quad& z) { return {fma2(x.a, y.a, z.a), fma2(x.b, y.b, z.b)}; }
__device__ __forceinline__ u64 rep(float v) { return pk(v, v); }
// (v, v) kept in a register pair: the compiler would rather rebuild a constant pair at every use
__device__ __forceinline__ u64 rep_kept(float v) {
    u64 d;
    asm volatile("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
    return d;
}
struct Pairs { u64 b0, b1, b2, b3, g0, g1, g2, hi, lo; };  // the coefficients (g_3 = b_3) and the scale, as (k, k)

// One row's z direction: the sums of the six output planes still open, the last value and the last first difference.
// A plane's second difference is added to the seven outputs it belongs to as it becomes known, each sum moving to its
// neighbour's register in the same FMA, so the march needs no queue of values and no register moves.
struct ZRow {
    Quad p0, p1, p2, p3, p4, p5, f, e;
    __device__ __forceinline__ void start(const Quad& f0, const Quad& f1) {
        const Quad z = {0, 0};
        p0 = p1 = p2 = p3 = p4 = p5 = z;
        e = f1 - f0;
        f = f1;
    }
    // the next plane's values in, the finished sum of the plane four below out
    __device__ __forceinline__ Quad push(const Quad& fn, const Pairs& k) {
        const Quad en = fn - f, s = en - e;
        f = fn;
        e = en;
        const Quad done = fmaq(k.b3, s, p0);
        p0 = fmaq(k.g2, s, p1);
        p1 = fmaq(k.g1, s, p2);
        p2 = fmaq(k.g0, s, p3);
        p3 = fmaq(k.g1, s, p4);
        p4 = fmaq(k.g2, s, p5);
        p5 = mulq(k.b3, s);
        return done;
    }
};

// the x direction's e_j - e_-1-j, j = 0..3, of the quad c between its neighbour quads l and r. The pairs of odd offsets
// straddle two registers, so these are scalar subtractions, each difference shared by the outputs it belongs to.
__device__ __forceinline__ void x_terms(const Quad& l, const Quad& c, const Quad& r, Quad (&d)[4]) {
    const float xs[12] = {lo_of(l.a), hi_of(l.a), lo_of(l.b), hi_of(l.b), lo_of(c.a), hi_of(c.a),
                          lo_of(c.b), hi_of(c.b), lo_of(r.a), hi_of(r.a), lo_of(r.b), hi_of(r.b)};
    float e[11];
#pragma unroll
    for (int i = 0; i < 11; ++i) e[i] = xs[i + 1] - xs[i];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        d[j].a = pk(e[4 + j] - e[3 - j], e[5 + j] - e[4 - j]);
        d[j].b = pk(e[6 + j] - e[5 - j], e[7 + j] - e[6 - j]);
    }
}

// f64 sum of f0 * o over the valid elements of a quad (the Poisson p.Ap and the kinetic <psi, lap psi>)
__device__ __forceinline__ double quad_dot(const Quad& f, const Quad& o, bool e1, bool e2, bool e3) {
    double d = (double)lo_of(f.a) * (double)lo_of(o.a);
    if (e1) d += (double)hi_of(f.a) * (double)hi_of(o.a);
    if (e2) d += (double)lo_of(f.b) * (double)lo_of(o.b);
    if (e3) d += (double)hi_of(f.b) * (double)hi_of(o.b);
    return d;
}
__device__ __forceinline__ void store_quad(float* dst, const Quad& o, bool e1, bool e2, bool e3) {
    *reinterpret_cast<float4*>(dst) = make_float4(lo_of(o.a), e1 ? hi_of(o.a) : 0.f, e2 ? lo_of(o.b) : 0.f, e3 ? hi_of(o.b) : 0.f);
}

template <int MODE, bool DOT, int BX>
__global__ void __launch_bounds__(Tile<BX>::THREADS, Tile<BX>::CTAS_PER_SM) stencil_kernel(const __grid_constant__ CUtensorMap tmap, Params p, float* __restrict__ out) {
    constexpr int HXW = Tile<BX>::HXW, PLANE_FLOATS = Tile<BX>::PLANE_FLOATS, THREADS = Tile<BX>::THREADS, NS = ring_depth<MODE>();
    constexpr unsigned PLANE_BYTES = Tile<BX>::PLANE_BYTES;
    extern __shared__ __align__(1024) float ring[];  // NS planes of HXW x 24
    __shared__ __align__(8) uint64_t bar[NS];

    const int vec = blockIdx.y;
    int b = blockIdx.x;
    const int tile_x = b % p.tiles_x;
    b /= p.tiles_x;
    const int tile_y = b % p.tiles_y;
    const int chunk = b / p.tiles_y;
    const int x0 = tile_x * BX, y0 = tile_y * BY;
    const int z0 = chunk * p.zc;
    const int nz = min(z0 + p.zc, p.n) - z0;
    const int nplanes = nz + 8;  // relative plane q <-> z = z0 - 4 + q
    const int tx = threadIdx.x % Tile<BX>::QX, ty = threadIdx.x / Tile<BX>::QX;
    const int gx = x0 + 4 * tx, gy = y0 + ROWS * ty;
    // the quad's elements inside the box (gx is a multiple of 4 below n <= P, so the whole quad lies inside the
    // row's P floats; elements at or past n are pad columns and are stored as 0)
    const bool ok[ROWS] = {gx < p.n && gy < p.n, gx < p.n && gy + 1 < p.n};
    const bool e1 = gx + 1 < p.n, e2 = gx + 2 < p.n, e3 = gx + 3 < p.n;
    const int ci = (ROWS * ty + 4) * HXW + 4 * tx + 4;

    if (threadIdx.x == 0) {
        for (int i = 0; i < NS; ++i) mbar_init(&bar[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    auto issue = [&](int q) {
        const int bb = q % NS;
        mbar_expect_tx(&bar[bb], PLANE_BYTES);
        tma_load_plane(ring + bb * PLANE_FLOATS, &tmap, x0 - 4, y0 - 4, z0 - 4 + q, p.vec0 + vec, &bar[bb]);
    };
    // A wait that gives up raises the error flag and marks the thread dead: a dead thread waits no longer than a poll
    // for later planes, thread 0 issues no further loads once dead, and before exiting thread 0 waits a bounded time
    // for its copies still in flight. The CTA's outputs are then undefined (the host reports the error).
    int issued = 0;  // planes issued so far (thread 0's count)
    if (threadIdx.x == 0)
        for (; issued < min(NS, nplanes); ++issued) issue(issued);

    // 32-bit offsets inside a field (F < 2^31) from per-vector bases: one address instruction per access
    const int plane = p.n * p.P;
    const int row0 = (z0 * p.n + gy) * p.P + gx;
    const long long vbase = (long long)vec * p.F;
    const float* rbase = p.R ? p.R + vbase : nullptr;
    float* obase = out + vbase;
    float* obase2 = (MODE == ST_HAM_RESIDUAL) ? p.out2 + vbase : nullptr;
    float* dbase = p.dinv ? p.dinv + vbase : nullptr;
    // the side ring, [SD][NSIDE][ROWS][THREADS] float4 after the plane ring: slot t % SD holds this thread's V (r, factor)
    // quads of output plane t. Each thread reads only its own copies, after its own wait_group, and refills a slot
    // only after the step that read it has consumed the values.
    constexpr int NSIDE = n_side<MODE>();
    float4* side = reinterpret_cast<float4*>(ring + NS * PLANE_FLOATS) + threadIdx.x;
    auto side_issue = [&](int t, int off) {
        if (NSIDE > 0) {
            if (t < nz) {
                float4* dst = side + (t % SD) * NSIDE * ROWS * THREADS;
#pragma unroll
                for (int w = 0; w < ROWS; ++w)
                    if (ok[w]) {
                        cp_async16(dst + w * THREADS, p.V + (off + w * p.P));
                        if (MODE == ST_JACOBI) {
                            cp_async16(dst + (ROWS + w) * THREADS, rbase + (off + w * p.P));
                            if (dbase) cp_async16(dst + (2 * ROWS + w) * THREADS, dbase + (off + w * p.P));
                        }
                    }
            }
            cp_async_commit();  // one group per plane, empty or not, so that wait_group counts planes
        }
    };
#pragma unroll
    for (int t = 0; t < SD - 1; ++t) side_issue(t, row0 + t * plane);

    const Pairs k = {rep_kept(CB0), rep_kept(CB1), rep_kept(CB2), rep_kept(CB3), rep_kept(CG0), rep_kept(CG1), rep_kept(CG2),
                     rep_kept(p.scale_hi), rep_kept(p.scale_lo)};
    ZRow zr[ROWS];
    bool alive = true;
    auto plane_in = [&](int q) {  // planes 0..7 of the march's start
        alive = mbar_wait(&bar[q % NS], (unsigned)((q / NS) & 1), p.err, alive ? WAIT_LIMIT : 1) && alive;
        return ring + (q % NS) * PLANE_FLOATS + ci;
    };
    {
        Quad f0[ROWS];
        const float* at = plane_in(0);
#pragma unroll
        for (int w = 0; w < ROWS; ++w) f0[w] = ldq(at + w * HXW);
        at = plane_in(1);
#pragma unroll
        for (int w = 0; w < ROWS; ++w) zr[w].start(f0[w], ldq(at + w * HXW));
    }
#pragma unroll
    for (int i = 2; i < 8; ++i) {
        if (i == 4) {
            __syncthreads();  // planes 0..3 are consumed: their buffers take the next four
            if (alive && threadIdx.x == 0) {
                proxy_fence();
                for (; issued < min(NS + 4, nplanes); ++issued) issue(issued);
            }
        }
        const float* at = plane_in(i);
#pragma unroll
        for (int w = 0; w < ROWS; ++w) zr[w].push(ldq(at + w * HXW), k);
    }

    const float lam = (MODE == ST_JACOBI || MODE == ST_HAM_RESIDUAL) ? (float)p.lambda[vec] : 0.0f;
    // theta split into f32 hi + lo, as the residual kernel does: r = fma(-lo, x, fma(-hi, x, Hx))
    const double th = (MODE == ST_HAM_RESIDUAL) ? p.theta[vec] : 0.0;
    const float th_hi = (float)th, th_lo = (float)(th - (double)th_hi);
    double dot = 0.0;
    // two steps per iteration where the side ring is read or two fields are stored (95^3 k = 8: the sweep 29.1 -> 28.3 us, the
    // residual form 41.4 -> 39.8), one for H and the Laplacian, which gained nothing
    constexpr int STEPS = MODE == ST_JACOBI || MODE == ST_HAM_RESIDUAL ? 2 : 1;
    int sn = 8 % NS, sc = 4 % NS;  // ring slots of the newest and the centre plane
    unsigned pn = (8 / NS) & 1;    // parity of the newest plane's round
    int off = row0;
#pragma unroll STEPS
    for (int s = 0; s < nz; ++s, off += plane) {
        alive = mbar_wait(&bar[sn], pn, p.err, alive ? WAIT_LIMIT : 1) && alive;
        // the next plane's side copies go out before this plane's are read
        side_issue(s + SD - 1, off + (SD - 1) * plane);
        const float* fresh = ring + sn * PLANE_FLOATS + ci;
        const float* cpl = ring + sc * PLANE_FLOATS + ci;
        Quad acc[ROWS], f[ROWS];
#pragma unroll
        for (int w = 0; w < ROWS; ++w) {
            acc[w] = zr[w].push(ldq(fresh + w * HXW), k);
            f[w] = ldq(cpl + w * HXW);
        }
        Quad dx[ROWS][4];
#pragma unroll
        for (int w = 0; w < ROWS; ++w) x_terms(ldq(cpl + w * HXW - 4), f[w], ldq(cpl + w * HXW + 4), dx[w]);
        // first differences along y of the rows gy - 4 .. gy + 5: ey[i] between rows gy + i - 4 and gy + i - 3
        Quad ey[9];
        {
            Quad prev = ldq(cpl - 4 * HXW);
#pragma unroll
            for (int i = 0; i < 9; ++i) {
                const int rr = i - 3;
                const Quad next = rr == 0 ? f[0] : rr == 1 ? f[1] : ldq(cpl + rr * HXW);
                ey[i] = next - prev;
                prev = next;
            }
        }
#pragma unroll
        for (int j = 3; j >= 0; --j) {
#pragma unroll
            for (int w = 0; w < ROWS; ++w) {
                const Quad d = (ey[4 + w + j] - ey[3 + w - j]) + dx[w][j];
                acc[w] = fmaq(j == 3 ? k.b3 : j == 2 ? k.b2 : j == 1 ? k.b1 : k.b0, d, acc[w]);
            }
        }
        if (NSIDE > 0) cp_async_wait<SD - 1>();
        const float4* sl = side + (s % SD) * NSIDE * ROWS * THREADS;
#pragma unroll
        for (int w = 0; w < ROWS; ++w) {
            Quad o = fmaq(k.hi, acc[w], mulq(k.lo, acc[w]));
            if (MODE != ST_LAPLACIAN && ok[w]) {
                const float4 v = sl[w * THREADS];
                const Quad h = fmaq(ldq(sl + w * THREADS), f[w], o);
                if (MODE == ST_HAMILTONIAN) {
                    o = h;
                } else if (MODE == ST_HAM_RESIDUAL) {
                    // r = Hx - theta x (hi and lo parts of theta), w0 = r / max(diag_t + V - lambda, 0.1)
                    o = fmaq(rep(-th_lo), f[w], fmaq(rep(-th_hi), f[w], h));
                    const float w0 = lo_of(o.a) / fmaxf(p.diag_t + v.x - lam, 0.1f);
                    const float w1 = hi_of(o.a) / fmaxf(p.diag_t + v.y - lam, 0.1f);
                    const float w2 = lo_of(o.b) / fmaxf(p.diag_t + v.z - lam, 0.1f);
                    const float w3 = hi_of(o.b) / fmaxf(p.diag_t + v.w - lam, 0.1f);
                    *reinterpret_cast<float4*>(obase2 + (off + w * p.P)) = make_float4(w0, e1 ? w1 : 0.f, e2 ? w2 : 0.f, e3 ? w3 : 0.f);
                    if (dbase) {  // the sweeps' factor, as the JACOBI mode computes it
                        const float d0 = p.omega * (1.0f / fmaxf(p.diag_t + v.x - lam, 0.1f));
                        const float d1 = p.omega * (1.0f / fmaxf(p.diag_t + v.y - lam, 0.1f));
                        const float d2 = p.omega * (1.0f / fmaxf(p.diag_t + v.z - lam, 0.1f));
                        const float d3 = p.omega * (1.0f / fmaxf(p.diag_t + v.w - lam, 0.1f));
                        *reinterpret_cast<float4*>(dbase + (off + w * p.P)) = make_float4(d0, e1 ? d1 : 0.f, e2 ? d2 : 0.f, e3 ? d3 : 0.f);
                    }
                } else {
                    // w + (omega / max(diag_t + V - lambda, 0.1)) (r - (H w - lambda w)), as the scalar sweep (an
                    // approximate division measured 2 % faster per solve but moved the NH3 96^3 finite-difference check
                    // of the adjoint past its bound: the sweep keeps the IEEE division)
                    const Quad u = ldq(sl + (ROWS + w) * THREADS) - fmaq(rep(-lam), f[w], h);
                    Quad fac;
                    if (dbase) {  // the factor stored by the residual pass of this iteration
                        fac = ldq(sl + (2 * ROWS + w) * THREADS);
                    } else {
                        fac.a = pk(p.omega * (1.0f / fmaxf(p.diag_t + v.x - lam, 0.1f)), p.omega * (1.0f / fmaxf(p.diag_t + v.y - lam, 0.1f)));
                        fac.b = pk(p.omega * (1.0f / fmaxf(p.diag_t + v.z - lam, 0.1f)), p.omega * (1.0f / fmaxf(p.diag_t + v.w - lam, 0.1f)));
                    }
                    o = fmaq(fac, u, f[w]);
                }
            }
            if (ok[w]) {
                store_quad(obase + (off + w * p.P), o, e1, e2, e3);
                if (DOT) dot += quad_dot(MODE == ST_HAM_RESIDUAL ? o : f[w], o, e1, e2, e3);
            }
        }
        __syncthreads();  // the centre plane's buffer is free
        if (alive && threadIdx.x == 0 && s + 4 + NS < nplanes) {
            proxy_fence();
            issue(s + 4 + NS);
            issued = s + 5 + NS;
        }
        if (++sn == NS) { sn = 0; pn ^= 1u; }
        if (++sc == NS) sc = 0;
    }
    // after a wait gave up: the latest copy issued into each slot may still be in flight (a parity wait on a slot's
    // latest copy is unambiguous, and returns at once for one that arrived)
    if (threadIdx.x == 0 && !alive)
        for (int qq = max(0, issued - NS); qq < issued; ++qq) mbar_wait(&bar[qq % NS], (unsigned)((qq / NS) & 1), nullptr, DRAIN_LIMIT);
    if (DOT) {
        const double sum = block_sum(dot);
        // [vector][CTA] for the Laplacian / H dots; [CTA][vector] for the residual norms (the residual kernel's layout)
        if (threadIdx.x == 0) {
            if (MODE == ST_HAM_RESIDUAL) p.dot_partials[(size_t)blockIdx.x * gridDim.y + blockIdx.y] = sum;
            else p.dot_partials[blockIdx.x + (size_t)gridDim.x * blockIdx.y] = sum;
        }
    }
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    // resolved once (thread-safe static initialisation)
    static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        cudaDriverEntryPointQueryResult q;
        void* ptr = nullptr;
        KS_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q));
        if (q != cudaDriverEntryPointSuccess || !ptr) throw DeviceError("cuTensorMapEncodeTiled is not available");
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
    }();
    return fn;
}

struct Shape { int tiles_x, tiles_y, chunks, zc; };

// The tile width of an n^3 grid: the fewest tile columns for the work in them. A tile's plane costs its arithmetic, which
// grows with the width, but no less than a fixed part (the 24 TMA rows, the barrier), about that of 42 columns: a row of tiles
// costs tiles x max(264, 6.25 BX). Measured with every width forced to 32 / 48 / 64 (us, events around each launch of a solve,
// which add up to 5 us to the shortest): the sweep at 48^3 k = 4 10.9 / 10.7 / 10.7 and H at k = 8 12.9 / 10.7 / 12.7; 64^3 k = 8
// 16.2 / 18.9 / 14.8; 95^3 k = 8 31.2 / 29.1 / 36.7; 128^3 k = 20 147 / 158 / 125; H at 128^3 k = 40 177 / 197 / 176.
int tile_width(int n) {
    int best = 32;
    double cost = 1e30;
    for (int bx : {32, 48, 64}) {
        const double c = ceil_div(n, bx) * std::max(264.0, 6.25 * bx);
        if (c < cost) {
            cost = c;
            best = bx;
        }
    }
    return best;
}

// shared memory of a launch, and the CTAs of it that an SM holds: 228 KB with 1 KB reserved per CTA, of which the
// kernel's static part is under 1 KB
template <int MODE, int BX>
constexpr int smem_bytes() { return ring_depth<MODE>() * (int)Tile<BX>::PLANE_BYTES + SD * n_side<MODE>() * ROWS * Tile<BX>::THREADS * 16; }
template <int MODE, int BX>
constexpr int ctas_of() {
    const int by_smem = (228 * 1024) / (smem_bytes<MODE, BX>() + 1536);
    return by_smem < Tile<BX>::CTAS_PER_SM ? by_smem : Tile<BX>::CTAS_PER_SM;
}
int ctas_per_sm(int mode, int bx) {
    if (mode == ST_JACOBI) return bx == 32 ? ctas_of<ST_JACOBI, 32>() : bx == 48 ? ctas_of<ST_JACOBI, 48>() : ctas_of<ST_JACOBI, 64>();
    return bx == 32 ? ctas_of<ST_HAMILTONIAN, 32>() : bx == 48 ? ctas_of<ST_HAMILTONIAN, 48>() : ctas_of<ST_HAMILTONIAN, 64>();
}

// The grid: (x, y) tiles x vectors x z-chunks. A CTA's time is about (its planes + prologue) steps
// whatever else runs, and the launch takes ceil(CTAs / resident slots) such rounds, so the chunk count minimises
// waves x (zc + c) with c the fixed cost of a chunk in plane steps (its 8 halo planes, partly hidden behind the other
// resident CTAs; c = 8 measured best against 12 and 4). Chunks go down to 4 planes, which only grids that leave the chip
// idle reach. Device time of a call there: 33^3 x 3 with 7 chunks of 5 planes 4.9 us, with 4 of 9 6.8 us; 48^3 x 4 with 12 of
// 4 planes 4.5 us, with 6 of 8 6.3 us.
Shape shape_for(const Layout& L, int count, int mode) {
    const int bx = tile_width(L.n);
    Shape sh;
    sh.tiles_x = ceil_div(L.n, bx);
    sh.tiles_y = ceil_div(L.n, BY);
    const long long per_chunk = (long long)sh.tiles_x * sh.tiles_y * count;
    const long long slots = (long long)ctas_per_sm(mode, bx) * sm_count();
    long long best = -1;
    for (int c = 1; c <= stencil_max_chunks(L); ++c) {
        const int zc = ceil_div(L.n, c);
        const int cc = ceil_div(L.n, zc);
        const long long waves = (cc * per_chunk + slots - 1) / slots;
        const long long cost = waves * (zc + 8);
        if (best < 0 || cost < best) {
            best = cost;
            sh.zc = zc;
            sh.chunks = cc;
        }
    }
    return sh;
}

// the shape of a launch with c z-chunks per tile column
Shape shape_with_chunks(const Layout& L, int c) {
    Shape sh;
    sh.tiles_x = ceil_div(L.n, tile_width(L.n));
    sh.tiles_y = ceil_div(L.n, BY);
    sh.zc = ceil_div(L.n, std::max(1, std::min(c, L.n)));
    sh.chunks = ceil_div(L.n, sh.zc);
    return sh;
}

// the autotuner's table: (device, n, count, mode) -> z-chunks
std::mutex tune_mu;
std::atomic<int> tune_entries{0};  // table size, read without the lock by every tunable launch
std::map<std::tuple<int, int, int, int>, int>& tune_table() {
    static std::map<std::tuple<int, int, int, int>, int> t;
    return t;
}
int current_device() {
    int d = 0;
    KS_CUDA(cudaGetDevice(&d));
    return d;
}

template <int MODE, bool DOT, int BX>
void launch_tile(const Shape& sh, int count, const CUtensorMap& tmap, const Params& p, float* out, cudaStream_t s) {
    constexpr int smem = smem_bytes<MODE, BX>();
    static std::atomic<unsigned long long> attr_set{0};
    once_per_device(attr_set, [] {
        KS_CUDA(cudaFuncSetAttribute(stencil_kernel<MODE, DOT, BX>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        // the rings of an SM's CTAs need the large shared-memory carveout
        KS_CUDA(cudaFuncSetAttribute(stencil_kernel<MODE, DOT, BX>, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    });
    dim3 grid(sh.tiles_x * sh.tiles_y * sh.chunks, count);
    stencil_kernel<MODE, DOT, BX><<<grid, Tile<BX>::THREADS, smem, s>>>(tmap, p, out);
    KS_LAUNCH_CHECK();
}

template <int MODE, bool DOT>
void launch_mode(const Shape& sh, int count, const CUtensorMap& tmap, const Params& p, float* out, cudaStream_t s) {
    const int bx = tile_width(p.n);
    if (bx == 32) launch_tile<MODE, DOT, 32>(sh, count, tmap, p, out, s);
    else if (bx == 48) launch_tile<MODE, DOT, 48>(sh, count, tmap, p, out, s);
    else launch_tile<MODE, DOT, 64>(sh, count, tmap, p, out, s);
}

}  // namespace

void make_field_tmap(CUtensorMap* map, const Layout& L, const float* base, int count) {
    cuuint64_t dims[4] = {(cuuint64_t)L.n, (cuuint64_t)L.n, (cuuint64_t)L.n, (cuuint64_t)count};
    cuuint64_t strides[3] = {(cuuint64_t)L.P * 4, (cuuint64_t)L.n * L.P * 4, (cuuint64_t)L.F * 4};
    cuuint32_t box[4] = {(cuuint32_t)(tile_width(L.n) + 8), HYW, 1, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(base), dims, strides, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw DeviceError("cuTensorMapEncodeTiled failed (code " + std::to_string((int)r) + ")");
}

void stencil_set_tuned_chunks(int n, int count, int mode, int chunks) {
    if (mode != ST_HAMILTONIAN && mode != ST_JACOBI) throw std::invalid_argument("stencil tuning: only H psi and the Jacobi sweep are tuned");
    if (n < 1 || count < 1 || chunks < 1 || chunks > n) throw std::invalid_argument("stencil tuning: need n, count >= 1 and 1 <= chunks <= n");
    std::lock_guard<std::mutex> g(tune_mu);
    tune_table()[std::make_tuple(current_device(), n, count, mode)] = chunks;
    tune_entries.store((int)tune_table().size());
}

int stencil_tuned_chunks(int n, int count, int mode) {
    if (tune_entries.load() == 0) return 0;
    const int dev = current_device();
    std::lock_guard<std::mutex> g(tune_mu);
    auto it = tune_table().find(std::make_tuple(dev, n, count, mode));
    return it == tune_table().end() ? 0 : it->second;
}

// chunks of 4 planes at least: what the cost model searches and the autotuner times
int stencil_max_chunks(const Layout& L) { return std::max(1, L.n / 4); }

int stencil_model_chunks(const Layout& L, int count, int mode) { return shape_for(L, count, mode).chunks; }

std::vector<std::array<int, 4>> stencil_tuning_entries() {
    const int dev = current_device();
    std::lock_guard<std::mutex> g(tune_mu);
    std::vector<std::array<int, 4>> out;
    for (const auto& e : tune_table())
        if (std::get<0>(e.first) == dev) out.push_back({std::get<1>(e.first), std::get<2>(e.first), std::get<3>(e.first), e.second});
    return out;
}

void stencil_tuning_clear() {
    const int dev = current_device();
    std::lock_guard<std::mutex> g(tune_mu);
    for (auto it = tune_table().begin(); it != tune_table().end();)
        it = std::get<0>(it->first) == dev ? tune_table().erase(it) : std::next(it);
    tune_entries.store((int)tune_table().size());
}

int stencil_ctas_per_vector(const Layout& L, int count) {
    Shape sh = shape_for(L, count, ST_HAM_RESIDUAL);
    return sh.tiles_x * sh.tiles_y * sh.chunks;
}

int launch_stencil(const Layout& L, const CUtensorMap& tmap, int count, const StencilArgs& a, float* out, cudaStream_t s) {
    if (count <= 0) return 0;
    // the quads' 16-byte loads and stores need 16-byte aligned fields (P is a multiple of 4 floats)
    if ((reinterpret_cast<uintptr_t>(out) & 15) || (a.V && (reinterpret_cast<uintptr_t>(a.V) & 15)) ||
        (a.R && (reinterpret_cast<uintptr_t>(a.R) & 15)) || (a.out2 && (reinterpret_cast<uintptr_t>(a.out2) & 15)) ||
        (a.dinv && (reinterpret_cast<uintptr_t>(a.dinv) & 15)))
        throw std::invalid_argument("stencil: fields must be 16-byte aligned");
    const bool dot = a.dot_partials != nullptr;
    // the chunking: the caller's, else the autotuner's for the modes whose outputs do not depend on it, else the model's
    int chunks = a.chunks;
    if (chunks <= 0 && !dot && (a.mode == ST_HAMILTONIAN || a.mode == ST_JACOBI)) chunks = stencil_tuned_chunks(L.n, count, a.mode);
    if (chunks > 0 && dot) throw std::invalid_argument("stencil: a forced chunking is for the launches without dot partials");
    Shape sh = chunks > 0 ? shape_with_chunks(L, chunks) : shape_for(L, count, a.mode);
    Params p;
    p.n = L.n;
    p.P = L.P;
    p.F = L.F;
    p.tiles_x = sh.tiles_x;
    p.tiles_y = sh.tiles_y;
    p.zc = sh.zc;
    const double scale = a.scale * KAPPA;
    p.scale_hi = (float)scale;
    p.scale_lo = (float)(scale - (double)p.scale_hi);
    p.omega = a.omega;
    p.diag_t = a.diag_t;
    p.V = a.V;
    p.R = a.R;
    p.lambda = a.lambda;
    p.dot_partials = a.dot_partials;
    p.err = device_error_flag();
    p.vec0 = a.vec0;
    p.theta = a.theta;
    p.out2 = a.out2;
    p.dinv = a.dinv;
    switch (a.mode) {
        case ST_LAPLACIAN:
            if (dot) launch_mode<ST_LAPLACIAN, true>(sh, count, tmap, p, out, s);
            else launch_mode<ST_LAPLACIAN, false>(sh, count, tmap, p, out, s);
            break;
        case ST_HAMILTONIAN:
            if (dot) launch_mode<ST_HAMILTONIAN, true>(sh, count, tmap, p, out, s);
            else launch_mode<ST_HAMILTONIAN, false>(sh, count, tmap, p, out, s);
            break;
        case ST_HAM_RESIDUAL:
            if (!dot || !a.theta || !a.lambda || !a.out2 || !a.V) throw std::invalid_argument("stencil: the residual form needs theta, lambda, V, W0 and partials");
            launch_mode<ST_HAM_RESIDUAL, true>(sh, count, tmap, p, out, s);
            break;
        default:
            if (dot) throw std::invalid_argument("stencil: dot partials are for the Laplacian, H and the residual form only");
            launch_mode<ST_JACOBI, false>(sh, count, tmap, p, out, s);
            break;
    }
    return sh.tiles_x * sh.tiles_y * sh.chunks * count;
}

}  // namespace ks
