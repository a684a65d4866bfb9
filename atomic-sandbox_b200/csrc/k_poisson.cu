// k_poisson.cu -- Hartree solve pieces on sm_100a: the multipole boundary right-hand side, the
// geometric-multigrid V-cycle kernels and the device-side CG scalar updates.
//
// Equation and boundary split: crates/qm/src/poisson.rs:1-70 (A V = b, A = -L_int,
// b = 4 pi rho + L_bc, ghost values from the l <= 6 solid-harmonic expansion). Multigrid:
// crates/qm-gpu/src/multigrid.rs:1-60 and shaders/multigrid.wgsl -- 2nd-order 7-point operator per
// level, coarse points at odd fine indices, Dirichlet boundary d spacings beyond the end points
// (linear extrapolation of the missing neighbour, x_ghost = (1 - 1/d) x_0), damped Jacobi with
// omega = 6/7, full weighting and trilinear prolongation. No ghost cells are stored: a missing
// neighbour reads as zero. A level's fields stay in the L2, so a step costs its launch latency and its instructions: the
// kernels take one thread per (x, y) column of 4 points with 32-bit indices from the grid, march z with the neighbours in
// registers, and the first two sweeps (from x = 0) are one kernel that reads only b. Levels at or below 12^3 run as one
// single-CTA kernel whose fields never leave shared memory. Fusing a level's whole descent and ascent into one kernel
// each over shared-memory tiles with recomputed halos measured slower (95^3: 30 + 28 us).
#include <cmath>
#include "kernels.cuh"
#include "reduce_util.cuh"
#include "harmonics.cuh"

namespace ks {

namespace {

constexpr int TPB = 256;
constexpr double PI = 3.14159265358979323846;

inline int blocks_for(long long work) {
    long long b = (work + TPB - 1) / TPB;
    long long cap = 8LL * sm_count();
    return (int)std::max(1LL, std::min(b, cap));
}

// two block sums of a 2-D CTA (as block_sum: fixed shuffle tree, fixed warp order); valid in thread (0, 0)
__device__ __forceinline__ double2 block_sum_xy(double a, double b) {
    __shared__ double2 part[32];
    const int t = threadIdx.y * blockDim.x + threadIdx.x, lane = t & 31, warp = t >> 5, nw = (blockDim.x * blockDim.y + 31) >> 5;
    a = warp_sum(a);
    b = warp_sum(b);
    if (lane == 0) part[warp] = make_double2(a, b);
    __syncthreads();
    double2 s = make_double2(0.0, 0.0);
    if (warp == 0) {
        if (lane < nw) s = part[lane];
        s.x = warp_sum(s.x);
        s.y = warp_sum(s.y);
    }
    return s;
}

// V_bc(r) = sum_l (sum_m Q_lm R_lm(r)) / |r|^(2l+1)  (crates/qm/src/poisson.rs:185-199)
__device__ double bc_value(const double* q, double x, double y, double z) {
    double d2 = x * x + y * y + z * z;
    double hv[49];
    solid_harmonics_dev(x, y, z, hv);
    double acc = 0.0, inv_pow = 1.0 / sqrt(d2);
    for (int l = 0; l <= 6; ++l) {
        double s = 0.0;
        for (int m = -l; m <= l; ++m) s += q[l * l + l + m] * hv[l * l + l + m];
        acc += s * inv_pow;
        inv_pow /= d2;
    }
    return acc;
}

// ghost table: face = 2*axis + (high side), depth 1..4 beyond the face, (u, v) = the other two
// axes in increasing order
__global__ void ghost_kernel(int n, double h, double origin, const double* __restrict__ q, double* __restrict__ ghost) {
    const long long per = (long long)n * n;
    const long long total = 6LL * 4 * per;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
        int face = (int)(t / (4 * per));
        long long rem = t % (4 * per);
        int depth = (int)(rem / per) + 1;
        long long uv = rem % per;
        int u = (int)(uv % n), v = (int)(uv / n);
        int axis = face >> 1;
        bool high = face & 1;
        int c[3];
        int ua = axis == 0 ? 1 : 0, va = axis == 2 ? 1 : 2;
        c[ua] = u;
        c[va] = v;
        c[axis] = high ? n - 1 + depth : -depth;
        ghost[t] = bc_value(q, origin + c[0] * h, origin + c[1] * h, origin + c[2] * h);
    }
}

__global__ void rhs_kernel(int n, int P, long long F, double h, const float* __restrict__ rho, const double* __restrict__ ghost,
                           float* __restrict__ b) {
    const double COEFF[5] = {-205.0 / 72.0, 8.0 / 5.0, -1.0 / 5.0, 8.0 / 315.0, -1.0 / 560.0};
    const double inv_h2 = 1.0 / (h * h);
    const long long per = (long long)n * n;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < F; e += (long long)gridDim.x * blockDim.x) {
        int i = (int)(e % P);
        long long row = e / P;
        int j = (int)(row % n), k = (int)(row / n);
        if (i >= n) { b[e] = 0.0f; continue; }
        double val = 4.0 * PI * (double)rho[e];
        int pos[3] = {i, j, k};
        bool near = false;
        for (int a = 0; a < 3; ++a) near = near || pos[a] < 4 || pos[a] >= n - 4;
        if (near) {
            double acc = 0.0;
            for (int axis = 0; axis < 3; ++axis) {
                int ua = axis == 0 ? 1 : 0, va = axis == 2 ? 1 : 2;
                long long uv = pos[ua] + (long long)n * pos[va];
                for (int m = 1; m <= 4; ++m) {
                    // sign -1 then +1 (crates/qm/src/poisson.rs:166-176)
                    if (pos[axis] - m < 0) {
                        int depth = m - pos[axis];
                        acc += COEFF[m] * ghost[((long long)(2 * axis) * 4 + (depth - 1)) * per + uv];
                    }
                    if (pos[axis] + m >= n) {
                        int depth = pos[axis] + m - (n - 1);
                        acc += COEFF[m] * ghost[((long long)(2 * axis + 1) * 4 + (depth - 1)) * per + uv];
                    }
                }
            }
            val += acc * inv_h2;
        }
        b[e] = (float)val;
    }
}

// ---- multigrid (7-point A_2 per level with boundary-distance ghost factors)
// the diagonal of A_2 (times h^2) at a point: 6 minus the factors of its missing neighbours
__device__ __forceinline__ float mg_diag(const MgLevel& L, int i, int j, int k) {
    float g = 0.f;
    if (i == 0) g += L.g_low;
    if (j == 0) g += L.g_low;
    if (k == 0) g += L.g_low;
    if (i == L.n - 1) g += L.g_high;
    if (j == L.n - 1) g += L.g_high;
    if (k == L.n - 1) g += L.g_high;
    return 6.0f - g;
}
__device__ __forceinline__ bool mg_inside(int n, int i, int j, int k) {
    return (unsigned)i < (unsigned)n && (unsigned)j < (unsigned)n && (unsigned)k < (unsigned)n;
}
// omega / diag: the division only where a neighbour is missing
__device__ __forceinline__ float mg_weight(float omega, float w6, float diag) { return diag == 6.0f ? w6 : omega / diag; }
// one damped sweep and the residual of a point, nb the sum of its neighbours: the same roundings on every level and form
__device__ __forceinline__ float mg_swept(float xq, float b, float nb, float diag, float w, float h2) {
    return fmaf(w, fmaf(-diag, xq, fmaf(h2, b, nb)), xq);
}
__device__ __forceinline__ float mg_res(float xq, float b, float nb, float diag, float h2) { return b + fmaf(-diag, xq, nb) / h2; }

constexpr int MX = 32, MY = 8, MZ = 4;  // threads in x and y, points per thread in z
// body(i, j, k, e): the thread's points, e the element index (F < 2^31)
template <class F>
__device__ __forceinline__ void mg_points(const MgLevel& L, F&& body) {
    const int i = blockIdx.x * MX + threadIdx.x, j = blockIdx.y * MY + threadIdx.y;
    if (i >= L.n || j >= L.n) return;
    const int k0 = blockIdx.z * MZ;
#pragma unroll
    for (int t = 0; t < MZ; ++t) {
        const int k = k0 + t;
        if (k < L.n) body(i, j, k, (k * L.n + j) * L.P + i);
    }
}
// the sum of the six neighbours of x[e] (0 beyond the box)
__device__ __forceinline__ float mg_neighbours(const MgLevel& L, const float* __restrict__ x, int i, int j, int k, int e) {
    const int sy = L.P, sz = L.n * L.P;
    const float xm = i > 0 ? x[e - 1] : 0.f, xp = i < L.n - 1 ? x[e + 1] : 0.f;
    const float ym = j > 0 ? x[e - sy] : 0.f, yp = j < L.n - 1 ? x[e + sy] : 0.f;
    const float zm = k > 0 ? x[e - sz] : 0.f, zp = k < L.n - 1 ? x[e + sz] : 0.f;
    return ((xp + xm) + (yp + ym)) + (zp + zm);
}

// x = two damped Jacobi sweeps from zero: the first, x1 = (omega / diag) h^2 b, is formed at the seven points it is read at
__global__ void __launch_bounds__(MX * MY) mg_first_kernel(MgLevel L, const float* __restrict__ b, float* __restrict__ x, float omega) {
    const float h2 = (float)(L.h * L.h), w6 = omega / 6.0f;
    auto x1 = [&](int i, int j, int k, int e) { return __fmul_rn(mg_weight(omega, w6, mg_diag(L, i, j, k)), h2 * b[e]); };
    mg_points(L, [&](int i, int j, int k, int e) {
        const int n = L.n, sy = L.P, sz = n * L.P;
        const float xm = i > 0 ? x1(i - 1, j, k, e - 1) : 0.f, xp = i < n - 1 ? x1(i + 1, j, k, e + 1) : 0.f;
        const float ym = j > 0 ? x1(i, j - 1, k, e - sy) : 0.f, yp = j < n - 1 ? x1(i, j + 1, k, e + sy) : 0.f;
        const float zm = k > 0 ? x1(i, j, k - 1, e - sz) : 0.f, zp = k < n - 1 ? x1(i, j, k + 1, e + sz) : 0.f;
        const float nb = ((xp + xm) + (yp + ym)) + (zp + zm);
        const float diag = mg_diag(L, i, j, k), w = mg_weight(omega, w6, diag), bv = b[e];
        x[e] = mg_swept(w * (h2 * bv), bv, nb, diag, w, h2);
    });
}

// out = one sweep on x; with DOT also the CTA's partial sums of b.out and b.b (the PCG's r.z and r.r)
template <bool DOT>
__global__ void __launch_bounds__(MX * MY) mg_sweep_kernel(MgLevel L, const float* __restrict__ x, const float* __restrict__ b,
                                                           float* __restrict__ out, float omega, double* __restrict__ partials) {
    const float h2 = (float)(L.h * L.h), w6 = omega / 6.0f;
    double rz = 0.0, rr = 0.0;
    mg_points(L, [&](int i, int j, int k, int e) {
        const float diag = mg_diag(L, i, j, k), xq = x[e], bv = b[e];
        const float v = mg_swept(xq, bv, mg_neighbours(L, x, i, j, k, e), diag, mg_weight(omega, w6, diag), h2);
        out[e] = v;
        if (DOT) {
            rz += (double)bv * v;
            rr += (double)bv * bv;
        }
    });
    if (DOT) {
        const double2 s = block_sum_xy(rz, rr);
        if (threadIdx.x == 0 && threadIdx.y == 0) {
            const size_t cta = blockIdx.x + (size_t)gridDim.x * (blockIdx.y + (size_t)gridDim.y * blockIdx.z);
            partials[2 * cta] = s.x;
            partials[2 * cta + 1] = s.y;
        }
    }
}

__global__ void __launch_bounds__(MX * MY) mg_residual_kernel(MgLevel L, const float* __restrict__ x, const float* __restrict__ b,
                                                              float* __restrict__ out) {
    const float h2 = (float)(L.h * L.h);
    mg_points(L, [&](int i, int j, int k, int e) {
        out[e] = mg_res(x[e], b[e], mg_neighbours(L, x, i, j, k, e), mg_diag(L, i, j, k), h2);
    });
}

// bc = the full-weighted residual at the coarse points (fine index 2 c + 1; only the high side can lie beyond the box)
__global__ void __launch_bounds__(MX * MY) mg_restrict_kernel(MgLevel C, MgLevel L, const float* __restrict__ r, float* __restrict__ bc) {
    const int i = blockIdx.x * MX + threadIdx.x, j = blockIdx.y * MY + threadIdx.y, k = blockIdx.z;
    if (i >= C.n || j >= C.n) return;
    const bool hx = 2 * i + 2 < L.n;
    float s = 0.f;
#pragma unroll
    for (int dz = 0; dz < 3; ++dz) {
        if (2 * k + dz >= L.n) continue;
#pragma unroll
        for (int dy = 0; dy < 3; ++dy) {
            if (2 * j + dy >= L.n) continue;
            const float w = (dy == 1 ? 0.5f : 0.25f) * (dz == 1 ? 0.5f : 0.25f);
            const float* q = r + ((2 * k + dz) * L.n + 2 * j + dy) * L.P + 2 * i;
            s += 0.25f * w * q[0];
            s += 0.5f * w * q[1];
            if (hx) s += 0.25f * w * q[2];
        }
    }
    bc[(k * C.n + j) * C.P + i] = s;
}

// P xc at a fine point: odd index 2 c + 1 takes coarse c, even 2 c half of c - 1 and of c (zero beyond the box)
template <class X>
__device__ __forceinline__ float mg_interpolated(int n, int i, int j, int k, X&& xc) {
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const int ci = (c & 1) ? i >> 1 : (i - 1) >> 1, cj = (c & 2) ? j >> 1 : (j - 1) >> 1, ck = (c & 4) ? k >> 1 : (k - 1) >> 1;
        if (((c & 1) && (i & 1)) || ((c & 2) && (j & 1)) || ((c & 4) && (k & 1))) continue;  // the one neighbour of an odd index
        const float w = ((i & 1) ? 1.f : 0.5f) * ((j & 1) ? 1.f : 0.5f) * ((k & 1) ? 1.f : 0.5f);
        if (mg_inside(n, ci, cj, ck)) s = fmaf(w, xc(ci, cj, ck), s);
    }
    return s;
}
// x += P xc
__global__ void __launch_bounds__(MX * MY) mg_prolong_kernel(MgLevel C, MgLevel L, const float* __restrict__ xc, float* __restrict__ x) {
    mg_points(L, [&](int i, int j, int k, int e) {
        x[e] += mg_interpolated(C.n, i, j, k, [&](int ci, int cj, int ck) { return xc[(ck * C.n + cj) * C.P + ci]; });
    });
}

// The bottom of the V-cycle (levels of at most 12^3) in one CTA with every field in shared memory: level 0's right-hand
// side is read from b, its solution written to x. Same sequence as the larger levels (two sweeps from zero, residual,
// restriction, recursion, prolongation, two sweeps; the coarsest level does `coarsest` sweeps). A thread owns a (i, j)
// column of a level, or a part of one where the level has few columns, and marches k with the z-neighbours in registers.
constexpr int CT = 1024;  // threads
struct CLevel { int n, nn, groups; float h2, gl, gh; float *x, *b, *t; };
template <class F>
__device__ __forceinline__ void c_columns(const CLevel& L, F&& body) {  // body(c, i, j, k0, k1): the thread's column part
    const int c = threadIdx.x % L.nn, g = threadIdx.x / L.nn;
    if (g >= L.groups) return;
    const int per = (L.n + L.groups - 1) / L.groups;
    body(c, c % L.n, c / L.n, g * per, min(L.n, (g + 1) * per));
}
__device__ __forceinline__ float c_diag(const CLevel& L, int i, int j, int k) {  // as mg_diag
    float g = 0.f;
    if (i == 0) g += L.gl;
    if (j == 0) g += L.gl;
    if (k == 0) g += L.gl;
    if (i == L.n - 1) g += L.gh;
    if (j == L.n - 1) g += L.gh;
    if (k == L.n - 1) g += L.gh;
    return 6.0f - g;
}
// out = sweep(src) (RES false) or the residual b - A src (RES true)
template <bool RES>
__device__ __forceinline__ void c_apply(const CLevel& L, const float* src, float* out, float omega) {
    const float w6 = omega / 6.0f;
    c_columns(L, [&](int c, int i, int j, int k0, int k1) {
        const int n = L.n, nn = L.nn;
        if (k0 >= k1) return;
        float zm = k0 > 0 ? src[(k0 - 1) * nn + c] : 0.f, xq = src[k0 * nn + c];
        for (int k = k0; k < k1; ++k) {
            const int e = k * nn + c;
            const float zp = k + 1 < n ? src[e + nn] : 0.f;
            const float xm = i > 0 ? src[e - 1] : 0.f, xp = i < n - 1 ? src[e + 1] : 0.f;
            const float ym = j > 0 ? src[e - n] : 0.f, yp = j < n - 1 ? src[e + n] : 0.f;
            const float nb = ((xp + xm) + (yp + ym)) + (zp + zm);
            const float diag = c_diag(L, i, j, k);
            out[e] = RES ? mg_res(xq, L.b[e], nb, diag, L.h2) : mg_swept(xq, L.b[e], nb, diag, mg_weight(omega, w6, diag), L.h2);
            zm = xq;
            xq = zp;
        }
    });
    __syncthreads();
}
// the first sweep from x = 0
__device__ __forceinline__ void c_first(const CLevel& L, float* out, float omega) {
    const float w6 = omega / 6.0f;
    c_columns(L, [&](int c, int i, int j, int k0, int k1) {
        for (int k = k0; k < k1; ++k) out[k * L.nn + c] = mg_weight(omega, w6, c_diag(L, i, j, k)) * (L.h2 * L.b[k * L.nn + c]);
    });
    __syncthreads();
}

__global__ void __launch_bounds__(CT) mg_coarse_kernel(MgCoarse c, const float* __restrict__ b, float* __restrict__ x, float omega,
                                                       int coarsest) {
    extern __shared__ float sm[];
    const int nl = c.nlev;
    auto level = [&](int l) {
        CLevel L;
        float* p = sm;
        for (int q = 0; q < l; ++q) p += 3 * c.lv[q].n * c.lv[q].n * c.lv[q].n;
        L.n = c.lv[l].n;
        L.nn = L.n * L.n;
        L.groups = min(L.n, CT / L.nn);
        L.h2 = (float)(c.lv[l].h * c.lv[l].h);
        L.gl = c.lv[l].g_low;
        L.gh = c.lv[l].g_high;
        L.x = p;
        L.b = p + L.nn * L.n;
        L.t = p + 2 * L.nn * L.n;
        return L;
    };
    {
        const CLevel L = level(0);
        c_columns(L, [&](int col, int i, int j, int k0, int k1) {
            for (int k = k0; k < k1; ++k) L.b[k * L.nn + col] = b[((long long)k * L.n + j) * c.lv[0].P + i];
        });
        __syncthreads();
    }
    for (int l = 0; l < nl; ++l) {  // descend
        const CLevel L = level(l);
        c_first(L, L.t, omega);
        if (l == nl - 1) {  // the rest of the coarsest level's sweeps, the last one into x
            float* src = L.t;
            float* dst = L.x;
            for (int s = 1; s < coarsest; ++s) {
                c_apply<false>(L, src, dst, omega);
                float* o = src;
                src = dst;
                dst = o;
            }
            if (src != L.x) {
                c_columns(L, [&](int col, int, int, int k0, int k1) {
                    for (int k = k0; k < k1; ++k) L.x[k * L.nn + col] = src[k * L.nn + col];
                });
                __syncthreads();
            }
            break;
        }
        c_apply<false>(L, L.t, L.x, omega);
        c_apply<true>(L, L.x, L.t, omega);
        const CLevel N = level(l + 1);
        c_columns(N, [&](int col, int i, int j, int k0, int k1) {
            for (int k = k0; k < k1; ++k) {
                float s = 0.f;
                for (int dz = -1; dz <= 1; ++dz) {
                    const int z = 2 * k + 1 + dz;
                    if (z >= L.n) continue;
                    for (int dy = -1; dy <= 1; ++dy) {
                        const int y = 2 * j + 1 + dy;
                        if (y >= L.n) continue;
                        for (int dx = -1; dx <= 1; ++dx) {
                            const int xx = 2 * i + 1 + dx;
                            if (xx >= L.n) continue;
                            s += (dx == 0 ? 0.5f : 0.25f) * (dy == 0 ? 0.5f : 0.25f) * (dz == 0 ? 0.5f : 0.25f) * L.t[(z * L.n + y) * L.n + xx];
                        }
                    }
                }
                N.b[k * N.nn + col] = s;
            }
        });
        __syncthreads();
    }
    for (int l = nl - 2; l >= 0; --l) {  // ascend
        const CLevel L = level(l), N = level(l + 1);
        c_columns(L, [&](int col, int i, int j, int k0, int k1) {
            for (int k = k0; k < k1; ++k)
                L.x[k * L.nn + col] += mg_interpolated(N.n, i, j, k, [&](int ci, int cj, int ck) { return N.x[(ck * N.n + cj) * N.n + ci]; });
        });
        __syncthreads();
        c_apply<false>(L, L.x, L.t, omega);
        c_apply<false>(L, L.t, L.x, omega);
    }
    const CLevel L = level(0);
    c_columns(L, [&](int col, int i, int j, int k0, int k1) {
        for (int k = k0; k < k1; ++k) x[((long long)k * L.n + j) * c.lv[0].P + i] = L.x[k * L.nn + col];
    });
}

// ---- CG updates. scal layout: [1], [3] r.z and [2], [4] r.r (alternating). The dot products arrive as one f64 partial per
// CTA of the kernel that formed them: every CTA sums the same partials in the same order (a few KB from L2, cheaper than a
// launch of its own), CTA 0 also stores the sums.
__device__ double partial_sum(const double* __restrict__ partials, int count, int stride) {
    __shared__ double total;
    double s = 0.0;
    for (int t = threadIdx.x; t < count; t += TPB) s += partials[(size_t)t * stride];
    s = block_sum(s);
    if (threadIdx.x == 0) total = s;
    __syncthreads();
    const double r = total;
    __syncthreads();  // total is reused by the next call
    return r;
}

// partials: the Laplacian's sums of p.(L p), so p.Ap = -sum
__global__ void __launch_bounds__(TPB) cg_update_kernel(long long F4, float4* __restrict__ v, float4* __restrict__ r,
                                                        const float4* __restrict__ p, const float4* __restrict__ ap,
                                                        const double* __restrict__ partials, int count, const double* __restrict__ scal,
                                                        int rz_slot, double* __restrict__ pap_out) {
    const double pap = -partial_sum(partials, count, 1), rz = scal[rz_slot];
    if (blockIdx.x == 0 && threadIdx.x == 0) *pap_out = pap;
    const bool ok = pap > 0.0 && rz > 0.0;
    const float alpha = ok ? (float)(rz / pap) : 0.0f;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < F4; e += (long long)gridDim.x * blockDim.x) {
        float4 pv = p[e], a = ap[e], vv = v[e], rv = r[e];
        // v += alpha p; r -= alpha A p = r + alpha L p  (ap holds L p)
        vv.x = fmaf(alpha, pv.x, vv.x); vv.y = fmaf(alpha, pv.y, vv.y); vv.z = fmaf(alpha, pv.z, vv.z); vv.w = fmaf(alpha, pv.w, vv.w);
        rv.x = fmaf(alpha, a.x, rv.x); rv.y = fmaf(alpha, a.y, rv.y); rv.z = fmaf(alpha, a.z, rv.z); rv.w = fmaf(alpha, a.w, rv.w);
        v[e] = vv;
        r[e] = rv;
    }
}

// partials: pairs (r.z, r.r). rz_old < 0: the first direction, p = z.
__global__ void __launch_bounds__(TPB) cg_direction_kernel(long long F4, float4* __restrict__ p, const float4* __restrict__ z,
                                                           const double* __restrict__ partials, int count, double* __restrict__ scal,
                                                           int rz_old, int rz_new, double* __restrict__ dots_out) {
    const double rz = partial_sum(partials, count, 2), rr = partial_sum(partials + 1, count, 2);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        scal[rz_new] = rz;
        scal[rz_new + 1] = rr;
        dots_out[0] = rz;
        dots_out[1] = rr;
    }
    const float beta = rz_old < 0 ? 0.f : (float)(rz / scal[rz_old]);
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < F4; e += (long long)gridDim.x * blockDim.x) {
        float4 zz = z[e];
        if (rz_old >= 0) {
            const float4 pp = p[e];
            zz.x = fmaf(beta, pp.x, zz.x); zz.y = fmaf(beta, pp.y, zz.y); zz.z = fmaf(beta, pp.z, zz.z); zz.w = fmaf(beta, pp.w, zz.w);
        }
        p[e] = zz;
    }
}

}  // namespace

void launch_poisson_rhs(const Layout& L, const float* rho, const double* q, double* ghost, float* b, cudaStream_t s) {
    const long long need = 24LL * L.n * L.n;
    ghost_kernel<<<blocks_for(need), TPB, 0, s>>>(L.n, L.h, L.origin, q, ghost);
    KS_LAUNCH_CHECK();
    rhs_kernel<<<blocks_for(L.F), TPB, 0, s>>>(L.n, L.P, L.F, L.h, rho, ghost, b);
    KS_LAUNCH_CHECK();
}

static dim3 mg_grid(int n, int per_z) { return dim3(ceil_div(n, MX), ceil_div(n, MY), ceil_div(n, per_z)); }
int mg_sweep_ctas(const MgLevel& lv) {
    const dim3 g = mg_grid(lv.n, MZ);
    return (int)(g.x * g.y * g.z);
}
void launch_mg_first(const MgLevel& lv, const float* b, float* x, float omega, cudaStream_t s) {
    mg_first_kernel<<<mg_grid(lv.n, MZ), dim3(MX, MY), 0, s>>>(lv, b, x, omega);
    KS_LAUNCH_CHECK();
}
void launch_mg_sweep(const MgLevel& lv, const float* x, const float* b, float* out, float omega, double* partials, cudaStream_t s) {
    if (partials) mg_sweep_kernel<true><<<mg_grid(lv.n, MZ), dim3(MX, MY), 0, s>>>(lv, x, b, out, omega, partials);
    else mg_sweep_kernel<false><<<mg_grid(lv.n, MZ), dim3(MX, MY), 0, s>>>(lv, x, b, out, omega, nullptr);
    KS_LAUNCH_CHECK();
}
void launch_mg_residual(const MgLevel& lv, const float* x, const float* b, float* out, cudaStream_t s) {
    mg_residual_kernel<<<mg_grid(lv.n, MZ), dim3(MX, MY), 0, s>>>(lv, x, b, out);
    KS_LAUNCH_CHECK();
}
void launch_mg_restrict(const MgLevel& coarse, const MgLevel& fine, const float* r, float* bc, cudaStream_t s) {
    mg_restrict_kernel<<<mg_grid(coarse.n, 1), dim3(MX, MY), 0, s>>>(coarse, fine, r, bc);
    KS_LAUNCH_CHECK();
}
void launch_mg_prolong_add(const MgLevel& coarse, const MgLevel& fine, const float* xc, float* x, cudaStream_t s) {
    mg_prolong_kernel<<<mg_grid(fine.n, MZ), dim3(MX, MY), 0, s>>>(coarse, fine, xc, x);
    KS_LAUNCH_CHECK();
}
void launch_mg_coarse(const MgCoarse& c, const float* b, float* x, float omega, int coarsest_sweeps, cudaStream_t s) {
    if (c.nlev <= 0) return;
    size_t floats = 0;
    for (int l = 0; l < c.nlev; ++l) floats += 3 * (size_t)c.lv[l].n * c.lv[l].n * c.lv[l].n;
    constexpr int cap = 227 * 1024 - 1024;
    if (floats * 4 > (size_t)cap) throw std::logic_error("multigrid: the coarse levels do not fit one CTA");
    static std::atomic<unsigned long long> attr_set{0};
    once_per_device(attr_set, [] { KS_CUDA(cudaFuncSetAttribute(mg_coarse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, cap)); });
    mg_coarse_kernel<<<1, CT, floats * 4, s>>>(c, b, x, omega, coarsest_sweeps);
    KS_LAUNCH_CHECK();
}

void launch_cg_update(long long F, float* v, float* r, const float* p, const float* ap, const double* partials, int count, const double* scal,
                      int rz_slot, double* pap_out, cudaStream_t s) {
    cg_update_kernel<<<blocks_for(F / 4), TPB, 0, s>>>(F / 4, reinterpret_cast<float4*>(v), reinterpret_cast<float4*>(r),
                                                      reinterpret_cast<const float4*>(p), reinterpret_cast<const float4*>(ap), partials,
                                                      count, scal, rz_slot, pap_out);
    KS_LAUNCH_CHECK();
}
void launch_cg_direction(long long F, float* p, const float* z, const double* partials, int count, double* scal, int rz_old, int rz_new,
                         double* dots_out, cudaStream_t s) {
    cg_direction_kernel<<<blocks_for(F / 4), TPB, 0, s>>>(F / 4, reinterpret_cast<float4*>(p), reinterpret_cast<const float4*>(z), partials,
                                                         count, scal, rz_old, rz_new, dots_out);
    KS_LAUNCH_CHECK();
}

}  // namespace ks
