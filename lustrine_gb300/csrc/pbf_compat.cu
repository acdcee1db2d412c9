// pbf_compat.cu -- the reference's fluid step (mode R) on the GPU.
//
// Semantics of Lustrine::simulate_fluid (Simulate.cpp:27-115) with its
// neighbour search (Neighbors.cpp:366-450) and cubic kernel (Kernels.cpp:6-41),
// float operation for float operation.  This translation unit is compiled with
// --fmad=false: the reference's arithmetic has no fused multiply-adds, and
// with the same operation order the neighbour sets, lambdas and positions
// are bit-identical to the reference's.  The one intended difference is the
// position update, which is Jacobi (every particle reads its neighbours'
// positions from before the pass) instead of the reference's in-place
// Gauss-Seidel sweep, which has no parallel form.
#include "pbf_common.cuh"
#include "pbf_compat.cuh"
#include "pbf_kernels.h"

namespace lgb {

// a / b correctly rounded from y = 1 / b correctly rounded, the divisor known
// in advance (Brisebarre, Muller and Raina, "Accelerating correctly rounded
// floating-point division when the divisor is known in advance", IEEE Trans.
// Comput. 2004): a product, its remainder, one correction, where a division
// that knows neither takes some 13 instructions.  The remainder has to be
// exact: a not below 2^-100 or zero (its sign kept), b within 2^-60 .. 2^60.
__device__ __forceinline__ float div_known(float a, float b, float y) {
    const float q = __fmul_rn(a, y);
    return __fmaf_rn(-__fmaf_rn(b, q, -a), y, q);
}

// q = r kfac / h of the kernels.  rcp_h: 1 / h, or 0 where h is out of
// div_known's range.  (Below 2^-100 the quotient's last bits may differ: W is
// then its value at 0 and the gradient 0 either way.)
__device__ __forceinline__ float q_ref(const StepParams& p, float r) {
    const float rl = r * p.kfac;
    return p.rcp_h != 0.0f ? div_known(rl, p.h, p.rcp_h) : rl / p.h;
}

// cubic_kernel (Kernels.cpp:6-19)
__device__ __forceinline__ float W_ref(const StepParams& p, float r) {
    float q = q_ref(p, r);
    float result = 0.0f;
    if (q <= 1.0f) {
        if (q <= 0.5f) {
            float q2 = q * q;
            float q3 = q2 * q;
            float a = 6.0f * q3;
            float b = 6.0f * q2;
            result = p.cubic_k * ((a - b) + 1.0f);
        } else {
            result = p.cubic_k * (2.0f * ipow_rn(1.0f - q, 3));
        }
    }
    return result;
}

// cubic_kernel_grad (Kernels.cpp:26-41); len = glm::length(r), which the
// callers already hold (the same expression, so the same bits)
__device__ __forceinline__ float3 gradW_ref(const StepParams& p, float rx, float ry, float rz, float len) {
    float rl = len * p.kfac;
    float q = q_ref(p, len);
    float3 out = make_float3(0.0f, 0.0f, 0.0f);
    // the reference compares with the double 1.0e-5, which lies between the
    // float 1.0e-5f and the next: the same comparison
    if (rl > 1.0e-5f && q <= 1.0f) {
        float s = 1.0f / (rl * p.h);
        float gx = s * rx, gy = s * ry, gz = s * rz;
        float c;
        if (q <= 0.5f) {
            c = (p.cubic_l * q) * (3.0f * q - 2.0f);
        } else {
            float f = 1.0f - q;
            c = p.cubic_l * ((-f) * f);
        }
        out = make_float3(c * gx, c * gy, c * gz);
    }
    return out;
}

// s_coor (Simulate.cpp:7-9): -k * pow(W(r) / W(dq), n).  rcp_w: 1 / W(dq) at
// the exponent 4, or 0 where W(dq) is out of div_known's range (a W(r) below
// it gives a power that underflows to 0 either way).
__device__ __forceinline__ float scorr_ref(const StepParams& p, float rl, float w_dq, float rcp_w) {
    const float w = W_ref(p, rl);
    float ratio = rcp_w != 0.0f ? div_known(w, w_dq, rcp_w) : w / w_dq;
    float pw = p.sn_int == 4 ? pow4_rn(ratio) : (p.sn_int >= 0 ? ipow_rn(ratio, p.sn_int) : powf(ratio, p.sn));
    return (-p.sk) * pw;
}

// resolve_collision (Simulate.cpp:13-24)
__device__ __forceinline__ float resolve_collision(float value, float lo, float hi) {
    const float eps = 0.01f;
    if (value <= lo) return eps;
    if (value > hi) return hi - eps;
    return value;
}

// Simulate.cpp:48-51 plus the cell key and histogram of the counting sort.
__global__ void k_predict_ref(StepParams p, const float4* __restrict__ x, float4* __restrict__ v,
                              float4* __restrict__ xs, int* __restrict__ key,
                              int* __restrict__ rank, int* __restrict__ count, int* status) {
    pdl_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    float4 xi = x[i], vi = v[i];
    float gmx = p.gxv * p.mass, gmy = p.gyv * p.mass, gmz = p.gzv * p.mass;
    vi.x = vi.x + gmx * p.dt;
    vi.y = vi.y + gmy * p.dt;
    vi.z = vi.z + gmz * p.dt;
    float4 s = make_float4(xi.x + vi.x * p.dt, xi.y + vi.y * p.dt, xi.z + vi.z * p.dt, 0.0f);
    v[i] = vi;
    xs[i] = s;
    int k = cell_ref(p, s.x, s.y, s.z, status);
    key[i] = k;
    rank[i] = atomicAdd(&count[k], 1);
}

__global__ void k_key_ref(StepParams p, const float4* __restrict__ pos, int m, int* __restrict__ key,
                          int* __restrict__ rank, int* __restrict__ count, int* status) {
    pdl_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    float4 s = pos[i];
    int k = cell_ref(p, s.x, s.y, s.z, status);
    key[i] = k;
    rank[i] = atomicAdd(&count[k], 1);
}

// Neighbours in the reference's list order: the 27 cells around the
// particle's cell in y -> x -> z offset order (Neighbors.cpp:401-403); in each
// cell its fluid particles by ascending id, then its solids by ascending
// storage index (Neighbors.cpp:374-384).  The three cells of a row are
// consecutive ids: a row without solids is one range of fluid slots, walked
// in one loop; the solids' table is read only near solids (near, set per
// cell).  Each row's bounds are loaded while the one before is walked.  Bound by
// instruction issue at the few warps a scene of this mode has (100,000
// particles, h = 1.55: 36.2 us cell by cell with a store to the list's row per
// accepted candidate, 19.5 us like this).  G lanes share a particle's rows where
// a scene has few (as the sand lists do).
constexpr int REF_BLOCK = 128;
constexpr int REF_STAGE = 24;  // list entries staged in shared memory
template <int G>
__global__ void __launch_bounds__(REF_BLOCK) k_lists_ref(StepParams p, const float4* __restrict__ xs,
                                                         const int* __restrict__ key,
                                                         const int* __restrict__ fstart,
                                                         const float4* __restrict__ solid,
                                                         const int* __restrict__ sstart, int* __restrict__ nbr,
                                                         int* __restrict__ cnt, int* status) {
    pdl_wait();
    constexpr int STAGE = G == 1 ? REF_STAGE : 12;
    __shared__ int stage[STAGE * REF_BLOCK];
    const int s = (blockIdx.x * REF_BLOCK + threadIdx.x) / G, g = threadIdx.x % G;
    if (s >= p.n) return;
    const float4 self = xs[s];
    const int id = key[s];
    const int slab = p.gx * p.gz;
    const int yy = id / slab, xx = (id % slab) / p.gz, zz = id % p.gz;
    const int z0 = max(zz - 1, 0), z1 = min(zz + 1, p.gz - 1);
    const bool near = p.ns > 0 && p.solid_near[id];
    auto fluid_entry = [](int t) { return t; };
    auto solid_entry = [](int u) { return -1 - u; };
    // this lane's rows: two or three of the nine
    const int q0 = G == 1 ? 0 : (g ? 2 * g + 1 : 0), q1 = G == 1 ? 9 : 2 * g + 3;
    auto walk = [&](auto& out) {
        int next = 0, row = 0, a_next = 0, b_next = 0, s_next = 0, e_next = 0;
        auto bounds = [&](int r) {
            for (; r < q1; r++) {
                const int y = yy + r / 3 - 1, x = xx + r % 3 - 1;
                if (y < 0 || y >= p.gy || x < 0 || x >= p.gx) continue;
                row = y * slab + x * p.gz;
                a_next = fstart[row + z0];
                b_next = fstart[row + z1 + 1];
                if (near) {
                    s_next = sstart[row + z0];
                    e_next = sstart[row + z1 + 1];
                }
                break;
            }
            next = r;
        };
        bounds(q0);
        while (next < q1) {
            const int a = a_next, b = b_next, sa = s_next, sb = e_next, r0 = row;
            bounds(next + 1);
            if (sa == sb) {
                walk_span(xs, a, b, self, p.h2, out, fluid_entry);
            } else if (a == b) {
                walk_span(solid, sa, sb, self, p.h2, out, solid_entry);
            } else {
                int f0 = a, s0 = sa;
                for (int c = r0 + z0; c <= r0 + z1; c++) {
                    const int f1 = fstart[c + 1], s1 = sstart[c + 1];
                    walk_span(xs, f0, f1, self, p.h2, out, fluid_entry);
                    walk_span(solid, s0, s1, self, p.h2, out, solid_entry);
                    f0 = f1;
                    s0 = s1;
                }
            }
        }
    };
    StagedList<STAGE, REF_BLOCK, G> out(stage, nbr, p, s);
    walk(out);
    int off, c_n = group_offset<G>(out.count(), off);
    out.write(off);
    if (G > 1 && out.extra) {
        LateEntries<STAGE> late{nbr + s, (size_t)p.n, off, p.max_nbrs, 0};
        walk(late);
    }
    if (c_n > p.max_nbrs) {
        set_status(status, ST_NBR_OVERFLOW);
        c_n = p.max_nbrs;
    }
    if (g == 0) cnt[s] = c_n;
}

__device__ __forceinline__ float4 nbr_pos(int j, const float4* __restrict__ xs,
                                          const float4* __restrict__ solid) {
    return j >= 0 ? xs[j] : solid[-1 - j];
}

// f(k, position) for every entry k of a list, in order: REF_CHUNK entries and
// then their positions are loaded together, the next chunk's entries while
// this one is used (2 or 8: no faster).
constexpr int REF_CHUNK = 4;
template <class F>
__device__ __forceinline__ void for_each_nbr(const StepParams& p, const int* __restrict__ nbr, int s, int c,
                                             const float4* __restrict__ xs, const float4* __restrict__ solid, F&& f) {
    int e[REF_CHUNK];
#pragma unroll
    for (int u = 0; u < REF_CHUNK; u++) e[u] = c > 0 ? __ldg(&nbr[(size_t)min(u, c - 1) * p.n + s]) : 0;
    for (int k = 0; k < c; k += REF_CHUNK) {
        float4 o[REF_CHUNK];
#pragma unroll
        for (int u = 0; u < REF_CHUNK; u++) o[u] = nbr_pos(e[u], xs, solid);
#pragma unroll
        for (int u = 0; u < REF_CHUNK; u++) e[u] = __ldg(&nbr[(size_t)min(k + REF_CHUNK + u, c - 1) * p.n + s]);
#pragma unroll
        for (int u = 0; u < REF_CHUNK; u++)
            if (k + u < c) f(k + u, o[u]);
    }
}

// Simulate.cpp:58-88; lambdas are stored by the caller's particle id because
// the position pass indexes them by list position (Simulate.cpp:97).  The
// reference's two loops over the list (density, then gradients) run as one:
// each sum still takes its terms in list order, so the bits are the same,
// with one gather per neighbour instead of two.
__global__ void k_lambda_ref(StepParams p, const float4* __restrict__ xs, const int* __restrict__ id,
                             const int* __restrict__ nbr, const int* __restrict__ cnt,
                             const float4* __restrict__ solid, float* __restrict__ lam_by_id,
                             float* __restrict__ rho) {
    pdl_wait();
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= p.n) return;
    const float4 self = xs[s];
    const int c = cnt[s];
    float density = 0.0f;
    float gsum = 0.0f;
    float gcx = 0.0f, gcy = 0.0f, gcz = 0.0f;
    const float coef = -(p.mass / p.rho0);
    for_each_nbr(p, nbr, s, c, xs, solid, [&](int, float4 o) {
        float ix = self.x - o.x, iy = self.y - o.y, iz = self.z - o.z;
        float len = sqrtf((ix * ix + iy * iy) + iz * iz);
        density += p.mass * W_ref(p, len);
        float3 g = gradW_ref(p, ix, iy, iz, len);
        float nx = coef * g.x, ny = coef * g.y, nz = coef * g.z;
        gsum += (nx * nx + ny * ny) + nz * nz;
        gcx -= nx;
        gcy -= ny;
        gcz -= nz;
    });
    density += p.mass * W_ref(p, 0.0f);
    float constraint = density / p.rho0 - 1.0f;  // exact in the reference's double, then rounded: the same value
    gsum += (gcx * gcx + gcy * gcy) + gcz * gcz;
    float lam = 0.0f;
    if (gsum > 0.0f) lam = (-constraint) / (gsum + p.eps);
    lam_by_id[id[s]] = lam;
    if (rho) rho[s] = density;
}

// Simulate.cpp:90-113 with a Jacobi read of the neighbours' positions.  Bound
// by instruction issue; s_corr's power in double and the two divisions took
// more than half of it (100,000 particles of 27 neighbours: 47.4 us, now 20.6).
__global__ void k_delta_ref(StepParams p, const float4* __restrict__ xs, float4* __restrict__ xs_out,
                            float4* __restrict__ x, float4* __restrict__ v,
                            const int* __restrict__ id, const int* __restrict__ nbr,
                            const int* __restrict__ cnt, const float4* __restrict__ solid,
                            const float* __restrict__ lam_by_id) {
    pdl_wait();
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= p.n) return;
    const float4 self = xs[s];
    const float li = lam_by_id[id[s]];
    const float w_dq = W_ref(p, p.dq);
    const float rcp_w = p.sn_int == 4 && w_dq >= 0x1p-40f && w_dq <= 0x1p60f ? __frcp_rn(w_dq) : 0.0f;
    const int c = cnt[s];
    float px = 0.0f, py = 0.0f, pz = 0.0f;
    for_each_nbr(p, nbr, s, c, xs, solid, [&](int k, float4 o) {
        float ix = self.x - o.x, iy = self.y - o.y, iz = self.z - o.z;
        float len = sqrtf((ix * ix + iy * iy) + iz * iz);
        float sc = scorr_ref(p, len, w_dq, rcp_w);
        float3 g = gradW_ref(p, ix, iy, iz, len);
        float w = (li + lam_by_id[k]) + sc;
        px += w * g.x;
        py += w * g.y;
        pz += w * g.z;
    });
    px = px / p.rho0;
    py = py / p.rho0;
    pz = pz / p.rho0;
    float nx = self.x + px, ny = self.y + py, nz = self.z + pz;
    nx = resolve_collision(nx, p.lox, p.hix);
    ny = resolve_collision(ny, p.loy, p.hiy);
    nz = resolve_collision(nz, p.loz, p.hiz);
    const float4 xo = x[s];
    v[s] = make_float4((nx - xo.x) / p.dt, (ny - xo.y) / p.dt, (nz - xo.z) / p.dt, 0.0f);
    const float4 xn = make_float4(nx, ny, nz, 0.0f);
    x[s] = xn;
    xs_out[s] = xn;
}

// ------------------------------------------------------------------ launch --

static inline int blocks_for(int n, int t) { return (n + t - 1) / t; }

// Up to this many particles a list is built by four lanes.  Measured, us a step
// with one lane / with four: 3,000 particles of kernel radius 1.55 46.7 / 43.1,
// 10,000 47.2 / 45.2 (of radius 2.0 66.1 / 60.9), 20,000 47.1 / 46.1, 40,000
// 48.7 / 55.2, 100,000 67.9 / 79.5: with more particles than lanes at work the
// group's idle lanes and second walks cost more than the shorter chain gives.
constexpr int REF_LISTS_GROUP_MAX = 16000;

void launch_predict_ref(const StepParams& p, const float4* x, float4* v, float4* xs, int* key,
                        int* rank, int* count, int* status, cudaStream_t st) {
    if (p.n <= 0) return;
    launch_k(k_predict_ref, blocks_for(p.n, 256), 256, st, pdl_enabled(), p, x, v, xs, key, rank, count, status);
}

void launch_key_ref(const StepParams& p, const float4* pos, int m, int* key, int* rank, int* count,
                    int* status, cudaStream_t st) {
    if (m <= 0) return;
    launch_k(k_key_ref, blocks_for(m, 256), 256, st, pdl_enabled(), p, pos, m, key, rank, count, status);
}

void launch_lists_ref(const StepParams& p, const float4* xs, const int* key, const int* fstart,
                      const float4* solid, const int* sstart, int* nbr, int* cnt, int* status,
                      cudaStream_t st) {
    if (p.n <= 0) return;
    if (p.n <= REF_LISTS_GROUP_MAX)
        launch_k(k_lists_ref<4>, blocks_for(p.n, REF_BLOCK / 4), REF_BLOCK, st, pdl_enabled(), p, xs, key, fstart, solid,
                 sstart, nbr, cnt, status);
    else
        launch_k(k_lists_ref<1>, blocks_for(p.n, REF_BLOCK), REF_BLOCK, st, pdl_enabled(), p, xs, key, fstart, solid,
                 sstart, nbr, cnt, status);
}

void launch_lambda_ref(const StepParams& p, const float4* xs, const int* id, const int* nbr,
                       const int* cnt, const float4* solid, float* lam_by_id, float* rho,
                       cudaStream_t st) {
    if (p.n <= 0) return;
    launch_k(k_lambda_ref, blocks_for(p.n, 128), 128, st, pdl_enabled(), p, xs, id, nbr, cnt, solid, lam_by_id,
             rho);
}

void launch_delta_ref(const StepParams& p, const float4* xs, float4* xs_out, float4* x, float4* v,
                      const int* id, const int* nbr, const int* cnt, const float4* solid,
                      const float* lam_by_id, cudaStream_t st) {
    if (p.n <= 0) return;
    launch_k(k_delta_ref, blocks_for(p.n, 128), 128, st, pdl_enabled(), p, xs, xs_out, x, v, id, nbr, cnt, solid,
             lam_by_id);
}

}  // namespace lgb
