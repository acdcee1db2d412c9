// sand.cu -- the reference's sand step (LUSTRINE_MODE_SAND) on the GPU.
//
// Semantics of Lustrine::simulate_sand (Simulate.cpp:156-325) with its
// neighbour search find_neighbors_uniform_grid_v1 (Neighbors.cpp:262-361),
// float operation for float operation.  This translation unit is compiled
// with --fmad=false and evaluates every expression in the reference's order
// (glm 0.9.9.8: dot = (x*x + y*y) + z*z, length = sqrt(dot),
// normalize = v * (1 / sqrt(dot(v, v))), clamp = min(max(v, lo), hi)), so
// positions, velocities, attract flags and list order equal the reference's
// bit for bit.  The reference's contact/friction substeps already read a
// snapshot of the positions (positions_tmp), so the GPU's Jacobi passes are
// its exact parallel form.
//
// Step: k_sand_predict (integration, attract and blow, box clamp, cell key,
// histogram) -> cell scan -> stable scatter/gather of x, x*, attract flags
// into cell order -> k_sand_lists (symmetric lists in the reference's push
// order) -> 4 x k_sand_substep; the last substep commits x, v and the flags
// back into the side the step started from.
#include "pbf_common.cuh"
#include "pbf_compat.cuh"
#include "pbf_kernels.h"

namespace lgb {

// simulate_sand's constants (Simulate.cpp:159-163)
constexpr float SAND_COLLISION = 0.8f;
constexpr float SAND_FRICTION = 0.7f;
constexpr float SAND_MU_S = 0.95f;
constexpr float SAND_MU_K = 0.9f;

__device__ __forceinline__ float sdot(float x, float y, float z) { return (x * x + y * y) + z * z; }
__device__ __forceinline__ float slen(float x, float y, float z) { return sqrtf(sdot(x, y, z)); }
__device__ __forceinline__ float sdot2(float ax, float ay, float az, float bx, float by, float bz) {
    return (ax * bx + ay * by) + az * bz;
}
// glm::max / glm::min on floats
__device__ __forceinline__ float smax(float a, float b) { return a < b ? b : a; }
__device__ __forceinline__ float smin(float a, float b) { return b < a ? b : a; }

// glm::clamp(v, vec3(r), vec3(X, Y, Z) - vec3(r)) (Simulate.cpp:208, 298)
__device__ __forceinline__ float4 sand_clamp(const StepParams& p, float x, float y, float z) {
    return make_float4(smin(smax(x, p.lox), p.hix), smin(smax(y, p.loy), p.hiy),
                       smin(smax(z, p.loz), p.hiz), 0.0f);
}

// Integration (Simulate.cpp:183-209) plus the cell key and histogram of the
// counting sort (Neighbors.cpp:275-278).
__global__ void k_sand_predict(StepParams p, SandParams q, const float4* __restrict__ x,
                               float4* __restrict__ v, float4* __restrict__ xs, int* __restrict__ att,
                               int* __restrict__ key, int* __restrict__ rank, int* __restrict__ count,
                               int* status) {
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const float4 xi = x[i];
    float4 vi = v[i];
    vi.x = vi.x + p.gxv * p.dt;
    vi.y = vi.y + p.gyv * p.dt;
    vi.z = vi.z + p.gzv * p.dt;
    int a = att[i];
    if (q.prev_attract && !q.attract) a = 0;
    if (q.attract) {
        if (slen(q.px - xi.x, q.py - xi.y, q.pz - xi.z) < q.attract_radius) a = 1;
        if (a) {
            // towards 1.5 above the player's position
            const float ox = (q.px + 0.0f) - xi.x, oy = (q.py + 1.5f) - xi.y, oz = (q.pz + 0.0f) - xi.z;
            const float s = 1.0f / sqrtf(sdot(ox, oy, oz));
            vi.x = vi.x + ((((ox * s) * 1.0f) * q.attract_coeff) * q.radius * p.dt) * q.w;
            vi.y = vi.y + ((((oy * s) * 1.0f) * q.attract_coeff) * q.radius * p.dt) * q.w;
            vi.z = vi.z + ((((oz * s) * 1.0f) * q.attract_coeff) * q.radius * p.dt) * q.w;
        }
    }
    if (q.blow) {
        const float dx = q.px - xi.x, dy = q.py - xi.y, dz = q.pz - xi.z;
        const float ld = slen(dx, dy, dz);
        if (ld < q.blow_radius) {
            const float s = 1.0f / sqrtf(sdot(dx, dy, dz));
            // blow_kernel (Simulate.cpp:143-154)
            const float bk = ld > q.blow_radius ? 0.0f : 1.0f - ld / q.blow_radius;
            vi.x = vi.x + (((-(dx * s) * bk) * q.blow_coeff) * q.radius) * q.w;
            vi.y = vi.y + (((-(dy * s) * bk) * q.blow_coeff) * q.radius) * q.w;
            vi.z = vi.z + (((-(dz * s) * bk) * q.blow_coeff) * q.radius) * q.w;
        }
    }
    const float4 s = sand_clamp(p, xi.x + vi.x * p.dt, xi.y + vi.y * p.dt, xi.z + vi.z * p.dt);
    v[i] = vi;
    xs[i] = s;
    att[i] = a;
    const int k = cell_ref(p, s.x, s.y, s.z, status);
    key[i] = k;
    rank[i] = atomicAdd(&count[k], 1);
}

// The reference's lists in its push order (Neighbors.cpp:306-358), built per
// particle without the symmetric pushes: particle i's list is first the sand
// particles k < i whose own walk found i, in ascending k -- the 27-cell walk
// in y -> x -> z order visits cells by ascending id and the sorted slots of a
// cell ascend, so that is the walk itself restricted to slots below i -- then
// its own walk over j >= i, each cell's static particles before its sand.
// The reference also lists i itself twice; the substeps skip it
// (Simulate.cpp:226), so it is left out.  Entries: sand slot t >= 0, static
// slot u as -1 - u.
//
// The three cells of a row (dy, dx) are consecutive ids, so their sand is one
// slot range.  Away from static particles (near, set per cell) the two parts
// together are the nine ranges in order without i: one pass over the
// candidates (two passes cell by cell took 64.6 us for 262,144 particles of a
// heap, h = 1.55; this one takes 41.5, bound by instruction issue: 100
// candidates a particle, of which it lists 17).  Near some, the lower slots'
// ranges come first, then every row's static particles with its sand above i,
// cell by cell only in rows that hold both.
//
// G lanes share a particle's walk (its ranges and rows in order, in G
// stretches): a small scene has fewer warps than the GPU has schedulers, and a
// particle's walk is a chain of dependent loads.
constexpr int SAND_BLOCK = 128;
// List entries staged in shared memory (16-18 a particle in a heap): at 32 the
// larger stage leaves the L1 too small for the candidates (hit rate 80 -> 56 %,
// 46 us), at 12 most lists leave it (49 us).
constexpr int SAND_STAGE = 20;
template <int G>
__global__ void __launch_bounds__(SAND_BLOCK) k_sand_lists(StepParams p, const float4* __restrict__ xs,
                                                           const int* __restrict__ key,
                                                           const int* __restrict__ fstart,
                                                           const float4* __restrict__ solid,
                                                           const int* __restrict__ sstart, int* __restrict__ nbr,
                                                           int* __restrict__ cnt, int* status) {
    pdl_wait();
    constexpr int STAGE = G == 1 ? SAND_STAGE : 12;
    __shared__ int stage[STAGE * SAND_BLOCK];
    const int i = (blockIdx.x * SAND_BLOCK + threadIdx.x) / G, g = threadIdx.x % G;
    if (i >= p.n) return;
    const float4 self = xs[i];
    const int id = key[i];
    const int slab = p.gx * p.gz;
    const int yy = id / slab;
    const int t0 = id - yy * slab;
    const int zz = t0 % p.gz, xx = t0 / p.gz;
    const int z0 = max(zz - 1, 0), z1 = min(zz + 1, p.gz - 1);
    const bool near = p.ns > 0 && p.solid_near[id];
    auto sand_entry = [](int t) { return t; };
    auto static_entry = [](int u) { return -1 - u; };
    // The walk's items: away from static particles the ten ranges (i's own row
    // cut at i into two); near some the five ranges up to i, then the nine rows.
    // An item's bounds are loaded while the one before is walked.
    const int items = near ? 14 : 10;
    int q0 = 0, q1 = items;
    if (G == 4) {  // three rows each at most
        q0 = g == 0 ? 0 : (g == 1 ? 3 : (g == 2 ? (near ? 8 : 5) : (near ? 11 : 7)));
        q1 = g == 0 ? 3 : (g == 1 ? (near ? 8 : 5) : (g == 2 ? (near ? 11 : 7) : items));
    }
    auto walk = [&](auto& out) {
        int next = 0, row = 0, a_next = 0, b_next = 0, s_next = 0, e_next = 0;
        auto to_row = [&](int k) {  // row k of the stencil, if the grid has it
            const int y = yy + k / 3 - 1, x = xx + k % 3 - 1;
            row = y * slab + x * p.gz;
            return y >= 0 && y < p.gy && x >= 0 && x < p.gx;
        };
        auto range = [&](int q, int end) {  // the next range from q on
            for (; q < end; q++) {
                if (!to_row(q > 4 ? q - 1 : q)) continue;
                a_next = q == 5 ? i + 1 : fstart[row + z0];
                b_next = q == 4 ? i : fstart[row + z1 + 1];
                break;
            }
            next = q;
        };
        const int ranges = min(q1, near ? 5 : 10);
        range(q0, ranges);
        while (next < ranges) {
            const int a = a_next, b = b_next;
            range(next + 1, ranges);
            walk_span(xs, a, b, self, p.h2, out, sand_entry);
        }
        if (!near || q1 <= 5) return;
        auto next_row = [&](int q) {  // the next row from item q on: its static particles, its sand above i
            for (; q < q1; q++) {
                if (!to_row(q - 5)) continue;
                s_next = sstart[row + z0];
                e_next = sstart[row + z1 + 1];
                a_next = q < 9 ? 0 : (q == 9 ? i + 1 : fstart[row + z0]);
                b_next = q < 9 ? 0 : fstart[row + z1 + 1];
                if (s_next < e_next || a_next < b_next) break;
            }
            next = q;
        };
        next_row(max(q0, 5));
        while (next < q1) {
            const int r0 = row, a = a_next, b = b_next, sa = s_next, sb = e_next;
            next_row(next + 1);
            if (sa == sb) {
                walk_span(xs, a, b, self, p.h2, out, sand_entry);
            } else if (a >= b) {
                walk_span(solid, sa, sb, self, p.h2, out, static_entry);
            } else {
                int s0 = sa, f0 = a;  // both advance cell by cell
                for (int c = r0 + z0; c <= r0 + z1; c++) {
                    const int s1 = sstart[c + 1], f1 = fstart[c + 1];
                    walk_span(solid, s0, s1, self, p.h2, out, static_entry);
                    walk_span(xs, f0, f1, self, p.h2, out, sand_entry);
                    s0 = s1;
                    f0 = max(f0, f1);
                }
            }
        }
    };
    StagedList<STAGE, SAND_BLOCK, G> out(stage, nbr, p, i);
    walk(out);
    int off, c_n = group_offset<G>(out.count(), off);
    out.write(off);
    if (G > 1 && out.extra) {
        LateEntries<STAGE> late{nbr + i, (size_t)p.n, off, p.max_nbrs, 0};
        walk(late);
    }
    if (c_n > p.max_nbrs) {
        set_status(status, ST_NBR_OVERFLOW);
        c_n = p.max_nbrs;
    }
    if (g == 0) cnt[i] = c_n;
}

// One contact and friction term (Simulate.cpp:236-266 for a sand neighbour,
// 268-286 for a static one): the displacements that the reference subtracts
// one after the other, the contact's t and the friction's f.  coef: the
// contact's share, collision m / (m + m) between two sand particles,
// collision against a static one (whose own displacement is zero).
struct SandTerm {
    float tx, ty, tz, fx, fy, fz;
};
__device__ __forceinline__ SandTerm sand_pair(const SandParams& q, bool sand_j, float coef, float4 pi, float4 pj,
                                              float4 xi, float4 xj) {
    SandTerm o = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    float ix = pi.x - pj.x, iy = pi.y - pj.y, iz = pi.z - pj.z;
    float d2 = sdot(ix, iy, iz);
    if (d2 == 0.0f) {
        ix = 0.0f;
        iy = 0.00001f;
        iz = 0.0f;
        d2 = sdot(ix, iy, iz);
    }
    const float len = sqrtf(d2);
    if (len > q.diameter) return o;
    const float s = coef * (len - q.diameter);
    o.tx = (s * ix) / len;
    o.ty = (s * iy) / len;
    o.tz = (s * iz) / len;
    const float d = slen(o.tx, o.ty, o.tz);
    const float ax = pi.x - o.tx, ay = pi.y - o.ty, az = pi.z - o.tz;  // pi - tmp
    // pj + tmp and its displacement; a static particle stays
    const float bx = sand_j ? pj.x + o.tx : pj.x, by = sand_j ? pj.y + o.ty : pj.y,
                bz = sand_j ? pj.z + o.tz : pj.z;
    const float rx = (ax - xi.x) - (sand_j ? bx - xj.x : 0.0f);
    const float ry = (ay - xi.y) - (sand_j ? by - xj.y : 0.0f);
    const float rz = (az - xi.z) - (sand_j ? bz - xj.z : 0.0f);
    float nx = ax - bx, ny = ay - by, nz = az - bz;
    const float inv = 1.0f / sqrtf(sdot(nx, ny, nz));
    nx = nx * inv;
    ny = ny * inv;
    nz = nz * inv;
    const float dr = sdot2(rx, ry, rz, nx, ny, nz);
    const float ux = rx - dr * nx, uy = ry - dr * ny, uz = rz - dr * nz;  // tangential part
    const float lt = slen(ux, uy, uz);
    o.fx = SAND_FRICTION * ux;
    o.fy = SAND_FRICTION * uy;
    o.fz = SAND_FRICTION * uz;
    if (!((d * SAND_MU_S) > lt + 1e-9f)) {
        const float r = (SAND_MU_K * d) / (lt + 1e-9f);
        const float ratio = r < 1 ? r : 1;
        o.fx = o.fx * ratio;
        o.fy = o.fy * ratio;
        o.fz = o.fz * ratio;
    }
    return o;
}

// One contact/friction substep (Simulate.cpp:221-303): every particle reads
// positions_tmp (tmp_in) and the pre-step positions (xpre), writes its new
// clamped position.  The last substep commits instead: x = x*,
// v = (x* - x) / dt (Simulate.cpp:309-313), the attract flags and the
// particle's index -- its slot in this step's cell order, as the reference
// re-orders its arrays -- into the side the step started from (whose
// contents the sort already consumed).
//
// A list holds every particle within h, a third of them in contact (within a
// diameter), and a contact term costs some 150 instructions (four square
// roots and five divisions, each correctly rounded).  Evaluated entry by entry a
// warp pays for a term wherever any lane has a contact (13 of 32 lanes active).
// So a thread first collects its contacts: SAND_CHUNK positions loaded
// together (2 or 8: 10 % slower) and tested by d^2 against reach2, the largest
// float whose square root rounds to at most the diameter (the same test
// without the root); then it evaluates them in list order, the next contact's
// positions loaded ahead.
constexpr int SAND_CHUNK = 4;
constexpr int SAND_HITS = 16;  // contacts collected before they are evaluated
__global__ void __launch_bounds__(SAND_BLOCK) k_sand_substep(
    StepParams p, SandParams q, const float4* __restrict__ tmp_in, float4* __restrict__ star_out,
    const float4* __restrict__ xpre, const int* __restrict__ nbr, const int* __restrict__ cnt,
    const float4* __restrict__ solid, float4* __restrict__ x_commit, float4* __restrict__ v_commit,
    const int* __restrict__ att_in, int* __restrict__ att_commit, int* __restrict__ id_commit) {
    pdl_wait();
    __shared__ int hits[SAND_HITS * SAND_BLOCK];
    const int i = blockIdx.x * SAND_BLOCK + threadIdx.x;
    if (i >= p.n) return;
    int* hit = hits + threadIdx.x;
    const float4 pi = tmp_in[i];
    const float4 xi = xpre[i];
    const float sand_coef = (SAND_COLLISION * p.mass) / (p.mass + p.mass);
    float dpx = 0.0f, dpy = 0.0f, dpz = 0.0f;
    const int c = cnt[i];
    auto pos = [&](int e) { return e >= 0 ? tmp_in[e] : __ldg(&solid[-1 - e]); };
    for (int k = 0; k < c;) {
        int m = 0;
        for (; k < c && m <= SAND_HITS - SAND_CHUNK; k += SAND_CHUNK) {
            int e[SAND_CHUNK];
            float4 o[SAND_CHUNK];
#pragma unroll
            for (int u = 0; u < SAND_CHUNK; u++) e[u] = nbr[(size_t)min(k + u, c - 1) * p.n + i];
#pragma unroll
            for (int u = 0; u < SAND_CHUNK; u++) o[u] = pos(e[u]);
#pragma unroll
            for (int u = 0; u < SAND_CHUNK; u++) {
                const float d2 = sdot(pi.x - o[u].x, pi.y - o[u].y, pi.z - o[u].z);
                if (k + u < c && !(d2 > q.reach2)) hit[SAND_BLOCK * m++] = e[u];
            }
        }
        if (!m) continue;
        int e = hit[0];
        float4 pj = pos(e), xj = e >= 0 ? xpre[e] : pj;
        for (int h = 0; h < m; h++) {
            const bool sand_j = e >= 0;
            const float4 pc = pj, xc = xj;
            if (h + 1 < m) {
                e = hit[SAND_BLOCK * (h + 1)];
                pj = pos(e);
                xj = e >= 0 ? xpre[e] : pj;
            }
            const SandTerm o = sand_pair(q, sand_j, sand_j ? sand_coef : SAND_COLLISION, pi, pc, xi, xc);
            dpx = (dpx - o.tx) - o.fx;
            dpy = (dpy - o.ty) - o.fy;
            dpz = (dpz - o.tz) - o.fz;
        }
    }
    const float4 s = sand_clamp(p, pi.x + dpx, pi.y + dpy, pi.z + dpz);
    if (!x_commit) {
        star_out[i] = s;
        return;
    }
    x_commit[i] = s;
    v_commit[i] = make_float4((s.x - xi.x) / p.dt, (s.y - xi.y) / p.dt, (s.z - xi.z) / p.dt, 0.0f);
    att_commit[i] = att_in[i];
    id_commit[i] = i;
}

// ------------------------------------------------------------------ launch --

static inline int blocks_for(int n, int t) { return (n + t - 1) / t; }

// Largest scenes whose list build gives each particle four lanes.  Measured, us a
// step with one lane / with four: 5,000 particles 52.3 / 47.3, 10,000 (h = 1.55)
// 73.9 / 63.6, 20,011 54.4 / 49.7, 41,000 56.8 / 53.5, 81,000 65.2 / 65.8; 96
// contexts of 2,000 to 20,000 at once 398 / 365 (h = 1.55: 469 / 505).  (Four lanes in
// the substeps too gave a single scene of 5,000 43.8, but the 96 contexts 541.)
constexpr int SAND_LISTS_GROUP_MAX = 45000;

void launch_sand_predict(const StepParams& p, const SandParams& q, const float4* x, float4* v, float4* xs,
                         int* att, int* key, int* rank, int* count, int* status, cudaStream_t st) {
    if (p.n <= 0) return;
    launch_k(k_sand_predict, blocks_for(p.n, 256), 256, st, pdl_enabled(), p, q, x, v, xs, att, key, rank,
             count, status);
}

void launch_sand_lists(const StepParams& p, const float4* xs, const int* key, const int* fstart,
                       const float4* solid, const int* sstart, int* nbr, int* cnt, int* status,
                       cudaStream_t st) {
    if (p.n <= 0) return;
    if (p.n <= SAND_LISTS_GROUP_MAX)
        launch_k(k_sand_lists<4>, blocks_for(p.n, SAND_BLOCK / 4), SAND_BLOCK, st, pdl_enabled(), p, xs, key, fstart,
                 solid, sstart, nbr, cnt, status);
    else
        launch_k(k_sand_lists<1>, blocks_for(p.n, SAND_BLOCK), SAND_BLOCK, st, pdl_enabled(), p, xs, key, fstart,
                 solid, sstart, nbr, cnt, status);
}

void launch_sand_substep(const StepParams& p, const SandParams& q, const float4* tmp_in, float4* star_out,
                         const float4* xpre, const int* nbr, const int* cnt, const float4* solid,
                         float4* x_commit, float4* v_commit, const int* att_in, int* att_commit,
                         int* id_commit, cudaStream_t st) {
    if (p.n <= 0) return;
    launch_k(k_sand_substep, blocks_for(p.n, SAND_BLOCK), SAND_BLOCK, st, pdl_enabled(), p, q, tmp_in, star_out,
             xpre, nbr, cnt, solid, x_commit, v_commit, att_in, att_commit, id_commit);
}

}  // namespace lgb
