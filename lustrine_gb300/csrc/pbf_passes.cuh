// pbf_passes.cuh -- the kernels of the PBF step (mode P): the
// position-based-fluids solver the reference's parameters describe
// (Simulation.hpp:157-171: rest density, relaxation epsilon, s_corr, XSPH) on
// the poly6 / spiky kernels of Kernels.cpp:43-67, with N Jacobi solver
// iterations over neighbour lists built once per step.  Templates only: the
// launchers in pbf_solver.cu (column lists) and pbf_compact.cu (compact lists)
// instantiate them.
//
// Position representations (template parameter MIXED):
//   plain  float4 xyz = absolute position;
//   mixed  xyz = offset from the particle's cell corner, the cell being the
//          sorted key of the step (fixed during the step's iterations, so an
//          offset may leave [0, cell) until the next prediction renormalises
//          it); the committed state keeps the cell packed in w.  Neighbour
//          offsets are (o_i - o_j) + (c_i - c_j) * cell with the cell
//          difference cached in the neighbour list entry, so their precision
//          does not depend on the distance to the origin; density sums use
//          compensated (Kahan) accumulation.
// During the iterations w of the predicted positions holds the particle's
// lambda, written in place by the lambda pass, so the position pass gathers
// one float4 per neighbour.
//
// Neighbour list entry (int32, column lists): bits 0-24 slot, then the
// neighbour's cell offset from the particle's cell, 2 bits per axis as d + 1
// (x in 25-26, y in 27-28, z in 29-30), bit 31 set for solids.  Compact
// lists (no cell codes, no solids): 16-byte records, see COMPACT_INLINE in
// pbf_common.cuh.
//
// Grids: dense (cell id = offset + y gX gZ + x gZ + z; the three cells of a
// stencil row are consecutive ids) or hashed (the counting sort runs over
// hash buckets of cells, see cell_bucket; each slot keeps its packed cell,
// so the 27-cell walk rejects particles of other cells sharing a bucket --
// used for domains with more cells than fit a dense table).
#pragma once

#include "pbf_common.cuh"
#include "pbf_device.cuh"
#include "pbf_kernels.h"

namespace lgb {

template <bool MIXED>
__global__ void k_predict(StepParams p, CellPack cp, const float4* __restrict__ x,
                          const float4* __restrict__ v, float4* __restrict__ xs, int* __restrict__ key,
                          int* __restrict__ rank, int* __restrict__ count, int* __restrict__ cellk,
                          int* __restrict__ tile_count) {
    __shared__ TileSum tiles;
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = i < p.n;
    int k = 0;
    if (live) k = predict_one<MIXED>(p, cp, geo_slot(p, i), x[i], v[i], i, xs, key, rank, count, cellk);
    if (threadIdx.x == 0) open_tile_sum(tiles, k);
    __syncthreads();
    if (live) add_tile(tiles, tile_count, k, i, p.n);
}

// Cell key and histogram of static particles (solids; scene from solid_scene_of).
template <bool MIXED>
__global__ void k_key(StepParams p, CellPack cp, const float4* __restrict__ pos, int m,
                      int* __restrict__ key, int* __restrict__ rank, int* __restrict__ count,
                      int* __restrict__ cellk) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    float4 q = pos[i];
    const Geo g = p.scenes ? geo_scene(p, p.solid_scene_of[i]) : geo_single(p);
    int3 c = MIXED ? unpack_cell(cp, q.w) : plain_cell(p, g, q.x, q.y, q.z);
    int k = cell_key(p, cp, g, c, cellk, i);
    key[i] = k;
    rank[i] = atomicAdd(&count[k], 1);
}

// Cells (hash buckets) with a static particle in their 27-cell
// neighbourhood, marked once when the solids are set: the list build walks
// the solids only from those (a bucket shared with another cell is a false
// positive, which only costs a walk).
template <bool MIXED>
__global__ void k_mark_solid_near(StepParams p, CellPack cp, const float4* __restrict__ pos, int m,
                                  unsigned char* __restrict__ near) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    float4 q = pos[i];
    const Geo g = p.scenes ? geo_scene(p, p.solid_scene_of[i]) : geo_single(p);
    int3 c = MIXED ? unpack_cell(cp, q.w) : plain_cell(p, g, q.x, q.y, q.z);
    if (p.hash_bits) c = make_int3(min(c.x, (int)cp.mx), min(c.y, (int)cp.my), min(c.z, (int)cp.mz));
    for (int dy = -1; dy <= 1; dy++)
        for (int dx = -1; dx <= 1; dx++)
            for (int dz = -1; dz <= 1; dz++) {
                const int3 cn = make_int3(c.x + dx, c.y + dy, c.z + dz);
                if (cn.x < 0 || cn.y < 0 || cn.z < 0 || cn.x >= g.gx || cn.y >= g.gy || cn.z >= g.gz) continue;
                if (p.hash_bits) {
                    if (cn.x > (int)cp.mx || cn.y > (int)cp.my || cn.z > (int)cp.mz) continue;
                    near[cell_bucket(cn, p.hash_bits)] = 1;
                } else {
                    near[linear_cell(g, cn)] = 1;
                }
            }
}

// List formats: column lists, or compact lists in one of three records
// (pbf_common.cuh): 16-bit offsets from the scene's first slot,
// 24-bit slots, 32-bit slots.
enum : int { L_COLUMN = 0, L_C16 = 1, L_C24 = 2, L_C32 = 3 };

// Entries a compact list keeps in its two records: inline (first record),
// second record, both.
template <int FMT>
struct RecordFormat {
    static constexpr int INLINE = FMT == L_C16 ? COMPACT_INLINE : (FMT == L_C24 ? WIDE24_INLINE : WIDE_INLINE);
    static constexpr int EXT = FMT == L_C16 ? COMPACT_EXT : (FMT == L_C24 ? WIDE24_EXT : WIDE_EXT);
    static constexpr int RECORDS = INLINE + EXT;
};

// The high bytes of three words as a 24-bit value, and a 24-bit value's byte b
// as a word's high byte: where a 24-bit record keeps its fifth entry.
__device__ __forceinline__ int high_bytes(unsigned a, unsigned b, unsigned c) {
    return (int)__byte_perm(__byte_perm(a, b, 0x0073), c >> 24, 0x5410);
}
__device__ __forceinline__ unsigned as_high_byte(unsigned e, int b) { return (e >> (8 * b)) << 24; }

// Entry k of a record (FIRST: the first, else the second); 16-bit records:
// the offset.
template <int FMT, bool FIRST>
__device__ __forceinline__ unsigned record_entry(const uint4& r, int k) {
    constexpr unsigned M = 0xFFFFFFu;
    if (FMT == L_C24) {
        if (FIRST)
            return k == 0 ? r.x >> 8 : (k == 1 ? r.y & M : (k == 2 ? r.z & M : (k == 3 ? r.w & M
                                                                                        : (unsigned)high_bytes(r.y, r.z, r.w))));
        return k == 0 ? r.x & M : (k == 1 ? r.y & M : (k == 2 ? r.z & M : (k == 3 ? r.w
                                                                                  : (unsigned)high_bytes(r.x, r.y, r.z))));
    }
    const int j = (FMT == L_C16 ? k >> 1 : k) + (FIRST ? 1 : 0);  // the word
    const unsigned x = j == 0 ? r.x : (j == 1 ? r.y : (j == 2 ? r.z : r.w));
    if (FMT == L_C32) return x;
    return (k & 1) ? x >> 16 : x & 0xFFFFu;
}

// A thread's list while the stencil is walked: column lists (entry k of slot s
// at nbr[k n + s] with its cell codes and solid flag) or compact lists.  The
// first CAP accepted entries wait in shared memory, the 32-bit ones with entry
// k at [k][thread]; the 16-bit ones take COMPACT_STRIDE consecutive words a
// thread (an odd stride: no bank conflicts among equal k), read back as the
// records' words.  Entries past CAP go to their rows of nbr at once.
// STAGED (column lists on a dense grid): a candidate costs one store to the next
// free place and a conditional step of the pointer, a refused one overwritten
// by the next, where a store under a branch runs the branch for the warp
// whenever a lane accepts.  That pays for rows of several particles a cell
// (262,144 particles on voxels, 1.6 a cell: 35.5 us with the first lambda
// summed in the branch, 31.9 like this, 32.2 with the store in it), not for
// compact lists at unit density (2 M particles: 105 against 101 us) or hashed
// rows (1 M particles: 120 against 113 us).
constexpr int COMPACT_STRIDE = 9;
template <int FORMAT, int B, bool STAGED>
struct StagedEntries {
    static constexpr int CAP = FORMAT == L_C16 ? 2 * COMPACT_STRIDE : 16;
    static constexpr int WORDS = FORMAT == L_C16 ? COMPACT_STRIDE * B : CAP * B;  // of the block
    static constexpr int STEP = FORMAT == L_C16 ? 1 : B;
    static constexpr int ROW0 = FORMAT == L_COLUMN ? 0 : RecordFormat<FORMAT>::RECORDS;  // entry of nbr's row 0
    using T = typename std::conditional<FORMAT == L_C16, unsigned short, int>::type;
    T* first;  // entry 0
    T* at;     // the next place
    int* row;  // nbr + s
    int base;  // 16-bit entries: the scene's first slot
    int extra = 0;  // entries past CAP
    // init: else the list was begun by other threads, its count set by set_count
    __device__ __forceinline__ StagedEntries(unsigned* smem, int at_thread, int* nbr, const StepParams& p, int s,
                                             int slot0, bool init = true)
        : row(nbr + s), base(slot0) {
        if (FORMAT == L_C16)
            first = reinterpret_cast<T*>(smem + COMPACT_STRIDE * at_thread);
        else
            first = reinterpret_cast<T*>(smem) + at_thread;
        at = first;
        if (!init) return;
        // places past the count hold the sentinel in the records
        if (FORMAT == L_C16) {
#pragma unroll
            for (int q = 0; q < COMPACT_RECORDS / 2; q++) reinterpret_cast<unsigned*>(first)[q] = 0xFFFFFFFFu;
        } else {
#pragma unroll
            for (int q = 0; q < ROW0; q++) first[q * STEP] = (T)p.n;
        }
    }
    __device__ __forceinline__ bool room(int w) const { return at <= first + (CAP - w) * STEP; }
    __device__ __forceinline__ void put(int e, bool in) {  // with room only
        *at = (T)(FORMAT == L_C16 ? e - base : e);
        at += in ? STEP : 0;
    }
    __device__ __forceinline__ void push(const StepParams& p, int e) {
        if (at < first + CAP * STEP) {
            put(e, true);
        } else {
            if (CAP + extra < p.max_nbrs) row[(size_t)(CAP - ROW0 + extra) * p.n] = e;
            extra++;
        }
    }
    template <int W>
    __device__ __forceinline__ void take(const StepParams& p, const int (&e)[W], const bool (&in)[W]) {
        if (STAGED && room(W)) {
#pragma unroll
            for (int u = 0; u < W; u++) put(e[u], in[u]);
        } else {
#pragma unroll
            for (int u = 0; u < W; u++)
                if (in[u]) push(p, e[u]);
        }
    }
    // entry k set by itself, and the number of entries then (lists built by a group)
    __device__ __forceinline__ void place(const StepParams& p, int k, int e) {
        if (k < CAP) first[k * STEP] = (T)(FORMAT == L_C16 ? e - base : e);
        else if (k < p.max_nbrs) row[(size_t)(k - ROW0) * p.n] = e;
    }
    __device__ __forceinline__ void set_count(int c) {
        at = first + min(c, CAP) * STEP;
        extra = max(c - CAP, 0);
    }
    __device__ __forceinline__ int staged() const { return (int)(at - first) / STEP; }
    __device__ __forceinline__ int count() const { return staged() + extra; }
    // entry k below the count and the capacity
    __device__ __forceinline__ int get(const StepParams& p, int k) const {
        if (k >= CAP) return row[(size_t)(k - ROW0) * p.n];
        return (FORMAT == L_C16 ? base : 0) + (int)first[k * STEP];
    }
    // The list's c_n entries: records and rows, and the rows' sentinel entries
    // up to a multiple of the passes' chunk (pad divides the buffer's rows:
    // max_nbrs rounded up to LIST_PAD_MAX).  solid: a column list holds some.
    __device__ __forceinline__ void close(const StepParams& p, int s, int* __restrict__ cnt, int c_n, bool solid) {
        const int m = min(staged(), c_n);
        if (FORMAT == L_COLUMN) {
            cnt[s] = c_n | (solid ? CNT_SOLID : 0);
            for (int k = 0; k < m; k++) row[(size_t)k * p.n] = (int)first[k * STEP];
            for (int k = c_n; k % p.pad != 0; k++) row[(size_t)k * p.n] = sentinel_entry(p);
            return;
        }
        for (int k = ROW0; k < m; k++) row[(size_t)(k - ROW0) * p.n] = get(p, k);
        // places from the count on: the last refused candidate's, or entries
        // cut at the capacity
        for (int k = m; k < min(staged() + 1, ROW0); k++) first[k * STEP] = (T)(FORMAT == L_C16 ? 0xFFFF : p.n);
        uint4 r, r2;
        if (FORMAT == L_C16) {
            const unsigned* w = reinterpret_cast<const unsigned*>(first);
            r = make_uint4((unsigned)c_n | ((unsigned)base << 8), w[0], w[1], w[2]);
            r2 = make_uint4(w[3], w[4], w[5], w[6]);
        } else {
            auto e = [&](int k) { return (unsigned)first[k * STEP]; };
            if (FORMAT == L_C24) {
                r = make_uint4((unsigned)c_n | (e(0) << 8), e(1) | as_high_byte(e(4), 0), e(2) | as_high_byte(e(4), 1),
                               e(3) | as_high_byte(e(4), 2));
                r2 = make_uint4(e(5) | as_high_byte(e(9), 0), e(6) | as_high_byte(e(9), 1),
                                e(7) | as_high_byte(e(9), 2), e(8));
            } else {
                r = make_uint4((unsigned)c_n, e(0), e(1), e(2));
                r2 = make_uint4(e(3), e(4), e(5), e(6));
            }
        }
        p.rec[s] = r;
        if (c_n > ROW0 - RecordFormat<FORMAT>::EXT) p.rec2[s] = r2;
        for (int k = c_n - ROW0; k > 0 && k % p.pad != 0; k++) row[(size_t)k * p.n] = p.n;
    }
};

// One lane's part of a list that a group of lanes builds: the accepted
// candidates of its rows in order, k at [k][thread]; those past CAP are only
// counted, and LatePart collects them once the lane's place is known.
template <int B>
struct LanePart {
    static constexpr int CAP = 8;
    int* first;
    int c = 0;
    template <int W>
    __device__ __forceinline__ void take(const StepParams&, const int (&e)[W], const bool (&in)[W]) {
#pragma unroll
        for (int u = 0; u < W; u++)
            if (in[u]) {
                if (c < CAP) first[c * B] = e[u];
                c++;
            }
    }
};
template <int CAP, class Staged>
struct LatePart {
    Staged& list;
    int off, c;
    template <int W>
    __device__ __forceinline__ void take(const StepParams& p, const int (&e)[W], const bool (&in)[W]) {
#pragma unroll
        for (int u = 0; u < W; u++)
            if (in[u]) {
                if (c >= CAP) list.place(p, off + c, e[u]);
                c++;
            }
    }
};

// x_i - x_j of a pair from the list entry e of its neighbour q, as the walk formed it.
template <bool MIXED>
__device__ __forceinline__ float3 rel_entry(const StepParams& p, const float4& self, const float4& q, int e) {
    float3 d = make_float3(__fsub_rn(self.x, q.x), __fsub_rn(self.y, q.y), __fsub_rn(self.z, q.z));
    if (MIXED) {
        d.x = __fadd_rn(d.x, axis_shift(p.cell, e, 25));
        d.y = __fadd_rn(d.y, axis_shift(p.cell, e, 27));
        d.z = __fadd_rn(d.z, axis_shift(p.cell, e, 29));
    }
    return d;
}

// The entries a list dropped at its capacity, summed into the first lambda
// after the listed ones (a second walk, only where a list was cut).
template <bool MIXED, bool KAHAN>
struct DroppedEntries {
    LambdaAcc& a;
    const float4& self;
    const float4* xs;
    const float4* solid;
    int c;
    template <int W>
    __device__ __forceinline__ void take(const StepParams& p, const int (&e)[W], const bool (&in)[W]) {
#pragma unroll
        for (int u = 0; u < W; u++)
            if (in[u] && c++ >= p.max_nbrs)
                lambda_accumulate<KAHAN, MIXED>(p, a, rel_entry<MIXED>(p, self, load_entry(e[u], xs, solid), e[u]),
                                                entry_solid(e[u]));
    }
};

// The candidates [t0, t1) of one stencil row (its three cells' ids are
// consecutive, so their particles are one slot range), tested in slot order:
// W positions loaded together (past t1 too: the buffers are SPAN_PAD
// longer), each within h offered to out.  code: the entry's cell code of the
// row (dx, dy; dz = 0) and its solid flag; MIXED: b1, b2 are the bounds of the row's
// second and third cell, which give the entry's dz code and the cell shift.
// fp32 entries carry dz = 0, which no fp32 pass reads.
static_assert(4 <= SPAN_PAD, "a range reads at most SPAN_PAD positions past its end");
template <bool MIXED, int W, class L>
__device__ __forceinline__ void walk_range(const StepParams& p, const float4& self, int skip, const float4* pos,
                                           int t0, int t1, int b1, int b2, int dz0, int code, L& out) {
    for (int t = t0; t < t1; t += W) {
        float4 q[W];
        int e[W];
        bool in[W];
#pragma unroll
        for (int u = 0; u < W; u++) q[u] = pos[t + u];
        const int left = t1 - t, self_at = skip - t;
#pragma unroll
        for (int u = 0; u < W; u++) {
            float3 d = make_float3(__fsub_rn(self.x, q[u].x), __fsub_rn(self.y, q[u].y), __fsub_rn(self.z, q[u].z));
            e[u] = t + u + code;
            if (MIXED) {
                const int cz = dz0 + (t + u >= b1) + (t + u >= b2);
                e[u] += cz << 29;
                d.x = __fadd_rn(d.x, axis_shift(p.cell, code, 25));
                d.y = __fadd_rn(d.y, axis_shift(p.cell, code, 27));
                d.z = __fadd_rn(d.z, -(float)cz * p.cell);
            }
            in[u] = u < left && u != self_at && dot3e(d.x, d.y, d.z) <= p.h2;
        }
        out.take(p, e, in);
    }
}

// One stencil row on a hashed grid, the cells z0..z1 of (x, y): one slot range
// (two where the table's end cuts it), tested in slot order, W candidates
// loaded together.  A candidate belongs to the row if its packed cell is k
// cells above z0's: lines that share buckets put other cells' particles in the
// range.  code: the entry's cell code of the row (dx, dy; dz = 0) and its solid
// flag; zc: the particle's own z.  Bound by instruction issue (1 M particles,
// 16 blobs, first lambda included: a walk of each cell's bucket took 173 us
// mixed and 152 compact; this one 113 and 86; one candidate at a time 128 and
// 99).
template <bool MIXED, bool CODES, class L>
__device__ __forceinline__ void walk_hashed_row(const StepParams& p, const CellPack& cp, const float4& self, int skip,
                                                int x, int y, int z0, int z1, int zc, const float4* pos,
                                                const int* __restrict__ cells, const int* __restrict__ start, int code,
                                                L& out) {
    constexpr int W = 2;
    const f32x2 sxy = pack2(self.x, self.y);
    const f32x2 shift = pack2(axis_shift(p.cell, code, 25), axis_shift(p.cell, code, 27));
    while (z0 <= z1) {
        const int bucket = cell_bucket(make_int3(x, y, z0), p.hash_bits);
        const int m = min(z1 + 1 - z0, (1 << p.hash_bits) - bucket), dz0 = z0 - zc;
        const int t0 = start[bucket], t1 = start[bucket + m];
        const unsigned packed = pack_bits(cp, make_int3(x, y, z0));
        const int row_code = code + (CODES ? (dz0 + 1) << 29 : 0);
        for (int t = t0; t < t1; t += W) {
            int tw[W], e[W];
            unsigned k[W];
            ulonglong2 o[W];
            bool in[W];
#pragma unroll
            for (int w = 0; w < W; w++) {
                tw[w] = w ? min(t + w, t1 - 1) : t;
                k[w] = (unsigned)__ldg(&cells[tw[w]]) - packed;
                o[w] = reinterpret_cast<const ulonglong2*>(pos)[tw[w]];
            }
#pragma unroll
            for (int w = 0; w < W; w++) {
                k[w] = __funnelshift_r(k[w], k[w], cp.bz_shift);  // another x or y: above any k
                f32x2 dxy = sub2(sxy, o[w].x);
                float dz = __fsub_rn(self.z, lo2(o[w].y));
                if (MIXED) {
                    dxy = add2(dxy, shift);
                    dz = __fmaf_rn(-(float)(dz0 + (int)k[w]), p.cell, dz);  // by -1, 0 or 1: one rounding
                }
                e[w] = tw[w] + row_code + (CODES ? (int)(k[w] << 29) : 0);
                in[w] = (w == 0 || t + w < t1) && tw[w] != skip && k[w] < (unsigned)m &&
                        dot3e(lo2(dxy), hi2(dxy), dz) <= p.h2;
            }
            out.take(p, e, in);
        }
        z0 += m;
    }
}

// The stencil's candidates of fluid slot s in cell c, in list order, offered to
// out: on a dense grid the nine rows (with the static particles of each row
// after its fluid ones where the neighbourhood holds some, near); on a hashed
// grid the rows' bucket ranges.  CODES: entries with cell codes (column lists).
// A row's bounds are loaded just before its walk (fewer live registers, more
// resident warps).
template <bool MIXED, bool HASHED, bool SOLIDS, bool CODES, int G = 1, class L>
__device__ __forceinline__ void walk_stencil(const StepParams& p, const CellPack& cp, const float4& self, int s,
                                             const int3& c, const Geo& g, const float4* xs,
                                             const int* __restrict__ cell_sorted, const int* __restrict__ fstart,
                                             const float4* __restrict__ solid, const int* __restrict__ solid_cell,
                                             const int* __restrict__ sstart, bool near, L& out) {
    if constexpr (!HASHED) {
        // 4 candidates at a time for column lists, 2 for compact ones (their
        // build is held to 40 registers)
        constexpr int W = CODES ? 4 : 2;
        const int slab = g.gx * g.gz;
        const int z0 = max(c.z - 1, 0), z1 = min(c.z + 1, g.gz - 1);
        auto row_of = [&](int dy, int y, int dx) {
            const int x = c.x + dx;
            if (x < 0 || x >= g.gx) return;
            const int row = g.off + y * slab + x * g.gz;
            const int i1 = row + z0 + 1, i2 = row + min(z0 + 2, z1 + 1);  // the second and third cell
            const int code = CODES ? ((dx + 1) << 25) | ((dy + 1) << 27) | (1 << 29) : 0;
            walk_range<MIXED, W>(p, self, s, xs, fstart[row + z0], fstart[row + z1 + 1], MIXED ? fstart[i1] : 0,
                                 MIXED ? fstart[i2] : 0, z0 - c.z, code, out);
            if (SOLIDS && near)
                walk_range<MIXED, W>(p, self, -1, solid, sstart[row + z0], sstart[row + z1 + 1],
                                     MIXED ? sstart[i1] : 0, MIXED ? sstart[i2] : 0, z0 - c.z,
                                     code | (int)0x80000000u, out);
        };
        if constexpr (G == 4) {  // a lane's two or three rows
            const int lane = threadIdx.x % G;
#pragma unroll 1
            for (int r = lane ? 2 * lane + 1 : 0; r < 2 * lane + 3; r++) {
                const int dy = r / 3 - 1, y = c.y + dy;
                if (y >= 0 && y < g.gy) row_of(dy, y, r % 3 - 1);
            }
        } else {
#pragma unroll 1
            for (int dy = -1; dy <= 1; dy++) {
                const int y = c.y + dy;
                if (y < 0 || y >= g.gy) continue;
#pragma unroll 1
                for (int dx = -1; dx <= 1; dx++) row_of(dy, y, dx);
            }
        }
    } else {
        // cells past the packed field widths hold no particle; the dense
        // walk's entry order: a row's fluid cells, then its solid cells
        const int z0 = max(c.z - 1, 0), z1 = min(min(c.z + 1, g.gz - 1), (int)cp.mz);
#pragma unroll 1
        for (int dy = -1; dy <= 1; dy++) {
            const int y = c.y + dy;
            if (y < 0 || y >= g.gy || y > (int)cp.my) continue;
#pragma unroll 1
            for (int dx = -1; dx <= 1; dx++) {
                const int x = c.x + dx;
                if (x < 0 || x >= g.gx || x > (int)cp.mx) continue;
                const int code = CODES ? ((dx + 1) << 25) | ((dy + 1) << 27) : 0;
                walk_hashed_row<MIXED, CODES>(p, cp, self, s, x, y, z0, z1, c.z, xs, cell_sorted, fstart, code, out);
                if (SOLIDS && near)
                    walk_hashed_row<MIXED, CODES>(p, cp, self, -1, x, y, z0, z1, c.z, solid, solid_cell, sstart,
                                                  code | (int)0x80000000u, out);
            }
        }
    }
}

// FRAME: mixed storage with the iterations in the scene frame (positions
// relative to the box corner, compensated density sums; the walk's cell is
// the step's key, which rounding of the frame position could move).
// FORMAT: StagedEntries (compact lists hold no static particles and no cell
// codes).  The stencil is walked first, only listing the accepted candidates
// (no sums live across the walk: fewer registers, so more resident warps, and
// no pair term evaluated for the few lanes of a warp that accept), then the
// first lambda sums over the finished list, two entries' positions loaded
// together (in the cache from the walk); a list cut at the capacity walks once
// more to sum the dropped entries after the listed ones, so that the terms
// and their order do not depend on the capacity or the format.
// G = 4 (dense grids): four lanes share a particle's rows, each collecting its
// part; then the block's first warps sum and close the lists, a lane each (one lane
// of every group instead leaves four warps with eight lanes at work: 512 contexts
// of up to 45,000 particles overlapping 2.13 ms a step against 2.00).
template <bool MIXED, bool HASHED, bool FRAME, int FORMAT, bool SOLIDS, int B, int G = 1>
__device__ __forceinline__ void lists_lambda(const StepParams& p, const CellPack& cp, float4* __restrict__ xs,
                                             const int* __restrict__ key_sorted, const int* __restrict__ cell_sorted,
                                             const int* __restrict__ fstart, const float4* __restrict__ solid,
                                             const int* __restrict__ solid_cell, const int* __restrict__ sstart,
                                             int* __restrict__ nbr, int* __restrict__ cnt, float* __restrict__ rho,
                                             int* status) {
    static_assert(FORMAT == L_COLUMN || (!MIXED && !SOLIDS), "compact lists");
    constexpr bool CODES = FORMAT == L_COLUMN;
    using Staged = StagedEntries<FORMAT, B / G, FORMAT == L_COLUMN && !HASHED>;
    __shared__ unsigned stage[Staged::WORDS];
    // the cell shifts of the entries: from a table on a dense grid, formed per
    // entry on a hashed one (whose walk leaves it no registers)
    constexpr bool TABLE = MIXED && !HASHED;
    __shared__ float4 shift_tab[TABLE ? 64 : 1];
    pdl_wait();
    if (TABLE) fill_shift_table(p, shift_tab);
    int s = (blockIdx.x * B + threadIdx.x) / G;
    constexpr bool KAHAN = MIXED || FRAME;
    __shared__ int totals[G > 1 ? B / G : 1];  // the lists' lengths
    if constexpr (G > 1) {
        using Lane = LanePart<B>;
        __shared__ int part[Lane::CAP * B];
        if (s < p.n) {
            const float4 self = xs[s];
            const Geo g = geo_slot(p, s);
            const int3 c = KAHAN ? slot_cell(p, cp, g, key_sorted, cell_sorted, s)
                                 : plain_cell(p, g, self.x, self.y, self.z);
            const bool near = SOLIDS && p.ns > 0 && p.solid_near && __ldg(&p.solid_near[__ldg(&key_sorted[s])]);
            Staged list(stage, threadIdx.x / G, nbr, p, s, g.slot0, threadIdx.x % G == 0);
            Lane mine{part + threadIdx.x};
            walk_stencil<MIXED, HASHED, SOLIDS, CODES, G>(p, cp, self, s, c, g, xs, cell_sorted, fstart, solid,
                                                          solid_cell, sstart, near, mine);
            int off;
            const int total = group_offset<G>(mine.c, off);
            __syncwarp(((1u << G) - 1u) << ((threadIdx.x & 31) & ~(G - 1)));  // the list's sentinels are set
            for (int k = 0; k < min(mine.c, Lane::CAP); k++) list.place(p, off + k, mine.first[k * B]);
            if (mine.c > Lane::CAP) {
                LatePart<Lane::CAP, Staged> late{list, off, 0};
                walk_stencil<MIXED, HASHED, SOLIDS, CODES, G>(p, cp, self, s, c, g, xs, cell_sorted, fstart, solid,
                                                              solid_cell, sstart, near, late);
            }
            if (threadIdx.x % G == 0) totals[threadIdx.x / G] = total;
        }
        __syncthreads();
        if (threadIdx.x >= B / G) return;
        s = blockIdx.x * (B / G) + threadIdx.x;
    }
    if (s >= p.n) return;
    const float4 self = xs[s];
    const Geo g = geo_slot(p, s);
    // fp32 on a dense grid: the cell the prediction keyed this position by
    const int3 c = (MIXED || HASHED || FRAME) ? slot_cell(p, cp, g, key_sorted, cell_sorted, s)
                                              : plain_cell(p, g, self.x, self.y, self.z);
    Staged out(stage, threadIdx.x, nbr, p, s, g.slot0, G == 1);
    // static particles only where the cell's neighbourhood holds some
    const bool near = SOLIDS && p.ns > 0 && p.solid_near && __ldg(&p.solid_near[__ldg(&key_sorted[s])]);
    if constexpr (G == 1) {
        walk_stencil<MIXED, HASHED, SOLIDS, CODES>(p, cp, self, s, c, g, xs, cell_sorted, fstart, solid, solid_cell,
                                                   sstart, near, out);
    } else {
        out.set_count(totals[threadIdx.x]);
    }
    int c_n = out.count();
    const int m = min(c_n, p.max_nbrs);
    LambdaAcc a = lambda_init(p);
    auto position = [&](int e) {
        if (FORMAT != L_COLUMN) return xs[e];  // compact entries are slots
        return SOLIDS ? load_entry(e, xs, solid) : xs[entry_slot(e)];
    };
    int solids = 0;  // the sign bit: a static particle among the entries
    for (int k = 0; k < m; k += 2) {
        const bool two = k + 1 < m;
        const int e0 = out.get(p, k), e1 = two ? out.get(p, k + 1) : e0;
        const float4 q0 = position(e0), q1 = position(e1);
        if (SOLIDS) solids |= e0 | e1;
        auto rel = [&](const float4& q, int e) {
            return TABLE ? rel_t<TABLE>(self, q, e, shift_tab) : rel_entry<MIXED>(p, self, q, e);
        };
        lambda_accumulate<KAHAN, MIXED>(p, a, rel(q0, e0), SOLIDS && entry_solid(e0));
        if (two) lambda_accumulate<KAHAN, MIXED>(p, a, rel(q1, e1), SOLIDS && entry_solid(e1));
    }
    if (c_n > p.max_nbrs) {
        DroppedEntries<MIXED, KAHAN> rest{a, self, xs, solid, 0};
        walk_stencil<MIXED, HASHED, SOLIDS, CODES>(p, cp, self, s, c, g, xs, cell_sorted, fstart, solid, solid_cell,
                                                   sstart, near, rest);
        set_status(status, ST_NBR_OVERFLOW);
        c_n = p.max_nbrs;
    }
    out.close(p, s, cnt, c_n, solids < 0);
    // lambda into w in place: neighbours read only xyz of this element here
    reinterpret_cast<float*>(xs)[4 * (size_t)s + 3] = lambda_of(p, a);
    if (rho) rho[s] = density_of(p, a);
}

template <bool MIXED, bool HASHED, int B, bool FRAME = false, int G = 1>
__global__ void __launch_bounds__(B) k_lists_lambda(StepParams p, CellPack cp, float4* __restrict__ xs,
                                                    const int* __restrict__ key_sorted,
                                                    const int* __restrict__ cell_sorted,
                                                    const int* __restrict__ fstart,
                                                    const float4* __restrict__ solid,
                                                    const int* __restrict__ solid_cell,
                                                    const int* __restrict__ sstart,
                                                    int* __restrict__ nbr, int* __restrict__ cnt,
                                                    float* __restrict__ rho, int* status) {
    lists_lambda<MIXED, HASHED, FRAME, 0, true, B, G>(p, cp, xs, key_sorted, cell_sorted, fstart, solid, solid_cell,
                                                   sstart, nbr, cnt, rho, status);
}

// Compact 16-bit lists by four lanes a particle (small dense scenes).
template <int B, bool FRAME>
__global__ void __launch_bounds__(B) k_lists_compact_group(StepParams p, CellPack cp, float4* __restrict__ xs,
                                                           const int* __restrict__ key_sorted,
                                                           const int* __restrict__ cell_sorted,
                                                           const int* __restrict__ fstart, int* __restrict__ nbr,
                                                           int* __restrict__ cnt, float* __restrict__ rho, int* status) {
    lists_lambda<false, false, FRAME, L_C16, false, B, 4>(p, cp, xs, key_sorted, cell_sorted, fstart, nullptr, nullptr,
                                                          nullptr, nbr, cnt, rho, status);
}

// Compact lists (no static particles, fp32 pair offsets).
// Held to 12 blocks of 128 threads per SM (40 registers, at most 36 bytes
// spilled): the extra resident warps hide more of the gathers' latency
// (config 3: 0.382 -> 0.353 ms a step; a walk that loads the next row's
// bounds ahead, or 4 gathers in flight, was slower).
template <bool HASHED, int B, bool FRAME, int FMT>
__global__ void __launch_bounds__(B, 1536 / B) k_lists_compact(StepParams p, CellPack cp, float4* __restrict__ xs,
                                                             const int* __restrict__ key_sorted,
                                                             const int* __restrict__ cell_sorted,
                                                             const int* __restrict__ fstart,
                                                             const float4* __restrict__ solid,
                                                             const int* __restrict__ solid_cell,
                                                             const int* __restrict__ sstart,
                                                             int* __restrict__ nbr, int* __restrict__ cnt,
                                                             float* __restrict__ rho, int* status) {
    lists_lambda<false, HASHED, FRAME, FMT, false, B>(p, cp, xs, key_sorted, cell_sorted, fstart, solid, solid_cell,
                                                      sstart, nbr, cnt, rho, status);
}

// Walk a particle's list U entries at a time, calling f(entry, position)
// for each (SOL: the scene has static particles, whose entries read solid).
// E entries (U or LIST_PAD_MAX) are loaded together with the count, the
// rest a chunk ahead of their gathers: with E = LIST_PAD_MAX a list of up to
// 8 neighbours waits for one round trip to DRAM for its entries and then one
// to L2 per chunk of gathers, at the price of loading 8 entries for shorter
// lists (the position pass gains, measured; the lambda pass, with fewer
// instructions per pair to hide the latency behind, loses and keeps E = U).
// The list is padded with sentinel entries to a multiple of U (the list
// build's pad) and the buffer holds at least LIST_PAD_MAX rows (2
// LIST_PAD_MAX when a count exceeds LIST_PAD_MAX), so every entry a chunk
// below the count reads is valid and every load in bounds.
template <int U, bool SOL, int E, class F>
__device__ __forceinline__ void walk_column(const StepParams& p, const int* __restrict__ col, const int (&e0)[E], int c,
                                            const float4* __restrict__ xs, const float4* __restrict__ solid, F&& f) {
    if (E > U) {
#pragma unroll
        for (int k = 0; k < E; k += U) {
            if (k >= c) return;
            float4 q[U];
#pragma unroll
            for (int u = 0; u < U; u++) q[u] = SOL ? load_entry(e0[k + u], xs, solid) : xs[entry_slot(e0[k + u])];
#pragma unroll
            for (int u = 0; u < U; u++) f(e0[k + u], q[u]);
        }
        if (c <= E) return;
    }
    // the chunks from E on (E = U: from the first), each chunk's entries
    // loaded while the one before is gathered
    int nx[U];
#pragma unroll
    for (int u = 0; u < U; u++) nx[u] = E > U ? __ldg(&col[(size_t)(E + u) * p.n]) : e0[u];
    for (int k = E > U ? E : 0; k < c; k += U) {
        int e[U];
        float4 q[U];
#pragma unroll
        for (int u = 0; u < U; u++) e[u] = nx[u];
        if (k + U < c) {
#pragma unroll
            for (int u = 0; u < U; u++) nx[u] = __ldg(&col[(size_t)(k + U + u) * p.n]);
        }
#pragma unroll
        for (int u = 0; u < U; u++) q[u] = SOL ? load_entry(e[u], xs, solid) : xs[entry_slot(e[u])];
#pragma unroll
        for (int u = 0; u < U; u++) f(e[u], q[u]);
    }
}
// SOL: f is called as f(entry, position, true_type or false_type), whether the
// entry may be a static particle: warps whose lists hold none (nine in ten
// of a block lying on voxels) run the walk without the tests.
template <int U, bool SOL, int E, class F>
__device__ __forceinline__ void for_each_entry(const StepParams& p, const int* __restrict__ col, const int (&e0)[E],
                                               int raw, const float4* __restrict__ xs,
                                               const float4* __restrict__ solid, F&& f) {
    static_assert(E % U == 0 && E <= LIST_PAD_MAX, "prefetch depth");
    const int c = raw & ~CNT_SOLID;
    if (SOL && __any_sync(__activemask(), raw & CNT_SOLID))
        walk_column<U, true>(p, col, e0, c, xs, solid, [&](int e, const float4& q) { f(e, q, std::true_type()); });
    else
        walk_column<U, false>(p, col, e0, c, xs, solid, [&](int e, const float4& q) { f(e, q, std::false_type()); });
}

// The start of a particle's list: its record, or its count and first E column
// entries.  The lists are older than the pass's predecessor in the stream
// (list build, position pass, lambda pass, position pass, ...), so a pass
// launched behind it loads them before it waits for it: when its blocks start,
// every block of the predecessor has passed its own wait, so whatever ran before
// that has completed.  (The first position pass follows the list build: it
// waits first, StepParams::early unset.)  One dependent load less a pass where
// launches and latency count: host frames of 77,777 particles 420 -> 397 us for
// four, 157,443 in 37 scenes 382 -> 371 for four steps; 2 M: no change.
template <int FMT, int E>
struct ListHead {
    uint4 rec;
    int raw, e0[E];
    __device__ __forceinline__ void load(const StepParams& p, const int* __restrict__ nbr,
                                         const int* __restrict__ cnt, int s) {
        if (FMT != L_COLUMN) {
            rec = __ldg(&p.rec[s]);
        } else {
#pragma unroll
            for (int u = 0; u < E; u++) e0[u] = __ldg(&nbr[(size_t)u * p.n + s]);
            raw = __ldg(&cnt[s]);
        }
    }
};

// P particles per thread: the lists of slots s[0..P) walked together, U
// entries of each per round, so the loads of all P lists and their gathers
// are in flight at once; f(r, entry, position) per entry of particle r in
// list order.  Past its own count a particle reads the sentinel entry (every
// pair term with it is exactly zero), so the lists may differ in length.
template <int U, int P, bool SOL, class F>
__device__ __forceinline__ void for_each_entry_p(const StepParams& p, const int* __restrict__ nbr,
                                                 const int (&s)[P], const int (&c)[P],
                                                 const float4* __restrict__ xs, const float4* __restrict__ solid,
                                                 F&& f) {
    int cmax = 0;
#pragma unroll
    for (int r = 0; r < P; r++) cmax = max(cmax, c[r]);
    const int sent = sentinel_entry(p);
    for (int k = 0; k < cmax; k += U) {
        int e[P][U];
        float4 q[P][U];
#pragma unroll
        for (int r = 0; r < P; r++)
#pragma unroll
            for (int u = 0; u < U; u++) e[r][u] = k + u < c[r] ? __ldg(&nbr[(size_t)(k + u) * p.n + s[r]]) : sent;
#pragma unroll
        for (int r = 0; r < P; r++)
#pragma unroll
            for (int u = 0; u < U; u++) q[r][u] = SOL ? load_entry(e[r][u], xs, solid) : xs[entry_slot(e[r][u])];
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int r = 0; r < P; r++) f(r, e[r][u], q[r][u]);
    }
}

// The entries [K0, K0 + M) of a compact list from record r (K0 = 0: the
// first record), min(U, M) gathers at a time; false once the count is
// reached.
template <int U, int M, int K0, int FMT, class T, class G, class F>
__device__ __forceinline__ bool walk_record(const StepParams& p, const uint4& r, int c, int base, G&& gather,
                                            F&& f) {
    constexpr int V = U < M ? U : M;
    // each chunk decodes its own entries (a short list decodes only those it uses)
#pragma unroll
    for (int k = 0; k < M; k += V) {
        if (K0 + k >= c) return false;
        int sl[V];
        T q[V];
#pragma unroll
        for (int u = 0; u < V; u++)
            if (k + u < M) {
                const unsigned x = record_entry<FMT, K0 == 0>(r, k + u);
                // one gather at a time never reads past the count
                sl[u] = FMT != L_C16 ? (int)x : (V == 1 ? base + (int)x : compact_slot(p, base, x));
                q[u] = gather(sl[u]);
            }
#pragma unroll
        for (int u = 0; u < V; u++)
            if (k + u < M) f(sl[u], q[u]);
    }
    return K0 + M < c;
}

// Walk a compact list (record r of slot s, r2 its second record; col =
// nbr + s, its overflow rows): gather(slot) loads what f(slot, value) needs
// of each neighbour.  A record's entries go min(U, its entries) at a time,
// all gathers of a chunk in flight together, so with U >= 4 a list of up to
// 4 neighbours (3 in 32-bit records) waits for one round trip to DRAM (the
// record, with the particle's own loads) and one to L2 for the neighbours;
// the second record is loaded only for a longer list.  Past the count an
// entry reads the sentinel slot, whose terms are exactly zero; the overflow
// rows are padded with it to a multiple of U (the list build's pad).
template <int U, int FMT, class T, class G, class F>
__device__ __forceinline__ void walk_compact(const StepParams& p, const uint4& r, const uint4* __restrict__ r2,
                                             const int* __restrict__ col, G&& gather, F&& f) {
    using RF = RecordFormat<FMT>;
    const int c = FMT == L_C32 ? (int)r.x : (int)(r.x & 0xFFu);
    const int base = FMT == L_C16 ? (int)(r.x >> 8) : 0;
    if (!walk_record<U, RF::INLINE, 0, FMT, T>(p, r, c, base, gather, f)) return;
    if (!walk_record<U, RF::EXT, RF::INLINE, FMT, T>(p, __ldg(r2), c, base, gather, f)) return;
    constexpr int R = RF::RECORDS;
    int nx[U];
#pragma unroll
    for (int u = 0; u < U; u++) nx[u] = __ldg(&col[(size_t)u * p.n]);
    for (int k = R; k < c; k += U) {
        int e[U];
        T q[U];
#pragma unroll
        for (int u = 0; u < U; u++) e[u] = nx[u];
        if (k + U < c) {
#pragma unroll
            for (int u = 0; u < U; u++) nx[u] = __ldg(&col[(size_t)(k - R + U + u) * p.n]);
        }
#pragma unroll
        for (int u = 0; u < U; u++) q[u] = gather(e[u]);
#pragma unroll
        for (int u = 0; u < U; u++) f(e[u], q[u]);
    }
}

// The list format of a pass: F bit 3 compact, with bit 4 24-bit, with bit 5
// 32-bit records.
template <int F>
struct ListFormatOf {
    static constexpr int value = !(F & 8) ? L_COLUMN : ((F & 32) ? L_C32 : ((F & 16) ? L_C24 : L_C16));
};

// Lambda pass over the lists (iterations after the first); U neighbour
// gathers in flight per thread.
// F: bit 0 mixed precision, bit 1 the scene has static particles (the
// solid-free kernels skip the per-entry solid tests).
template <int F, int U, int B, int P = 1>
__global__ void __launch_bounds__(B) k_lambda(StepParams p, float4* __restrict__ xs,
                                              const int* __restrict__ nbr, const int* __restrict__ cnt,
                                              const float4* __restrict__ solid,
                                              float* __restrict__ rho) {
    // F bit 2: the scene frame (fp32 pair offsets, compensated density sums)
    // F bits 3-5: compact lists (fp32 pair offsets, no static particles), ListFormatOf
    constexpr bool MIXED = (F & 1) != 0, SOL = (F & 2) != 0, KAHAN = MIXED || (F & 4) != 0;
    constexpr int FMT = ListFormatOf<F>::value;
    constexpr bool COMPACT = FMT != L_COLUMN;
    static_assert(!COMPACT || (!MIXED && !SOL && P == 1), "compact lists");
    __shared__ float4 shift_tab[MIXED ? 64 : 1];
    if (P == 1) {
        const int s = blockIdx.x * B + threadIdx.x;
        const bool live = s < p.n;
        ListHead<FMT, U> head;
        if (live) head.load(p, nbr, cnt, s);
        pdl_wait();
        if (MIXED) fill_shift_table(p, shift_tab);
        if (!live) return;
        const float4 self = xs[s];
        LambdaAcc a = lambda_init(p);
        if (COMPACT) {
            walk_compact<U, FMT, float4>(
                p, head.rec, p.rec2 + s, nbr + s, [&](int t) { return xs[t]; },
                [&](int, float4 q) { lambda_accumulate<KAHAN>(p, a, rel_t<false>(self, q, 0, shift_tab), false); });
        } else {
            for_each_entry<U, SOL>(p, nbr + s, head.e0, head.raw, xs, solid, [&](int e, float4 q, auto sol) {
                float3 d = rel_t<MIXED>(self, q, e, shift_tab);
                lambda_accumulate<KAHAN, MIXED>(p, a, d, decltype(sol)::value && entry_solid(e));
            });
        }
        reinterpret_cast<float*>(xs)[4 * (size_t)s + 3] = lambda_of(p, a);
        if (rho) rho[s] = density_of(p, a);
        return;
    }
    pdl_wait();
    if (MIXED) fill_shift_table(p, shift_tab);
    // P slots per thread, B apart (each load of the block coalesced)
    int s[P], c[P];
    float4 self[P];
    LambdaAcc a[P];
#pragma unroll
    for (int r = 0; r < P; r++) {
        s[r] = (blockIdx.x * P + r) * B + threadIdx.x;
        const bool ok = s[r] < p.n;
        c[r] = ok ? __ldg(&cnt[s[r]]) & ~CNT_SOLID : 0;
        self[r] = ok ? xs[s[r]] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        a[r] = lambda_init(p);
    }
    for_each_entry_p<U, P, SOL>(p, nbr, s, c, xs, solid, [&](int r, int e, float4 q) {
        float3 d = rel_t<MIXED>(self[r], q, e, shift_tab);
        lambda_accumulate<KAHAN, MIXED>(p, a[r], d, SOL && entry_solid(e));
    });
#pragma unroll
    for (int r = 0; r < P; r++) {
        if (s[r] >= p.n) continue;
        reinterpret_cast<float*>(xs)[4 * (size_t)s[r] + 3] = lambda_of(p, a[r]);
        if (rho) rho[s[r]] = density_of(p, a[r]);
    }
}

// Position correction with s_corr, solid push-out and box clamp (Jacobi).
// The last iteration also writes v = (x* - x) / dt.
struct DeltaAcc {
    float px, py, pz, cx, cy, cz;
    int nct;
};

template <bool MIXED, bool SOL, bool POW = true>
__device__ __forceinline__ void delta_pair(const StepParams& p, DeltaAcc& a, const float4& self, int e, float4 q,
                                           const float4* tab) {
    const float li = self.w;
    const bool sol = SOL && entry_solid(e);
    float3 d = rel_t<MIXED>(self, q, e, tab);
    const float r2 = dot3e(d.x, d.y, d.z);
    const float inv_r = inv_r_of<MIXED>(r2);
    const float r = __fmul_rn(r2, inv_r);
    const float lj = sol ? li : q.w;
    const float w = __fmul_rn(__fadd_rn(__fadd_rn(li, lj), scorr_hd<POW>(p, hdiff(p, r2))), spiky_g(p, r, inv_r));
    a.px = __fmaf_rn(w, d.x, a.px);
    a.py = __fmaf_rn(w, d.y, a.py);
    a.pz = __fmaf_rn(w, d.z, a.pz);
    if (sol && r < p.contact && r2 > 0.0f) {
        const float t = __fmul_rn(__fsub_rn(p.contact, r), inv_r);
        a.cx = __fmaf_rn(t, d.x, a.cx);
        a.cy = __fmaf_rn(t, d.y, a.cy);
        a.cz = __fmaf_rn(t, d.z, a.cz);
        a.nct++;
    }
}

// dp = (m / rho0) sum (lambda_i + lambda_j + s_corr) dW, dW = -Ks g d; the
// solid push-out averaged; the box clamp; x* and (last pass) v written.
// scene: the slot's scene index (scene_index); packed: its packed cell in
// mixed precision on a sorted packed-cell array (else unused), both loaded
// before the neighbour walk.
template <bool MIXED>
__device__ __forceinline__ void delta_finish(const StepParams& p, const CellPack& cp, int s, const float4& self,
                                             const DeltaAcc& a, float4* __restrict__ xs_out,
                                             const int* __restrict__ key_sorted, const float4* __restrict__ x,
                                             float4* __restrict__ v_out, int scene, int packed) {
    const float kd = __fmul_rn(-p.ks, p.mr);
    float dx = __fmul_rn(a.px, kd), dy = __fmul_rn(a.py, kd), dz = __fmul_rn(a.pz, kd);
    if (a.nct) {
        const float inv = __frcp_rn((float)a.nct);
        dx = __fmaf_rn(a.cx, inv, dx);
        dy = __fmaf_rn(a.cy, inv, dy);
        dz = __fmaf_rn(a.cz, inv, dz);
    }
    float4 out;
    int3 cs = make_int3(0, 0, 0);
    const Geo g = geo_of(p, scene);
    if (!MIXED) {
        out = make_float4(clampf(__fadd_rn(self.x, dx), g.lox, g.hix), clampf(__fadd_rn(self.y, dy), g.loy, g.hiy),
                          clampf(__fadd_rn(self.z, dz), g.loz, g.hiz), 0.0f);
    } else {
        if (p.cell_sorted) {
            const unsigned u = (unsigned)packed;
            cs = make_int3((int)(u & cp.mx), (int)((u >> cp.by_shift) & cp.my), (int)((u >> cp.bz_shift) & cp.mz));
        } else {
            cs = slot_cell(p, cp, g, key_sorted, nullptr, s);
        }
        out = make_float4(clamp_offset(p, __fadd_rn(self.x, dx), cs.x, g.lox, g.hix),
                          clamp_offset(p, __fadd_rn(self.y, dy), cs.y, g.loy, g.hiy),
                          clamp_offset(p, __fadd_rn(self.z, dz), cs.z, g.loz, g.hiz), 0.0f);
    }
    xs_out[s] = out;
    if (v_out) {
        float4 xo = x[p.src ? __ldg(&p.src[s]) : s];  // the committed position, unsorted when src is set
        if (!MIXED && p.frame) {  // the committed state is cell + offset: into the scene frame
            const int3 co = unpack_cell(cp, xo.w);
            xo = make_float4(__fmaf_rn((float)co.x, p.cell, xo.x), __fmaf_rn((float)co.y, p.cell, xo.y),
                             __fmaf_rn((float)co.z, p.cell, xo.z), 0.0f);
        }
        float3 d = make_float3(__fsub_rn(out.x, xo.x), __fsub_rn(out.y, xo.y), __fsub_rn(out.z, xo.z));
        if (MIXED) {
            int3 co = unpack_cell(cp, xo.w);
            d.x = __fmaf_rn((float)(cs.x - co.x), p.cell, d.x);
            d.y = __fmaf_rn((float)(cs.y - co.y), p.cell, d.y);
            d.z = __fmaf_rn((float)(cs.z - co.z), p.cell, d.z);
        }
        v_out[s] = make_float4(__fmul_rn(d.x, p.inv_dt), __fmul_rn(d.y, p.inv_dt), __fmul_rn(d.z, p.inv_dt), 0.0f);
    }
}

// With one particle per thread and up to 2 gathers in flight the kernel
// fits 40 registers without spilling: 6 blocks of 256 threads per SM instead
// of 5 (a 262,144-particle pass then takes 1.12 waves of the GPU instead of
// 1.35).  Compact lists with one gather in flight fit 32 registers with at
// most 20 bytes spilled (their steps have an integer s_corr exponent: no powf):
// 16 blocks of 128 threads per SM, the whole SM's warps.  P = 2:
// two particles per thread (B apart), their lists walked together.
template <int F, int U, int B, int P = 1>
__global__ void __launch_bounds__(B, ((F & 8) && U == 1) ? 2048 / B : ((U <= 2 && P == 1) ? 1536 / B : 1))
    k_delta(StepParams p, CellPack cp, const float4* __restrict__ xs, float4* __restrict__ xs_out,
            const int* __restrict__ nbr, const int* __restrict__ cnt, const float4* __restrict__ solid,
            const int* __restrict__ key_sorted, const float4* __restrict__ x, float4* __restrict__ v_out) {
    constexpr bool MIXED = (F & 1) != 0, SOL = (F & 2) != 0;
    constexpr int FMT = ListFormatOf<F>::value;
    constexpr bool COMPACT = FMT != L_COLUMN;
    static_assert(!COMPACT || (!MIXED && !SOL && P == 1), "compact lists");
    __shared__ float4 shift_tab[MIXED ? 64 : 1];
    if (P == 1) {
        const int s = blockIdx.x * B + threadIdx.x;
        const bool live = s < p.n;
        ListHead<FMT, LIST_PAD_MAX> head;
        if (live && p.early) head.load(p, nbr, cnt, s);
        pdl_wait();
        if (MIXED) fill_shift_table(p, shift_tab);
        if (!live) return;
        if (!p.early) head.load(p, nbr, cnt, s);
        const float4 self = xs[s];
        const int scene = FMT == L_C16 ? scene_of_record(p, head.rec.x) : scene_index(p, s);
        const int packed = (MIXED && p.cell_sorted) ? __ldg(&p.cell_sorted[s]) : 0;
        DeltaAcc a{0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0};
        if (COMPACT) {
            walk_compact<U, FMT, float4>(
                p, head.rec, p.rec2 + s, nbr + s, [&](int t) { return xs[t]; },
                [&](int t, float4 q) { delta_pair<false, false, false>(p, a, self, t, q, shift_tab); });
        } else {
            for_each_entry<U, SOL>(p, nbr + s, head.e0, head.raw, xs, solid, [&](int e, float4 q, auto sol) {
                delta_pair<MIXED, decltype(sol)::value>(p, a, self, e, q, shift_tab);
            });
        }
        delta_finish<MIXED>(p, cp, s, self, a, xs_out, key_sorted, x, v_out, scene, packed);
        return;
    }
    pdl_wait();
    if (MIXED) fill_shift_table(p, shift_tab);
    int s[P], c[P];
    float4 self[P];
    DeltaAcc a[P];
#pragma unroll
    for (int r = 0; r < P; r++) {
        s[r] = (blockIdx.x * P + r) * B + threadIdx.x;
        const bool ok = s[r] < p.n;
        c[r] = ok ? __ldg(&cnt[s[r]]) & ~CNT_SOLID : 0;
        self[r] = ok ? xs[s[r]] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        a[r] = DeltaAcc{0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0};
    }
    for_each_entry_p<U, P, SOL>(p, nbr, s, c, xs, solid, [&](int r, int e, float4 q) {
        delta_pair<MIXED, SOL>(p, a[r], self[r], e, q, shift_tab);
    });
#pragma unroll
    for (int r = 0; r < P; r++)
        if (s[r] < p.n)
            delta_finish<MIXED>(p, cp, s[r], self[r], a[r], xs_out, key_sorted, x, v_out, scene_index(p, s[r]),
                                (MIXED && p.cell_sorted) ? __ldg(&p.cell_sorted[s[r]]) : 0);
}

// A neighbour's predicted position and velocity (the XSPH gathers).
struct PosVel {
    float4 x, v;
};

// One XSPH pair: a += (v_j - v_i) hd^3 (the sum is scaled by c K6 once).
template <bool MIXED>
__device__ __forceinline__ void xsph_pair(const StepParams& p, const float4& self, const float4& vi,
                                          const float4& q, const float4& vj, int e, const float4* tab, float& ax,
                                          float& ay, float& az) {
    float3 d = rel_t<MIXED>(self, q, e, tab);
    const float hd = hdiff(p, dot3e(d.x, d.y, d.z));
    const float w = __fmul_rn(__fmul_rn(hd, hd), hd);
    ax = __fmaf_rn(__fsub_rn(vj.x, vi.x), w, ax);
    ay = __fmaf_rn(__fsub_rn(vj.y, vi.y), w, ay);
    az = __fmaf_rn(__fsub_rn(vj.z, vi.z), w, az);
}

// XSPH viscosity (Macklin & Mueller eq. 17) and commit x = x*.
// With xs_next, also the next step's prediction from the state it commits
// (into xs_next, key, rank, count, cellk; count is zero here, the step's
// scan having consumed it).
template <int F, int U>
__device__ __forceinline__ void xsph_commit(const StepParams& p, const CellPack& cp, const float4* __restrict__ xs,
                                            const float4* __restrict__ v_in, const int* __restrict__ nbr,
                                            const int* __restrict__ cnt, const int* __restrict__ key_sorted,
                                            float4* __restrict__ x_out, float4* __restrict__ v_out,
                                            float4* __restrict__ xs_next, int* __restrict__ key,
                                            int* __restrict__ rank, int* __restrict__ count, int* __restrict__ cellk,
                                            int* __restrict__ tile_count) {
    constexpr bool MIXED = (F & 1) != 0, SOL = (F & 2) != 0;
    constexpr int FMT = ListFormatOf<F>::value;
    constexpr bool COMPACT = FMT != L_COLUMN;
    static_assert(!COMPACT || (!MIXED && !SOL), "compact lists");
    __shared__ float4 shift_tab[MIXED ? 64 : 1];
    __shared__ TileSum tiles;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = s < p.n;
    // older than the last position pass (ListHead): loaded before the wait for
    // it, but where the 32-register kernel would spill for it
    constexpr bool AHEAD = !(FMT == L_C24 && U == 1);
    uint4 rec = make_uint4(0u, 0u, 0u, 0u);
    if (COMPACT && AHEAD) rec = __ldg(&p.rec[live ? s : 0]);
    const int raw = COMPACT ? 0 : __ldg(&cnt[live ? s : 0]);
    // the block's tile: that of its first particle's cell in this step
    if (xs_next && threadIdx.x == 0) open_tile_sum(tiles, __ldg(&key_sorted[s]));
    pdl_wait();
    const float4 self = xs[live ? s : 0];  // in flight across the barrier
    const float4 vi = v_in[live ? s : 0];
    if (COMPACT && !AHEAD) rec = __ldg(&p.rec[live ? s : 0]);
    if (MIXED)
        fill_shift_table(p, shift_tab);
    else if (xs_next)
        __syncthreads();
    if (!live) return;
    const int* __restrict__ col = nbr + s;
    float ax = 0.0f, ay = 0.0f, az = 0.0f;
    if (COMPACT && p.c_xsph != 0.0f) {
        walk_compact<U, FMT, PosVel>(
            p, rec, p.rec2 + s, col, [&](int t) { return PosVel{xs[t], v_in[t]}; },
            [&](int t, const PosVel& q) { xsph_pair<false>(p, self, vi, q.x, q.v, t, shift_tab, ax, ay, az); });
    } else if (p.c_xsph != 0.0f) {
        const int c = raw & ~CNT_SOLID;
        const int sent = sentinel_entry(p);
        for (int k = 0; k < c; k += U) {
            int e[U];
            float4 q[U], vj[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int t = __ldg(&col[(size_t)(k + u) * p.n]);  // padded list: valid below roundup(c, U)
                e[u] = (SOL && entry_solid(t)) ? sent : t;  // solids take no part (the sentinel's zero term)
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                q[u] = xs[entry_slot(e[u])];
                vj[u] = v_in[entry_slot(e[u])];
            }
#pragma unroll
            for (int u = 0; u < U; u++) xsph_pair<MIXED>(p, self, vi, q[u], vj[u], e[u], shift_tab, ax, ay, az);
        }
    }
    // v += c sum (v_j - v_i) W, W = K6 hd^3
    const float cx = __fmul_rn(p.c_xsph, p.k6);
    const float4 vc = make_float4(__fmaf_rn(cx, ax, vi.x), __fmaf_rn(cx, ay, vi.y), __fmaf_rn(cx, az, vi.z), 0.0f);
    v_out[s] = vc;
    const Geo g = FMT == L_C16 ? geo_of(p, scene_of_record(p, rec.x))
                                     : geo_slot(p, s);
    float4 xc;
    if (!MIXED && !p.frame) {
        xc = make_float4(self.x, self.y, self.z, 0.0f);
    } else {
        const int3 cs = slot_cell(p, cp, g, key_sorted, p.cell_sorted, s);
        if (MIXED)
            xc = make_float4(self.x, self.y, self.z, pack_cell(cp, cs.x, cs.y, cs.z));
        else  // scene frame: back to the offset from the step's cell
            xc = make_float4(__fsub_rn(self.x, __fmul_rn((float)cs.x, p.cell)),
                             __fsub_rn(self.y, __fmul_rn((float)cs.y, p.cell)),
                             __fsub_rn(self.z, __fmul_rn((float)cs.z, p.cell)), pack_cell(cp, cs.x, cs.y, cs.z));
    }
    x_out[s] = xc;
    if (xs_next) {
        int k;
        if (MIXED || p.frame)
            k = predict_one<true>(p, cp, g, xc, vc, s, xs_next, key, rank, count, cellk);
        else
            k = predict_one<false>(p, cp, g, xc, vc, s, xs_next, key, rank, count, cellk);
        add_tile(tiles, tile_count, k, s, p.n);
    }
}

template <int F, int U, int B>
__global__ void __launch_bounds__(B) k_xsph(StepParams p, CellPack cp, const float4* __restrict__ xs,
                                            const float4* __restrict__ v_in,
                                            const int* __restrict__ nbr, const int* __restrict__ cnt,
                                            const int* __restrict__ key_sorted,
                                            float4* __restrict__ x_out, float4* __restrict__ v_out,
                                            float4* __restrict__ xs_next, int* __restrict__ key,
                                            int* __restrict__ rank, int* __restrict__ count,
                                            int* __restrict__ cellk, int* __restrict__ tile_count) {
    xsph_commit<F, U>(p, cp, xs, v_in, nbr, cnt, key_sorted, x_out, v_out, xs_next, key, rank, count, cellk,
                      tile_count);
}

// Compact lists (F = 8, 24, 40) with one gather in flight: registers capped at 32
// for every warp slot of the SM (8 bytes spilled with 16-bit records, 88 with
// 24-bit ones, none with 32-bit ones; config 3 XSPH 0.175 -> 0.141 ms at step 5,
// 0.239 -> 0.219 ms at step 100 against the best uncapped shape).  More
// gathers in flight keep k_xsph.
template <int F, int U, int B>
__global__ void __launch_bounds__(B, 2048 / B) k_xsph_compact(
    StepParams p, CellPack cp, const float4* __restrict__ xs, const float4* __restrict__ v_in,
    const int* __restrict__ nbr, const int* __restrict__ cnt, const int* __restrict__ key_sorted,
    float4* __restrict__ x_out, float4* __restrict__ v_out, float4* __restrict__ xs_next, int* __restrict__ key,
    int* __restrict__ rank, int* __restrict__ count, int* __restrict__ cellk, int* __restrict__ tile_count) {
    xsph_commit<F, U>(p, cp, xs, v_in, nbr, cnt, key_sorted, x_out, v_out, xs_next, key, rank, count, cellk,
                      tile_count);
}

// ------------------------------------------------------------- launch shape --

static inline int blocks_for(int n, int t) { return (n + t - 1) / t; }

// Kernels templated on (F, U, B) are instantiated for F in {0..3} (mixed,
// solids), U in {1, 2, 4, 8} and B in {64, 128, 256}; the tuning and the
// scene pick one (TUNE_DISPATCH expands the switch).
#define TUNE_LAUNCH(KERNEL, MIX, U_, B_, N, ST, ...)                                            \
    launch_k(KERNEL<MIX, U_, B_>, blocks_for(N, B_), B_, ST, pdl_enabled(), __VA_ARGS__)
// two particles per thread (the lambda and delta-p passes), U in {1, 2}
#define TUNE_LAUNCH_P2(KERNEL, MIX, U_, B_, N, ST, ...)                                         \
    launch_k(KERNEL<MIX, U_, B_, 2>, blocks_for(N, 2 * B_), B_, ST, pdl_enabled(), __VA_ARGS__)
#define TUNE_BLOCKS_P2(KERNEL, MIX, U_, tu, N, ST, ...)                                         \
    do {                                                                                        \
        if (tu.block <= 64)                                                                     \
            TUNE_LAUNCH_P2(KERNEL, MIX, U_, 64, N, ST, __VA_ARGS__);                            \
        else if (tu.block <= 128)                                                               \
            TUNE_LAUNCH_P2(KERNEL, MIX, U_, 128, N, ST, __VA_ARGS__);                           \
        else                                                                                    \
            TUNE_LAUNCH_P2(KERNEL, MIX, U_, 256, N, ST, __VA_ARGS__);                           \
    } while (0)
#define TUNE_CASE_P2(KERNEL, MIX, tu, N, ST, ...)                                               \
    do {                                                                                        \
        if (tu.unroll <= 1)                                                                     \
            TUNE_BLOCKS_P2(KERNEL, MIX, 1, tu, N, ST, __VA_ARGS__);                             \
        else                                                                                    \
            TUNE_BLOCKS_P2(KERNEL, MIX, 2, tu, N, ST, __VA_ARGS__);                             \
    } while (0)
#define TUNE_DISPATCH_PPT(KERNEL, fcode, tu, N, ST, ...)                                        \
    do {                                                                                        \
        if (tu.ppt != 2) {                                                                      \
            TUNE_DISPATCH(KERNEL, fcode, tu, N, ST, __VA_ARGS__);                               \
            break;                                                                              \
        }                                                                                       \
        switch (fcode) {                                                                        \
            case 0: TUNE_CASE_P2(KERNEL, 0, tu, N, ST, __VA_ARGS__); break;                     \
            case 1: TUNE_CASE_P2(KERNEL, 1, tu, N, ST, __VA_ARGS__); break;                     \
            case 2: TUNE_CASE_P2(KERNEL, 2, tu, N, ST, __VA_ARGS__); break;                     \
            default: TUNE_CASE_P2(KERNEL, 3, tu, N, ST, __VA_ARGS__); break;                    \
        }                                                                                       \
    } while (0)
#define TUNE_BLOCKS(KERNEL, MIX, U_, tu, N, ST, ...)                                            \
    do {                                                                                        \
        if (tu.block <= 64)                                                                     \
            TUNE_LAUNCH(KERNEL, MIX, U_, 64, N, ST, __VA_ARGS__);                               \
        else if (tu.block <= 128)                                                               \
            TUNE_LAUNCH(KERNEL, MIX, U_, 128, N, ST, __VA_ARGS__);                              \
        else                                                                                    \
            TUNE_LAUNCH(KERNEL, MIX, U_, 256, N, ST, __VA_ARGS__);                              \
    } while (0)
#define TUNE_CASE(KERNEL, MIX, tu, N, ST, ...)                                                  \
    do {                                                                                        \
        if (tu.unroll <= 1)                                                                     \
            TUNE_BLOCKS(KERNEL, MIX, 1, tu, N, ST, __VA_ARGS__);                                \
        else if (tu.unroll == 2)                                                                \
            TUNE_BLOCKS(KERNEL, MIX, 2, tu, N, ST, __VA_ARGS__);                                \
        else if (tu.unroll == 4)                                                                \
            TUNE_BLOCKS(KERNEL, MIX, 4, tu, N, ST, __VA_ARGS__);                                \
        else                                                                                    \
            TUNE_BLOCKS(KERNEL, MIX, 8, tu, N, ST, __VA_ARGS__);                                \
    } while (0)
// fcode: bit 0 mixed (cell-relative pair offsets), bit 1 static particles,
// bit 2 (the lambda pass only) the scene frame's compensated sums, bit 3
// compact lists (with bit 2 at most), bit 4 their 24-bit and bit 5 their 32-bit
// records
#define TUNE_DISPATCH(KERNEL, fcode, tu, N, ST, ...)                                            \
    do {                                                                                        \
        switch (fcode) {                                                                        \
            case 0: TUNE_CASE(KERNEL, 0, tu, N, ST, __VA_ARGS__); break;                        \
            case 1: TUNE_CASE(KERNEL, 1, tu, N, ST, __VA_ARGS__); break;                        \
            case 2: TUNE_CASE(KERNEL, 2, tu, N, ST, __VA_ARGS__); break;                        \
            default: TUNE_CASE(KERNEL, 3, tu, N, ST, __VA_ARGS__); break;                       \
        }                                                                                       \
    } while (0)
#define TUNE_DISPATCH_FRAME(KERNEL, fcode, tu, N, ST, ...)                                      \
    do {                                                                                        \
        if (fcode == 4) TUNE_CASE(KERNEL, 4, tu, N, ST, __VA_ARGS__);                           \
        else if (fcode == 6) TUNE_CASE(KERNEL, 6, tu, N, ST, __VA_ARGS__);                      \
        else TUNE_DISPATCH(KERNEL, fcode, tu, N, ST, __VA_ARGS__);                              \
    } while (0)


}  // namespace lgb
