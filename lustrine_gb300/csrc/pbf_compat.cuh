// pbf_compat.cuh -- the reference's cell mapping and the list entries' way
// through shared memory, shared by the reference-semantics steps (fluid,
// pbf_compat.cu; sand, sand.cu).  Both are compiled with --fmad=false.
#pragma once

#include "pbf_common.cuh"

namespace lgb {

// get_cell_id (Utils.hpp:24-33): truncating division per axis; optional clamp.
__device__ __forceinline__ int cell_ref(const StepParams& p, float x, float y, float z, int* status) {
    int cx = (int)(x / p.cell);
    int cy = (int)(y / p.cell);
    int cz = (int)(z / p.cell);
    if (p.clamp_cells) {
        cx = min(max(cx, 0), p.gx - 1);
        cy = min(max(cy, 0), p.gy - 1);
        cz = min(max(cz, 0), p.gz - 1);
    }
    long long id = (long long)cy * p.gx * p.gz + (long long)cx * p.gz + cz;
    if (id < 0 || id >= p.num_cells) {
        // The reference writes past its cell table here; record it and clamp.
        cx = min(max(cx, 0), p.gx - 1);
        cy = min(max(cy, 0), p.gy - 1);
        cz = min(max(cz, 0), p.gz - 1);
        id = (long long)cy * p.gx * p.gz + (long long)cx * p.gz + cz;
        set_status(status, ST_CELL_RANGE);
    }
    return (int)id;
}

// A thread's list entries on their way to the column rows of nbr (entry k of
// particle i at k n + i): the first CAP wait in shared memory, entry k at
// [k][thread], so that a candidate costs one store and a conditional step of
// the pointer (a refused one is overwritten by the next) where a store to
// the row under a branch would run the branch for the whole warp whenever
// one lane accepts.  Entries past CAP (rare) go to their rows at once.
//
// G lanes may build one particle's list together, each a stretch of the walk:
// a lane's place in the list is known when all have finished, so entries past
// CAP are only counted, and a lane that has some walks its stretch again
// (LateEntries).
template <int CAP, int B, int G>
struct StagedList {
    int* first;  // this thread's entry 0
    int* at;     // its next entry
    int* row;    // nbr + i
    size_t n;
    int extra, max_nbrs;
    __device__ __forceinline__ StagedList(int* smem, int* nbr, const StepParams& p, int i)
        : first(smem + threadIdx.x), at(first), row(nbr + i), n((size_t)p.n), extra(0), max_nbrs(p.max_nbrs) {}
    __device__ __forceinline__ bool room(int w) const { return at <= first + (CAP - w) * B; }
    __device__ __forceinline__ void put(int e, bool in) {  // with room only
        *at = e;
        at += in ? B : 0;
    }
    __device__ __forceinline__ void push(int e) {
        if (at < first + CAP * B) {
            *at = e;
            at += B;
        } else {
            if (G == 1 && CAP + extra < max_nbrs) row[(size_t)(CAP + extra) * n] = e;
            extra++;
        }
    }
    __device__ __forceinline__ int count() const { return (int)(at - first) / B + extra; }
    // the staged entries to their rows, the list's place of the first being off
    __device__ __forceinline__ void write(int off) {
        const int m = min((int)(at - first) / B, max_nbrs - off);
        for (int k = 0; k < m; k++) row[(size_t)(off + k) * n] = first[k * B];
    }
};

// The entries of a lane's stretch from the CAP-th on, straight to their rows.
template <int CAP>
struct LateEntries {
    int* row;
    size_t n;
    int at, max_nbrs, seen;  // at: the place of the stretch's first entry
    __device__ __forceinline__ bool room(int) const { return false; }
    __device__ __forceinline__ void put(int, bool) {}
    __device__ __forceinline__ void push(int e) {
        if (seen >= CAP && at + seen < max_nbrs) row[(size_t)(at + seen) * n] = e;
        seen++;
    }
};

// The particles of slots [t0, t1) of pos within h of self, in slot order,
// entry(t) listed for each: SPAN_W positions are loaded together (past t1 too:
// the buffers are SPAN_PAD longer), then tested in order.  The squared
// distance is the reference's expression ((dx dx + dy dy) + dz dz, no
// contraction), the same bits from either particle's side.
constexpr int SPAN_W = 4;
static_assert(SPAN_W <= SPAN_PAD, "a span reads at most SPAN_PAD positions past its end");
template <class L, class E>
__device__ __forceinline__ void walk_span(const float4* __restrict__ pos, int t0, int t1, const float4& self,
                                          float h2, L& out, E&& entry) {
    const f32x2 sxy = pack2(self.x, self.y);
    for (int t = t0; t < t1; t += SPAN_W) {
        const ulonglong2* __restrict__ q = reinterpret_cast<const ulonglong2*>(pos + t);
        ulonglong2 o[SPAN_W];
        bool in[SPAN_W];
#pragma unroll
        for (int u = 0; u < SPAN_W; u++) o[u] = q[u];
        const int left = t1 - t;
#pragma unroll
        for (int u = 0; u < SPAN_W; u++) {
            const f32x2 d = sub2(sxy, o[u].x), d2 = mul2(d, d);
            const float dz = self.z - lo2(o[u].y);
            in[u] = u < left && (lo2(d2) + hi2(d2)) + dz * dz <= h2;
        }
        if (out.room(SPAN_W)) {
#pragma unroll
            for (int u = 0; u < SPAN_W; u++) out.put(entry(t + u), in[u]);
        } else {
#pragma unroll
            for (int u = 0; u < SPAN_W; u++)
                if (in[u]) out.push(entry(t + u));
        }
    }
}

}  // namespace lgb
