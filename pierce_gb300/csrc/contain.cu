// Parity of first vertices by object pairs, and containment by candidate
// pairs (mesh_intersection_anyhit.cu:46-240, mesh_containment.cu:179-293).
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "grid.cuh"
#include "hash.cuh"
#include "predicates.cuh"

namespace pgpu {

// ---- parity by object pairs ----------------------------------------------------
// A warp per source object: the lanes take the entries of the object's grid
// cell (candidate targets: box contains the first vertex in x and y and
// reaches above it), then for each candidate the lanes take its 32-triangle
// chunk boxes and the triangles of the chunks the +Z ray's column meets, and
// count the crossings.  A source's targets each come up once, so an odd pair
// goes straight to where it is wanted -- the join's pair set, or a list --
// and no parity table (12 MB per direction at 50,000 objects) is filled,
// scanned and read back.  Both directions in one launch.  Bound by the chain
// of dependent loads per source (cell, entries, chunk boxes, indices,
// vertices; 17 % of issue slots used).  2 x 50,000 rays took 0.60 ms; with the
// candidates found lane by lane and four chunks' loads in flight 0.38 (10
// blocks of 128 per SM, 48 registers; 8 blocks 0.40, 6 0.47, 12 0.37), with the
// objects' boxes and ranges in the grid's entries 0.355, with 64 chunks' boxes
// and kAhead chunks' triangles in flight 0.335.
struct ParitySide {
    DevDataset src;      // first vertices, partitions
    ColumnGrid grid;     // the target's column grid
    DevDataset tgt;      // the target's triangles (verts, idx, obj_range)
    int64_t lo, hi;      // source objects [lo, hi) cast rays (a shard)
    int swap;            // keys (target, source)
};
struct ParityObjParams {
    ParitySide side[2];
    int64_t rays0;       // of the launch's rays, those of side 0 come first
    int64_t rays;
    PairSet set;         // odd pairs into the set ...
    uint64_t* out;       // ... or (no table) appended to a list
    unsigned long long* out_count;
    uint64_t out_cap;
    uint32_t* err;
    DevCounters* ctr;
    // k_parity_objects<true> (diagnostics, side 0) writes, instead of pairs,
    // per source object s: the targets its ray crosses an odd number of times
    // with their crossing counts (slots s * track_k ..., in candidate order),
    // the number of targets it crosses at all, and the odd targets that found
    // no slot
    int32_t track_k;
    int32_t* track_ids;
    uint32_t* track_hits;
    uint32_t* track_crossed;
    uint32_t* track_overflow;
};

__device__ __forceinline__ float3 vertex(const DevDataset& d, uint32_t i) {
    return make_float3(__ldg(d.verts + 3 * (size_t)i), __ldg(d.verts + 3 * (size_t)i + 1),
                       __ldg(d.verts + 3 * (size_t)i + 2));
}
__device__ __forceinline__ float3 tri_vertex(const DevDataset& d, uint32_t tri, int k) {
    return vertex(d, __ldg(d.idx + 3 * (size_t)tri + k));
}
// out of line: one or two lanes run it per chunk, and its registers would
// halve the warps in flight
__device__ __noinline__ bool zray_cross_call(float3 p, float3 a, float3 b, float3 c, PredCounters& pc) {
    return zray_cross(p, a, b, c, pc);
}

constexpr int kAhead = 6;
template <bool TRACK>
__global__ void __launch_bounds__(128, 10) k_parity_objects(ParityObjParams P) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    uint32_t n_tests = 0, n_rays = 0, probes = 0;
    PredCounters pc{0, 0};
    for (int64_t ray = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); ray < P.rays; ray += warps) {
        const ParitySide& S = P.side[ray < P.rays0 ? 0 : 1];
        const int64_t s = S.lo + (ray < P.rays0 ? ray : ray - P.rays0);
        const float4 fv = __ldg(S.src.first_vertex + s);
        if (fv.w != 0.0f) continue;  // object without triangles (warp-uniform)
        ++n_rays;
        const float3 p = make_float3(fv.x, fv.y, fv.z);
        const DevDataset& T = S.tgt;
        uint32_t n_crossed = 0, n_odd = 0;  // TRACK: lane 0's tallies of this source
        int cx, cx1, cy, cy1;
        grid_cell_range(S.grid.bounds, S.grid.nx, S.grid.ny, p.x, p.x, 0, cx, cx1);
        grid_cell_range(S.grid.bounds, S.grid.nx, S.grid.ny, p.y, p.y, 1, cy, cy1);
        const int cell = cy * S.grid.nx + cx;
        const int32_t e0 = __ldg(S.grid.offsets + cell), e1 = __ldg(S.grid.offsets + cell + 1);
        const int32_t part = T.obj_part ? __ldg(S.src.obj_part + s) : 0;
        for (int32_t base = e0; base < e1; base += 32) {
            int4 cand = make_int4(0, -1, 0, 0);  // (hi.z bits), object, first triangle, count
            if (base + lane < e1) {
                const float4* e = reinterpret_cast<const float4*>(S.grid.entries + base + lane);
                const float4 xy = __ldg(e);
                cand = __ldg(reinterpret_cast<const int4*>(e + 1));
                if (!(xy.x <= p.x && p.x <= xy.y && xy.z <= p.y && p.y <= xy.w && __int_as_float(cand.x) >= p.z &&
                      (!T.obj_part || __ldg(T.obj_part + cand.y) == part)))
                    cand.y = -1;
            }
            for (unsigned left = __ballot_sync(0xFFFFFFFFu, cand.y >= 0); left; left &= left - 1) {
                const int from = __ffs(left) - 1;
                const int32_t t = __shfl_sync(0xFFFFFFFFu, cand.y, from);
                const int2 r = make_int2(__shfl_sync(0xFFFFFFFFu, cand.z, from), __shfl_sync(0xFFFFFFFFu, cand.w, from));
                const int64_t end = (int64_t)r.x + r.y, c_last = (end - 1) / 32;
                uint32_t crossings = 0;  // this lane's
                for (int64_t c0 = (int64_t)r.x / 32; c0 <= c_last; c0 += 64) {
                    // 64 chunks' boxes in flight together
                    bool hit[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int64_t c = c0 + 32 * h + lane;
                        hit[h] = false;
                        if (c <= c_last) {
                            const float* bb = T.tri_chunk_box + 6 * c;
                            hit[h] = __ldg(bb) <= p.x && p.x <= __ldg(bb + 3) && __ldg(bb + 1) <= p.y &&
                                     p.y <= __ldg(bb + 4) && __ldg(bb + 5) >= p.z;
                        }
                    }
                    const unsigned m_hi = __ballot_sync(0xFFFFFFFFu, hit[1]);
                    for (unsigned long long m = ((unsigned long long)m_hi << 32) | __ballot_sync(0xFFFFFFFFu, hit[0]); m;) {
                        // the triangles of up to kAhead chunks, their loads in
                        // flight together; those whose box the ray meets (one
                        // or two lanes per chunk) are tested after, together
                        int64_t tri[kAhead];
                        uint32_t id[kAhead][3];
                        unsigned pass = 0;
#pragma unroll
                        for (int q = 0; q < kAhead; ++q) {
                            tri[q] = m ? (c0 + __ffsll((long long)m) - 1) * 32 + lane : -1;
                            m &= m - 1;
                            if (tri[q] < r.x || tri[q] >= end) tri[q] = -1;
                        }
#pragma unroll
                        for (int q = 0; q < kAhead; ++q)
                            if (tri[q] >= 0)
                                for (int v = 0; v < 3; ++v) id[q][v] = __ldg(T.idx + 3 * tri[q] + v);
#pragma unroll
                        for (int q = 0; q < kAhead; ++q)
                            if (tri[q] >= 0) {
                                const float3 a = vertex(T, id[q][0]), b = vertex(T, id[q][1]), d = vertex(T, id[q][2]);
                                if (!(fminf(a.x, fminf(b.x, d.x)) > p.x || fmaxf(a.x, fmaxf(b.x, d.x)) < p.x ||
                                      fminf(a.y, fminf(b.y, d.y)) > p.y || fmaxf(a.y, fmaxf(b.y, d.y)) < p.y ||
                                      fmaxf(a.z, fmaxf(b.z, d.z)) < p.z))
                                    pass |= 1u << q;
                            }
                        for (; pass; pass &= pass - 1) {
                            const int q = __ffs(pass) - 1;
                            int64_t t3 = tri[0];
#pragma unroll
                            for (int k = 1; k < kAhead; ++k)
                                if (q == k) t3 = tri[k];
                            ++n_tests;
                            if (zray_cross_call(p, tri_vertex(T, (uint32_t)t3, 0), tri_vertex(T, (uint32_t)t3, 1),
                                                tri_vertex(T, (uint32_t)t3, 2), pc))
                                ++crossings;
                        }
                        __syncwarp();
                    }
                }
                const uint32_t hits = __reduce_add_sync(0xFFFFFFFFu, crossings);
                if constexpr (TRACK) {
                    if (hits && lane == 0) {
                        ++n_crossed;
                        if (hits & 1u) {
                            if (n_odd < (uint32_t)P.track_k) {
                                const int64_t at = s * (int64_t)P.track_k + n_odd;
                                P.track_ids[at] = t;
                                P.track_hits[at] = hits;
                            }
                            ++n_odd;
                        }
                    }
                } else if ((hits & 1u) && lane == 0) {
                    const uint64_t key = S.swap ? pack_key(t, (int32_t)s) : pack_key((int32_t)s, t);
                    if (P.set.table) {
                        hash_add(P.set, key, P.err, probes);
                    } else {
                        const unsigned long long pos = atomicAdd(P.out_count, 1ull);
                        if (pos < P.out_cap) P.out[pos] = key;
                    }
                }
            }
        }
        if constexpr (TRACK) {
            if (lane == 0) {
                P.track_crossed[s] = n_crossed;
                P.track_overflow[s] = n_odd > (uint32_t)P.track_k ? n_odd - (uint32_t)P.track_k : 0u;
            }
        }
    }
    // per-lane test and ambiguity counts; rays once per warp
    flush_counter(&P.ctr->tri_tests, n_tests);
    flush_counter(&P.ctr->fp32_ambiguous, pc.fp32_ambiguous);
    flush_counter(&P.ctr->fp64_ambiguous, pc.fp64_ambiguous);
    flush_counter(&P.ctr->parity_rays, lane == 0 ? n_rays : 0u);
}

static unsigned parity_blocks(pierce_ctx* ctx, int64_t rays) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((rays + 3) / 4, (int64_t)ctx->sm_count * 32));
}

int launch_parity_objects(pierce_ctx* ctx, const ParityRays* side0, const ParityRays* side1, const PairSet& set,
                          uint64_t* out, unsigned long long* out_count, uint64_t out_cap) {
    ParityObjParams P{};
    const ParityRays* sides[2] = {side0, side1};
    for (int d = 0; d < 2; ++d) {
        if (!sides[d] || !sides[d]->tgt.obj_range || sides[d]->grid.nx <= 0) continue;
        ParitySide& S = P.side[d];
        S.src = sides[d]->src;
        S.grid = sides[d]->grid;
        S.tgt = sides[d]->tgt;
        S.swap = sides[d]->swap;
        S.lo = std::max<int64_t>(sides[d]->lo, 0);
        S.hi = std::min<int64_t>(sides[d]->hi, S.src.num_objects);
        const int64_t n = std::max<int64_t>(S.hi - S.lo, 0);
        if (d == 0) P.rays0 = n;
        P.rays += n;
    }
    if (P.rays == 0) return PIERCE_OK;
    P.set = set;
    P.out = out;
    P.out_count = out_count;
    P.out_cap = out_cap;
    P.err = ctx->d_err;
    P.ctr = ctx->d_counters;
    k_parity_objects<false><<<parity_blocks(ctx, P.rays), 128, 0, ctx->stream>>>(P);
    ctx->launches += 1;
    return check_cuda(cudaGetLastError(), "parity (object pairs) kernel");
}

// Parity-ray diagnostics of src's objects against tgt over tgt's column
// grid: ids[src.num_objects * k] (preset to -1 by the caller), hits (same
// shape), crossed and overflow (src.num_objects each; entries of objects
// without triangles are left as they are).
int launch_parity_tracking(pierce_ctx* ctx, const DevDataset& src, const DevDataset& tgt, const ColumnGrid& grid,
                           int32_t k, int32_t* ids, uint32_t* hits, uint32_t* crossed, uint32_t* overflow) {
    if (src.num_objects <= 0 || !tgt.obj_range || grid.nx <= 0) return PIERCE_OK;
    ParityObjParams P{};
    P.side[0].src = src;
    P.side[0].grid = grid;
    P.side[0].tgt = tgt;
    P.side[0].hi = src.num_objects;
    P.rays0 = P.rays = src.num_objects;
    P.err = ctx->d_err;
    P.ctr = ctx->d_counters;
    P.track_k = k;
    P.track_ids = ids;
    P.track_hits = hits;
    P.track_crossed = crossed;
    P.track_overflow = overflow;
    k_parity_objects<true><<<parity_blocks(ctx, P.rays), 128, 0, ctx->stream>>>(P);
    ctx->launches += 1;
    return check_cuda(cudaGetLastError(), "parity tracking kernel");
}

// The exact closed triangle-triangle predicate, float32 first.
__device__ __noinline__ bool tri_tri_meet(const float3& a0, const float3& a1, const float3& a2, const float3& b0,
                                             const float3& b1, const float3& b2, PredCounters& pc) {
    const int cls = tri_tri_fp32_class(a0, a1, a2, b0, b1, b2);
    if (cls != SEG_AMBIGUOUS) return cls == SEG_HIT;
    pc.fp32_ambiguous++;
    return tri_tri_exact(a0, a1, a2, b0, b1, b2, pc);
}

// ---- containment by candidate pairs -------------------------------------------
// Containment is parity(B in A) \ overlap (pierce_containment_main.cpp:
// 385-550), so only the odd-parity pairs (a, b) need an overlap answer.
// k_containment_warps answers the ordinary ones, a warp each; the others go
// to k_containment_pairs, a block of kPairThreads each, so that one large
// pair does not hold a lone warp for the whole launch.  A block lists the triangles of a
// (those of a's 32-triangle chunks whose boxes meet, read first) whose boxes
// meet the intersection of the two object boxes (a patch of a's
// surface; the vertices of up to kPairVerts of them are kept in shared
// memory), shrinks the box to that patch's box, and streams b's triangles
// past them, one per thread (a triangle whose 32-triangle chunk box misses
// the patch is skipped unread), each tested against the listed triangles whose
// boxes meet its own with the exact closed triangle-triangle predicate.  The pair is a containment pair when none meets;
// a b deep inside a lists nothing and costs one pass over a's triangles.  A
// patch larger than kPairList is read from a's range in place.  A pair whose
// objects hold more than kPairScanMax triangles together, or whose unlisted
// patch would cost more than kPairStreamMax triangle pairs, is counted in
// *fallback and the join takes the culling pipeline instead.
constexpr int kPairThreads = 256;
constexpr int kPairList = 1024;
constexpr int kPairVerts = 512;
constexpr int kPairChunkList = 512;  // listed chunks of the container (more: its whole range)
constexpr int kPairSeg = 16;           // listed triangles with one box together
constexpr int kPairScanMax = 1 << 16;
constexpr int64_t kPairStreamMax = 1 << 22;

struct ContainParams {
    const uint64_t* pairs;                // odd-parity pairs (a << 32 | b) ...
    const unsigned long long* n_pairs;    // ... and their number
    uint64_t pairs_cap;
    uint64_t* big;                        // pairs left for the block kernel (as many as pairs)
    unsigned long long* n_big;
    DevDataset a, b;  // vertices, indices, object ranges and boxes
    uint64_t* out;
    unsigned long long* count;
    uint64_t cap;
    unsigned long long* fallback;
    DevCounters* ctr;
};

__device__ __forceinline__ bool tri_box_meets(const float3& p, const float3& q, const float3& r, const float3& lo,
                                              const float3& hi) {
    return box_overlap(fminf(p.x, fminf(q.x, r.x)), fmaxf(p.x, fmaxf(q.x, r.x)), fminf(p.y, fminf(q.y, r.y)),
                       fmaxf(p.y, fmaxf(q.y, r.y)), fminf(p.z, fminf(q.z, r.z)), fmaxf(p.z, fmaxf(q.z, r.z)), lo, hi);
}

// Box over the block's threads, each bringing [lo, hi].
__device__ __forceinline__ void block_box(float3& lo, float3& hi, float (*red)[6]) {
    for (int off = 16; off; off >>= 1) {
        lo.x = fminf(lo.x, __shfl_xor_sync(0xFFFFFFFFu, lo.x, off));
        lo.y = fminf(lo.y, __shfl_xor_sync(0xFFFFFFFFu, lo.y, off));
        lo.z = fminf(lo.z, __shfl_xor_sync(0xFFFFFFFFu, lo.z, off));
        hi.x = fmaxf(hi.x, __shfl_xor_sync(0xFFFFFFFFu, hi.x, off));
        hi.y = fmaxf(hi.y, __shfl_xor_sync(0xFFFFFFFFu, hi.y, off));
        hi.z = fmaxf(hi.z, __shfl_xor_sync(0xFFFFFFFFu, hi.z, off));
    }
    if ((threadIdx.x & 31) == 0) {
        float* r = red[threadIdx.x >> 5];
        r[0] = lo.x; r[1] = lo.y; r[2] = lo.z;
        r[3] = hi.x; r[4] = hi.y; r[5] = hi.z;
    }
    __syncthreads();
    for (int k = 0; k < kPairThreads / 32; ++k) {
        const float* r = red[k];
        lo = make_float3(fminf(lo.x, r[0]), fminf(lo.y, r[1]), fminf(lo.z, r[2]));
        hi = make_float3(fmaxf(hi.x, r[3]), fmaxf(hi.y, r[4]), fmaxf(hi.z, r[5]));
    }
    __syncthreads();
}

// Position of this thread's flag among the block's set flags, after `base`
// (warp ballots; per-warp counts in s_warp), and the block's total.
__device__ __forceinline__ int block_compact(bool flag, int base, int* s_warp) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned m = __ballot_sync(0xFFFFFFFFu, flag);
    if (lane == 0) s_warp[w] = __popc(m);
    __syncthreads();
    int before = base;
    for (int q = 0; q < w; ++q) before += s_warp[q];
    return before + __popc(m & ((1u << lane) - 1u));
}
__device__ __forceinline__ int block_total(const int* s_warp) {
    int total = 0;
    for (int q = 0; q < kPairThreads / 32; ++q) total += s_warp[q];
    return total;
}

__global__ void __launch_bounds__(kPairThreads) k_containment_pairs(ContainParams P) {
    __shared__ uint32_t s_list[kPairList];
    __shared__ uint32_t s_chunk[kPairChunkList];
    __shared__ float4 s_tri[kPairVerts][3];
    __shared__ float s_seg[kPairList / kPairSeg][6];
    __shared__ int s_warp[kPairThreads / 32];
    __shared__ float s_red[kPairThreads / 32][6];
    const int tid = threadIdx.x;
    PredCounters pc{0, 0};
    uint32_t tests = 0;
    const int64_t n = (int64_t)min(*P.n_big, (unsigned long long)P.pairs_cap);
    for (int64_t q = blockIdx.x; q < n; q += gridDim.x) {
        {
            const uint64_t key = P.big[q];
            const uint32_t a = (uint32_t)(key >> 32), b = (uint32_t)key;
            const float* ba = P.a.obj_box + 6 * (size_t)a;
            const float* bb = P.b.obj_box + 6 * (size_t)b;
            float3 lo = make_float3(fmaxf(__ldg(ba), __ldg(bb)), fmaxf(__ldg(ba + 1), __ldg(bb + 1)),
                                    fmaxf(__ldg(ba + 2), __ldg(bb + 2)));
            float3 hi = make_float3(fminf(__ldg(ba + 3), __ldg(bb + 3)), fminf(__ldg(ba + 4), __ldg(bb + 4)),
                                    fminf(__ldg(ba + 5), __ldg(bb + 5)));
            bool meets = false, undecided = false;
            if (lo.x <= hi.x && lo.y <= hi.y && lo.z <= hi.z) {
                const int2 ra = __ldg(P.a.obj_range + a), rb = __ldg(P.b.obj_range + b);
                if ((int64_t)ra.y + rb.y > kPairScanMax) {
                    undecided = true;
                } else {
                    // a's 32-triangle chunks whose boxes meet the common box, then
                    // the triangles of those chunks that do: the list (block-wide
                    // compaction) and the patch box
                    const int c0 = ra.x >> 5, c1 = (ra.x + ra.y - 1) >> 5;
                    int nmc = 0;
                    for (int base = c0; base <= c1; base += kPairThreads) {
                        const int c = base + tid;
                        bool meet = true;  // no chunk boxes: every chunk
                        if (c > c1) meet = false;
                        else if (P.a.tri_chunk_box) {
                            const float* cb = P.a.tri_chunk_box + 6 * (size_t)c;
                            meet = box_overlap(__ldg(cb), __ldg(cb + 3), __ldg(cb + 1), __ldg(cb + 4), __ldg(cb + 2),
                                               __ldg(cb + 5), lo, hi);
                        }
                        const int pos = block_compact(meet, nmc, s_warp);
                        if (meet && pos < kPairChunkList) s_chunk[pos] = (uint32_t)c;
                        nmc += block_total(s_warp);
                        __syncthreads();
                    }
                    int na = 0;
                    float3 plo = make_float3(3.4e38f, 3.4e38f, 3.4e38f), phi = make_float3(-3.4e38f, -3.4e38f, -3.4e38f);
                    const bool by_chunks = nmc <= kPairChunkList;
                    const int slots = by_chunks ? 32 * nmc : ra.y;
                    for (int base = 0; base < slots; base += kPairThreads) {
                        const int k = base + tid;
                        bool meet = false;
                        uint32_t t = 0;
                        if (k < slots) {
                            const int tt = by_chunks ? (int)(s_chunk[k >> 5] << 5) + (k & 31) : ra.x + k;
                            if (tt >= ra.x && tt < ra.x + ra.y) {
                                t = (uint32_t)tt;
                                const float3 v0 = tri_vertex(P.a, t, 0), v1 = tri_vertex(P.a, t, 1),
                                             v2 = tri_vertex(P.a, t, 2);
                                meet = tri_box_meets(v0, v1, v2, lo, hi);
                                if (meet) {
                                    plo = make_float3(fminf(plo.x, fminf(v0.x, fminf(v1.x, v2.x))),
                                                      fminf(plo.y, fminf(v0.y, fminf(v1.y, v2.y))),
                                                      fminf(plo.z, fminf(v0.z, fminf(v1.z, v2.z))));
                                    phi = make_float3(fmaxf(phi.x, fmaxf(v0.x, fmaxf(v1.x, v2.x))),
                                                      fmaxf(phi.y, fmaxf(v0.y, fmaxf(v1.y, v2.y))),
                                                      fmaxf(phi.z, fmaxf(v0.z, fmaxf(v1.z, v2.z))));
                                }
                            }
                        }
                        const int pos = block_compact(meet, na, s_warp);
                        if (meet && pos < kPairList) s_list[pos] = t;
                        na += block_total(s_warp);
                        __syncthreads();
                    }
                    block_box(plo, phi, s_red);
                    const bool listed = na <= kPairList;
                    const bool cached = na <= kPairVerts;
                    if (listed) {
                        const int segs = (na + kPairSeg - 1) / kPairSeg;
                        for (int g = tid; g < segs; g += kPairThreads) {
                            float3 slo = make_float3(3.4e38f, 3.4e38f, 3.4e38f), shi = make_float3(-3.4e38f, -3.4e38f, -3.4e38f);
                            for (int j = g * kPairSeg; j < min(g * kPairSeg + kPairSeg, na); ++j)
                                for (int v = 0; v < 3; ++v) {
                                    const float3 x = tri_vertex(P.a, s_list[j], v);
                                    slo = make_float3(fminf(slo.x, x.x), fminf(slo.y, x.y), fminf(slo.z, x.z));
                                    shi = make_float3(fmaxf(shi.x, x.x), fmaxf(shi.y, x.y), fmaxf(shi.z, x.z));
                                }
                            float* w = s_seg[g];
                            w[0] = slo.x; w[1] = slo.y; w[2] = slo.z;
                            w[3] = shi.x; w[4] = shi.y; w[5] = shi.z;
                        }
                        if (!cached) __syncthreads();
                    }
                    if (cached) {
                        for (int k = tid; k < na; k += kPairThreads) {
                            const uint32_t t = s_list[k];
                            for (int v = 0; v < 3; ++v) {
                                const float3 x = tri_vertex(P.a, t, v);
                                s_tri[k][v] = make_float4(x.x, x.y, x.z, 0.0f);
                            }
                        }
                        __syncthreads();
                    }
                    if (!listed && (int64_t)ra.y * rb.y > kPairStreamMax) {
                        undecided = true;
                    } else if (na > 0) {
                        lo = make_float3(fmaxf(lo.x, plo.x), fmaxf(lo.y, plo.y), fmaxf(lo.z, plo.z));
                        hi = make_float3(fminf(hi.x, phi.x), fminf(hi.y, phi.y), fminf(hi.z, phi.z));
                        const int nj = listed ? na : ra.y;
                        // b's triangles, one per thread, against the patch
                        for (int base = 0; base < rb.y && !meets; base += kPairThreads) {
                            const int k = base + tid;
                            bool hit = false;
                            bool near = k < rb.y;
                            if (near && P.b.tri_chunk_box) {  // the triangle's chunk box first
                                const float* cb = P.b.tri_chunk_box + 6 * (size_t)((rb.x + k) >> 5);
                                near = box_overlap(__ldg(cb), __ldg(cb + 3), __ldg(cb + 1), __ldg(cb + 4), __ldg(cb + 2),
                                                   __ldg(cb + 5), lo, hi);
                            }
                            float3 b0{}, b1{}, b2{}, blo{}, bhi{};
                            if (near) {
                                const uint32_t tb = (uint32_t)(rb.x + k);
                                b0 = tri_vertex(P.b, tb, 0);
                                b1 = tri_vertex(P.b, tb, 1);
                                b2 = tri_vertex(P.b, tb, 2);
                                blo = make_float3(fminf(b0.x, fminf(b1.x, b2.x)), fminf(b0.y, fminf(b1.y, b2.y)),
                                                  fminf(b0.z, fminf(b1.z, b2.z)));
                                bhi = make_float3(fmaxf(b0.x, fmaxf(b1.x, b2.x)), fmaxf(b0.y, fmaxf(b1.y, b2.y)),
                                                  fmaxf(b0.z, fmaxf(b1.z, b2.z)));
                                near = box_overlap(blo.x, bhi.x, blo.y, bhi.y, blo.z, bhi.z, lo, hi);
                            }
                            if (!__syncthreads_or(near)) continue;
                            // 64 of a's triangles at a time, by the boxes of
                            // 16 (of a chunk's 32 in place): one hit ends the pair
                            for (int j0 = 0; j0 < nj && !meets; j0 += 64) {
                                for (int s0 = j0; near && s0 < min(j0 + 64, nj) && !hit;) {
                                    int s1 = min(s0 + kPairSeg, nj);
                                    bool seg;
                                    if (listed) {
                                        const float* w = s_seg[s0 / kPairSeg];
                                        seg = box_overlap(w[0], w[3], w[1], w[4], w[2], w[5], blo, bhi);
                                    } else {
                                        // up to the end of the triangle's chunk
                                        s1 = min(min((((ra.x + s0) >> 5) + 1) * 32 - ra.x, j0 + 64), nj);
                                        const float* w = P.a.tri_chunk_box + 6 * (size_t)((ra.x + s0) >> 5);
                                        seg = box_overlap(__ldg(w), __ldg(w + 3), __ldg(w + 1), __ldg(w + 4), __ldg(w + 2),
                                                          __ldg(w + 5), blo, bhi);
                                    }
                                    for (int j = s0; seg && j < s1 && !hit; ++j) {
                                        float3 a0, a1, a2;
                                        if (cached) {
                                            const float4 x0 = s_tri[j][0], x1 = s_tri[j][1], x2 = s_tri[j][2];
                                            a0 = make_float3(x0.x, x0.y, x0.z);
                                            a1 = make_float3(x1.x, x1.y, x1.z);
                                            a2 = make_float3(x2.x, x2.y, x2.z);
                                        } else {
                                            const uint32_t ta = listed ? s_list[j] : (uint32_t)(ra.x + j);
                                            a0 = tri_vertex(P.a, ta, 0);
                                            a1 = tri_vertex(P.a, ta, 1);
                                            a2 = tri_vertex(P.a, ta, 2);
                                        }
                                        if (!tri_box_meets(a0, a1, a2, blo, bhi)) continue;
                                        ++tests;
                                        hit = tri_tri_meet(a0, a1, a2, b0, b1, b2, pc);
                                    }
                                    s0 = s1;
                                }
                                meets = __syncthreads_or(hit) != 0;
                            }
                        }
                    }
                }
            }
            if (tid == 0) {
                if (undecided) {
                    atomicAdd(P.fallback, 1ull);
                } else if (!meets) {
                    const unsigned long long pos = atomicAdd(P.count, 1ull);
                    if (pos < P.cap) P.out[pos] = key;
                }
            }
            __syncthreads();
        }
    }
    flush_counter(&P.ctr->tri_tests, tests);
    flush_counter(&P.ctr->fp32_ambiguous, pc.fp32_ambiguous);
    flush_counter(&P.ctr->fp64_ambiguous, pc.fp64_ambiguous);
}


// An ordinary pair, a warp each: the lanes take a's 32-triangle chunk boxes,
// then the triangles of the chunks that meet the common box of the two
// objects; those that meet it too (a patch of a's surface) are kept in shared
// memory, the box shrinks to theirs, and b's chunks and triangles are taken
// the same way and tested against the patch.  A b deep inside a ends after
// a's chunk boxes.  Pairs of more than kWarpTris triangles, with a patch of
// more than kWarpPatch or more than kWarpWork boxes to compare go to the
// block kernel: a lone warp would hold the launch up (kWarpWork 1,024: 63 us
// here and 182 in the block kernel on the 12,000 odd pairs of 2 x 50,000
// ellipsoids; 2,048: 60 and 182; 4,096: 74 and 177; 16,384: 133 and 187; all
// pairs in blocks that read each patch triangle's vertices for every triangle
// of b: 605).
constexpr int kWarpTris = 8192, kWarpPatch = 64, kWarpNear = 512;
constexpr int kWarpWork = 2048;  // patch triangles x b triangles near them
struct WarpPatch {
    float tri[kWarpPatch][9];
    float box[kWarpPatch][6];
    uint32_t near[kWarpNear];  // b triangles that meet the patch's box
};
__global__ void __launch_bounds__(128, 6) k_containment_warps(ContainParams P) {
    __shared__ WarpPatch patches[4];
    WarpPatch& W = patches[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const int64_t n = (int64_t)min(*P.n_pairs, (unsigned long long)P.pairs_cap);
    PredCounters pc{0, 0};
    uint32_t tests = 0;
    for (int64_t q = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5); q < n; q += (int64_t)gridDim.x * 4) {
        const uint64_t key = P.pairs[q];
        const uint32_t a = (uint32_t)(key >> 32), b = (uint32_t)key;
        const float* ba = P.a.obj_box + 6 * (size_t)a;
        const float* bb = P.b.obj_box + 6 * (size_t)b;
        const int2 ra = __ldg(P.a.obj_range + a), rb = __ldg(P.b.obj_range + b);
        float3 lo = make_float3(fmaxf(__ldg(ba), __ldg(bb)), fmaxf(__ldg(ba + 1), __ldg(bb + 1)),
                                fmaxf(__ldg(ba + 2), __ldg(bb + 2)));
        float3 hi = make_float3(fminf(__ldg(ba + 3), __ldg(bb + 3)), fminf(__ldg(ba + 4), __ldg(bb + 4)),
                                fminf(__ldg(ba + 5), __ldg(bb + 5)));
        bool meets = false, big = false;
        if (lo.x <= hi.x && lo.y <= hi.y && lo.z <= hi.z) {
            big = (int64_t)ra.y + rb.y > kWarpTris;
            int na = 0;
            const int a_last = (ra.x + ra.y - 1) >> 5;
            for (int c0 = ra.x >> 5; c0 <= a_last && !big; c0 += 32) {
                bool near = false;
                if (c0 + lane <= a_last) {
                    const float* cb = P.a.tri_chunk_box + 6 * (size_t)(c0 + lane);
                    near = box_overlap(__ldg(cb), __ldg(cb + 3), __ldg(cb + 1), __ldg(cb + 4), __ldg(cb + 2),
                                       __ldg(cb + 5), lo, hi);
                }
                for (unsigned m = __ballot_sync(0xFFFFFFFFu, near); m && !big;) {
                    // two chunks at a time
                    int t[2];
                    float3 v[2][3];
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        t[k] = m ? ((c0 + __ffs(m) - 1) << 5) + lane : -1;
                        m &= m - 1;
                        if (t[k] < ra.x || t[k] >= ra.x + ra.y) t[k] = -1;
                    }
#pragma unroll
                    for (int k = 0; k < 2; ++k)
                        if (t[k] >= 0)
                            for (int d = 0; d < 3; ++d) v[k][d] = tri_vertex(P.a, (uint32_t)t[k], d);
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const bool meet = t[k] >= 0 && tri_box_meets(v[k][0], v[k][1], v[k][2], lo, hi);
                        const unsigned mm = __ballot_sync(0xFFFFFFFFu, meet);
                        const int pos = na + __popc(mm & below);
                        na += __popc(mm);
                        if (meet && pos < kWarpPatch)
                            for (int d = 0; d < 3; ++d) {
                                W.tri[pos][3 * d] = v[k][d].x;
                                W.tri[pos][3 * d + 1] = v[k][d].y;
                                W.tri[pos][3 * d + 2] = v[k][d].z;
                            }
                    }
                    big = na > kWarpPatch;
                }
            }
            __syncwarp();
            if (!big && na > 0) {
                // boxes of the patch's triangles, and the patch's box
                float3 plo = make_float3(3.4e38f, 3.4e38f, 3.4e38f), phi = make_float3(-3.4e38f, -3.4e38f, -3.4e38f);
                for (int j = lane; j < na; j += 32) {
                    const float* w = W.tri[j];
                    float* g = W.box[j];
                    for (int d = 0; d < 3; ++d) {
                        g[d] = fminf(w[d], fminf(w[3 + d], w[6 + d]));
                        g[3 + d] = fmaxf(w[d], fmaxf(w[3 + d], w[6 + d]));
                    }
                    plo = make_float3(fminf(plo.x, g[0]), fminf(plo.y, g[1]), fminf(plo.z, g[2]));
                    phi = make_float3(fmaxf(phi.x, g[3]), fmaxf(phi.y, g[4]), fmaxf(phi.z, g[5]));
                }
                for (int off = 16; off; off >>= 1) {
                    plo.x = fminf(plo.x, __shfl_xor_sync(0xFFFFFFFFu, plo.x, off));
                    plo.y = fminf(plo.y, __shfl_xor_sync(0xFFFFFFFFu, plo.y, off));
                    plo.z = fminf(plo.z, __shfl_xor_sync(0xFFFFFFFFu, plo.z, off));
                    phi.x = fmaxf(phi.x, __shfl_xor_sync(0xFFFFFFFFu, phi.x, off));
                    phi.y = fmaxf(phi.y, __shfl_xor_sync(0xFFFFFFFFu, phi.y, off));
                    phi.z = fmaxf(phi.z, __shfl_xor_sync(0xFFFFFFFFu, phi.z, off));
                }
                lo = make_float3(fmaxf(lo.x, plo.x), fmaxf(lo.y, plo.y), fmaxf(lo.z, plo.z));
                hi = make_float3(fminf(hi.x, phi.x), fminf(hi.y, phi.y), fminf(hi.z, phi.z));
                __syncwarp();
                // b's triangles that meet the patch's box
                int nn = 0;
                const int limit = min(kWarpNear, kWarpWork / na);
                const int b_last = (rb.x + rb.y - 1) >> 5;
                for (int c0 = rb.x >> 5; c0 <= b_last && !big; c0 += 32) {
                    bool near = false;
                    if (c0 + lane <= b_last) {
                        const float* cb = P.b.tri_chunk_box + 6 * (size_t)(c0 + lane);
                        near = box_overlap(__ldg(cb), __ldg(cb + 3), __ldg(cb + 1), __ldg(cb + 4), __ldg(cb + 2),
                                           __ldg(cb + 5), lo, hi);
                    }
                    for (unsigned m = __ballot_sync(0xFFFFFFFFu, near); m && !big; m &= m - 1) {
                        const int t = ((c0 + __ffs(m) - 1) << 5) + lane;
                        const bool meet = t >= rb.x && t < rb.x + rb.y &&
                                          tri_box_meets(tri_vertex(P.b, (uint32_t)t, 0), tri_vertex(P.b, (uint32_t)t, 1),
                                                        tri_vertex(P.b, (uint32_t)t, 2), lo, hi);
                        const unsigned mm = __ballot_sync(0xFFFFFFFFu, meet);
                        const int pos = nn + __popc(mm & below);
                        nn += __popc(mm);
                        if (meet && pos < limit) W.near[pos] = (uint32_t)t;
                        big = nn > limit;
                    }
                }
                __syncwarp();
                // 32 of them at a time against the patch; one hit ends the pair
                for (int n0 = 0; n0 < nn && !meets && !big; n0 += 32) {
                    const bool in = n0 + lane < nn;
                    bool hit = false;
                    float3 b0{}, b1{}, b2{}, blo{}, bhi{};
                    if (in) {
                        const uint32_t t = W.near[n0 + lane];
                        b0 = tri_vertex(P.b, t, 0);
                        b1 = tri_vertex(P.b, t, 1);
                        b2 = tri_vertex(P.b, t, 2);
                        blo = make_float3(fminf(b0.x, fminf(b1.x, b2.x)), fminf(b0.y, fminf(b1.y, b2.y)),
                                          fminf(b0.z, fminf(b1.z, b2.z)));
                        bhi = make_float3(fmaxf(b0.x, fmaxf(b1.x, b2.x)), fmaxf(b0.y, fmaxf(b1.y, b2.y)),
                                          fmaxf(b0.z, fmaxf(b1.z, b2.z)));
                    }
                    for (int j = 0; in && j < na && !hit; ++j) {
                        const float* g = W.box[j];
                        if (!box_overlap(g[0], g[3], g[1], g[4], g[2], g[5], blo, bhi)) continue;
                        const float* v = W.tri[j];
                        ++tests;
                        hit = tri_tri_meet(make_float3(v[0], v[1], v[2]), make_float3(v[3], v[4], v[5]),
                                           make_float3(v[6], v[7], v[8]), b0, b1, b2, pc);
                    }
                    meets = __any_sync(0xFFFFFFFFu, hit);
                }
                __syncwarp();
            }
        }
        if (lane == 0) {
            if (big) {
                P.big[atomicAdd(P.n_big, 1ull)] = key;
            } else if (!meets) {
                const unsigned long long pos = atomicAdd(P.count, 1ull);
                if (pos < P.cap) P.out[pos] = key;
            }
        }
        __syncwarp();
    }
    flush_counter(&P.ctr->tri_tests, tests);
    flush_counter(&P.ctr->fp32_ambiguous, pc.fp32_ambiguous);
    flush_counter(&P.ctr->fp64_ambiguous, pc.fp64_ambiguous);
}

int launch_containment_pairs(pierce_ctx* ctx, const uint64_t* pairs, const unsigned long long* n_pairs,
                             uint64_t pairs_cap, int64_t bound, uint64_t* big, unsigned long long* n_big,
                             const DevDataset& a, const DevDataset& b, uint64_t* out, unsigned long long* count,
                             uint64_t cap, unsigned long long* fallback) {
    if (!a.obj_range || !b.obj_range)
        return set_error(PIERCE_ERR_INVALID_ARGUMENT, "containment by pairs: objects must be stored contiguously");
    ContainParams P;
    P.pairs = pairs;
    P.n_pairs = n_pairs;
    P.pairs_cap = pairs_cap;
    P.big = big;
    P.n_big = n_big;
    P.a = a;
    P.b = b;
    P.out = out;
    P.count = count;
    P.cap = cap;
    P.fallback = fallback;
    P.ctr = ctx->d_counters;
    const int64_t blocks = std::min<int64_t>((bound + 3) / 4, (int64_t)ctx->sm_count * 16);
    k_containment_warps<<<(unsigned)std::max<int64_t>(blocks, 1), 128, 0, ctx->stream>>>(P);
    const int64_t big_blocks = std::min<int64_t>(bound, (int64_t)ctx->sm_count * 7);
    k_containment_pairs<<<(unsigned)std::max<int64_t>(big_blocks, 1), kPairThreads, 0, ctx->stream>>>(P);
    ctx->launches += 2;
    return check_cuda(cudaGetLastError(), "containment by pairs");
}

}  // namespace pgpu
