// Batched BFS / SSSP queries over many graphs in one persistent cooperative
// kernel (no counterpart in the reference, which runs one query per process).
//
// Every round of the kernel advances every unfinished query by one iteration:
//   pull    warps take items from the work queue, across all queries.  Sparse
//           pulls relax the out-edges of the vertices the last iteration changed
//           (items of PUSH_CHUNK listed vertices, whose out-edges are spread over
//           the lanes, and PUSH_PIECE-edge pieces of long lists); dense pulls
//           take 32 destinations, and WO_PIECE-edge pieces of the ones with more
//           in-edges: BFS the first source in the frontier, SSSP weight-ordered
//           in-edges up to the first weight that cannot lower the destination;
//           graphs without byte weights (SSSP) or with chunk ids take tiles
//           of 256 in-edges.  Changed vertices are listed as they change, and the
//           bitmap the next round writes is cleared.
//   decide  (block 0) per query: done when no mass changed, else the plain rule
//           (mass > t% of the query's edges: dense) picks the next pull; the
//           queries' item counts become one offset table, the work queue
// with a grid-wide barrier after each.  Queries on graphs whose CSRI holds chunk
// ids (beyond 2^32 in-edges) have two more phases before the pull:
//   build   the out-edge chunks of the listed vertices are marked
//           (wedge.c:63-155) and newly marked ones listed
//   prefix  (block 0) the offset table with those
// All blocks leave the loop together: the exit flag is written by block 0
// before a barrier and read by every block after it.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <pthread.h>
#include <stdlib.h>
#include <string.h>
#include <unistd.h>

#include "engine.cuh"
#include "pull.cuh"

namespace cg = cooperative_groups;

namespace wedge {

constexpr int BT = 256;                       // threads per persistent block
constexpr uint32_t BATCH_MAX_ROUNDS = 1u << 20; // iteration cap of the slowest query
constexpr uint32_t PUSH_CHUNK = 4;              // listed vertices per item
constexpr uint32_t PUSH_PIECE = 128;            // out-edges of a long list per item
constexpr uint32_t WO_GROUP = WO_MANY;          // in-edges of the longest destination a group of 32 pulls
constexpr uint32_t WO_PIECE = 512;              // in-edges per item of the longer ones
constexpr uint32_t SWEEP = 1024;                // bitmap words per clearing piece

struct BGraph {
    const uint32_t* src;
    const unsigned long long* w;
    const uint32_t* dst_id;
    const unsigned long long* dst_off;
    const uint32_t* chunk_dst0;  // [nchunks+1] compressed destination owning edge 32*c (Vne past the end)
    const uint32_t* dst_start;   // destination-start bitmap of the graph handle
    const uint8_t* w8;           // byte-wide weights, or null
    const uint32_t* wsrc;        // weight-ordered sources and weights, or null
    const uint8_t* ww8;
    const uint32_t* wo_src;      // every destination's first weight-ordered source (bit 31: its only one)
    const uint16_t* wo_w;        // and first two weights
    const uint32_t* first_src;   // every destination's first source
    const uint2* wo_long;        // (destination, first in-edge) pieces of the destinations past WO_GROUP in-edges
    uint32_t nlong;
    const uint32_t* outdeg;      // with push: the out-lists' lengths (a shard's are shorter than its out-degrees)
    const unsigned long long* csri_off;
    const uint32_t* csri;
    const uint8_t* cw8;          // out-edge weights (push): byte-wide, or
    const unsigned long long* cw; // 64-bit words
    const uint32_t* new2old;
    const uint32_t* old2new;
    uint64_t V, E;
    uint32_t Vne, nchunks, weight_kind;
    uint32_t push;               // sparse pulls relax out-edges (CSRI of destinations)
};

struct BQuery {
    uint32_t graph, app, root_in, pad;
    unsigned long long* prop; // [V] BFS parent (engine id; the root holds itself) / SSSP distance
    uint32_t* front[3];       // [V/32+1] activation bitmaps in turn by iteration: read, written, cleared
    uint32_t* list[2];        // [V] the same vertices as lists (with push: but for those of long out-lists)
    uint32_t* chunk_bits;     // [nchunks/32+1] Wedge frontier
    uint32_t* chunk_list;     // [nchunks] its marked chunks
    uint2* items[2];          // [E/(PUSH_PIECE/2) + 1] (vertex, piece) items of long out-lists
};

struct BCtl {
    unsigned long long mass;
    uint32_t nlist[3]; // by iteration modulo 3
    uint32_t nitem[3];
    unsigned long long fmin, next_fmin; // SSSP: no vertex the last (this) iteration changed is nearer
    uint32_t items; // work items of the next pull
    uint32_t mode;
    uint32_t iter;
    uint32_t done;
    uint32_t root; // engine id
};

struct BShared {
    uint32_t active;
    uint32_t rounds;
    unsigned long long grab_pull, grab_build;
    unsigned long long chunks_pulled;
};

struct BArgs {
    const BGraph* graphs;
    const BQuery* q;
    BCtl* ctl;
    BShared* sh;
    unsigned long long* pull_off;  // [Q+1]
    unsigned long long* build_off; // [Q+1]
    const uint32_t* sweep_off;     // [Q+1] SWEEP-word pieces of the queries' bitmaps
    uint32_t Q, threshold_pct, grab, split, max_rounds, chunks;  // chunks: some graph's CSRI holds chunk ids
};

template <class T>
__device__ __forceinline__ uint32_t find_owner(const T* off, uint32_t Q, T i)
{
    // last q with off[q] <= i (off[0] = 0, off[Q] > i)
    uint32_t lo = 0, hi = Q;
    while (hi - lo > 1u) {
        const uint32_t mid = (lo + hi) >> 1;
        if (off[mid] <= i)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// exclusive prefix of f(q) over q < Q into off[0..Q] by the threads of one block
template <class F>
__device__ void block_prefix(unsigned long long* off, uint32_t Q, F f)
{
    __shared__ unsigned long long part[BT / 32];
    const uint32_t per = (Q + BT - 1) / BT;
    const uint32_t q0 = threadIdx.x * per, q1 = min(Q, q0 + per);
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    unsigned long long s = 0;
    for (uint32_t q = q0; q < q1; ++q)
        s += f(q);
    unsigned long long incl = s;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long y = __shfl_up_sync(FULL, incl, d);
        if (lane >= d)
            incl += y;
    }
    if (lane == 31)
        part[wib] = incl;
    __syncthreads();
    unsigned long long run = incl - s;
    for (int w = 0; w < wib; ++w)
        run += part[w];
    if (threadIdx.x == BT - 1)
        off[Q] = run + s;
    for (uint32_t q = q0; q < q1; ++q) {
        off[q] = run;
        run += f(q);
    }
    __syncthreads();
}

__device__ __forceinline__ void mark_batch_chunk(const BQuery& qq, BCtl& c, uint32_t ch)
{
    const uint32_t bit = 1u << (ch & 31u);
    if (!(qq.chunk_bits[ch >> 5] & bit)) {
        const uint32_t old = atomicOr(&qq.chunk_bits[ch >> 5], bit);
        if (!(old & bit)) {
            const uint32_t pos = atomicAdd(&c.items, 1u);
            qq.chunk_list[pos] = ch;
        }
    }
}

// ---------------------------------------------------------------- build (chunk graphs)
__device__ void phase_build(const BArgs& a)
{
    const int lane = threadIdx.x & 31;
    const unsigned long long total = a.build_off[a.Q];
    for (;;) {
        unsigned long long base = 0;
        if (lane == 0)
            base = atomicAdd(&a.sh->grab_build, 32ull);
        base = __shfl_sync(FULL, base, 0);
        if (base >= total)
            break;
        const unsigned long long i = base + (unsigned long long)lane;
        const bool valid = i < total;
        uint32_t q = 0, v = 0;
        unsigned long long start = 0, len = 0;
        if (valid) {
            q = find_owner(a.build_off, a.Q, i);
            const BCtl& c = a.ctl[q];
            v = a.q[q].list[c.iter & 1u][i - a.build_off[q]];
            const BGraph& G = a.graphs[a.q[q].graph];
            start = G.csri_off[v];
            len = G.csri_off[v + 1] - start;
        }
        // short lists: one lane each
        if (valid && len <= a.split) {
            const BGraph& G = a.graphs[a.q[q].graph];
            for (unsigned long long j = 0; j < len; ++j)
                mark_batch_chunk(a.q[q], a.ctl[q], G.csri[start + j]);
        }
        // long lists: the whole warp, one list at a time
        uint32_t longs = __ballot_sync(FULL, valid && len > a.split);
        while (longs) {
            const int l = __ffs(longs) - 1;
            longs &= longs - 1u;
            const uint32_t lq = __shfl_sync(FULL, q, l);
            const unsigned long long ls = __shfl_sync(FULL, start, l), ll = __shfl_sync(FULL, len, l);
            const BGraph& G = a.graphs[a.q[lq].graph];
            for (unsigned long long j = lane; j < ll; j += 32)
                mark_batch_chunk(a.q[lq], a.ctl[lq], G.csri[ls + j]);
        }
    }
}

// ---------------------------------------------------------------- prefix (block 0)
__device__ void phase_prefix(const BArgs& a)
{
    block_prefix(a.pull_off, a.Q, [&](uint32_t q) -> unsigned long long {
        const BCtl& c = a.ctl[q];
        return c.done ? 0ull : (unsigned long long)c.items;
    });
    bool act = false;
    for (uint32_t q = threadIdx.x; q < a.Q; q += blockDim.x)
        act = act || !a.ctl[q].done;
    const int any = __syncthreads_or(act);
    if (threadIdx.x == 0) {
        a.sh->grab_pull = 0ull;
        a.sh->active = any ? 1u : 0u;
        if (any)
            a.sh->rounds += 1u;
    }
}

// ---------------------------------------------------------------- pull
// vertex v of out-degree od into the next iteration's list, or its items; one lane
__device__ __forceinline__ void list_one(const BQuery& qq, BCtl& c, const BGraph& G, uint32_t v, uint32_t od)
{
    const uint32_t nx = (c.iter + 1u) % 3u, buf = (c.iter + 1u) & 1u;
    if (G.push && od > PUSH_PIECE) {
        const uint32_t np = (od + PUSH_PIECE - 1u) / PUSH_PIECE;
        const uint32_t at = atomicAdd(&c.nitem[nx], np);
        for (uint32_t j = 0; j < np; ++j)
            qq.items[buf][at + j] = make_uint2(v, j);
    } else {
        qq.list[buf][atomicAdd(&c.nlist[nx], 1u)] = v;
    }
}

// the same for the lanes of a warp together
__device__ __forceinline__ void list_warp(const BQuery& qq, BCtl& c, const BGraph& G, bool on, uint32_t v, uint32_t od)
{
    const int lane = threadIdx.x & 31;
    const bool shrt = on && od <= PUSH_PIECE;
    const uint32_t m = __ballot_sync(FULL, shrt);
    if (m) {
        uint32_t at = 0u;
        if (lane == 0)
            at = atomicAdd(&c.nlist[(c.iter + 1u) % 3u], (uint32_t)__popc(m));
        at = __shfl_sync(FULL, at, 0) + (uint32_t)__popc(m & ((1u << lane) - 1u));
        if (shrt)
            qq.list[(c.iter + 1u) & 1u][at] = v;
    }
    if (on && !shrt)
        list_one(qq, c, G, v, od);
}

__device__ void pull_chunk(const BArgs& a, uint32_t q, uint32_t ch, uint32_t* heads, unsigned long long& mass)
{
    const int lane = threadIdx.x & 31;
    const BQuery& qq = a.q[q];
    BCtl& c = a.ctl[q];
    const BGraph& G = a.graphs[qq.graph];
    const unsigned long long p = 32ull * ch + (unsigned long long)lane;
    const bool valid = p < G.E;
    const uint32_t s = valid ? G.src[p] : NONE32;
    DevGraph dg;
    dg.Vne = G.Vne;
    dg.dst_off = G.dst_off;
    TileGeo<1> tg;
    tile_geometry<1>(dg, 32ull * ch, ch + 1u >= G.nchunks, G.chunk_dst0[ch], G.chunk_dst0[ch + 1], lane, heads, tg,
                     [](uint32_t, uint32_t) {});
    const uint32_t k = pos_dst(tg, 0);
    const uint32_t* cur = qq.front[c.iter % 3u];
    uint32_t* nxt = qq.front[(c.iter + 1u) % 3u];
    auto activate = [&](uint32_t vtx) {
        const uint32_t b = 1u << (vtx & 31u);
        if (!(atomicOr(&nxt[vtx >> 5], b) & b)) {
            const uint32_t od = G.outdeg[vtx];
            list_one(qq, c, G, vtx, od);
            mass += od;
        }
    };
    if (qq.app == WEDGE_APP_BFS) {
        uint32_t v[1];
        v[0] = NONE32;
        if (valid && ((cur[s >> 5] >> (s & 31u)) & 1u)) {
            const uint32_t vtx = G.dst_id[k];
            if (qq.prop[vtx] == NONE64) /* unvisited */
                v[0] = s;
        }
        seg_reduce<1>(v, tg, lane, MinU32(), [&](uint32_t kk, uint32_t val, int) {
            if (val == NONE32)
                return;
            const uint32_t vtx = G.dst_id[kk];
            if (atomicMin(&qq.prop[vtx], (unsigned long long)val) == NONE64)
                activate(vtx);
        });
    } else {
        unsigned long long v[1];
        v[0] = NONE64;
        if (valid) {
            const unsigned long long d = qq.prop[s];
            const unsigned long long wt = G.w8 ? (unsigned long long)G.w8[p] : G.w[p];
            if (G.weight_kind == WEDGE_WEIGHTS_F64)
                v[0] = (unsigned long long)__double_as_longlong(
                    __dadd_rn(__longlong_as_double((long long)d), __longlong_as_double((long long)wt)));
            else
                v[0] = (d == NONE64) ? NONE64 : d + wt; /* phase_edge_pull_sssp.c:136-137 */
        }
        seg_reduce<1>(v, tg, lane, MinU64(), [&](uint32_t kk, unsigned long long val, int) {
            if (val == NONE64)
                return;
            const uint32_t vtx = G.dst_id[kk];
            if (val < qq.prop[vtx] && val < atomicMin(&qq.prop[vtx], val))
                activate(vtx);
        });
    }
}

// A dense pull's item: a tile of BTILE_CH chunks (32*BEPL in-edges), lane l
// holding BEPL consecutive ones, with the single-query engine's tile machinery
// (destination-start bitmap geometry, segmented reduction).  BFS gathers the
// frontier bits of the sources and claims an unvisited destination for the
// least frontier source with one compare-and-swap; SSSP gathers distances,
// adds the weights and lowers the destination with atomicMin.  Per
// destination, not per in-edge: the visited test, the property write and the
// activation.
constexpr int BEPL = 8;
constexpr uint32_t BTILE_CH = BEPL; /* 32-edge chunks per tile */

__device__ void pull_tile(const BArgs& a, uint32_t q, uint32_t t, unsigned long long& mass)
{
    const int lane = threadIdx.x & 31;
    const BQuery& qq = a.q[q];
    BCtl& c = a.ctl[q];
    const BGraph& G = a.graphs[qq.graph];
    const uint64_t base = (uint64_t)t * (32u * BEPL);
    const uint32_t ch0 = t * BTILE_CH;
    const uint32_t k0 = G.chunk_dst0[ch0];
    const uint32_t kend = G.chunk_dst0[min(ch0 + BTILE_CH, G.nchunks)];
    const bool last = base + 32u * BEPL >= G.E;
    uint32_t sa[BEPL];
    {
        const uint64_t p0 = base + (uint64_t)lane * BEPL;
        uint32_t x[8];
        ld_stream_v8(G.src + p0, x);
#pragma unroll
        for (int j = 0; j < BEPL; ++j)
            sa[j] = (p0 + (uint64_t)j < G.E) ? x[j] : NONE32;
    }
    DevGraph dg;
    dg.dst_start = G.dst_start;
    TileGeo<BEPL> tg;
    const uint32_t* cur = qq.front[c.iter % 3u];
    uint32_t* nxt = qq.front[(c.iter + 1u) % 3u];
    auto activate = [&](uint32_t vtx) {
        const uint32_t b = 1u << (vtx & 31u);
        if (!(atomicOr(&nxt[vtx >> 5], b) & b)) {
            const uint32_t od = G.outdeg[vtx];
            list_one(qq, c, G, vtx, od);
            mass += od;
        }
    };
    if (qq.app == WEDGE_APP_BFS) {
        uint32_t v[BEPL];
#pragma unroll
        for (int j = 0; j < BEPL; ++j) {
            const uint32_t x = sa[j];
            v[j] = (x != NONE32 && ((cur[x >> 5] >> (x & 31u)) & 1u)) ? x : NONE32;
        }
        tile_geometry_bits<BEPL>(dg, base, last, k0, kend, lane, tg);
        seg_reduce<BEPL>(v, tg, lane, MinU32(), [&](uint32_t k, uint32_t val, int) {
            if (val == NONE32)
                return;
            const uint32_t vtx = G.dst_id[k];
            /* the least frontier source of this tile claims an unvisited destination */
            if (qq.prop[vtx] == NONE64 && atomicCAS(&qq.prop[vtx], NONE64, (unsigned long long)val) == NONE64)
                activate(vtx);
        });
    } else {
        const bool f64 = G.weight_kind == WEDGE_WEIGHTS_F64;
        unsigned long long v[BEPL];
        const uint64_t p0 = base + (uint64_t)lane * BEPL;
#pragma unroll
        for (int j = 0; j < BEPL; ++j) {
            const uint32_t x = sa[j];
            v[j] = NONE64;
            if (x != NONE32) {
                const unsigned long long d = qq.prop[x];
                const unsigned long long wt = G.w8 ? (unsigned long long)G.w8[p0 + j] : G.w[p0 + j];
                if (f64)
                    v[j] = (unsigned long long)__double_as_longlong(
                        __dadd_rn(__longlong_as_double((long long)d), __longlong_as_double((long long)wt)));
                else
                    v[j] = (d == NONE64) ? NONE64 : d + wt; /* phase_edge_pull_sssp.c:136-137 */
            }
        }
        tile_geometry_bits<BEPL>(dg, base, last, k0, kend, lane, tg);
        seg_reduce<BEPL>(v, tg, lane, MinU64(), [&](uint32_t k, unsigned long long val, int) {
            if (val == NONE64)
                return;
            const uint32_t vtx = G.dst_id[k];
            if (val < qq.prop[vtx] && val < atomicMin(&qq.prop[vtx], val))
                activate(vtx);
        });
    }
}

// Four out-edges per lane of changed vertices with values x (BFS: the vertex;
// SSSP: its distance): destinations, their present state, the atomics and the
// listing in stages, so that the four chains are in flight together.  BFS: an
// unvisited destination takes the vertex as its parent; SSSP: min-plus.
__device__ __forceinline__ void push4(const BQuery& qq, BCtl& c, const BGraph& G, const bool (&on)[4],
                                      const unsigned long long (&x)[4], const uint32_t (&e)[4], unsigned long long& mass,
                                      unsigned long long& least)
{
    uint32_t* nxt = qq.front[(c.iter + 1u) % 3u];
    const bool bfs = qq.app == WEDGE_APP_BFS, f64 = G.weight_kind == WEDGE_WEIGHTS_F64;
    uint32_t d[4];
    unsigned long long nd[4], p[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        d[u] = on[u] ? G.csri[e[u]] : 0u;
        nd[u] = x[u];
        if (on[u] && !bfs) {
            const unsigned long long wt = G.cw8 ? (unsigned long long)G.cw8[e[u]] : G.cw[e[u]];
            nd[u] = f64 ? (unsigned long long)__double_as_longlong(
                              __dadd_rn(__longlong_as_double((long long)x[u]), __longlong_as_double((long long)wt)))
                        : x[u] + wt; /* phase_edge_pull_sssp.c:136-137; an activated source is reached */
        }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
        p[u] = on[u] ? qq.prop[d[u]] : 0ull;
    bool low[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        low[u] = bfs ? p[u] == NONE64 : nd[u] < p[u];
        if (low[u])
            p[u] = bfs ? atomicCAS(&qq.prop[d[u]], NONE64, nd[u]) : atomicMin(&qq.prop[d[u]], nd[u]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        low[u] = low[u] && (bfs ? p[u] == NONE64 : nd[u] < p[u]);
        if (low[u])
            least = min(least, nd[u]);
    }
    if (!__any_sync(FULL, low[0] || low[1] || low[2] || low[3]))
        return;
    uint32_t o[4], od[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        o[u] = FULL;
        od[u] = 0u;
        if (low[u]) {
            o[u] = atomicOr(&nxt[d[u] >> 5], 1u << (d[u] & 31u));
            od[u] = G.outdeg[d[u]];
        }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const bool first = low[u] && !((o[u] >> (d[u] & 31u)) & 1u);
        mass += first ? od[u] : 0u;
        list_warp(qq, c, G, first, d[u], od[u]);
    }
}

__device__ __forceinline__ unsigned long long push_value(const BQuery& qq, uint32_t v)
{
    return qq.app == WEDGE_APP_BFS ? (unsigned long long)v : qq.prop[v];
}

// one PUSH_PIECE of a long out-list
__device__ void push_piece(const BArgs& a, uint32_t q, uint2 it, unsigned long long& mass, unsigned long long& least)
{
    const int lane = threadIdx.x & 31;
    const BQuery& qq = a.q[q];
    BCtl& c = a.ctl[q];
    const BGraph& G = a.graphs[qq.graph];
    const uint32_t lo = (uint32_t)G.csri_off[it.x] + it.y * PUSH_PIECE, end = (uint32_t)G.csri_off[it.x + 1u];
    const uint32_t hi = end - lo > PUSH_PIECE ? lo + PUSH_PIECE : end;
    const unsigned long long x0 = push_value(qq, it.x);
    const unsigned long long x[4] = {x0, x0, x0, x0};
    for (uint32_t t = lo; t < hi; t += 128u) {
        bool on[4];
        uint32_t e[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            e[u] = t + 32u * u + (uint32_t)lane;
            on[u] = e[u] < hi;
        }
        push4(qq, c, G, on, x, e, mass, least);
    }
}

// PUSH_CHUNK listed vertices: their out-edges spread over the lanes by a prefix sum
struct PushShared {
    uint32_t pre[PUSH_CHUNK], beg[PUSH_CHUNK];
    unsigned long long val[PUSH_CHUNK];
};

__device__ void push_chunk(const BArgs& a, uint32_t q, uint32_t i0, uint32_t n, PushShared& sh, unsigned long long& mass,
                           unsigned long long& least)
{
    const int lane = threadIdx.x & 31;
    const BQuery& qq = a.q[q];
    BCtl& c = a.ctl[q];
    const BGraph& G = a.graphs[qq.graph];
    uint32_t lo = 0u, len = 0u;
    __syncwarp();
    if ((uint32_t)lane < PUSH_CHUNK && i0 + (uint32_t)lane < n) {
        const uint32_t v = qq.list[c.iter & 1u][i0 + (uint32_t)lane];
        lo = (uint32_t)G.csri_off[v];
        len = (uint32_t)G.csri_off[v + 1u] - lo;
        sh.val[lane] = push_value(qq, v);
    }
    uint32_t incl = len;
#pragma unroll
    for (int d = 1; d < (int)PUSH_CHUNK; d <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, incl, d);
        if (lane >= d)
            incl += y;
    }
    const uint32_t total = __shfl_sync(FULL, incl, PUSH_CHUNK - 1u);
    if ((uint32_t)lane < PUSH_CHUNK) {
        sh.pre[lane] = incl - len;
        sh.beg[lane] = lo - (incl - len);
    }
    __syncwarp();
    for (uint32_t t0 = 0; t0 < total; t0 += 128u) {
        bool on[4];
        uint32_t e[4];
        unsigned long long x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t t = t0 + 32u * u + (uint32_t)lane;
            on[u] = t < total;
            uint32_t o = 0u; /* the vertex: the last one whose out-edges begin at or before t */
#pragma unroll
            for (uint32_t h = PUSH_CHUNK / 2u; h > 0u; h >>= 1)
                if (sh.pre[o + h] <= t)
                    o += h;
            e[u] = sh.beg[o] + t;
            x[u] = sh.val[o];
        }
        push4(qq, c, G, on, x, e, mass, least);
    }
}

// the weights that may lower a distance: below this.  After a pull only the
// vertices it changed matter to the next; none of them, and none it lowers in
// turn, is nearer than fmin.
__device__ __forceinline__ unsigned long long wo_limit(unsigned long long dist, unsigned long long fmin)
{
    return dist > fmin ? dist - fmin : 0ull;
}

// four weight-ordered in-edges at position p (a multiple of 4), of which those
// in [lo, hi) are the destination's; returns the weight of position p + 3
__device__ __forceinline__ uint32_t wo_step(const BQuery& qq, const BGraph& G, uint32_t p, uint32_t lo, uint32_t hi,
                                            unsigned long long fmin, unsigned long long& dist)
{
    const unsigned long long lim = wo_limit(dist, fmin);
    const uint32_t ww = ld_ro_u32(reinterpret_cast<const uint32_t*>(G.ww8 + p));
    const uint4 xs = __ldg(reinterpret_cast<const uint4*>(G.wsrc + p));
    const uint32_t x[4] = {xs.x, xs.y, xs.z, xs.w};
    unsigned long long y[4];
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
        const uint32_t w = (ww >> (8 * j)) & 0xFFu;
        y[j] = (p + j >= lo && p + j < hi && w < lim) ? qq.prop[x[j]] : NONE64;
    }
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j)
        if (y[j] != NONE64)
            dist = min(dist, y[j] + ((ww >> (8 * j)) & 0xFFu)); /* phase_edge_pull_sssp.c:136-137 */
    return ww >> 24;
}

// weight-ordered in-edges [p, hi) by the warp, 128 a step, up to the first
// weight that cannot lower dist (p a multiple of 4; all warp-uniform)
__device__ __forceinline__ unsigned long long wo_run(const BQuery& qq, const BGraph& G, uint32_t p, uint32_t hi,
                                                     unsigned long long fmin, unsigned long long dist)
{
    const int lane = threadIdx.x & 31;
    const uint32_t lo = p;
    for (; p < hi; p += 128u) {
        const uint32_t at = p + 4u * (uint32_t)lane;
        const uint32_t last = at < hi ? wo_step(qq, G, at, lo, hi, fmin, dist) : 0xFFFFFFFFu;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1)
            dist = min(dist, __shfl_xor_sync(FULL, dist, d));
        if (__shfl_sync(FULL, last, 31) >= wo_limit(dist, fmin))
            break;
    }
    return dist;
}

// A dense SSSP pull's item: 32 destinations, one per lane.  Those of more than
// WO_GROUP in-edges are left to their pieces: a lane that reads on for long
// holds up 31 others (groups of up to 32, 64, 128 and 256 in-edges took 4.4,
// 3.7, 3.8 and 3.6 ms on the 32 SSSPs of phase_pull's comment, 2.06, 1.72, 1.80
// and 2.09 ms on 16 over graphs of scales 16 to 20).
__device__ void wo_group(const BArgs& a, uint32_t q, uint32_t group, unsigned long long& mass, unsigned long long& least)
{
    const int lane = threadIdx.x & 31;
    const BQuery& qq = a.q[q];
    BCtl& c = a.ctl[q];
    const BGraph& G = a.graphs[qq.graph];
    const uint32_t k = group * 32u + (uint32_t)lane;
    const unsigned long long fmin = c.fmin;
    unsigned long long before = 0ull, dist = 0ull;
    uint32_t d = 0u;
    bool more = false;
    if (k < G.Vne) { /* the first in-edge and the second's weight settle most */
        const uint32_t x = G.wo_src[k], w = G.wo_w[k];
        d = G.dst_id[k];
        before = dist = qq.prop[d];
        if (!(x & WO_MANY_BIT) && (w & 0xFFu) < wo_limit(dist, fmin)) { /* the long ones are left to their pieces */
            const unsigned long long y = qq.prop[x & WO_ID_BITS];
            if (y != NONE64)
                dist = min(dist, y + (w & 0xFFu));
            more = !(x & WO_ONLY_BIT) && (w >> 8) < wo_limit(dist, fmin);
        }
    }
    if (more) {
        const uint32_t lo = (uint32_t)G.dst_off[k], hi = (uint32_t)G.dst_off[k + 1u];
        for (uint32_t p = lo & ~3u; more;) {
            const uint32_t last = wo_step(qq, G, p, lo, hi, fmin, dist);
            p += 4u;
            more = p < hi && last < wo_limit(dist, fmin);
        }
    }
    const bool low = dist < before;
    uint32_t od = 0u;
    if (low) { /* the destination's only writer in this pull */
        qq.prop[d] = dist;
        least = min(least, dist);
        atomicOr(&qq.front[(c.iter + 1u) % 3u][d >> 5], 1u << (d & 31u));
        od = G.outdeg[d];
        mass += od;
    }
    list_warp(qq, c, G, low, d, od);
}

// a piece of a destination with many in-edges; the pieces combine with atomicMin
__device__ void wo_piece(const BArgs& a, uint32_t q, uint2 it, unsigned long long& mass, unsigned long long& least)
{
    const BQuery& qq = a.q[q];
    BCtl& c = a.ctl[q];
    const BGraph& G = a.graphs[qq.graph];
    const uint32_t d = G.dst_id[it.x], end = (uint32_t)G.dst_off[it.x + 1u];
    const uint32_t hi = end - it.y > WO_PIECE ? it.y + WO_PIECE : end;
    const unsigned long long before = __shfl_sync(FULL, qq.prop[d], 0);
    const unsigned long long fmin = c.fmin;
    unsigned long long dist = before;
    /* the piece's first in-edges up to a multiple of 4, on lane 0 */
    const uint32_t p = min(hi, (it.y + 3u) & ~3u);
    bool go = true;
    if (p != it.y) {
        uint32_t stop = 0u;
        if ((threadIdx.x & 31) == 0) {
            wo_step(qq, G, it.y & ~3u, it.y, p, fmin, dist);
            stop = G.ww8[p - 1u] >= wo_limit(dist, fmin) ? 1u : 0u;
        }
        dist = __shfl_sync(FULL, dist, 0);
        go = __shfl_sync(FULL, stop, 0) == 0u;
    }
    if (go)
        dist = wo_run(qq, G, p, hi, fmin, dist);
    if ((threadIdx.x & 31) == 0 && dist < before && dist < atomicMin(&qq.prop[d], dist)) {
        least = min(least, dist);
        const uint32_t b = 1u << (d & 31u);
        if (!(atomicOr(&qq.front[(c.iter + 1u) % 3u][d >> 5], b) & b)) {
            const uint32_t od = G.outdeg[d];
            list_one(qq, c, G, d, od);
            mass += od;
        }
    }
}

// dense pulls by destinations (and pieces of the long ones) instead of tiles
__device__ __forceinline__ bool by_destination(const BGraph& G, uint32_t app)
{
    return app == WEDGE_APP_BFS ? G.push != 0u : G.wsrc != nullptr;
}

// A dense BFS pull's item: 32 destinations, one per lane.  An unvisited one
// takes its first source in the frontier; for most that is the first of all,
// which first_src holds in order.  A destination's pieces and its lane claim it
// by compare-and-swap.
__device__ void bfs_group(const BArgs& a, uint32_t q, uint32_t group, unsigned long long& mass)
{
    const int lane = threadIdx.x & 31;
    const BQuery& qq = a.q[q];
    BCtl& c = a.ctl[q];
    const BGraph& G = a.graphs[qq.graph];
    const uint32_t k = group * 32u + (uint32_t)lane;
    const uint32_t* cur = qq.front[c.iter % 3u];
    uint32_t d = 0u, par = NONE32, od = 0u;
    if (k < G.Vne) {
        d = G.dst_id[k];
        const uint32_t x = G.first_src[k];
        if (qq.prop[d] == NONE64) {
            if ((cur[x >> 5] >> (x & 31u)) & 1u) {
                par = x;
            } else {
                const uint32_t lo = (uint32_t)G.dst_off[k], hi = (uint32_t)G.dst_off[k + 1u];
                if (hi - lo <= WO_GROUP) /* the others are left to their pieces */
                    for (uint32_t p = lo & ~3u; p < hi && par == NONE32; p += 4u) {
                        const uint4 xs = __ldg(reinterpret_cast<const uint4*>(G.src + p));
                        const uint32_t y[4] = {xs.x, xs.y, xs.z, xs.w};
                        uint32_t w[4];
#pragma unroll
                        for (uint32_t j = 0; j < 4; ++j)
                            w[j] = p + j > lo && p + j < hi ? cur[y[j] >> 5] : 0u;
#pragma unroll
                        for (int j = 3; j >= 0; --j)
                            if ((w[j] >> (y[j] & 31u)) & 1u)
                                par = y[j];
                    }
            }
        }
    }
    const bool hit = par != NONE32 && atomicCAS(&qq.prop[d], NONE64, (unsigned long long)par) == NONE64;
    if (hit) {
        atomicOr(&qq.front[(c.iter + 1u) % 3u][d >> 5], 1u << (d & 31u));
        od = G.outdeg[d];
        mass += od;
    }
    list_warp(qq, c, G, hit, d, od);
}

// a piece of a destination with many in-edges: the first source in the frontier
__device__ void bfs_piece(const BArgs& a, uint32_t q, uint2 it, unsigned long long& mass)
{
    const int lane = threadIdx.x & 31;
    const BQuery& qq = a.q[q];
    BCtl& c = a.ctl[q];
    const BGraph& G = a.graphs[qq.graph];
    const uint32_t d = G.dst_id[it.x], end = (uint32_t)G.dst_off[it.x + 1u];
    if (__shfl_sync(FULL, qq.prop[d], 0) != NONE64)
        return;
    const uint32_t* cur = qq.front[c.iter % 3u];
    const uint32_t hi = end - it.y > WO_PIECE ? it.y + WO_PIECE : end;
    for (uint32_t p = it.y; p < hi; p += 32u) {
        const uint32_t e = p + (uint32_t)lane;
        uint32_t x = 0u;
        bool on = false;
        if (e < hi) {
            x = G.src[e];
            on = (cur[x >> 5] >> (x & 31u)) & 1u;
        }
        const uint32_t m = __ballot_sync(FULL, on);
        if (m) {
            if (lane == __ffs(m) - 1 && atomicCAS(&qq.prop[d], NONE64, (unsigned long long)x) == NONE64) {
                const uint32_t od = G.outdeg[d];
                atomicOr(&qq.front[(c.iter + 1u) % 3u][d >> 5], 1u << (d & 31u));
                list_one(qq, c, G, d, od);
                mass += od;
            }
            return;
        }
    }
}

// The order of the groups in the queue: in-degrees fall with the destination
// number, and a warp takes up to 32 items at a time, so consecutive items are
// groups far apart (32 neighbouring hub groups kept one warp busy for 900 us of
// a 1.2 ms pull).  A permutation of [0, n): rows of 32, then what is left.
__device__ __forceinline__ uint32_t wo_spread(uint32_t i, uint32_t n)
{
    const uint32_t rows = n / 32u;
    return i < rows * 32u ? (i % 32u) * rows + i / 32u : i;
}

// Bound by the latency of the items' chains (weights and sources, distances of
// the sources; lists, out-edges, distances, claims) and by how evenly they
// spread: items are kept short, and a warp takes fewer of them towards the
// queue's end.  32 SSSPs over 8 graphs (scales 12 to 20, 177 M in-edges in
// all): 3.1 ms in 16 rounds (3.6 without wo_limit's bound and the first in-edges
// in arrays of their own), 13.3 with 256-edge tiles that streamed every in-edge
// of a dense pull; 16 BFS over scales 16 to 20: 0.61 ms, 1.5 in tiles; 16 BFS
// and 16 SSSP over scales 13 to 16: 0.55 ms, 2.8 before.
__device__ void phase_pull(const BArgs& a)
{
    __shared__ uint32_t heads_all[BT / 32];
    __shared__ PushShared push_all[BT / 32];
    const int lane = threadIdx.x & 31;
    uint32_t* heads = &heads_all[threadIdx.x >> 5];
    PushShared& push_sh = push_all[threadIdx.x >> 5];
    // the bitmaps the next round writes
    {
        const uint32_t nw = (gridDim.x * blockDim.x) >> 5, pieces = a.sweep_off[a.Q];
        for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < pieces; i += nw) {
            const uint32_t q = find_owner(a.sweep_off, a.Q, i);
            const BCtl& c = a.ctl[q];
            if (c.done)
                continue;
            const uint32_t words = (uint32_t)((a.graphs[a.q[q].graph].V + 31) / 32), w0 = (i - a.sweep_off[q]) * SWEEP;
            uint32_t* f = a.q[q].front[(c.iter + 2u) % 3u];
            for (uint32_t w = w0 + (uint32_t)lane; w < min(words, w0 + SWEEP); w += 32u)
                f[w] = 0u;
        }
    }
    const unsigned long long total = a.pull_off[a.Q];
    unsigned long long pulled = 0, mass = 0, least = NONE64;
    uint32_t q = 0;
    auto settle = [&]() { /* the mass of the items of query q so far */
        if (__any_sync(FULL, mass != 0ull)) {
#pragma unroll
            for (int d = 16; d > 0; d >>= 1)
                mass += __shfl_xor_sync(FULL, mass, d);
            if (lane == 0)
                atomicAdd(&a.ctl[q].mass, mass);
        }
        if (__any_sync(FULL, least != NONE64) && a.graphs[a.q[q].graph].wsrc) {
#pragma unroll
            for (int d = 16; d > 0; d >>= 1)
                least = min(least, __shfl_xor_sync(FULL, least, d));
            if (lane == 0 && least < *(volatile unsigned long long*)&a.ctl[q].next_fmin)
                atomicMin(&a.ctl[q].next_fmin, least);
        }
        mass = 0ull;
        least = NONE64;
    };
    const unsigned long long warps = 2ull * ((gridDim.x * blockDim.x) >> 5);
    unsigned long long base = 0;
    for (;;) {
        // up to a.grab items, fewer towards the queue's end: half an even share of what was left at the last grab
        const unsigned long long want = max(1ull, min((unsigned long long)a.grab, (total - base) / warps));
        if (lane == 0)
            base = atomicAdd(&a.sh->grab_pull, want);
        base = __shfl_sync(FULL, base, 0);
        if (base >= total)
            break;
        const unsigned long long end = min(total, base + want);
        for (unsigned long long i = base; i < end; ++i) {
            if (!(a.pull_off[q] <= i && i < a.pull_off[q + 1])) {
                settle();
                q = find_owner(a.pull_off, a.Q, i); /* warp-uniform */
            }
            const uint32_t local = (uint32_t)(i - a.pull_off[q]);
            const BCtl& c = a.ctl[q];
            const BQuery& qq = a.q[q];
            const BGraph& G = a.graphs[qq.graph];
            if (c.mode != MODE_WEDGE) {
                const uint32_t groups = (G.Vne + 31u) / 32u;
                if (!by_destination(G, qq.app))
                    pull_tile(a, q, local, mass); /* tiles of BTILE_CH chunks */
                else if (qq.app == WEDGE_APP_BFS && local < G.nlong)
                    bfs_piece(a, q, G.wo_long[local], mass);
                else if (qq.app == WEDGE_APP_BFS)
                    bfs_group(a, q, wo_spread(local - G.nlong, groups), mass);
                else if (local < G.nlong)
                    wo_piece(a, q, G.wo_long[local], mass, least);
                else
                    wo_group(a, q, wo_spread(local - G.nlong, groups), mass, least);
            } else if (G.push) {
                const uint32_t ni = c.nitem[c.iter % 3u];
                if (local < ni)
                    push_piece(a, q, qq.items[c.iter & 1u][local], mass, least);
                else
                    push_chunk(a, q, (local - ni) * PUSH_CHUNK, c.nlist[c.iter % 3u], push_sh, mass, least);
            } else {
                const uint32_t ch = qq.chunk_list[local];
                pull_chunk(a, q, ch, heads, mass);
                if (lane == 0)
                    atomicAnd(&qq.chunk_bits[ch >> 5], ~(1u << (ch & 31u))); /* consumed */
            }
            ++pulled;
        }
    }
    settle();
    if (lane == 0 && pulled)
        atomicAdd(&a.sh->chunks_pulled, pulled);
}

// ---------------------------------------------------------------- decide (block 0)
// the work items of a query's next pull (chunk graphs' sparse pulls: the build counts them)
__device__ __forceinline__ uint32_t pull_items(const BGraph& G, const BQuery& qq, const BCtl& c)
{
    if (c.mode == MODE_DENSE) {
        if (by_destination(G, qq.app))
            return (G.Vne + 31u) / 32u + G.nlong;
        return (G.nchunks + BTILE_CH - 1u) / BTILE_CH;
    }
    if (!G.push)
        return 0u;
    return c.nitem[c.iter % 3u] + (c.nlist[c.iter % 3u] + PUSH_CHUNK - 1u) / PUSH_CHUNK;
}

__device__ void phase_decide(const BArgs& a)
{
    for (uint32_t q = threadIdx.x; q < a.Q; q += blockDim.x) {
        BCtl& c = a.ctl[q];
        if (c.done)
            continue;
        const BGraph& G = a.graphs[a.q[q].graph];
        c.iter += 1u;
        const unsigned long long m = c.mass;
        c.mass = 0ull;
        c.fmin = c.next_fmin;
        c.next_fmin = NONE64;
        if (m == 0ull || c.iter >= a.max_rounds) { /* execution_bfs.c:239-251 */
            c.done = 1u;
            continue;
        }
        const unsigned long long thr = (G.E * (unsigned long long)a.threshold_pct) / 100ull; /* execution_bfs.c:132 */
        c.mode = m > thr ? MODE_DENSE : MODE_WEDGE;                                         /* execution_bfs.c:141 */
        c.nlist[(c.iter + 1u) % 3u] = 0u;
        c.nitem[(c.iter + 1u) % 3u] = 0u;
        c.items = pull_items(G, a.q[q], c);
    }
    __syncthreads();
    if (!a.chunks) {
        phase_prefix(a);
        return;
    }
    block_prefix(a.build_off, a.Q, [&](uint32_t q) -> unsigned long long {
        const BCtl& c = a.ctl[q];
        return (!c.done && c.mode == MODE_WEDGE && !a.graphs[a.q[q].graph].push) ? (unsigned long long)c.nlist[c.iter % 3u] : 0ull;
    });
    if (threadIdx.x == 0)
        a.sh->grab_build = 0ull;
}

__global__ void __launch_bounds__(BT, 4) batch_kernel(BArgs a)
{
    cg::grid_group grid = cg::this_grid();
    for (uint32_t round = 0; round < a.max_rounds + 1u; ++round) {
        if (a.chunks) {
            phase_build(a);
            grid.sync();
            if (blockIdx.x == 0)
                phase_prefix(a);
            grid.sync();
        }
        if (*(volatile uint32_t*)&a.sh->active == 0u) /* written before the barrier, uniform after it */
            break;
        phase_pull(a);
        grid.sync();
        if (blockIdx.x == 0)
            phase_decide(a);
        grid.sync();
    }
}

// ---------------------------------------------------------------- setup kernels
__global__ void batch_chunk_index_kernel(BGraph G, uint32_t* chunk_dst0)
{
    // chunk_dst0[c] = compressed destination owning edge 32c: last k with dst_off[k] <= 32c
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c <= G.nchunks; c += gridDim.x * blockDim.x) {
        const unsigned long long p = 32ull * c;
        uint32_t k;
        if (p >= G.E) {
            k = G.Vne;
        } else {
            uint32_t lo = 0, hi = G.Vne;
            while (hi - lo > 1u) {
                const uint32_t mid = (lo + hi) >> 1;
                if (G.dst_off[mid] <= p)
                    lo = mid;
                else
                    hi = mid;
            }
            k = lo;
        }
        chunk_dst0[c] = k;
    }
}

__global__ void batch_reset_kernel(const BGraph* graphs, const BQuery* qs, uint32_t Q)
{
    const uint32_t q = blockIdx.y;
    if (q >= Q)
        return;
    const BQuery& qq = qs[q];
    const BGraph& G = graphs[qq.graph];
    const unsigned long long inf = (qq.app == WEDGE_APP_SSSP && G.weight_kind == WEDGE_WEIGHTS_F64)
                                       ? 0x7FF0000000000000ull /* execution_sssp.c:78, as double */
                                       : NONE64;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t t0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    for (uint64_t v = t0; v < G.V; v += stride)
        qq.prop[v] = inf;
    for (uint64_t i = t0; i < (G.V + 31) / 32 + 1; i += stride) {
        qq.front[0][i] = 0u;
        qq.front[1][i] = 0u;
        qq.front[2][i] = 0u;
    }
    if (!G.push)
        for (uint64_t i = t0; i < (uint64_t)G.nchunks / 32 + 1; i += stride)
            qq.chunk_bits[i] = 0u;
}

__global__ void batch_seed_kernel(BArgs a)
{
    // roots (execution_bfs.c:110-117, execution_sssp.c:83-88), first modes, first offsets
    for (uint32_t q = threadIdx.x; q < a.Q; q += blockDim.x) {
        const BQuery& qq = a.q[q];
        const BGraph& G = a.graphs[qq.graph];
        BCtl& c = a.ctl[q];
        const uint32_t root_in = qq.root_in < G.V ? qq.root_in : 0u; /* main.c:81-85 */
        const uint32_t r = G.old2new[root_in];
        c.root = r;
        c.mass = 0ull;
        c.fmin = 0ull;
        c.next_fmin = NONE64;
        c.iter = 0u;
        c.done = G.E == 0ull ? 1u : 0u;
        qq.prop[r] = (qq.app == WEDGE_APP_BFS) ? (unsigned long long)r : 0ull;
        qq.front[0][r >> 5] |= 1u << (r & 31u);
        for (uint32_t j = 0; j < 3u; ++j) {
            c.nlist[j] = 0u;
            c.nitem[j] = 0u;
        }
        const uint32_t od = G.outdeg[r];
        if (G.push && od > PUSH_PIECE) {
            c.nitem[0] = (od + PUSH_PIECE - 1u) / PUSH_PIECE;
            for (uint32_t j = 0; j < c.nitem[0]; ++j)
                qq.items[0][j] = make_uint2(r, j);
        } else {
            qq.list[0][0] = r;
            c.nlist[0] = 1u;
        }
        const unsigned long long thr = (G.E * (unsigned long long)a.threshold_pct) / 100ull;
        c.mode = (unsigned long long)od > thr ? MODE_DENSE : MODE_WEDGE;
        c.items = pull_items(G, qq, c);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        a.sh->active = 0u;
        a.sh->rounds = 0u;
        a.sh->grab_pull = a.sh->grab_build = 0ull;
        a.sh->chunks_pulled = 0ull;
    }
    __syncthreads();
    if (a.chunks)
        block_prefix(a.build_off, a.Q, [&](uint32_t q) -> unsigned long long {
            const BCtl& c = a.ctl[q];
            return (!c.done && c.mode == MODE_WEDGE && !a.graphs[a.q[q].graph].push) ? 1ull : 0ull;
        });
    else
        phase_prefix(a);
}

// the pieces of the destinations past WO_GROUP in-edges: counted (out null), then listed
__global__ void batch_wo_long_kernel(const unsigned long long* dst_off, uint32_t Vne, uint32_t* count, uint2* out)
{
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < Vne; k += gridDim.x * blockDim.x) {
        const uint32_t lo = (uint32_t)dst_off[k], n = (uint32_t)(dst_off[k + 1u] - dst_off[k]);
        if (n <= WO_GROUP)
            continue;
        const uint32_t np = (n + WO_PIECE - 1u) / WO_PIECE, at = atomicAdd(count, np);
        for (uint32_t j = 0; out && j < np; ++j)
            out[at + j] = make_uint2(k, lo + j * WO_PIECE);
    }
}

// the lengths of a shard's out-lists
__global__ void batch_list_length_kernel(const unsigned long long* off, uint64_t V, uint32_t* len)
{
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x)
        len[v] = (uint32_t)(off[v + 1] - off[v]);
}

__global__ void batch_export_kernel(BGraph G, BQuery qq, unsigned long long* out)
{
    const uint32_t root = G.old2new[qq.root_in];
    for (uint64_t o = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; o < G.V; o += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = G.old2new[o];
        const unsigned long long x = qq.prop[v];
        if (qq.app == WEDGE_APP_BFS)
            out[o] = (x == NONE64 || v == root) ? NONE64 : (unsigned long long)G.new2old[(uint32_t)x];
        else
            out[o] = x;
    }
}

}  // namespace wedge

using namespace wedge;

static uint32_t bgrid(uint64_t work, uint32_t threads, uint32_t cap)
{
    const uint64_t g = (work + threads - 1) / threads;
    return (uint32_t)(g == 0 ? 1 : (g < cap ? g : cap));
}

struct wedge_batch {
    int device;
    int num_sms;
    cudaStream_t stream;
    cudaEvent_t ev[2];
    uint32_t Q, G;
    BGraph* d_graphs;
    BQuery* d_queries;
    BCtl* d_ctl;
    BShared* d_sh;
    unsigned long long* d_off; // 2 * (Q+1)
    uint32_t* d_sweep;         // [Q+1]
    uint32_t chunks;           // some graph's CSRI holds chunk ids
    unsigned long long* xbuf;  // staging of the result reads, the largest graph's (on first use)
    pthread_mutex_t xlock;     // one read at a time fills it
    BGraph* h_graphs;
    BQuery* h_queries;
    void* allocs[16];
    int nallocs;
    void** qallocs; // per-query buffers
    uint32_t nq_allocs;
    uint64_t maxV;
    cudaGraphExec_t exec;
    wedge_batch_tuning_t exec_tuning;
    uint32_t exec_blocks;
};

static void batch_release(wedge_batch* b)
{
    if (!b)
        return;
    if (b->stream)
        cudaStreamSynchronize(b->stream);
    if (b->exec)
        cudaGraphExecDestroy(b->exec);
    for (int i = 0; i < b->nallocs; ++i)
        cudaFree(b->allocs[i]);
    for (uint32_t i = 0; i < b->nq_allocs; ++i)
        cudaFree(b->qallocs[i]);
    if (b->xbuf)
        cudaFree(b->xbuf);
    free(b->qallocs);
    free(b->h_graphs);
    free(b->h_queries);
    for (int i = 0; i < 2; ++i)
        if (b->ev[i])
            cudaEventDestroy(b->ev[i]);
    if (b->stream)
        cudaStreamDestroy(b->stream);
    pthread_mutex_destroy(&b->xlock);
    free(b);
}

template <class T>
static int balloc(wedge_batch* b, T** p, uint64_t count, bool per_query)
{
    *p = nullptr;
    const cudaError_t e = cudaMalloc((void**)p, (size_t)(count ? count : 1) * sizeof(T));
    if (e != cudaSuccess)
        return cuda_status(e);
    if (per_query)
        b->qallocs[b->nq_allocs++] = *p;
    else
        b->allocs[b->nallocs++] = *p;
    return WEDGE_OK;
}

extern "C" int wedge_cuda_batch_create(wedge_graph_t* const* graphs, uint32_t num_graphs, const wedge_query_t* queries,
                                       uint32_t num_queries, wedge_batch_t** out)
{
    if (!out || !graphs || !queries || num_graphs == 0 || num_queries == 0 || num_queries > 65535u)
        return WEDGE_ERR_ARG; /* one grid row per query in the reset kernel */
    *out = nullptr;
    const int dev = graphs[0] ? graphs[0]->device : -1;
    for (uint32_t i = 0; i < num_graphs; ++i)
        if (!graphs[i] || graphs[i]->device != dev || graphs[i]->g.V > 0xFFFFFFFEull)
            return WEDGE_ERR_ARG;
    for (uint32_t i = 0; i < num_queries; ++i) {
        const wedge_query_t& q = queries[i];
        if (q.graph >= num_graphs || (q.app != WEDGE_APP_BFS && q.app != WEDGE_APP_SSSP))
            return WEDGE_ERR_ARG;
        if (q.app == WEDGE_APP_SSSP && graphs[q.graph]->weight_kind == WEDGE_WEIGHTS_NONE)
            return WEDGE_ERR_ARG; /* SSSP needs a weighted load (application.c:171) */
    }
    WEDGE_CHECK(cudaSetDevice(dev));
    wedge_batch* b = (wedge_batch*)calloc(1, sizeof(wedge_batch));
    if (!b)
        return WEDGE_ERR_OOM;
    pthread_mutex_init(&b->xlock, nullptr);
    b->device = dev;
    b->Q = num_queries;
    b->G = num_graphs;
    b->qallocs = (void**)calloc(2 * (size_t)num_graphs + 3, sizeof(void*)); /* two arrays per graph, the lists, the queries */
    b->h_graphs = (BGraph*)calloc(num_graphs, sizeof(BGraph));
    b->h_queries = (BQuery*)calloc(num_queries, sizeof(BQuery));
    int rc = WEDGE_OK;
    auto fail = [&](int r) {
        batch_release(b);
        return r;
    };
    if (!b->qallocs || !b->h_graphs || !b->h_queries)
        return fail(WEDGE_ERR_OOM);
    if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&b->ev[0]) != cudaSuccess || cudaEventCreate(&b->ev[1]) != cudaSuccess ||
        cudaDeviceGetAttribute(&b->num_sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return fail(WEDGE_ERR_CUDA);
    for (uint32_t i = 0; i < num_graphs; ++i) {
        const DevGraph& g = graphs[i]->g;
        BGraph& G = b->h_graphs[i];
        G.src = g.src;
        G.w = g.w;
        G.dst_id = g.dst_id;
        G.dst_off = g.dst_off;
        G.outdeg = g.outdeg;
        G.csri_off = g.csri_off;
        G.csri = g.csri;
        G.cw8 = g.cw8;
        G.cw = g.cw;
        G.push = g.csr;
        G.wsrc = g.csr ? g.wsrc : nullptr;
        G.ww8 = g.ww8;
        G.wo_src = g.wo_src;
        G.first_src = g.first_src;
        G.wo_w = g.wo_w;
        if (!g.csr)
            b->chunks = 1u;
        if (g.V > b->maxV)
            b->maxV = g.V;
        G.dst_start = g.dst_start;
        G.w8 = g.w8;
        G.new2old = g.new2old;
        G.old2new = g.old2new;
        G.V = g.V;
        G.E = g.E;
        G.Vne = g.Vne;
        G.nchunks = (uint32_t)((g.E + 31) / 32);
        G.weight_kind = g.weight_kind;
        uint32_t* cd = nullptr;
        if ((rc = balloc(b, &cd, (uint64_t)G.nchunks + 1, true)))
            return fail(rc);
        G.chunk_dst0 = cd;
        if (g.shard && g.csr) {
            uint32_t* len = nullptr;
            if ((rc = balloc(b, &len, g.V, true)))
                return fail(rc);
            batch_list_length_kernel<<<bgrid(g.V, 256, (uint32_t)b->num_sms * 8), 256, 0, b->stream>>>(g.csri_off, g.V, len);
            G.outdeg = len;
        }
        batch_chunk_index_kernel<<<bgrid((uint64_t)G.nchunks + 1, 256, (uint32_t)b->num_sms * 8), 256, 0, b->stream>>>(G, cd);
    }
    // pieces of the destinations with many in-edges (dense pulls): all graphs' counts, then their lists
    uint32_t* d_long = nullptr;
    if ((rc = balloc(b, &d_long, num_graphs, false)))
        return fail(rc);
    uint32_t* h_long = (uint32_t*)calloc(num_graphs, sizeof(uint32_t));
    if (!h_long)
        return fail(WEDGE_ERR_OOM);
    uint2* lists = nullptr; /* one after the other */
    for (int pass = 0; pass < 2 && !rc; ++pass) {
        if (cudaMemsetAsync(d_long, 0, num_graphs * sizeof(uint32_t), b->stream) != cudaSuccess)
            rc = WEDGE_ERR_CUDA;
        uint64_t at = 0;
        for (uint32_t i = 0; i < num_graphs && !rc; ++i) {
            BGraph& G = b->h_graphs[i];
            if (!G.push || (pass && !h_long[i]))
                continue;
            G.wo_long = lists + at;
            G.nlong = h_long[i];
            at += h_long[i];
            batch_wo_long_kernel<<<bgrid(G.Vne, 256, (uint32_t)b->num_sms * 8), 256, 0, b->stream>>>(
                G.dst_off, G.Vne, d_long + i, pass ? lists + (at - h_long[i]) : nullptr);
        }
        if (pass || rc)
            break;
        if (cudaMemcpyAsync(h_long, d_long, num_graphs * sizeof(uint32_t), cudaMemcpyDeviceToHost, b->stream) != cudaSuccess ||
            cudaStreamSynchronize(b->stream) != cudaSuccess) {
            rc = WEDGE_ERR_CUDA;
            break;
        }
        for (uint32_t i = 0; i < num_graphs; ++i)
            at += h_long[i];
        if (!at || (rc = balloc(b, &lists, at, true)))
            break;
    }
    free(h_long);
    if (rc)
        return fail(rc);
    uint32_t* h_sweep = (uint32_t*)calloc((size_t)num_queries + 1, sizeof(uint32_t));
    if (!h_sweep)
        return fail(WEDGE_ERR_OOM);
    unsigned char* base = nullptr; /* all queries' arrays, each on a 256-byte boundary */
    uint64_t size = 0;
    for (int pass = 0; pass < 2 && !rc; ++pass) {
        if (pass && (rc = balloc(b, &base, size, true)))
            break;
        size = 0;
        for (uint32_t i = 0; i < num_queries; ++i) {
            const BGraph& G = b->h_graphs[queries[i].graph];
            BQuery& q = b->h_queries[i];
            q.graph = queries[i].graph;
            q.app = (uint32_t)queries[i].app;
            q.root_in = queries[i].root < G.V ? (uint32_t)queries[i].root : 0u;
            const uint64_t words = (G.V + 31) / 32 + 1, chunks = G.push ? 0 : (uint64_t)G.nchunks,
                           nitems = G.push ? G.E / (PUSH_PIECE / 2u) + 1 : 0;
            h_sweep[i + 1] = h_sweep[i] + (uint32_t)((words + SWEEP - 1) / SWEEP);
            auto place = [&](uint64_t bytes) {
                const uint64_t at = size;
                size += (bytes + 255) & ~255ull;
                return at;
            };
            const uint64_t at_prop = place(8 * G.V), at_front = place(3 * ((4 * words + 255) & ~255ull)), at_l0 = place(4 * G.V),
                           at_l1 = place(4 * G.V), at_bits = place(4 * (chunks / 32 + 1)), at_list = place(4 * chunks),
                           at_i0 = place(8 * nitems), at_i1 = place(8 * nitems);
            if (!pass)
                continue;
            q.prop = (unsigned long long*)(base + at_prop);
            for (uint32_t f = 0; f < 3; ++f)
                q.front[f] = (uint32_t*)(base + at_front + f * ((4 * words + 255) & ~255ull));
            q.list[0] = (uint32_t*)(base + at_l0);
            q.list[1] = (uint32_t*)(base + at_l1);
            q.chunk_bits = (uint32_t*)(base + at_bits);
            q.chunk_list = (uint32_t*)(base + at_list);
            q.items[0] = (uint2*)(base + at_i0);
            q.items[1] = (uint2*)(base + at_i1);
        }
    }
    if (!rc && !(rc = balloc(b, &b->d_graphs, num_graphs, false)) && !(rc = balloc(b, &b->d_queries, num_queries, false)) &&
        !(rc = balloc(b, &b->d_ctl, num_queries, false)) && !(rc = balloc(b, &b->d_sh, 1, false)) &&
        !(rc = balloc(b, &b->d_off, 2ull * (num_queries + 1), false)) &&
        !(rc = balloc(b, &b->d_sweep, (uint64_t)num_queries + 1, false)) &&
        (cudaMemcpyAsync(b->d_sweep, h_sweep, sizeof(uint32_t) * ((size_t)num_queries + 1), cudaMemcpyHostToDevice, b->stream) !=
             cudaSuccess ||
         cudaStreamSynchronize(b->stream) != cudaSuccess))
        rc = WEDGE_ERR_CUDA;
    free(h_sweep);
    if (rc)
        return fail(rc);
    if (cudaMemcpyAsync(b->d_graphs, b->h_graphs, sizeof(BGraph) * num_graphs, cudaMemcpyHostToDevice, b->stream) !=
            cudaSuccess ||
        cudaMemcpyAsync(b->d_queries, b->h_queries, sizeof(BQuery) * num_queries, cudaMemcpyHostToDevice, b->stream) !=
            cudaSuccess ||
        cudaStreamSynchronize(b->stream) != cudaSuccess || cudaGetLastError() != cudaSuccess)
        return fail(WEDGE_ERR_CUDA);
    *out = b;
    return WEDGE_OK;
}

static void batch_tuning_defaults(const wedge_batch_tuning_t* in, int occ, wedge_batch_tuning_t* t)
{
    memset(t, 0, sizeof(*t));
    if (in)
        *t = *in;
    if (t->threshold_pct == 0 || t->threshold_pct > 100)
        t->threshold_pct = 20;
    if (t->grab == 0)
        t->grab = 8;
    if (t->blocks_per_sm == 0 || (int)t->blocks_per_sm > occ)
        t->blocks_per_sm = (uint32_t)occ;
    if (t->split == 0)
        t->split = 32;
}

static int batch_enqueue(wedge_batch* b, const wedge_batch_tuning_t& t, uint32_t blocks)
{
    BArgs a;
    memset(&a, 0, sizeof(a));
    a.graphs = b->d_graphs;
    a.q = b->d_queries;
    a.ctl = b->d_ctl;
    a.sh = b->d_sh;
    a.pull_off = b->d_off;
    a.build_off = b->d_off + (b->Q + 1);
    a.sweep_off = b->d_sweep;
    a.chunks = b->chunks;
    a.Q = b->Q;
    a.threshold_pct = t.threshold_pct;
    a.grab = t.grab;
    a.split = t.split;
    a.max_rounds = BATCH_MAX_ROUNDS;
    dim3 rgrid(64, b->Q);
    batch_reset_kernel<<<rgrid, 256, 0, b->stream>>>(b->d_graphs, b->d_queries, b->Q);
    batch_seed_kernel<<<1, BT, 0, b->stream>>>(a);
    void* args[] = {&a};
    WEDGE_CHECK(cudaLaunchCooperativeKernel((const void*)batch_kernel, dim3(blocks), dim3(BT), args, 0, b->stream));
    return WEDGE_OK;
}

extern "C" int wedge_cuda_batch_run(wedge_batch_t* b, const wedge_batch_tuning_t* tuning, uint32_t flags,
                                    wedge_batch_stats_t* stats)
{
    if (!b)
        return WEDGE_ERR_ARG;
    WEDGE_CHECK(cudaSetDevice(b->device));
    int occ = 0;
    WEDGE_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, batch_kernel, BT, 0));
    if (occ < 1)
        return WEDGE_ERR_CUDA;
    wedge_batch_tuning_t t;
    batch_tuning_defaults(tuning, occ, &t);
    const uint32_t blocks = (uint32_t)b->num_sms * t.blocks_per_sm;
    bool captured = false;
    WEDGE_CHECK(cudaEventRecord(b->ev[0], b->stream));
    if (flags & WEDGE_FLAG_GRAPH) {
        if (b->exec && memcmp(&b->exec_tuning, &t, sizeof(t)) != 0) {
            cudaGraphExecDestroy(b->exec);
            b->exec = nullptr;
        }
        if (!b->exec) {
            cudaGraph_t graph = nullptr;
            if (cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
                const int rc = batch_enqueue(b, t, blocks);
                const cudaError_t e = cudaStreamEndCapture(b->stream, &graph);
                if (rc == WEDGE_OK && e == cudaSuccess && graph &&
                    cudaGraphInstantiate(&b->exec, graph, 0) == cudaSuccess) {
                    b->exec_tuning = t;
                    b->exec_blocks = blocks;
                } else {
                    b->exec = nullptr;
                }
                if (graph)
                    cudaGraphDestroy(graph);
            }
            cudaGetLastError(); /* a refused capture falls back to direct launches */
        }
        if (b->exec) {
            WEDGE_CHECK(cudaGraphLaunch(b->exec, b->stream));
            captured = true;
        }
    }
    if (!captured) {
        const int rc = batch_enqueue(b, t, blocks);
        if (rc)
            return rc;
    }
    WEDGE_CHECK(cudaEventRecord(b->ev[1], b->stream));
    WEDGE_CHECK(cudaStreamSynchronize(b->stream));
    WEDGE_CHECK(cudaGetLastError());
    BShared sh;
    WEDGE_CHECK(cudaMemcpy(&sh, b->d_sh, sizeof(sh), cudaMemcpyDeviceToHost));
    if (stats) {
        memset(stats, 0, sizeof(*stats));
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, b->ev[0], b->ev[1]);
        stats->running_ms = ms;
        stats->rounds = sh.rounds;
        stats->chunks_pulled = sh.chunks_pulled;
        stats->captured = captured ? 1u : 0u;
        stats->blocks = blocks;
        BCtl* c = (BCtl*)malloc(sizeof(BCtl) * b->Q);
        if (!c)
            return WEDGE_ERR_OOM;
        cudaError_t e = cudaMemcpy(c, b->d_ctl, sizeof(BCtl) * b->Q, cudaMemcpyDeviceToHost);
        uint64_t it = 0;
        for (uint32_t i = 0; i < b->Q; ++i)
            it += c[i].iter;
        free(c);
        WEDGE_CHECK(e);
        stats->iterations = it;
    }
    return WEDGE_OK;
}

// The copy to pageable memory faults fresh pages in from the device's side, one
// by one: 82 MB of results into new buffers took 10.8 ms, 4.3 with the pages
// touched by the host first (1.1 where they were there already).
static void touch_pages(void* p, uint64_t bytes)
{
    cudaPointerAttributes pa;
    if (cudaPointerGetAttributes(&pa, p) != cudaSuccess || pa.type != cudaMemoryTypeUnregistered) {
        cudaGetLastError();
        return; /* page-locked, managed or device memory */
    }
    const long page = sysconf(_SC_PAGESIZE);
    volatile unsigned char* q = (volatile unsigned char*)p;
    for (uint64_t i = 0; i < bytes; i += page > 0 ? (uint64_t)page : 4096u)
        q[i] = 0; /* every byte is overwritten by the copy; read first, the pages took 27 ms */
}

extern "C" int wedge_cuda_batch_read_result(wedge_batch_t* b, uint32_t query, void* host_props, uint64_t bytes)
{
    if (!b || query >= b->Q || !host_props)
        return WEDGE_ERR_ARG;
    const BQuery& q = b->h_queries[query];
    const BGraph& G = b->h_graphs[q.graph];
    if (bytes < 8ull * G.V)
        return WEDGE_ERR_ARG;
    WEDGE_CHECK(cudaSetDevice(b->device));
    cudaError_t e = cudaSuccess;
    pthread_mutex_lock(&b->xlock);
    if (!b->xbuf) /* kept: an allocation and its release took 180 of a small read's 200 us */
        e = cudaMalloc((void**)&b->xbuf, 8ull * (b->maxV ? b->maxV : 1));
    if (e == cudaSuccess) {
        batch_export_kernel<<<bgrid(G.V, 256, (uint32_t)b->num_sms * 8), 256, 0, b->stream>>>(G, q, b->xbuf);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) { /* a call that fails leaves the caller's buffer as it is; the pages while the kernel runs */
        touch_pages(host_props, 8ull * G.V);
        e = cudaMemcpyAsync(host_props, b->xbuf, 8ull * G.V, cudaMemcpyDeviceToHost, b->stream);
    }
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(b->stream);
    pthread_mutex_unlock(&b->xlock);
    return e == cudaSuccess ? WEDGE_OK : cuda_status(e);
}

extern "C" int wedge_cuda_batch_iterations(wedge_batch_t* b, uint32_t* host_iterations, uint32_t num_queries)
{
    if (!b || !host_iterations || num_queries < b->Q)
        return WEDGE_ERR_ARG;
    WEDGE_CHECK(cudaSetDevice(b->device));
    BCtl* c = (BCtl*)malloc(sizeof(BCtl) * b->Q);
    if (!c)
        return WEDGE_ERR_OOM;
    const cudaError_t e = cudaMemcpy(c, b->d_ctl, sizeof(BCtl) * b->Q, cudaMemcpyDeviceToHost);
    for (uint32_t i = 0; i < b->Q && e == cudaSuccess; ++i)
        host_iterations[i] = c[i].iter;
    free(c);
    WEDGE_CHECK(e);
    return WEDGE_OK;
}

extern "C" void wedge_cuda_batch_free(wedge_batch_t* b) { batch_release(b); }
