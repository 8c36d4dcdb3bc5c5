// Graph colouring on the device (replaces coloring::colors,
// src/vbd/coloring.rs:5-43, which the reference runs serially on the CPU
// after every detection).
//
// The reference visits vertices 0..n in order and gives each the smallest
// colour not used by an already-coloured neighbour (material graph, contact
// co-vertices, grab). Already-coloured means lower index, so the result is
// the unique solution of  c(v) = mex { c(u) : u ~ v, u < v }.  A plain
// parallel fixed-point iteration of that system needs as many sweeps as the
// longest descending chain, and contact edges between folded layers make
// chains of length ~n; k_color_walk below bounds the work by walking
// index-ordered chunks instead.

#include <algorithm>

#include "color.cuh"

namespace cc {

__device__ __forceinline__ void mark(unsigned long long& mask, uint32_t c, bool& high) {
    if (c < 64) mask |= 1ull << c;
    else high = true;
}

// Greedy rule for one vertex: smallest colour not used by a lower-index
// neighbour (material graph, contact co-vertices, grab). color_of(u) gives a
// neighbour's current colour. One pass over the neighbours per 64 colours; with one
// per colour above 63, two colourings of a stack of 48 layers (85 colours) took
// 2,240 ms instead of 600.
template <class ColorOf>
__device__ __forceinline__ uint32_t greedy_color(const ColorView& g, uint32_t v, ColorOf color_of) {
    const bool in_grab = g.grab_active && (g.grab_v[0] == v || g.grab_v[1] == v || g.grab_v[2] == v);
    for (uint32_t base = 0;; base += 64) {
        unsigned long long mask = 0;
        auto used = [&](uint32_t u) {
            const uint32_t c = color_of(u) - base;
            if (c < 64) mask |= 1ull << c;
        };
        for (uint32_t k = g.lo_off[v]; k < g.lo_off[v + 1]; ++k) used(g.lo[k]);
        for (uint32_t k = g.contacts.inc_off[v]; k < g.contacts.inc_off[v + 1]; ++k) {
            uint32_t c = g.contacts.inc[k];
            uint32_t kind = g.contacts.kind[c];
            uint4 cv = g.contacts.verts[c];
            uint32_t ids[4] = {cv.x, cv.y, cv.z, cv.w};
            uint32_t cnt = kind == 0 ? 2u : (kind == 1 ? 3u : 4u);
            for (uint32_t j = 0; j < cnt; ++j)
                if (ids[j] < v) used(ids[j]);
        }
        if (in_grab)
            for (int j = 0; j < 3; ++j)
                if (g.grab_v[j] < v) used(g.grab_v[j]);
        if (~mask != 0ull) return min(base + (uint32_t)__ffsll((long long)~mask) - 1, (uint32_t)kMaxColors - 1);
        if (base + 64 >= kMaxColors) return kMaxColors - 1;
    }
}

// Distinct lower neighbours of every vertex, one row per vertex, built by the
// whole GPU before the walk (k_color_rows), so that the walk's one block reads
// each neighbour once: in layered cloth a vertex has the same neighbour in
// many contacts (the 201 x 311 roll: 40 contacts a vertex, ~120 entries, ~20
// distinct lower neighbours).
constexpr int kChunk = 1024;       // vertices of one walk step
constexpr int kRowSlots = 64;      // distinct lower neighbours a row can hold
constexpr uint32_t kRowSlow = ~0u;  // count word of a vertex that takes the full rule instead
constexpr int kRowLanes = 8;       // threads per row

struct ColorRows {
    uint32_t* adj;  // rows: neighbours below the vertex's chunk, then those in it (outside its 32-group)
    // [n] .x first entry of the row / 4; .y entries below the chunk | in the chunk << 16, or kRowSlow;
    // .z lower neighbours among the vertex's 32-aligned group, one bit each; .w unused
    uint4* head;
    uint32_t* dirty;  // [n / 32] one bit per vertex whose rule may not hold
};
// First entry of v's row, 16-byte aligned: a vertex has at most its material
// neighbours, 3 vertices per contact and 2 of the grab; 3 more are lost to the
// alignment.
__host__ __device__ __forceinline__ size_t row_bound(size_t lo, size_t inc, size_t v) { return lo + 3 * inc + 5 * v; }
__device__ __forceinline__ size_t row_start(const ColorView& g, uint32_t v) {
    return (row_bound(g.lo_off[v], g.contacts.inc_off[v], v) + 3) & ~(size_t)3;
}

// Rows, and the lowest vertex whose rule fails for the current colouring (as n
// less it in `first`, 0 if there is none). Eight threads per vertex put its lower neighbours into a 64-slot
// hash set in shared memory. Bound by the latency of inc -> contact -> colour. Where
// the row overflows they mark the colours of all the neighbours between them (a hub
// of 3,000 neighbours as the last vertex of its disc: a colouring that finds nothing
// to change 1.19 -> 0.28 ms against probing a full set and one thread's greedy rule).
__global__ void __launch_bounds__(128) k_color_rows(ColorView g, ColorRows r, const uint16_t* col, unsigned int* first) {
    __shared__ uint32_t slots[128 / kRowLanes][kRowSlots];
    __shared__ uint32_t group_bits[128 / kRowLanes];
    constexpr uint32_t kEmpty = ~0u;
    const uint32_t lane = threadIdx.x & (kRowLanes - 1), row = threadIdx.x / kRowLanes;
    const unsigned gmask = ((1u << kRowLanes) - 1u) << ((threadIdx.x & 31u) & ~(unsigned)(kRowLanes - 1));
    uint32_t* slot = slots[row];
    constexpr uint32_t kPer = 128 / kRowLanes;
    for (uint32_t v = blockIdx.x * kPer + row; v < g.n; v += gridDim.x * kPer) {  // whole groups step together
        for (int k = lane; k < kRowSlots; k += kRowLanes) slot[k] = kEmpty;
        if (lane == 0) group_bits[row] = 0u;
        __syncwarp(gmask);
        // more material neighbours (all distinct) than slots and the group hold
        bool full = g.lo_off[v + 1] - g.lo_off[v] > kRowSlots + 31;
        auto insert = [&](uint32_t u) {
            if (u >= v || full) return;
            if ((u >> 5) == (v >> 5)) {
                atomicOr(&group_bits[row], 1u << (u & 31u));
                return;
            }
            uint32_t h = (u * 2654435761u) >> 26;
            for (int tries = 0; tries < kRowSlots; ++tries, h = (h + 1) & (kRowSlots - 1)) {
                const uint32_t old = atomicCAS(&slot[h], kEmpty, u);
                if (old == kEmpty || old == u) return;
            }
            full = true;
        };
        // the lane's share of v's neighbours
        auto share = [&](auto take) {
            for (uint32_t k = g.lo_off[v] + lane; k < g.lo_off[v + 1]; k += kRowLanes) take(g.lo[k]);
            for (uint32_t k = g.contacts.inc_off[v] + lane; k < g.contacts.inc_off[v + 1]; k += kRowLanes) {
                uint32_t c = g.contacts.inc[k];
                uint32_t kind = g.contacts.kind[c];
                uint4 cv = g.contacts.verts[c];
                take(cv.x);
                take(cv.y);
                if (kind > 0) take(cv.z);
                if (kind > 1) take(cv.w);
            }
            if (lane == 0 && g.grab_active && (g.grab_v[0] == v || g.grab_v[1] == v || g.grab_v[2] == v))
                for (int j = 0; j < 3; ++j) take(g.grab_v[j]);
        };
        if (!full) share(insert);
        __syncwarp(gmask);
        full = __any_sync(gmask, full);
        const uint32_t bits = group_bits[row];
        const uint32_t base = v & ~(uint32_t)(kChunk - 1);
        // this lane's slots: those below the chunk, then those in it
        uint32_t n_out = 0, n_in = 0;
        unsigned long long mask = 0;
        bool high = false;
        if (full) {  // no row: every neighbour's colour, so that a hub of thousands is not one thread's work
            share([&](uint32_t u) { if (u < v) mark(mask, col[u], high); });
        } else {
            for (int k = lane; k < kRowSlots; k += kRowLanes) {
                const uint32_t u = slot[k];
                if (u == kEmpty) continue;
                if (u < base) ++n_out;
                else ++n_in;
                mark(mask, col[u], high);
            }
            for (uint32_t b = lane; b < 32; b += kRowLanes)
                if (bits >> b & 1u) mark(mask, col[(v & ~31u) + b], high);
        }
        uint32_t o0 = n_out, i0 = n_in;  // inclusive prefix over the group's lanes
        for (int o = 1; o < kRowLanes; o <<= 1) {
            const uint32_t a = __shfl_up_sync(gmask, o0, o, kRowLanes), c = __shfl_up_sync(gmask, i0, o, kRowLanes);
            if ((int)lane >= o) {
                o0 += a;
                i0 += c;
            }
        }
        const uint32_t outs = __shfl_sync(gmask, o0, kRowLanes - 1, kRowLanes);
        const uint32_t ins = __shfl_sync(gmask, i0, kRowLanes - 1, kRowLanes);
        o0 -= n_out;
        i0 -= n_in;
        if (!full) {
            uint32_t* out = r.adj + row_start(g, v);
            for (int k = lane; k < kRowSlots; k += kRowLanes) {
                const uint32_t u = slot[k];
                if (u == kEmpty) continue;
                if (u < base) out[o0++] = u;
                else out[outs + i0++] = u;
            }
        }
        for (int o = kRowLanes / 2; o > 0; o >>= 1) mask |= __shfl_xor_sync(gmask, mask, o, kRowLanes);
        high = __any_sync(gmask, high);
        if (lane == 0) {
            r.head[v] = make_uint4((uint32_t)(row_start(g, v) / 4), full ? kRowSlow : (outs | ins << 16), bits, 0u);
            const uint32_t c = (high || ~mask == 0ull) ? greedy_color(g, v, [&](uint32_t u) { return (uint32_t)col[u]; })
                                                       : (uint32_t)__ffsll((long long)~mask) - 1;
            if (c != col[v]) {
                atomicMax(first, g.n - v);
                atomicOr(&r.dirty[v >> 5], 1u << (v & 31u));
            }
        }
        __syncwarp(gmask);  // the slots are reused
    }
}

// Exact sequential-greedy colouring by one CTA: chunks of kChunk consecutive
// vertices are visited in index order, so every lower neighbour below the
// current chunk is already final; inside the chunk the greedy rule is iterated
// (rounds of one barrier, the chunk's colours double-buffered) until no colour
// changes. Each thread has one vertex. Once per chunk it folds the colours of
// its row's neighbours below the chunk into a 64-bit mask; a round adds the
// in-chunk neighbours of other warps from the last round's colours, and then
// each warp settles its own 32 vertices exactly (settle_chain, settle). A change
// therefore crosses a whole warp per round, and after round r the chunk's first
// r warps are final, so 32 rounds and one that finds no change bound the loop.
// From the second round on a warp whose neighbour warps did not change in the
// last one skips the evaluation: a round of all 32 warps is bound by instruction
// issue, one of a few by their latency alone. A vertex without a row, or with a
// colour >= 64 around it, takes the full rule (greedy_color) once a round
// instead; its chunk then needs at most kChunk + 1 rounds.
//
// The walk starts at the chunk of n - `first[0]`, the lowest vertex whose rule
// does not hold for the previous colouring (k_color_rows): every vertex
// below it already satisfies the rule against final lower neighbours, so it
// is final too. When the whole colouring fits (n <= kSmemColors) it is kept
// in shared memory for the walk.
//
// From there on only chunks with a vertex in `dirty` are visited: those whose
// rule failed for the previous colouring, and the higher neighbours of each
// vertex whose colour the walk has changed. Once a chunk changed more than
// kFewChanges vertices, or fewer than a fifth of the chunks were left out, all the
// following ones are visited: such changes run on through the mesh (a crumpling
// sheet, a roll), and the lookup of changed vertices' neighbours and the rows
// loaded on demand (~2 us a chunk) would save nothing. On the 40k-vertex garment,
// whose contacts change by a few between refreshes, it leaves out 40 % of the
// chunks: 0.22 -> 0.17 ms a colouring (host clock, with its sort and heads).
//
// What bounds it: the chain of chunks, each a row load, a gather of final
// colours and two to three barrier rounds; the next chunk's row is loaded
// before this one's rounds.
//
// settle: the rule for a warp's 32 consecutive vertices, each with the mask m
// of the colours of its neighbours outside the group and the bits wmask of its
// lower neighbours in it; c holds the current colours and receives the exact
// ones. At most kWarpTries evaluations of all lanes at once, each against the
// current colours (one suffices where nothing changes), else lane by lane.
// Returns false if a lane meets a colour that M has no bit for.
constexpr int kWarpTries = 3;
template <class M>
__device__ __forceinline__ bool settle(M m, uint32_t wmask, uint32_t steps, bool live, uint32_t& c) {
    constexpr uint32_t kBits = sizeof(M) == 8 ? 64 : 31;  // 32-bit masks keep bit 31 for the colours above 30
    auto mex = [](M x) { return sizeof(M) == 8 ? (uint32_t)__ffsll((long long)~x) - 1 : (uint32_t)__ffs((int)~x) - 1; };
    for (int tries = 0; tries < kWarpTries; ++tries) {
        M mw = m;
        bool out = false;
        uint32_t b = wmask;
        for (uint32_t k = 0; k < steps; ++k, b &= b - 1u) {
            const uint32_t cu = __shfl_sync(0xffffffffu, c, b ? __ffs((int)b) - 1 : 0);
            if (b && cu < kBits) mw |= (M)1 << cu;
            out = out || (b && cu >= kBits);
        }
        if (__any_sync(0xffffffffu, live && (out || mex(mw) >= kBits))) return false;
        const uint32_t cn = mex(mw);
        const bool same = !__any_sync(0xffffffffu, live && cn != c);
        if (live) c = cn;
        if (same) return true;
    }
    // lane k's colour is exact once those of lanes 0..k-1 are; a lane out of bits is found at the end
    M mw = m;
    for (uint32_t b = __reduce_or_sync(0xffffffffu, wmask); b; b &= b - 1u) {
        const uint32_t k = __ffs((int)b) - 1;
        const uint32_t ck = __shfl_sync(0xffffffffu, mex(mw), k);
        if ((wmask >> k & 1u) && ck < kBits) mw |= (M)1 << ck;
    }
    if (__any_sync(0xffffffffu, live && mex(mw) >= kBits)) return false;
    if (live) c = mex(mw);
    return true;
}

// The same where every lane's only neighbour in its group is the lane before it
// (or none), as in a row-major grid whose rows are longer than a warp: lane k's
// rule is then a function of one colour, x -> b if x == a else a, with a and b
// the first and second colour free of m. Such functions compose into (key, value
// if equal, value if not), so a prefix scan of five shuffles gives every lane's
// colour, ~250 cycles where lane by lane takes ~1,900. m: colours below 31.
// Returns false if a lane's colour may exceed 30.
__device__ __forceinline__ bool settle_chain(uint32_t m, uint32_t wmask, bool live, uint32_t& c) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t fa = ~m & (m + 1u), rest = m | fa, fb = ~rest & (rest + 1u);  // lowest clear bits
    const uint32_t a = (uint32_t)__ffs((int)fa) - 1, b = (uint32_t)__ffs((int)fb) - 1;
    if (__any_sync(0xffffffffu, live && rest >= 0x7fffffffu)) return false;  // the second free colour is above 30
    uint32_t key = wmask ? a : 255u, eq = wmask ? b : a, ne = a;
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, key | eq << 8 | ne << 16, d);
        if (lane >= (uint32_t)d) {
            const uint32_t oe = o >> 8 & 255u, on = o >> 16 & 255u;
            const uint32_t e = oe == key ? eq : ne, n = on == key ? eq : ne;
            key = o & 255u;
            eq = e;
            ne = n;
        }
    }
    if (live) c = ne;  // lane 0's function is constant, and so is every composition from it on
    return true;
}

// Marks the neighbours of v from `next` on; a call, so that its registers stay
// out of the walk's.
__device__ __noinline__ void mark_higher(const ColorView& g, uint32_t* dirty, uint32_t v, uint32_t next) {
    auto mark_dirty = [&](uint32_t u) {
        if (u >= next && u < g.n) atomicOr(&dirty[u >> 5], 1u << (u & 31u));
    };
    const uint4 h = g.head[2 * (size_t)v];
    for (uint32_t k = 0; k < h.y; ++k) mark_dirty(g.nb[h.x + k]);
    for (uint32_t k = g.contacts.inc_off[v]; k < g.contacts.inc_off[v + 1]; ++k) {
        const uint32_t c = g.contacts.inc[k];
        const uint32_t kind = g.contacts.kind[c];
        const uint4 cv = g.contacts.verts[c];
        mark_dirty(cv.x);
        mark_dirty(cv.y);
        if (kind > 0) mark_dirty(cv.z);
        if (kind > 1) mark_dirty(cv.w);
    }
    if (g.grab_active && (g.grab_v[0] == v || g.grab_v[1] == v || g.grab_v[2] == v))
        for (int j = 0; j < 3; ++j) mark_dirty(g.grab_v[j]);
    __threadfence_block();
}

constexpr int kAhead = 8;       // row entries loaded ahead
constexpr uint32_t kSmemColors = 90 * 1024;  // 180 KB of uint16 colours
// Dynamic shared memory: the colours (n <= kSmemColors) and, in what is left, a
// row of kChunk chunk-local indices for each of `inner_cap` in-chunk
// neighbours per vertex (17 at n = 92,160, 32 below 76k vertices and where the
// colours stay in global memory); further neighbours are read from the row. Up
// to four chunks take 12, which keeps the block below 48 KB: a step of a few
// dozen launches feels the SM's change to a large shared-memory carve-out.
constexpr int kFewChanges = 32;
constexpr int kMaxInner = 32;
constexpr size_t kWalkSmem = 214 * 1024;  // + 12 KB static
inline int walk_inner_cap(uint32_t n, size_t color_bytes) {
    if (n <= 4 * kChunk) return 12;
    return (int)std::min<size_t>(kMaxInner, (kWalkSmem - color_bytes) / (kChunk * sizeof(uint16_t)));
}
__global__ void __launch_bounds__(kChunk) k_color_walk(const __grid_constant__ ColorView g, ColorRows r, uint16_t* col_g,
                                                      const unsigned int* first, unsigned int* rounds_out,
                                                      unsigned int* err, uint32_t inner_cap) {
    extern __shared__ uint16_t walk_s[];
    uint16_t* inner = walk_s + threadIdx.x;  // [inner_cap][kChunk], this thread's column
    uint16_t* col_s = walk_s + inner_cap * kChunk;
    __shared__ uint16_t chunk_col[2][kChunk];   // the chunk's colours: the last round's and this one's
    // bit c of a colour c < 31, bit 31 for the others: what most rounds need
    __shared__ uint32_t chunk_bit[2][kChunk];
    __shared__ unsigned next_dirty;  // first dirty word of the scanned range
    __shared__ unsigned warp_changed[3];        // warps with a changed colour: this round's, the last one's, the next one's
    const uint32_t start = g.n - *first;
    const uint32_t t = threadIdx.x;
    if (start >= g.n) {  // already a fixed point
        if (t == 0) *rounds_out = 0;
        return;
    }
    const uint32_t chunk0 = start & ~(uint32_t)(kChunk - 1);
    const bool smem = g.n <= kSmemColors;
    uint16_t* col = col_g;
    if (smem) {
        for (uint32_t i = t; i < g.n; i += kChunk) col_s[i] = col_g[i];
        col = col_s;
    }
    // this chunk's rows: their first entries loaded one chunk ahead, their heads two
    uint4 head = make_uint4(0u, 0u, 0u, 0u), next_head = head;
    uint4 ahead_a = head, ahead_b = head;
    auto load_head = [&](uint32_t v) { return v < g.n ? r.head[v] : make_uint4(0u, 0u, 0u, 0u); };
    auto load_row = [&](uint4 h) {
        // 16-byte aligned; a row may have fewer than kAhead entries, the buffer is padded past its end
        const uint4* row = reinterpret_cast<const uint4*>(r.adj) + h.x;
        ahead_a = row[0];
        ahead_b = row[1];
    };
    head = load_head(chunk0 + t);
    load_row(head);
    if (t < 3) warp_changed[t] = 0u;
    __syncthreads();
    unsigned int rounds = 0;
    // one chunk; `ahead_next`: load the following chunk's rows meanwhile. Whether the thread's colour changed.
    auto visit_chunk = [&](uint32_t base, bool ahead_next) {
        const uint32_t v = base + t;
        const bool live = v < g.n;
        const bool slow = head.y == kRowSlow;
        const uint32_t n_out = slow ? 0u : (head.y & 0xffffu), n_in = slow ? 0u : (head.y >> 16);
        const uint32_t n_row = n_out + n_in, n_kept = min(n_in, inner_cap);
        const uint32_t wmask = head.z;
        const uint32_t* my_row = r.adj + 4 * (size_t)head.x;
        const uint32_t steps = __reduce_max_sync(0xffffffffu, (uint32_t)__popc(wmask));
        // final colours below the chunk into a mask, in-chunk neighbours into shared memory
        unsigned long long outer = 0;
        bool outer_high = slow;
        unsigned depends = slow ? ~0u : 0u;  // warps of this chunk that the colours depend on (all, without a row)
        auto take = [&](uint32_t k, uint32_t u) {
            if (k < n_out) {
                mark(outer, col[u], outer_high);
            } else {
                const uint32_t i = u - base, j = k - n_out;
                if (j < n_kept) inner[j * kChunk] = (uint16_t)i;
                depends |= 1u << (i >> 5);
            }
        };
        const uint32_t ahead[kAhead] = {ahead_a.x, ahead_a.y, ahead_a.z, ahead_a.w,
                                        ahead_b.x, ahead_b.y, ahead_b.z, ahead_b.w};
#pragma unroll
        for (uint32_t k = 0; k < kAhead; ++k)
            if (k < n_row) take(k, ahead[k]);
#pragma unroll 4
        for (uint32_t k = kAhead; k < n_row; ++k) take(k, my_row[k]);
        depends = __reduce_or_sync(0xffffffffu, depends);
        const bool chain = __all_sync(0xffffffffu, (wmask & ~(t & 31u ? 1u << ((t & 31u) - 1u) : 0u)) == 0u);
        const uint32_t outer32 = (uint32_t)(outer & 0x7fffffffull) | ((outer >> 31) != 0ull || outer_high ? 1u << 31 : 0u);
        uint32_t cur = live ? col[v] : 0u;
        auto bit_of = [](uint32_t c) { return 1u << min(c, 31u); };
        chunk_col[0][t] = (uint16_t)cur;
        chunk_bit[0][t] = bit_of(cur);
        if (ahead_next) {
            head = next_head;
            if (base + kChunk < g.n) load_row(head);
            next_head = load_head(v + 2 * kChunk);
        }
        __syncthreads();
        const uint32_t before = cur;
        int rd = 0, buf = 0;
        bool again = true;  // this warp has not settled: the first round, or it took the full rule
        uint32_t m_last = 0;
        for (; rd <= kChunk + 1; ++rd) {
            const uint16_t* now = chunk_col[buf];
            auto color_of = [&](uint32_t u) { return (uint32_t)(u >= base ? now[u - base] : col[u]); };
            uint32_t c = cur;
            const unsigned slot = rounds % 3;  // goes on over the chunks
            if (t == 0) warp_changed[(slot + 1) % 3] = 0u;  // last read in the last round
            if (again || (depends & warp_changed[(slot + 2) % 3])) {
                const uint32_t* bits = chunk_bit[buf];
                uint32_t m = outer32;
#pragma unroll 4
                for (uint32_t j = 0; j < n_kept; ++j) m |= bits[inner[j * kChunk]];
                for (uint32_t j = n_kept; j < n_in; ++j) m |= bits[my_row[n_out + j] - base];
                // nothing to do where the warp had settled and no lane's outside mask moved
                const bool wide = __any_sync(0xffffffffu, live && m >> 31);
                const bool moved = again || wide || __any_sync(0xffffffffu, live && m != m_last);
                m_last = m;
                bool full = false;
                unsigned long long m64 = outer;
                bool high = outer_high;
                if (moved && (wide || !(chain ? settle_chain(m, wmask, live, c)
                                              : settle<uint32_t>(m, wmask, steps, live, c)))) {
                    // colours above 30 around: 64-bit masks
                    for (uint32_t j = 0; j < n_in; ++j)
                        mark(m64, now[j < n_kept ? (uint32_t)inner[j * kChunk] : my_row[n_out + j] - base], high);
                    c = cur;
                    full = __any_sync(0xffffffffu, live && high) ||
                           !settle<unsigned long long>(m64, wmask, steps, live, c);
                }
                if (full && live) {
                    // a lane has no row or meets colours >= 64: the whole warp takes the rule on the last round's colours
                    unsigned long long ml = m64;
                    bool hl = high;
                    for (uint32_t b = wmask; b; b &= b - 1u) mark(ml, now[(t & ~31u) + __ffs((int)b) - 1], hl);
                    c = (hl || ~ml == 0ull) ? greedy_color(g, v, color_of) : (uint32_t)__ffsll((long long)~ml) - 1;
                }
                again = full;
            }
            const bool changed = live && c != cur;
            if (changed) {
                cur = c;
                col[v] = (uint16_t)c;
            }
            chunk_col[buf ^ 1][t] = (uint16_t)cur;
            chunk_bit[buf ^ 1][t] = bit_of(cur);
            buf ^= 1;
            ++rounds;
            if (__any_sync(0xffffffffu, changed) && (t & 31u) == 0) atomicOr(&warp_changed[slot], 1u << (t >> 5));
            __syncthreads();
            if (!warp_changed[slot]) break;
        }
        if (rd > kChunk + 1 && t == 0) atomicOr(err, 1u);
        return cur != before;
    };
    // dirty chunks only, while they change little
    uint32_t base = chunk0;
    bool many = false;
    for (uint32_t visited = 1, left_out = 0; base < g.n && !many; ++visited) {
        if (t == 0) next_dirty = ~0u;
        const bool changed = visit_chunk(base, false);
        uint32_t next = base + kChunk;
        many = __syncthreads_count(changed) > kFewChanges;
        if (!many) {
            if (changed) mark_higher(g, r.dirty, base + t, next);  // their rules may fail now
            __syncthreads();
            // the next chunk with a dirty vertex, 32 chunks (one word a thread) at a time
            for (; next < g.n; next += 32 * kChunk) {
                const uint32_t w = next / 32 + t;
                if (w < (g.n + 31) / 32 && __ldcg(&r.dirty[w])) atomicMin(&next_dirty, t);
                __syncthreads();
                const unsigned found = next_dirty;
                __syncthreads();  // every thread has read it before the next range writes it
                if (found != ~0u) {
                    next += found / 32 * kChunk;
                    break;
                }
            }
            left_out += (next - base) / kChunk - 1;
            many = visited >= 6 && 4 * left_out < visited;
        }
        base = next;
        head = load_head(base + t);
        if (base < g.n) load_row(head);
    }
    // then every chunk
    next_head = load_head(base + kChunk + t);
    for (; base < g.n; base += kChunk) visit_chunk(base, true);
    if (smem)
        for (uint32_t i = chunk0 + t; i < g.n; i += kChunk) col_g[i] = col_s[i];
    if (t == 0) *rounds_out = rounds;
}

// Vertices per colour: counted per block in shared memory (atomics on a few
// global counters took 23 us on the fold, 322 us on a 1024 x 1024 sheet).
__global__ void __launch_bounds__(256) k_color_count(uint32_t n, const uint16_t* col, uint32_t* counts) {
    constexpr uint32_t kLocal = 64;
    __shared__ uint32_t local[kLocal];
    if (threadIdx.x < kLocal) local[threadIdx.x] = 0u;
    __syncthreads();
    const uint32_t stride = gridDim.x * 256;
    for (uint32_t v0 = blockIdx.x * 256; v0 < n; v0 += stride) {
        const uint32_t v = v0 + threadIdx.x;
        const uint32_t c = v < n ? col[v] : ~0u;
        const unsigned same = __match_any_sync(0xffffffffu, c);
        if (v < n && (threadIdx.x & 31u) == (uint32_t)__ffs((int)same) - 1) {
            const uint32_t k = (uint32_t)__popc(same);
            if (c < kLocal) atomicAdd(&local[c], k);
            else atomicAdd(&counts[c], k);
        }
    }
    __syncthreads();
    if (threadIdx.x < kLocal && local[threadIdx.x]) atomicAdd(&counts[threadIdx.x], local[threadIdx.x]);
}

__global__ void k_iota(uint32_t n, uint32_t* out) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) out[v] = v;
}

void Coloring::init(uint32_t n, uint64_t lo_total, cudaStream_t s) {
    n_ = n;
    lo_total_ = lo_total;
    row_head_.reserve(n);
    a_.reserve(n);
    b_.reserve(n);
    order_.reserve(n);
    iota_.reserve(n);
    words_.reserve(kWords + ((size_t)n + 31) / 32);
    words_h_.reserve(kWords);
    CC_CUDA(cudaMemsetAsync(a_.ptr, 0, n * sizeof(uint16_t), s));
    if (n) k_iota<<<grid_for(n, 256), 256, 0, s>>>(n, iota_.ptr);
    CC_CUDA(cudaGetLastError());
    cur_ = a_.ptr;
}

void Coloring::compute(const ColorView& view, cudaStream_t s) {
    uint32_t n = n_;
    if (n == 0) {
        n_colors_ = 0;
        offsets_h_.assign(1, 0);
        return;
    }
    // the chunked walk updates the previous colouring in place, from the
    // first vertex the probe finds out of date
    CC_CUDA(cudaMemsetAsync(words_.ptr, 0, (kWords + ((size_t)n + 31) / 32) * sizeof(uint32_t), s));
    uint32_t* const counts = words_.ptr + 4;
    adj_.reserve(row_bound(lo_total_, view.n_incident, n) + 3 + kAhead);
    ColorRows rows{adj_.ptr, row_head_.ptr, words_.ptr + kWords};
    k_color_rows<<<grid_for((size_t)n * kRowLanes, 128), 128, 0, s>>>(view, rows, cur_, words_.ptr + 2);
    const size_t color_bytes = n <= kSmemColors ? n * sizeof(uint16_t) : 0;
    const int inner_cap = walk_inner_cap(n, color_bytes);
    const size_t smem = inner_cap * kChunk * sizeof(uint16_t) + color_bytes;
    static std::atomic<uint64_t> raised{0};  // devices on which the limit is raised
    allow_dynamic_smem_once(k_color_walk, kWalkSmem, raised);
    k_color_walk<<<1, kChunk, smem, s>>>(view, rows, cur_, words_.ptr + 2, words_.ptr, words_.ptr + 1,
                                         (uint32_t)inner_cap);
    launches_ += 2;
    CC_CUDA(cudaGetLastError());
    k_color_count<<<std::min(grid_for(n, 256), 148 * 2), 256, 0, s>>>(n, cur_, counts);
    CC_CUDA(cudaMemcpyAsync(words_h_.ptr, words_.ptr, kWords * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    CC_CUDA(cudaStreamSynchronize(s));
    const uint32_t* counts_h = words_h_.ptr + 4;
    last_iterations_ = words_h_.ptr[0];
    if (words_h_.ptr[1]) throw Failure{CC_ERR_CUDA, "colouring rounds exceeded their bound"};
    n_colors_ = 0;
    for (uint32_t c = 0; c < kMaxColors; ++c)
        if (counts_h[c]) n_colors_ = c + 1;
    if (n_colors_ >= kMaxColors) throw Failure{CC_ERR_CUDA, "colour limit exceeded"};
    offsets_h_.assign(n_colors_ + 1, 0);
    for (uint32_t c = 0; c < n_colors_; ++c) offsets_h_[c + 1] = offsets_h_[c] + counts_h[c];
    // vertices grouped by colour, in index order within a colour (a stable
    // sort on the colour bits): a warp's vertices are neighbours in the mesh
    // order, so the sweep's gathers share cache lines. The order within a
    // colour does not change any result (no two vertices of a colour interact).
    int bits = 1;
    while ((1u << bits) < n_colors_) ++bits;
    launches_ += sorter_.sort_pairs(cur_, b_.ptr, iota_.ptr, order_.ptr, n, bits, s, error_word_, DERR_SORT_WAIT);
    CC_CUDA(cudaGetLastError());
}

void Coloring::download(std::vector<uint32_t>& colors) {
    std::vector<uint16_t> c(n_);
    if (n_) CC_CUDA(cudaMemcpy(c.data(), cur_, n_ * sizeof(uint16_t), cudaMemcpyDeviceToHost));
    colors.assign(c.begin(), c.end());
}

}  // namespace cc
