// Kernels and host orchestration of the GB300 explicit-MPM substep (templated on the scalar type).
// Included by engine_f32.cu and engine_f64.cu, which instantiate one precision each.
//
// One substep (MpmSimulationBase::advanceOneTimeStep, MpmSimulationBase.cpp:262-357, with the
// AnisoFractureSimulation particlesToGrid override, AnisoFractureSimulation.h:129-141):
//   1. sort      the particle keys written by the previous G2P (or k_keys) merged into the previous order
//                (incremental sort; a radix sort after loads and aborts)
//   2. groups    the sorted range of every (scene, SPGrid page)
//   3. activate  every group inserts its page and the 7 pages at +1 block into a hash table; new
//                entries get a grid slot (MpmGrid::pollute, MpmGrid.h:153-193); in one kernel with the merge
//   4. p2g       one CTA per work item (a group, or a piece of a large one): stress V0*tau(F, g(d)) + APIC scatter of m, m v + m C (x_i - x_p),
//                -V0 tau grad w and the phase-field pair (d w, w) into a shared node tile, then
//                vector atomics into the 8 neighbouring grid blocks (MpmSimulationBase.cpp:669-855,
//                FBasedMpmForceHelper.cpp:43-63, AnisoFractureSimulation.h:161-176)
//   5. grid      v = m v / m, v += g dt + f dt / m, half-space BCs, phase field normalised; clears the
//                accumulators and the hash table for the next substep (MpmSimulationBase.cpp:655-666,
//                1179-1228, AnisoFractureSimulation.h:177-179)
//   6. g2p       one CTA per work item: gather v, C (APIC/RPIC blend), grad v and the damage Laplacian,
//                damage update with the old F, F <- (I + dt grad v) F, x += dt v, CFL / finiteness /
//                domain checks, next key; writes the particle to its sorted slot of the other buffer
//                (MpmSimulationBase.cpp:1269-1515, FBasedMpmForceHelper.cpp:95-108,
//                AnisoFractureSimulation.h:182-283)
//   7. end       time += dt per scene, substep counter (by the last CTA of G2P)
#pragma once
#include "common.cuh"
#include "engine.h"
#include "physics.cuh"
#include "tma.cuh"

#include <cub/cub.cuh>
#include <cuda_runtime.h>
#include <thrust/iterator/counting_iterator.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

namespace zr {

constexpr int NACC = 6; // m, m v + dt f (3), d w, w
constexpr int NVEL = 4; // v_new (3), normalised phase field
constexpr uint64_t HASH_EMPTY = ~0ULL;
constexpr int HASH_PROBES = 64;

// particle pool: field k of storage slot i at f[k * stride + i]
// P_MDT: the implicit damage solve's D~ history; P_DRV: the damage drive of the particle's current F (implicit
// scenes), kept by G2P and refilled after state writes
template <class T>
constexpr uint32_t P2G_CHUNK = sizeof(T) == 4 ? 512 : 256; // particles P2G stages at once: a whole block at 8 per cell
enum { P_X = 0, P_V = 3, P_C = 6, P_F = 15, P_M = 24, P_V0 = 25, P_D = 26, P_SC = 27, P_MDT = 28, P_DRV = 29, P_NF = 30 };

template <class T>
struct Pool {
    T* f;
    uint32_t* pid; // original index (low index_bits) | material << index_bits
    int64_t stride;
};

struct KeyLayout {
    int ib; // bits of the original particle index
    int cp; // bits of (offset >> data_bits): page and in-block cell
    int sb; // bits of the scene slot
    int block_bits;
    int wide; // keys are stored as 64-bit words; 0: as 32-bit words (total() <= 32), a third less sort traffic
    __host__ __device__ int total() const { return sb + cp + ib; }
    __host__ __device__ uint64_t at(const uint64_t* k, uint32_t i) const { return wide ? k[i] : (uint64_t)reinterpret_cast<const uint32_t*>(k)[i]; }
    __host__ __device__ void put(uint64_t* k, uint32_t i, uint64_t v) const
    {
        if (wide)
            k[i] = v;
        else
            reinterpret_cast<uint32_t*>(k)[i] = (uint32_t)v;
    }
    __host__ __device__ uint32_t scene(uint64_t k) const { return (uint32_t)(k >> (cp + ib)); }
    __host__ __device__ uint64_t page(uint64_t k) const { return (k >> (ib + block_bits)) & ((1ULL << (cp - block_bits)) - 1); }
    __host__ __device__ uint64_t group(uint64_t k) const { return k >> (ib + block_bits); }
    __host__ __device__ uint32_t orig(uint64_t k) const { return (uint32_t)(k & ((1ULL << ib) - 1)); }
};

// per-scene state of the implicit damage solve's conjugate gradients (ConjugateGradient.h), kept on the device
struct CgScalars {
    double zr; // r . z
    double zr_new;
    double pAp; // p . A p
    double tol; // min(|r0|_z, 1e-6)
    double alpha, beta; // step length; of the next search direction
    int32_t iter, done;
};

template <class T>
struct StepArgs {
    const uint64_t* keys_sorted;
    const uint32_t* vals_sorted;
    uint64_t* keys_next;
    Pool<T> pin, pout;
    uint32_t* g_start; // group heads after a full sort, in key order
    int32_t* g_nbr; // per group, at its first item's number: hash positions of its block and the +1 neighbours
    uint4* item; // work items of P2G and G2P: first sorted index, one past the last, the group's first item
    uint32_t item_max; // particles of an item (a group of up to 5/4 of it stays whole)
    int32_t* i_slot; // per item: grid slots of its block and the +1 neighbours (from P2G's set-up or k_nbr on)
    unsigned long long* open; // per hash position: a group's start or end while the other comes from another tile (see range_event)
    T* pay; // P2G payload, Pay<T>::N fields of pstride elements (also the implicit damage solve's particle scratch)
    int64_t pstride;
    T* cg; // implicit damage solve: CG_NF node vectors of b_cap * nodes
    CgScalars* cgs; // per scene
    uint64_t* b_key;
    T* acc;
    T* vel;
    uint64_t* h_keys;
    int32_t* h_vals;
    uint32_t h_mask;
    SceneParams<T>* scenes;
    double* grid_mass; // per scene, refreshed every substep
    uint32_t* sort_zero; // the incremental sort's counters, zero at the start of a substep
    uint32_t sort_zero_n; // words
    DevStatus* st;
    uint32_t n_total;
    uint32_t b_cap;
    int n_scenes;
    uint32_t opts; // OPT_* bits
    KeyLayout kl;
};
// OPT_PREFETCH: P2G prefetches the state of the groups ahead into L2
enum : uint32_t { OPT_PREFETCH = 1u };

__host__ __device__ inline uint64_t hash64(uint64_t k)
{
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdULL;
    k ^= k >> 33;
    k *= 0xc4ceb9fe1a85ec53ULL;
    k ^= k >> 33;
    return k;
}

__device__ inline void raise_flag(DevStatus* st, uint32_t f)
{
    uint32_t old = atomicOr(&st->flags, f | ((f & ABORTING) ? FLAG_ABORT : 0u));
    if ((f & ABORTING) && !(old & FLAG_ABORT)) atomicExch(&st->abort_step, (int32_t)st->step);
}

// an internal consistency check failed: record the first check's code, count, abort the substep
__device__ inline void check_failed(DevStatus* st, uint32_t code)
{
    atomicCAS(&st->check_code, 0u, code);
    atomicAdd(&st->check_count, 1u);
    raise_flag(st, FLAG_CHECK);
}

__device__ inline bool aborted(const DevStatus* st) { return (*(volatile const uint32_t*)&st->flags & FLAG_ABORT) != 0; }

// the same decision for every thread of the CTA (kernels with barriers or full-warp shuffles must not
// let some threads leave early)
__device__ inline bool aborted_cta(const DevStatus* st) { return __syncthreads_or(aborted(st) ? 1 : 0) != 0; }

// ---------------------------------------------------------------------------------------------------
// keys of the current particle positions (used after a load or a host upload; afterwards G2P writes
// the keys of the next substep). Also checks that every base node lies in its scene's domain. With a sort base (the
// 32-bit keys the storage order was sorted by) the particles whose key differs from it are counted into max_movers.
// ---------------------------------------------------------------------------------------------------
template <class T>
__global__ void k_keys(Pool<T> p, const SceneParams<T>* scenes, int n_scenes, uint64_t* keys, uint32_t n_total, KeyLayout kl, DevStatus* st,
    const uint32_t* base)
{
    using L = typename LayoutOf<T>::type;
    uint32_t movers = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_total; i += gridDim.x * blockDim.x) {
        int lo = 0, hi = n_scenes - 1; // scene owning storage slot i
        while (lo < hi) {
            int mid = (lo + hi + 1) >> 1;
            if (scenes[mid].first <= (int64_t)i) lo = mid;
            else hi = mid - 1;
        }
        const SceneParams<T>& sp = scenes[lo];
        int b[3];
        bool ok = true;
        for (int a = 0; a < 3; a++) {
            T x = p.f[(P_X + a) * p.stride + i];
            b[a] = base_node(x, sp.inv_dx);
            ok = ok && (x == x) && b[a] >= 0 && b[a] < sp.domain_cells - 3;
        }
        if (!ok) {
            raise_flag(st, FLAG_OUT_OF_DOMAIN);
            b[0] = b[1] = b[2] = 0;
        }
        const uint64_t k = ((uint64_t)lo << (kl.cp + kl.ib)) | ((L::offset(b[0], b[1], b[2]) >> L::data_bits) << kl.ib);
        kl.put(keys, i, k);
        if (base) movers += (uint32_t)k != base[i] ? 1u : 0u;
    }
    if (!base) return;
    for (int o = 16; o > 0; o >>= 1) movers += __shfl_down_sync(0xffffffffu, movers, o);
    if ((threadIdx.x & 31) == 0 && movers) atomicAdd(&st->max_movers, movers);
}

// The hot-path keys hold (scene, page, cell) only, so the radix sort needs 4 passes instead of 7; a
// stable sort of storage-ordered input leaves the particles of one cell in their previous order, which is
// deterministic and changes nothing in the substep but the order of floating-point sums. For the binning
// products (zr_scene_binning) this pass restores the reference's order inside each cell (ascending original
// index, the low bits of the reference key, MpmSimulationBase.cpp:1547-1552) with an insertion sort per run
// of equal keys; runs are short (~8) and nearly sorted.
template <class T>
__global__ void k_cellfix(const uint64_t* ks, uint32_t* vals, const uint32_t* pid, uint32_t n, KeyLayout kl)
{
    using L = typename LayoutOf<T>::type;
    const uint32_t mask = (1u << L::index_bits) - 1;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint64_t k = kl.at(ks, i);
        if (i > 0 && kl.at(ks, i - 1) == k) continue; // not the first of its run
        uint32_t e = i + 1;
        while (e < n && kl.at(ks, e) == k) e++;
        for (uint32_t q = i + 1; q < e; q++) {
            const uint32_t v = vals[q], o = pid[v] & mask;
            uint32_t r = q;
            while (r > i) {
                const uint32_t u = vals[r - 1];
                if ((pid[u] & mask) <= o) break;
                vals[r] = u;
                r--;
            }
            vals[r] = v;
        }
    }
}

// group heads of the sorted keys: first index of every (scene, page)
struct GroupHead {
    const uint64_t* k;
    KeyLayout kl;
    __device__ bool operator()(uint32_t i) const { return i == 0 || kl.group(kl.at(k, i)) != kl.group(kl.at(k, i - 1)); }
};

// ---------------------------------------------------------------------------------------------------
// Incremental sort (32-bit keys), hand-written. The storage order is the previous substep's sorted order, so the
// particles whose cell did not change ("stayers") are already sorted; only the particles that changed cell
// ("movers", ~2% per substep at the slab's speeds) need placing.
//
// Storage is cut into tiles (SortTile: 2,048 indices, or 512 in small scenes, see the host's sort_per). B[j] = the first old
// key of tile j (the old keys ascend with the storage index). Mover key k belongs to bucket b(k) = the largest j with B[j] <= k (0 when there is none): every
// element of bucket j (its movers) and tile j (its stayers) lies in [B[j], B[j+1]] and comes after every element of
// lower tiles and buckets, so tile j's merged output starts at (stayers in tiles < j) + (movers in buckets < j). Inside
// it, in the order (key, stayers first, storage index), a stayer goes to its rank among the tile's stayers plus the
// bucket's movers with a smaller key, a mover to its rank in the bucket plus the tile's stayers with a key not above its
// own. The order is fully determined by the keys and storage indices (no dependence on the order in which movers were
// found).
//
//   k_sort_tiles      per tile: stayer count and last stayer key; per mover its bucket (binary search over B), a ticket
//                     within it, the bucket's largest key, and (key, storage index) into the bucket's fixed slots
//   k_sort_merge      per tile: where its output starts and the key just before it (sums and maxima over the lower
//                     tiles and buckets, by the CTA itself), then the tile's stayers and its bucket's movers (sorted
//                     in shared memory) to their places; the groups that start in the tile's output take group
//                     numbers, and their blocks and +1 neighbours are activated in the grid hash
//
// Both kernels are chains of dependent memory round trips (about 0.7 us each) with little work behind them, so what they
// cost is the length of the chain. B comes from the old keys, known before the pass (B from the stayers put a second
// kernel between finding the movers and placing them), and groups are numbered as tiles finish (numbers in key order put
// a third kernel behind the merge, for the head counts of the lower tiles): as five nodes (a memset
// and four kernels) the substep took 57.0 us on 32,768 particles and 125.6 us on 425,984, with two 49.3 and 118.8 us.
//
// A bucket larger than its slots (SortTile::MAXM) raises FLAG_SORT: the host repeats the substep with a full radix sort, and sorts
// in full for longer each time that the sort behind it overflows again (SortBackoff). After a state write k_sort_probe tells
// beforehand.
// ---------------------------------------------------------------------------------------------------
constexpr int SORT_NT = 256, SORT_PER = 8, SORT_TILE = SORT_NT * SORT_PER; // the group-head pass, and tiles of large scenes
template <int PER>
struct SortTile { // PER items per thread: a tile, and its bucket's slots
    static constexpr int TILE = SORT_NT * PER, MAXM = PER > 4 ? TILE / 2 : TILE;
};
constexpr uint32_t SORT_NOKEY = 0xffffffffu; // keys of the incremental sort hold at most 31 bits

struct SortBufs {
    uint32_t* b_cnt; // [tiles] movers per bucket (zero at the start of a substep; k_grid clears it for the next one)
    uint32_t* b_max; // [tiles] largest mover key per bucket (likewise)
    uint32_t* stay_bits; // [ceil(n / 32)] bit i % 32 of word i / 32: storage index i keeps its key
    uint32_t* t_first; // [tiles] first old key per tile: B (k_group_heads or the previous merge wrote it)
    uint32_t* t_stay; // [tiles] stayers per tile
    uint32_t* t_last; // [tiles] last stayer key per tile (SORT_NOKEY: none)
    uint32_t* b_key; // [tiles * MAXM] movers' keys: bucket j's at j * MAXM + ticket
    uint32_t* b_idx; // [tiles * MAXM] movers' storage indices, likewise
    int64_t n;
    int tiles;
};
constexpr int SORT_FIRST = 4096; // tiles whose first keys a CTA copies to shared memory for its searches

// bucket of mover key k: the last tile whose first old key is not above it
__device__ __forceinline__ uint32_t bucket_of(const uint32_t* B, int tiles, uint32_t k)
{
    int lo = 0, hi = tiles; // first q with B[q] > k
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (B[mid] <= k) lo = mid + 1;
        else hi = mid;
    }
    return lo > 0 ? (uint32_t)(lo - 1) : 0u;
}

// After a state write: would a bucket of the next substep's sort hold more movers than its slots? Its movers counted by bucket
// (b_cnt, which the host clears again) with the keys, the base and the tiles that k_sort_tiles will see. Launched behind k_keys,
// whose count of movers says whether there is a question (sort_counted), so that both answers come back with one copy. One
// atomic per bucket and warp: neighbours in storage mostly go to one bucket.
template <int PER>
__host__ __device__ __forceinline__ bool sort_counted(int64_t movers, int64_t n) { return movers > SortTile<PER>::MAXM && 4 * movers <= n; }
template <int PER>
__global__ void __launch_bounds__(SORT_NT) k_sort_probe(const uint32_t* knew, const uint32_t* kold, SortBufs sb, DevStatus* st)
{
    constexpr uint32_t MAXM = SortTile<PER>::MAXM;
    __shared__ uint32_t s_first[SORT_FIRST];
    if (!sort_counted<PER>(st->max_movers, sb.n)) return;
    const int T = sb.tiles, lane = threadIdx.x & 31;
    if (T <= SORT_FIRST)
        for (int q = threadIdx.x; q < T; q += SORT_NT) s_first[q] = sb.t_first[q];
    __syncthreads();
    const uint32_t* B = T <= SORT_FIRST ? s_first : sb.t_first;
    for (int64_t i0 = blockIdx.x * (int64_t)SORT_NT + (threadIdx.x & ~31); i0 < sb.n; i0 += (int64_t)gridDim.x * SORT_NT) {
        const int64_t i = i0 + lane;
        const uint32_t k = i < sb.n ? knew[i] : 0u;
        const bool move = i < sb.n && k != kold[i];
        if (!__any_sync(0xffffffffu, move)) continue;
        const uint32_t b = move ? bucket_of(B, T, k) : SORT_NOKEY;
        const unsigned same = __match_any_sync(0xffffffffu, b);
        if (!move || lane != __ffs(same) - 1) continue;
        const uint32_t add = (uint32_t)__popc(same);
        if (atomicAdd(&sb.b_cnt[b], add) + add > MAXM) st->full_bucket = 1;
    }
}

template <int PER>
__global__ void __launch_bounds__(SORT_NT) k_sort_tiles(const uint32_t* knew, const uint32_t* kold, SortBufs sb, const DevStatus* st)
{
    constexpr int TILE = SortTile<PER>::TILE, MAXM = SortTile<PER>::MAXM;
    __shared__ uint32_t s_first[SORT_FIRST];
    __shared__ uint32_t s_cnt[SORT_NT / 32], s_last[SORT_NT / 32];
    const int j = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5, T = sb.tiles;
    const int64_t t0 = (int64_t)j * TILE;
    uint32_t nst = 0, last = SORT_NOKEY;
    unsigned moves = 0; // bit r: this thread's item of round r moved
    // items in storage order; a warp takes 256 consecutive ones, 32 at a time; every load issued first
    uint32_t kn[PER], ko[PER];
#pragma unroll
    for (int r = 0; r < PER; r++) {
        const int64_t i = t0 + (int64_t)w * (32 * PER) + r * 32 + lane;
        kn[r] = i < sb.n ? knew[i] : 0u;
        ko[r] = i < sb.n ? kold[i] : 1u;
    }
    const bool ab = aborted(st);
    if (T <= SORT_FIRST)
        for (int q = threadIdx.x; q < T; q += SORT_NT) s_first[q] = sb.t_first[q];
    const uint32_t* B = T <= SORT_FIRST ? s_first : sb.t_first;
#pragma unroll
    for (int r = 0; r < PER; r++) {
        const int64_t i = t0 + (int64_t)w * (32 * PER) + r * 32 + lane;
        const bool valid = i < sb.n, stay = valid && kn[r] == ko[r];
        const unsigned bs = __ballot_sync(0xffffffffu, stay);
        if (lane == 0 && valid) sb.stay_bits[i >> 5] = bs; // the merge reads these: it overwrites the old keys
        if (bs) last = __shfl_sync(0xffffffffu, kn[r], 31 - __clz(bs));
        nst += __popc(bs);
        if (valid && !stay) moves |= 1u << r;
    }
    if (lane == 0) {
        s_cnt[w] = nst;
        s_last[w] = last;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t c = 0, l = SORT_NOKEY;
        for (int q = 0; q < SORT_NT / 32; q++) {
            c += s_cnt[q];
            if (s_last[q] != SORT_NOKEY) l = s_last[q];
        }
        sb.t_stay[j] = c;
        sb.t_last[j] = l;
    }
    if (ab || !moves) return; // (an aborted substep's tickets would not be cleared)
#pragma unroll
    for (int r = 0; r < PER; r++) {
        if (!((moves >> r) & 1u)) continue;
        const uint32_t k = kn[r];
        const uint32_t b = bucket_of(B, T, k);
        const uint32_t t = atomicAdd(&sb.b_cnt[b], 1u);
        atomicMax(&sb.b_max[b], k);
        if (t < (uint32_t)MAXM) { // a fuller bucket makes the merge raise FLAG_SORT
            sb.b_key[(size_t)b * MAXM + t] = k;
            sb.b_idx[(size_t)b * MAXM + t] = (uint32_t)(t0 + (int64_t)w * (32 * PER) + r * 32 + lane);
        }
    }
}

// Block dl (x*4 + y*2 + z, at +1 block) of the group with key key0, into the block hash; a block seen for the first time
// takes the next grid slot (one slot counter atomic per group of converged lanes). Returns the block's hash position,
// whether this thread inserted the block or found it (-1: the probe failed and raised FLAG_CAPACITY). The slot behind it
// is written by the inserting thread, so it is read (nbr_slot) only by a later kernel.
template <class T>
__device__ __forceinline__ int32_t activate_block(const StepArgs<T>& a, uint64_t key0, uint32_t dl)
{
    using L = typename LayoutOf<T>::type;
    const uint64_t scene = a.kl.scene(key0);
    uint32_t bi, bj, bk;
    L::block_of_page(a.kl.page(key0), bi, bj, bk);
    const uint64_t hk = (scene << 40) | L::page_of_block(bi + (dl >> 2), bj + ((dl >> 1) & 1), bk + (dl & 1));
    uint32_t h = (uint32_t)hash64(hk) & a.h_mask;
    bool done = false, fresh = false;
    for (int p = 0; p < HASH_PROBES && !done; p++) {
        const unsigned long long prev = atomicCAS((unsigned long long*)&a.h_keys[h], (unsigned long long)HASH_EMPTY, (unsigned long long)hk);
        if (prev == HASH_EMPTY)
            done = fresh = true;
        else if (prev == hk)
            done = true;
        else
            h = (h + 1) & a.h_mask;
    }
    if (!done) raise_flag(a.st, FLAG_CAPACITY);
    const unsigned am = __activemask();
    const unsigned nw = __ballot_sync(am, fresh);
    if (nw) {
        const int lane = threadIdx.x & 31, leader = __ffs(nw) - 1;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(&a.st->n_blocks, (uint32_t)__popc(nw));
        base = __shfl_sync(am, base, leader);
        if (fresh) {
            const uint32_t slot = base + (uint32_t)__popc(nw & ((1u << lane) - 1u));
            if (slot >= a.b_cap) {
                raise_flag(a.st, FLAG_CAPACITY);
                a.h_vals[h] = -1;
            }
            else {
                a.h_vals[h] = (int32_t)slot;
                a.b_key[slot] = hk;
            }
        }
    }
    return done ? (int32_t)h : -1;
}

// Work items. P2G and G2P claim pieces of groups: a group of up to 5/4 of P2G's chunk is one item, a larger one is cut into
// equal items of at most a chunk. (One CTA per group made the group of a dense cluster the end of the kernel: 100,003
// particles in uneven blobs, P2G 107 k active cycles on the average SM and 463 k on the one with the fullest group. Items
// below 5/4 of a chunk would give the few blocks that hold a little more than 8 per cell a second node tile to flush.)
// Scenes too small for four items per SM at that size get smaller ones (item_max, see the host's item_size).
__device__ __forceinline__ uint32_t item_parts(uint32_t item_max, uint32_t count)
{
    return count <= item_max + item_max / 4 ? 1u : (count + item_max - 1) / item_max;
}
// the items of a group with sorted range [start, stop): the first at `first` (also the group's row in g_nbr), others from `rest` on
template <class T>
__device__ __forceinline__ void emit_items(const StepArgs<T>& a, uint32_t first, uint32_t rest, uint32_t start, uint32_t stop)
{
    const uint32_t n = stop - start, parts = item_parts(a.item_max, n);
    for (uint32_t p = 0; p < parts; p++) {
        const uint32_t at = p ? rest + p - 1 : first;
        if (at >= a.b_cap) { // the host grows the grid (and the item list with it) and repeats the substep
            raise_flag(a.st, FLAG_CAPACITY);
            return;
        }
        a.item[at] = make_uint4(start + (uint32_t)((uint64_t)n * p / parts), start + (uint32_t)((uint64_t)n * (p + 1) / parts), first, 0u);
    }
}
// A group whose range starts in one tile and ends in another: both tiles exchange what they know into the word of the
// group's block (hash position h): the start with the group's reserved item, or the end. The one that comes second finds the
// other's word, makes the items and clears the word.
constexpr unsigned long long RANGE_END = 1ull << 63;
template <class T>
__device__ __forceinline__ void range_event(const StepArgs<T>& a, int32_t h, unsigned long long mine)
{
    const unsigned long long other = atomicExch(a.open + h, mine);
    if (other == 0) return;
    a.open[h] = 0;
    const unsigned long long s = (mine & RANGE_END) ? other : mine, e = (mine & RANGE_END) ? mine : other;
    const uint32_t start = (uint32_t)s, first = (uint32_t)(s >> 32) - 1, stop = (uint32_t)e;
    if (!(e & RANGE_END) || (s & RANGE_END) || stop <= start) {
        check_failed(a.st, 10);
        return;
    }
    const uint32_t parts = item_parts(a.item_max, stop - start);
    emit_items(a, first, parts > 1 ? atomicAdd(&a.st->n_items, parts - 1) : 0u, start, stop);
}

// The shared buffers of k_sort_merge's two parts overlap.
template <int TILE, int MAXM>
union MergeShared {
    struct {
        uint32_t s_key[TILE], s_idx[TILE]; // the tile's stayers in storage (= key) order
        uint32_t m_key[MAXM], m_idx[MAXM], m_key2[MAXM], m_idx2[MAXM];
    } m;
    struct {
        uint32_t pos[TILE + MAXM]; // output positions of the tile's group heads, in order
        uint32_t off[TILE + MAXM]; // their first items, counted from the tile's first
    } h;
};

template <class T, int PER>
__global__ void __launch_bounds__(SORT_NT) k_sort_merge(StepArgs<T> a, const uint32_t* knew, SortBufs sb, uint32_t* out_keys, uint32_t* out_vals)
{
    constexpr int TILE = SortTile<PER>::TILE, MAXM = SortTile<PER>::MAXM, RMAX = (TILE + MAXM) / SORT_NT; // rounds over a tile's output
    __shared__ MergeShared<TILE, MAXM> sh;
    __shared__ uint32_t o_key[TILE + MAXM]; // the tile's output in order
    __shared__ uint32_t s_wcnt[RMAX][SORT_NT / 32];
    __shared__ uint32_t s_red[2][SORT_NT / 32];
    __shared__ uint32_t s_ns, s_nh, s_i0;
    uint32_t *s_key = sh.m.s_key, *s_idx = sh.m.s_idx, *m_key = sh.m.m_key, *m_idx = sh.m.m_idx, *m_key2 = sh.m.m_key2, *m_idx2 = sh.m.m_idx2;
    const int j = blockIdx.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    DevStatus* st = a.st;
    const KeyLayout kl = a.kl;
    if (blockIdx.x == 0) // the per-scene grid mass k_grid accumulates
        for (int s = tid; s < a.n_scenes; s += SORT_NT) a.grid_mass[s] = 0;
    // the tile's new keys and stay bits: issued ahead of everything that is tested. Item (r, w, lane) = t0 + r*256 + w*32 + lane
    const int64_t t0 = (int64_t)j * TILE;
    uint32_t keys[PER];
    unsigned mine = 0; // bit r: this thread's item of round r stays
#pragma unroll
    for (int r = 0; r < PER; r++) {
        const int64_t i = t0 + r * SORT_NT + tid;
        keys[r] = i < sb.n ? knew[i] : 0u;
        if (i < sb.n && ((sb.stay_bits[i >> 5] >> lane) & 1u)) mine |= 1u << r; // i % 32 == lane: rounds and warps start at multiples of 32
    }
    const uint32_t bc = sb.b_cnt[j];
    // the lower tiles and buckets: their element count (where this tile's output starts) and their largest key (the
    // key just before the output: stayer and bucket key ranges ascend with the tile). pk holds key + 1, 0 for none.
    uint32_t below = 0, pk = 0;
#pragma unroll 4
    for (int q = tid; q < j; q += SORT_NT) {
        const uint32_t c = sb.b_cnt[q], l = sb.t_last[q], mk = sb.b_max[q];
        below += sb.t_stay[q] + c;
        if (l != SORT_NOKEY) pk = max(pk, l + 1);
        if (c) pk = max(pk, mk + 1);
    }
    if (aborted_cta(st)) return;
    if (bc > (uint32_t)MAXM) { // the whole CTA: the substep is repeated with a full sort
        if (tid == 0) raise_flag(st, FLAG_SORT);
        return;
    }
    const int nm = (int)bc;
    for (int q = tid; q < nm; q += SORT_NT) {
        m_key[q] = sb.b_key[(size_t)j * MAXM + q];
        m_idx[q] = sb.b_idx[(size_t)j * MAXM + q];
    }
    for (int o = 16; o > 0; o >>= 1) {
        below += __shfl_down_sync(0xffffffffu, below, o);
        pk = max(pk, __shfl_down_sync(0xffffffffu, pk, o));
    }
    if (lane == 0) {
        s_red[0][w] = below;
        s_red[1][w] = pk;
    }
    // the tile's stayers, compacted in storage order
#pragma unroll
    for (int r = 0; r < PER; r++) {
        const unsigned b = __ballot_sync(0xffffffffu, (mine >> r) & 1u);
        if (lane == 0) s_wcnt[r][w] = __popc(b);
    }
    // exclusive offsets of the (round, warp) counts in order by the first warp, the total into *total: 8 per round
    auto scan_counts = [&](int rounds, uint32_t* total) {
        uint32_t* c = &s_wcnt[0][0];
        uint32_t carry = 0;
        for (int q0 = 0; q0 < rounds * (SORT_NT / 32); q0 += 32) {
            const uint32_t v = q0 + lane < rounds * (SORT_NT / 32) ? c[q0 + lane] : 0u;
            uint32_t x = v;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (q0 + lane < rounds * (SORT_NT / 32)) c[q0 + lane] = carry + x - v;
            carry += __shfl_sync(0xffffffffu, x, 31);
        }
        if (lane == 0) *total = carry;
    };
    __syncthreads();
    if (w == 0) scan_counts(PER, &s_ns);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < PER; r++) {
        const unsigned b = __ballot_sync(0xffffffffu, (mine >> r) & 1u);
        if ((mine >> r) & 1u) {
            const uint32_t pos = s_wcnt[r][w] + __popc(b & ((1u << lane) - 1u));
            s_key[pos] = keys[r];
            s_idx[pos] = (uint32_t)(t0 + r * SORT_NT + tid);
        }
    }
    // the bucket's movers ranked by (key, storage index): distinct pairs, so the ranks are a permutation
    for (int q = tid; q < nm; q += SORT_NT) {
        const uint32_t k = m_key[q], i = m_idx[q];
        int rank = 0;
        for (int o = 0; o < nm; o++) rank += (m_key[o] < k || (m_key[o] == k && m_idx[o] < i)) ? 1 : 0;
        m_key2[rank] = k;
        m_idx2[rank] = i;
    }
    __syncthreads();
    const int ns = (int)s_ns, cnt = ns + nm;
    uint32_t below_all = 0, pk_all = 0;
#pragma unroll
    for (int q = 0; q < SORT_NT / 32; q++) {
        below_all += s_red[0][q];
        pk_all = max(pk_all, s_red[1][q]);
    }
    const int64_t base = below_all; // elements of lower tiles and buckets
    if (base + cnt > sb.n) { // the counts cannot give this range (the whole CTA)
        if (tid == 0) check_failed(st, 8);
        return;
    }
    auto place = [&](int p, uint32_t k, uint32_t v) { // output p of the tile
        const int64_t pos = base + p;
        out_keys[pos] = k;
        out_vals[pos] = v;
        o_key[p] = k;
        if (pos % TILE == 0) sb.t_first[pos / TILE] = k; // B of the next substep
    };
    for (int t = tid; t < ns; t += SORT_NT) { // stayer: its rank + the bucket's movers with a smaller key
        const uint32_t k = s_key[t];
        int lo = 0, hi = nm;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (m_key2[mid] < k) lo = mid + 1;
            else hi = mid;
        }
        place(t + lo, k, s_idx[t]);
    }
    for (int r = tid; r < nm; r += SORT_NT) { // mover: its rank + the tile's stayers with a key not above its own
        const uint32_t k = m_key2[r];
        int lo = 0, hi = ns;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (s_key[mid] <= k) lo = mid + 1;
            else hi = mid;
        }
        place(r + lo, k, m_idx2[r]);
    }
    __syncthreads();
    // the groups that start in the tile's output: an output whose group differs from that of the key before it
    const uint32_t pred = pk_all ? pk_all - 1 : SORT_NOKEY; // the key before the tile's output (SORT_NOKEY: none)
    const int R = (cnt + SORT_NT - 1) / SORT_NT;
    unsigned heads = 0;
#pragma unroll
    for (int r = 0; r < RMAX; r++) {
        if (r >= R) break;
        const int p = r * SORT_NT + tid;
        bool head = false;
        if (p < cnt) {
            const uint32_t k = o_key[p], kp = p == 0 ? pred : o_key[p - 1];
            head = (p == 0 && pred == SORT_NOKEY) || kl.group(k) != kl.group(kp);
        }
        const unsigned b = __ballot_sync(0xffffffffu, head);
        if (head) heads |= 1u << r;
        if (lane == 0) s_wcnt[r][w] = __popc(b);
    }
    __syncthreads();
    if (w == 0) scan_counts(R, &s_nh);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RMAX; r++) {
        if (r >= R) break;
        const unsigned b = __ballot_sync(0xffffffffu, (heads >> r) & 1u);
        if ((heads >> r) & 1u) sh.h.pos[s_wcnt[r][w] + __popc(b & ((1u << lane) - 1u))] = (uint32_t)(r * SORT_NT + tid);
    }
    __syncthreads();
    const uint32_t nh = s_nh;
    const bool last_tile = j + 1 == sb.tiles;
    if (nh == 0 && !last_tile) return;
    // where head i's group ends, as an output position of the tile; ~0: in a later tile
    auto stop_of = [&](uint32_t i) { return i + 1 < nh ? sh.h.pos[i + 1] : (last_tile ? (uint32_t)cnt : ~0u); };
    // Tasks 8 i + q: block q of head i's group (q = 0 also makes the group's items, or reports its start); the last task
    // reports the end of the group that was open before the tile's first head, or that the particles end. The blocks go into
    // the hash while the last warp takes the items' numbers (one reserved for the group that stays open).
    const uint32_t tasks = 8 * nh + 1;
    for (uint32_t u0 = 0; u0 < tasks; u0 += SORT_NT) {
        const uint32_t t = u0 + tid, i = t >> 3, q = t & 7;
        int32_t h = -1;
        if (t < 8 * nh)
            h = activate_block(a, (uint64_t)o_key[sh.h.pos[i]], q);
        else if (t == 8 * nh && (nh ? pred != SORT_NOKEY : last_tile))
            h = activate_block(a, (uint64_t)(nh || !cnt ? pred : o_key[cnt - 1]), 0u);
        if (u0 == 0 && nh) {
            if (w == SORT_NT / 32 - 1) {
                uint32_t carry = 0;
                for (uint32_t k0 = 0; k0 < nh; k0 += 32) {
                    const uint32_t k = k0 + lane, stop = k < nh ? stop_of(k) : ~0u;
                    const uint32_t n = k >= nh ? 0u : (stop != ~0u ? item_parts(a.item_max, stop - sh.h.pos[k]) : 1u);
                    uint32_t x = n;
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                        if (lane >= o) x += y;
                    }
                    if (k < nh) sh.h.off[k] = carry + x - n;
                    carry += __shfl_sync(0xffffffffu, x, 31);
                }
                if (lane == 0) {
                    s_i0 = atomicAdd(&st->n_items, carry);
                    atomicAdd(&st->n_groups, nh);
                }
            }
            __syncthreads();
        }
        if (t > 8 * nh || h < 0) continue; // (a failed probe raised FLAG_CAPACITY)
        if (t == 8 * nh) {
            range_event(a, h, RANGE_END | (unsigned long long)(nh ? base + sh.h.pos[0] : sb.n));
            continue;
        }
        const uint32_t first = s_i0 + sh.h.off[i];
        if (first >= a.b_cap) { // more items than grid blocks: the host grows the grid and repeats the substep
            raise_flag(st, FLAG_CAPACITY);
            continue;
        }
        a.g_nbr[(size_t)first * 8 + q] = h;
        if (q == 0) {
            const uint32_t start = (uint32_t)base + sh.h.pos[i], stop = stop_of(i);
            if (stop != ~0u)
                emit_items(a, first, first + 1, start, (uint32_t)base + stop);
            else
                range_event(a, h, ((unsigned long long)(first + 1) << 32) | start);
        }
    }
}

// ---------------------------------------------------------------------------------------------------
// group heads: the first sorted index of every (scene, SPGrid page), compacted in order into g_start, their number
// into n_groups. One pass over the sorted keys with a decoupled look-back: tiles are taken in order from a counter
// (a tile's predecessors have started, so they publish), each publishes its head count, then the running total
// once its predecessors' is known. Waits are bounded; a wait that runs out raises FLAG_TIMEOUT.
// ---------------------------------------------------------------------------------------------------
constexpr uint64_t LB_AGG = 1ull << 62, LB_PREFIX = 2ull << 62, LB_VALUE = (1ull << 62) - 1;

static __global__ void __launch_bounds__(SORT_NT) k_group_heads(const uint64_t* keys, int64_t n, KeyLayout kl, uint64_t* status, uint32_t* counter,
    uint32_t* g_start, uint32_t cap, uint32_t* t_first, int first_tile, DevStatus* st)
{
    __shared__ uint32_t s_w[SORT_PER][SORT_NT / 32];
    __shared__ int s_tile;
    __shared__ uint64_t s_prefix;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tid == 0) s_tile = (int)atomicAdd(counter, 1u);
    __syncthreads();
    const int j = s_tile;
    const int64_t t0 = (int64_t)j * SORT_TILE;
    // B of the next substep's incremental sort (32-bit keys), whose tiles are first_tile items long
    for (int64_t i = t0 + (int64_t)tid * first_tile; i < min(n, t0 + SORT_TILE); i += (int64_t)SORT_NT * first_tile) t_first[i / first_tile] = (uint32_t)kl.at(keys, (uint32_t)i);
    unsigned mine = 0;
#pragma unroll
    for (int r = 0; r < SORT_PER; r++) {
        const int64_t i = t0 + r * SORT_NT + tid;
        const bool head = i < n && (i == 0 || kl.group(kl.at(keys, (uint32_t)i)) != kl.group(kl.at(keys, (uint32_t)(i - 1))));
        const unsigned b = __ballot_sync(0xffffffffu, head);
        if (head) mine |= 1u << r;
        if (lane == 0) s_w[r][w] = __popc(b);
    }
    __syncthreads();
    if (tid == 0) {
        uint32_t run = 0;
        for (int r = 0; r < SORT_PER; r++)
            for (int q = 0; q < SORT_NT / 32; q++) {
                const uint32_t c = s_w[r][q];
                s_w[r][q] = run;
                run += c;
            }
        s_prefix = run; // the tile's head count until the look-back below replaces it by the prefix
        volatile uint64_t* vs = status;
        vs[j] = (j == 0 ? LB_PREFIX : LB_AGG) | run;
    }
    __syncthreads();
    if (w == 0) { // look-back by the first warp: 32 predecessors per step, back to the nearest published prefix
        const uint32_t run = s_prefix;
        uint64_t prefix = 0;
        if (j > 0) {
            volatile uint64_t* vs = status;
            int q = j - 1;
            uint32_t spins = 0;
            bool timed_out = false;
            while (q >= 0 && !timed_out) {
                const int idx = q - lane;
                uint64_t v = LB_PREFIX + 0; // before tile 0: a prefix of zero
                if (idx >= 0) v = vs[idx];
                while (__any_sync(0xffffffffu, (v & (LB_AGG | LB_PREFIX)) == 0)) {
                    if (++spins > (1u << 22)) { // a predecessor never published: give up (the substep is aborted)
                        timed_out = true;
                        break;
                    }
                    __nanosleep(64);
                    if ((v & (LB_AGG | LB_PREFIX)) == 0) v = vs[idx];
                }
                if (timed_out) break;
                const unsigned pm = __ballot_sync(0xffffffffu, (v & LB_PREFIX) != 0);
                const int stop = pm ? __ffs(pm) - 1 : 31; // lanes 0..stop count (lane 0 is the nearest predecessor)
                uint64_t c = lane <= stop ? (v & LB_VALUE) : 0ull;
                for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
                prefix += __shfl_sync(0xffffffffu, c, 0);
                if (pm) break;
                q -= 32;
            }
            if (timed_out && lane == 0) raise_flag(st, FLAG_TIMEOUT);
            if (lane == 0) {
                __threadfence();
                vs[j] = LB_PREFIX | (prefix + run);
            }
        }
        if (lane == 0) {
            s_prefix = prefix;
            if ((int64_t)(j + 1) * SORT_TILE >= n) st->n_groups = st->n_items = (uint32_t)(prefix + run); // the last tile
        }
    }
    __syncthreads();
    const uint64_t prefix = s_prefix;
#pragma unroll
    for (int r = 0; r < SORT_PER; r++) {
        const unsigned b = __ballot_sync(0xffffffffu, (mine >> r) & 1u);
        if ((mine >> r) & 1u) {
            const uint64_t pos = prefix + s_w[r][w] + __popc(b & ((1u << lane) - 1u));
            if (pos < cap) g_start[pos] = (uint32_t)(t0 + r * SORT_NT + tid);
            else check_failed(st, 9);
        }
    }
}

// the blocks and items of every group (after a full sort and k_group_heads), 8 threads per group
template <class T>
__global__ void k_activate(StepArgs<T> a)
{
    if (blockIdx.x == 0) // the per-scene grid mass k_grid accumulates
        for (int s = threadIdx.x; s < a.n_scenes; s += blockDim.x) a.grid_mass[s] = 0;
    if (aborted(a.st)) return;
    const uint32_t G = a.st->n_groups;
    if (G > a.b_cap) {
        if (blockIdx.x == 0 && threadIdx.x == 0) raise_flag(a.st, FLAG_CAPACITY);
        return;
    }
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < G * 8; t += gridDim.x * blockDim.x) {
        const uint32_t g = t >> 3, start = a.g_start[g], stop = g + 1 < G ? a.g_start[g + 1] : a.n_total;
        a.g_nbr[t] = activate_block(a, a.kl.at(a.keys_sorted, start), t & 7); // (group g's first item is g)
        if ((t & 7) == 0) {
            const uint32_t parts = item_parts(a.item_max, stop - start);
            emit_items(a, g, parts > 1 ? atomicAdd(&a.st->n_items, parts - 1) : 0u, start, stop);
        }
    }
}

// ---------------------------------------------------------------------------------------------------
// neighbour slots: the grid slots of every item's block and its 7 neighbours at +1 block (read by P2G and G2P).
// Activation leaves the hash position of each of these blocks in the group's g_nbr; the slot behind it is final once
// activation has ended. The fused P2G translates its items' entries itself while it sets them up (and writes the slots
// back for G2P, into i_slot); the other P2G forms read those, so k_nbr translates every entry before them.
// ---------------------------------------------------------------------------------------------------
template <class T>
__device__ __forceinline__ int32_t nbr_slot(const StepArgs<T>& a, int32_t hpos)
{
    return (uint32_t)hpos <= a.h_mask ? a.h_vals[hpos] : -1; // -1: the probe failed and raised FLAG_CAPACITY
}

template <class T>
__global__ void k_nbr(StepArgs<T> a)
{
    if (aborted(a.st)) return;
    const uint32_t G = a.st->n_items;
    if (G > a.b_cap) return; // activation already raised FLAG_CAPACITY
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < G * 8; t += gridDim.x * blockDim.x) {
        const int32_t slot = nbr_slot(a, a.g_nbr[(size_t)a.item[t >> 3].z * 8 + (t & 7)]);
        if (slot < 0) raise_flag(a.st, FLAG_CAPACITY);
        a.i_slot[t] = slot;
    }
}

// ---------------------------------------------------------------------------------------------------
// P2G, in two kernels.
//
// k_stress (thread per sorted particle): stress V0 tau(F, g(d)) (FBasedMpmForceHelper.cpp:43-63) and a
// payload per particle, written in sorted order: fractional index-space position f = x/dx - base (or the weights it gives),
// m, A = m v - dx (m C) f, Bc = dx m C, K = -dt V0 tau / dx, d, and the particle's cell inside its block. With
// xm = (delta - f) dx for stencil offset delta,
//   m v + m C xm = A + Bc delta   and   dt f_i = K . (dw_i w_j w_k, w_i dw_j w_k, w_i w_j dw_k),
// so a node receives m w, w (A + Bc delta) + K grad-hat w, d w and w. The force enters the momentum
// directly (m v + dt f), which the grid update turns into v + f dt/m + g dt as the reference's
// gridVelocityExplicitUpdate does (MpmSimulationBase.cpp:1197-1226).
//
// k_scatter (a CTA per work item, persistent): a producer warp streams each chunk of an item's payload from
// HBM into shared memory with bulk asynchronous copies (double-buffered, mbarrier-synchronised); the
// consumer threads, one per (cell, stencil x-offset), accumulate the 9 nodes x 6 fields of their cell's
// particles in registers (all particles of a cell share the same 27 nodes), add them into a shared
// 6x6x6 node tile, and after the group's last chunk the tile goes to the 8 neighbouring grid blocks as
// vector atomics (MpmSimulationBase.cpp:669-855, AnisoFractureSimulation.h:161-176).
//
// Payload storage: field k of sorted particle q at pay[k * pstride + q + q/8]. The gap after every 8
// particles carries over into shared memory with the copy and staggers the shared-memory banks of the
// consumer lanes (one lane per cell, ~8 particles per cell).
// The Kirchhoff stress of every model here is symmetric (the energies are frame-indifferent), so K is
// its upper triangle: six fields instead of nine,
// three shared-memory loads fewer per particle and stencil x-offset in the accumulation.
// ---------------------------------------------------------------------------------------------------
//
// FP32 keeps the fractional position and evaluates the weights in each of a particle's three offset threads; FP64, whose
// pipe is 64 times slower than the FP32 one while shared memory is not, keeps the weights themselves, and per stencil
// z-offset k the vector Z_k = k wz_k B2 + dwz_k K2 (B2, K2: the third columns), which all of them use (accumulate_particle).
template <class T>
struct Pay {
    enum { F = 0, M = 3, A = 4, B = 7, K = 16, D = 22, CELL = 23, N = 24 };
};
template <>
struct Pay<double> { // WX .. WZ: 3 weights or derivatives per axis; B0, B1: the first columns; Z: 3 per z-offset
    enum { WX = 0, DWX = 3, WY = 6, DWY = 9, WZ = 12, M = 15, A = 16, B0 = 19, B1 = 22, K = 25, Z = 30, D = 39, CELL = 40, N = 41 };
};
enum { K_00 = 0, K_01 = 1, K_02 = 2, K_11 = 3, K_12 = 4, K_22 = 5 }; // offsets of the K entries (FP64 keeps the first five)

__host__ __device__ __forceinline__ uint64_t pay_pos(uint64_t q) { return q + (q >> 3); }

// Stress and payload of one particle (storage slot j of pool P): the fields of Pay<T> but CELL at y[f * S]; b gets the
// base node. V0 tau(F) of the particle's model (FBasedMpmForceHelper.cpp:43-63) with the degradation g(d).
template <class T, int MODELS>
__device__ __forceinline__ void particle_payload(const Pool<T>& P, uint32_t j, const SceneParams<T>& sp, T* y, int64_t S, int (&b)[3],
    uint32_t& fallbacks)
{
    using L = typename LayoutOf<T>::type;
    // The corotated stress's polar decomposition needs many registers: with it, v and C are loaded after the
    // stress (a second memory latency) instead of being held through it (spills)
    constexpr bool LATE_VC = (MODELS & 1) != 0;
    T x[3], v[3], Cm[9], F[9];
    auto load_vc = [&]() {
#pragma unroll
        for (int e = 0; e < 3; e++) v[e] = P.f[(P_V + e) * P.stride + j];
#pragma unroll
        for (int e = 0; e < 9; e++) Cm[e] = P.f[(P_C + e) * P.stride + j];
    };
#pragma unroll
    for (int e = 0; e < 3; e++) x[e] = P.f[(P_X + e) * P.stride + j];
#pragma unroll
    for (int e = 0; e < 9; e++) F[e] = P.f[(P_F + e) * P.stride + j];
    if constexpr (!LATE_VC) load_vc();
    const T mass = P.f[P_M * P.stride + j], V0 = P.f[P_V0 * P.stride + j];
    const bool damage = sp.damage != 0;
    const T dd = damage ? P.f[P_D * P.stride + j] : (T)0;
    const uint32_t mat = P.pid[j] >> L::index_bits;
    const Material<T>& mt = sp.materials[mat < (uint32_t)sp.n_materials ? mat : 0];
    T tau[9];
    const T g = (damage && mt.damage) ? degradation(dd, mt.residual) : (T)1;
    if (MODELS == 1 || (MODELS == 7 && mt.model == MODEL_COROTATED)) { // the reference degrades no corotated model
        if (tau_corotated(mt, F, tau)) fallbacks++;
    }
    else if (MODELS == 4 || (MODELS == 7 && mt.model == MODEL_QR_STABLE_NEOHOOKEAN))
        tau_qrnh(mt, F, g, tau);
    else
        tau_nhb(mt, F, g, tau);
    if constexpr (LATE_VC) load_vc();
    const T dx = sp.dx, inv_dx = sp.inv_dx, dt = sp.dt;
    T fr[3];
#pragma unroll
    for (int e = 0; e < 3; e++) {
        const T xs = mul_rn(x[e], inv_dx);
        b[e] = int_floor(sub_rn(xs, (T)0.5));
        fr[e] = xs - (T)b[e];
    }
    using Y = Pay<T>;
    const T kf = -dt * V0 * inv_dx;
    const T K[6] = { kf * tau[0], kf * tau[1], kf * tau[2], kf * tau[4], kf * tau[5], kf * tau[8] };
    y[Y::M * S] = mass;
    y[Y::D * S] = dd;
    if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int e = 0; e < 3; e++) y[(Y::F + e) * S] = fr[e];
#pragma unroll
        for (int r = 0; r < 3; r++) {
            const T m0 = mass * Cm[3 * r], m1 = mass * Cm[3 * r + 1], m2 = mass * Cm[3 * r + 2];
            y[(Y::A + r) * S] = mass * v[r] - dx * (m0 * fr[0] + m1 * fr[1] + m2 * fr[2]);
            y[(Y::B + 3 * r) * S] = dx * m0;
            y[(Y::B + 3 * r + 1) * S] = dx * m1;
            y[(Y::B + 3 * r + 2) * S] = dx * m2;
        }
#pragma unroll
        for (int e = 0; e < 6; e++) y[(Y::K + e) * S] = K[e];
    }
    else {
        T w[3][3], dw[3][3];
#pragma unroll
        for (int e = 0; e < 3; e++) {
            bspline_w(fr[e], 0, w[e], dw[e]);
#pragma unroll
            for (int k = 0; k < 3; k++) {
                y[((e == 0 ? Y::WX : e == 1 ? Y::WY : Y::WZ) + k) * S] = w[e][k];
                if (e < 2) y[((e == 0 ? Y::DWX : Y::DWY) + k) * S] = dw[e][k];
            }
        }
        const T kw2 = (T)2 * w[2][2], md = mass * dx;
#pragma unroll
        for (int r = 0; r < 3; r++) {
            const T b0 = md * Cm[3 * r], b1 = md * Cm[3 * r + 1], b2 = md * Cm[3 * r + 2];
            y[(Y::A + r) * S] = mass * v[r] - (b0 * fr[0] + b1 * fr[1] + b2 * fr[2]);
            y[(Y::B0 + r) * S] = b0;
            y[(Y::B1 + r) * S] = b1;
            const T k2 = K[r == 0 ? K_02 : r == 1 ? K_12 : K_22];
            y[(Y::Z + r) * S] = dw[2][0] * k2;
            y[(Y::Z + 3 + r) * S] = w[2][1] * b2 + dw[2][1] * k2;
            y[(Y::Z + 6 + r) * S] = kw2 * b2 + dw[2][2] * k2;
        }
#pragma unroll
        for (int e = 0; e < 5; e++) y[(Y::K + e) * S] = K[e];
    }
}

template <class T, int MODELS>
__global__ void __launch_bounds__(256) k_stress(StepArgs<T> a)
{
    using L = typename LayoutOf<T>::type;
    if (aborted(a.st)) return;
    const KeyLayout kl = a.kl;
    const uint64_t cmask = (1ULL << kl.cp) - 1;
    const int64_t S = a.pstride;
    uint32_t flags = 0, fallbacks = 0;
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < a.n_total; q += gridDim.x * blockDim.x) {
        const uint64_t key = a.kl.at(a.keys_sorted, q);
        T* y = a.pay + pay_pos(q);
        int b[3];
        particle_payload<T, MODELS>(a.pin, a.vals_sorted[q], a.scenes[kl.scene(key)], y, S, b, fallbacks);
        // the key was computed from this position by the previous G2P (or k_keys): they must agree
        const uint64_t want = (key >> kl.ib) & cmask;
        const bool ok = b[0] >= 0 && b[1] >= 0 && b[2] >= 0 && (L::offset(b[0], b[1], b[2]) >> L::data_bits) == want;
        if (!ok) flags |= FLAG_CAPACITY;
        y[Pay<T>::CELL * S] = ok ? (T)(int)(want & (L::nodes - 1)) : (T)255;
        if ((q & 7) == 7) { // the gap slot after every 8th particle: writing it keeps every 32-byte sector whole
#pragma unroll
            for (int f = 0; f < Pay<T>::N; f++) y[f * S + 1] = (T)0;
        }
    }
    if (flags) raise_flag(a.st, flags);
    if (fallbacks) atomicAdd(&a.st->fallback, fallbacks);
}

template <class T>
__device__ inline void flush_column(T* dst, const T* src, int n)
{
    if constexpr (std::is_same<T, float>::value) {
        if (n == 4) {
            float4 v = make_float4(src[0], src[1], src[2], src[3]);
            if (v.x != 0.f || v.y != 0.f || v.z != 0.f || v.w != 0.f) atomicAdd((float4*)dst, v);
        }
        else {
            float2 v = make_float2(src[0], src[1]);
            if (v.x != 0.f || v.y != 0.f) atomicAdd((float2*)dst, v);
        }
    }
    else {
        for (int q = 0; q < n; q++)
            if (src[q] != (T)0) atomicAdd(dst + q, src[q]);
    }
}

// Paired arithmetic: Blackwell issues two FP32 FMAs as one instruction on float2 operands (__ffma2_rn rounds each
// lane as fmaf does). The accumulators of a (cell, x-offset) thread are kept as pairs so that every update of
// two fields is one instruction; FP64 keeps scalar FMAs.
template <class T>
struct PairOf;
template <>
struct PairOf<float> {
    using type = float2;
};
template <>
struct PairOf<double> {
    using type = double2;
};
__device__ __forceinline__ float2 pfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
// 16 bytes of consecutive values (4 FP32 or 2 FP64), moved with one access
template <class T>
struct alignas(16) Vec16 {
    T v[16 / sizeof(T)];
};
// four values of one grid node read with one shared-memory access (velocity x, y, z and the phase field)
template <class T>
struct alignas(4 * sizeof(T)) Quad {
    T x, y, z, w;
};
__device__ __forceinline__ double2 pfma(double2 a, double2 b, double2 c) { return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y)); }
__device__ __forceinline__ float2 pmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ double2 pmul(double2 a, double2 b) { return make_double2(a.x * b.x, a.y * b.y); }
template <class P, class T>
__device__ __forceinline__ P pmake(T x, T y)
{
    P r;
    r.x = x;
    r.y = y;
    return r;
}

// The 9 nodes (jj, kk) x NACC fields of a (cell, stencil x-offset ii) thread, as pairs (p_x, p_y), (p_z, m), (d w, w)
template <class T>
struct NodeAcc {
    using P = typename PairOf<T>::type;
    P a[9][3];
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int n = 0; n < 9; n++)
#pragma unroll
            for (int k = 0; k < 3; k++) a[n][k] = pmake<P>((T)0, (T)0);
    }
    // field f of node n: 0 mass, 1-3 momentum, 4 d w, 5 w (the accumulator order of the grid)
    __device__ __forceinline__ T field(int n, int f) const
    {
        return f == 0 ? a[n][1].y : f == 1 ? a[n][0].x : f == 2 ? a[n][0].y : f == 3 ? a[n][1].x : f == 4 ? a[n][2].x : a[n][2].y;
    }
};

// One particle's contribution to the 9 nodes (ii, jj, kk) of a (cell, stencil x-offset ii) thread; y points
// at the particle's payload, fields STRIDE apart. Weights from the fractional position (BSplines.h:73-100).
// Node (ii, jj, kk) receives, per momentum component,
//   wz_k al(j) + e(j) Z_k   with   e = wx wy,   al = e (A + ii B0 + j B1) + dwx wy K0 + wx dwy K1,   Z_k = k wz_k B2 + dwz_k K2
// so the terms that depend on k through k wz_k and dwz_k are summed once per particle (Z), not per j, and a node takes two
// FMAs a component instead of three. What does not depend on (j, k) is folded first:
//   U = wx (A + ii B0) + dwx K0,  V = wx B1,  Wk = wx K1,   al = wy_j U + j wy_j V + dwy_j Wk.
// FP32 runs on pairs (two lanes per instruction): (x, y) and (z, m), and (d w, w). The mass lane has neither B nor K, so the
// z lane's terms with them are single FMAs.
template <class T, int STRIDE, bool DAMAGE>
__device__ __forceinline__ void accumulate_particle(NodeAcc<T>& acc, const T* y, int ii)
{
    using Y = Pay<T>;
    if constexpr (sizeof(T) == 4) {
        using P = typename NodeAcc<T>::P;
        T wy[3], dwy[3], wz[3], dwz[3];
        T wx, dwx;
        {
            const T d0 = y[Y::F * STRIDE];
            const T z = (T)1.5 - d0, d1 = d0 - (T)1, zz = d0 - (T)0.5;
            wx = ii == 0 ? (T)0.5 * z * z : (ii == 1 ? (T)0.75 - d1 * d1 : (T)0.5 * zz * zz);
            dwx = ii == 0 ? -z : (ii == 1 ? (T)-2 * d1 : zz);
        }
        bspline_w(y[(Y::F + 1) * STRIDE], 0, wy, dwy);
        bspline_w(y[(Y::F + 2) * STRIDE], 0, wz, dwz);
        const T mass = y[Y::M * STRIDE];
        const T dd = DAMAGE ? y[Y::D * STRIDE] : (T)0;
        const T fi = (T)ii;
        const P WX = pmake<P>(wx, wx), DWX = pmake<P>(dwx, dwx), FI = pmake<P>(fi, fi);
        auto f = [&](int k) { return y[k * STRIDE]; };
        auto pr = [&](int f0, int f1) { return pmake<P>(y[f0 * STRIDE], y[f1 * STRIDE]); };
        // K is symmetric: column c of it is (K0c, K1c, K2c) read from the upper triangle
        const P U01 = pfma(DWX, pr(Y::K + K_00, Y::K + K_01), pmul(WX, pfma(FI, pr(Y::B, Y::B + 3), pr(Y::A, Y::A + 1))));
        const P U2 = pmake<P>(dwx * f(Y::K + K_02) + wx * (fi * f(Y::B + 6) + f(Y::A + 2)), wx * mass);
        const P V01 = pmul(WX, pr(Y::B + 1, Y::B + 4)), K01 = pmul(WX, pr(Y::K + K_01, Y::K + K_11));
        const T V2 = wx * f(Y::B + 7), K2 = wx * f(Y::K + K_12);
        P Z01[3];
        T Z2[3];
        {
            const P b01 = pr(Y::B + 2, Y::B + 5), k01 = pr(Y::K + K_02, Y::K + K_12);
            const T b2 = f(Y::B + 8), k2 = f(Y::K + K_22);
#pragma unroll
            for (int kk = 0; kk < 3; kk++) {
                Z01[kk] = pmul(pmake<P>(dwz[kk], dwz[kk]), k01);
                Z2[kk] = dwz[kk] * k2;
                if (kk) {
                    const T kw = (T)kk * wz[kk];
                    Z01[kk] = pfma(pmake<P>(kw, kw), b01, Z01[kk]);
                    Z2[kk] = kw * b2 + Z2[kk];
                }
            }
        }
#pragma unroll
        for (int jj = 0; jj < 3; jj++) {
            const P WY = pmake<P>(wy[jj], wy[jj]), E = pmul(WY, WX);
            P AL0 = pfma(pmake<P>(dwy[jj], dwy[jj]), K01, pmul(WY, U01)), AL1 = pmul(WY, U2);
            AL1.x = dwy[jj] * K2 + AL1.x;
            if (jj) {
                const T jw = (T)jj * wy[jj];
                AL0 = pfma(pmake<P>(jw, jw), V01, AL0);
                AL1.x = jw * V2 + AL1.x;
            }
            const P DW = pmake<P>(E.x * dd, E.y);
#pragma unroll
            for (int kk = 0; kk < 3; kk++) {
                const P W = pmake<P>(wz[kk], wz[kk]);
                P* ac = acc.a[jj * 3 + kk];
                ac[0] = pfma(W, AL0, ac[0]);
                ac[0] = pfma(E, Z01[kk], ac[0]);
                ac[1] = pfma(W, AL1, ac[1]);
                ac[1].x = E.x * Z2[kk] + ac[1].x;
                if (DAMAGE) ac[2] = pfma(W, DW, ac[2]);
            }
        }
    }
    else {
        auto f = [&](int k) { return y[k * STRIDE]; };
        const T wx = f(Y::WX + ii), dwx = f(Y::DWX + ii), fi = (T)ii;
        T U[3], V[3], Wk[3];
#pragma unroll
        for (int r = 0; r < 3; r++) {
            U[r] = dwx * f(Y::K + r) + wx * (fi * f(Y::B0 + r) + f(Y::A + r)); // K's first column: 00, 01, 02
            V[r] = wx * f(Y::B1 + r);
            Wk[r] = wx * f(Y::K + (r == 0 ? K_01 : r == 1 ? K_11 : K_12));
        }
        const T mass = f(Y::M), dd = DAMAGE ? f(Y::D) : (T)0;
#pragma unroll
        for (int jj = 0; jj < 3; jj++) {
            const T wy = f(Y::WY + jj), dwy = f(Y::DWY + jj), e = wx * wy, em = e * mass, ed = e * dd, jw = (T)jj * wy;
            T al[3];
#pragma unroll
            for (int r = 0; r < 3; r++) {
                al[r] = dwy * Wk[r] + wy * U[r];
                if (jj) al[r] = jw * V[r] + al[r];
            }
#pragma unroll
            for (int kk = 0; kk < 3; kk++) {
                const T w = f(Y::WZ + kk);
                auto* ac = acc.a[jj * 3 + kk];
                ac[0].x = e * f(Y::Z + 3 * kk) + (w * al[0] + ac[0].x);
                ac[0].y = e * f(Y::Z + 3 * kk + 1) + (w * al[1] + ac[0].y);
                ac[1].x = e * f(Y::Z + 3 * kk + 2) + (w * al[2] + ac[1].x);
                ac[1].y = w * em + ac[1].y;
                if (DAMAGE) {
                    ac[2].x = w * ed + ac[2].x;
                    ac[2].y = w * e + ac[2].y;
                }
            }
        }
    }
}

// registers -> shared node tile of the block plus its +2 halo (distinct nodes within a warp: no contention)
template <class T, class L>
__device__ __forceinline__ void add_to_tile(const NodeAcc<T>& acc, T* tile, int cx, int cy, int cz, int ii, int nf)
{
    constexpr int TY = L::sy + 2, TZ = L::sz + 2, TN = (L::sx + 2) * TY * TZ;
#pragma unroll
    for (int jj = 0; jj < 3; jj++)
#pragma unroll
        for (int kk = 0; kk < 3; kk++) {
            T* t = tile + ((cx + ii) * TY + (cy + jj)) * TZ + (cz + kk);
#pragma unroll
            for (int f = 0; f < NACC; f++)
                if (f < nf) atomicAdd(t + f * TN, acc.field(jj * 3 + kk, f));
        }
}

// tile -> the 8 neighbouring grid blocks: z columns split at the block boundary (4 + 2 nodes), vector atomics;
// the tile is cleared behind the flush. nbr: grid slots of the block and its +1 neighbours (x*4 + y*2 + z).
template <class T, class L>
__device__ __forceinline__ void flush_tile(const StepArgs<T>& a, T* tile, const int32_t* nbr, int nf, int tid, int nthreads)
{
    constexpr int TX = L::sx + 2, TY = L::sy + 2, TZ = L::sz + 2, TN = TX * TY * TZ;
    for (int q = tid; q < nf * TX * TY * 2; q += nthreads) {
        const int half = q & 1, col = q >> 1;
        const int f = col / (TX * TY), ab = col % (TX * TY), ta = ab / TY, tb = ab % TY;
        const int ax = ta >= L::sx, ay = tb >= L::sy;
        const int slot = nbr[ax * 4 + ay * 2 + half];
        if ((uint32_t)slot >= a.b_cap) {
            check_failed(a.st, 5);
            continue;
        }
        T* dst = a.acc + ((size_t)slot * NACC + f) * L::nodes + L::element(ta - ax * L::sx, tb - ay * L::sy, 0);
        T* src = tile + f * TN + (ta * TY + tb) * TZ + half * L::sz;
        const int n = half ? TZ - L::sz : L::sz;
        flush_column(dst, src, n);
        for (int z = 0; z < n; z++) src[z] = (T)0;
    }
}

// The fused P2G's node tiles, one per stencil x-offset ii: tile ii holds nodes x = cx + ii for cx in [0, sx), all
// y and z of the block plus its +2 halo. The warps of one offset cover disjoint cx, and within a warp the lanes'
// cells are distinct, so each of the 9 node steps below touches distinct nodes: a plain read-modify-write
// replaces the shared-memory float atomics (about twice their throughput). Lanes of one warp reach the same
// node in different steps, so the steps are separated by __syncwarp (it orders the lanes' shared accesses).
// Every lane of the warp must call it.
template <class L>
struct OffsetTiles {
    static constexpr int TY = L::sy + 2, TZ = L::sz + 2;
    static constexpr int TS = L::sx * TY * TZ; // nodes of one offset's tile (per field)
    static constexpr int ELEMS = 3 * NACC * TS;
    // tile index of cell c's first node (of any offset)
    __device__ static __forceinline__ int corner(int c)
    {
        const int cx = c >> (L::zbits + L::ybits), cy = (c >> L::zbits) & (L::sy - 1), cz = c & (L::sz - 1);
        return (cx * TY + cy) * TZ + cz;
    }
};

// The same sums where several lanes hold pieces of one cell (split_cells): the pieces of a cell take turns, `parts` of them at
// most. Every lane of the warp must call it.
template <class T, class L>
__device__ __forceinline__ void add_pieces_to_offset_tile(const NodeAcc<T>& acc, T* tiles, int cell, int ii, int nf, bool used, int part, int parts)
{
    using OT = OffsetTiles<L>;
    T* base = tiles + ii * NACC * OT::TS + OT::corner(cell);
    for (int turn = 0; turn < parts; turn++) {
#pragma unroll
        for (int jj = 0; jj < 3; jj++)
#pragma unroll
            for (int kk = 0; kk < 3; kk++) {
                T* t = base + jj * OT::TZ + kk;
                if (used && part == turn) {
#pragma unroll
                    for (int f = 0; f < NACC; f++)
                        if (f < nf) t[f * OT::TS] += acc.field(jj * 3 + kk, f);
                }
                __syncwarp();
            }
    }
}

// Work of the accumulation's (cell, x-offset) threads where cells hold unequal numbers of particles. A warp's 32 cells take as
// long as the fullest of them, and a cell without particles leaves its lane idle: so the cells are cut into pieces of at
// most R particles, a piece per lane, R the smallest count for which the pieces fit (but not so small that the turns of a
// cell's pieces in the tile take longer than they save). It all happens inside the warp: the cells of an x-offset's two warps
// (FP32) cover disjoint x of the tile, so no warp touches another's nodes. (Pieces dealt over both warps need shared-memory
// atomics in the tile: on chunks of 19 crowded cells, 27 particles per cell, that made P2G 198 us, no pieces at all 171, these
// 142. At 8 per cell they change P2G by less than 1%: 53.4 against 53.5 us at 425,984 particles, 307 against 307 at 3,407,872.)
// [qa, qb): in the particles of the lane's cell c, out those of its piece. Returns the piece: cell (PIECE_NONE: no piece) | number
// in the cell << 8 | most pieces of a cell << 20 (0: nothing was cut, the piece is the cell).
constexpr uint32_t PIECE_NONE = 0xff;
template <class T>
__device__ __forceinline__ uint32_t split_cells(int c, int& qa, int& qb)
{
    const unsigned all = 0xffffffffu;
    const int lane = threadIdx.x & 31, n = qb - qa;
    const unsigned occupied = __ballot_sync(all, n > 0);
    if (occupied == all || occupied == 0) return (uint32_t)c; // no lane to give a piece to
    const int most = __reduce_max_sync(all, n), cnt = __reduce_add_sync(all, n);
    if (most <= 2) return (uint32_t)c;
    int R = max((cnt + 31) / 32, (int)sqrtf((float)most)), p;
    for (;; R++) { // (R = most always fits: at most one piece per cell)
        p = (int)(((float)(n + R - 1) + 0.5f) * (1.0f / (float)R)); // ceil(n / R), exact for these sizes
        if (__reduce_add_sync(all, p) <= 32) break;
    }
    const int parts = (most + R - 1) / R;
    // a turn in the tile takes about half a particle's accumulation in FP64 and one in FP32
    if (sizeof(T) == 8 ? 2 * most <= 2 * R + parts - 1 : most < R + parts + 1) return (uint32_t)c;
    int x = p; // exclusive offsets of the cells' pieces
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(all, x, o);
        if (lane >= o) x += y;
    }
    const int total = __shfl_sync(all, x, 31);
    x -= p;
    int l = 0; // the cell (lane) of piece `lane`: the last one whose pieces start at or before it
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const int y = __shfl_sync(all, x, l + o);
        if (y <= lane) l += o;
    }
    const int part = lane - __shfl_sync(all, x, l), q0 = __shfl_sync(all, qa, l), q1 = __shfl_sync(all, qb, l);
    qa = min(q0 + part * R, q1);
    qb = min(qa + R, q1);
    if (lane >= total) {
        qa = qb = q0;
        return PIECE_NONE | (uint32_t)parts << 20;
    }
    return (uint32_t)((c & ~31) + l) | (uint32_t)part << 8 | (uint32_t)parts << 20;
}

template <class T, class L>
__device__ __forceinline__ void add_to_offset_tile(const NodeAcc<T>& acc, T* tiles, int cell, int ii, int nf)
{
    using OT = OffsetTiles<L>;
    T* base = tiles + ii * NACC * OT::TS + OT::corner(cell);
#pragma unroll
    for (int jj = 0; jj < 3; jj++)
#pragma unroll
        for (int kk = 0; kk < 3; kk++) {
            T* t = base + jj * OT::TZ + kk;
#pragma unroll
            for (int f = 0; f < NACC; f++)
                if (f < nf) t[f * OT::TS] += acc.field(jj * 3 + kk, f);
            __syncwarp();
        }
}

// node (X, Y, z-column) of the block's 6x6x6 tile = the sum over the offsets ii with X - ii in [0, sx); written to
// the 8 neighbouring grid blocks as flush_tile does, the offset tiles cleared behind the flush
template <class T, int N>
__device__ __forceinline__ void flush_offset_column(T* dst, T* tiles, int f, int X, int Y, int z0)
{
    using L = typename LayoutOf<T>::type;
    using OT = OffsetTiles<L>;
    T v[N];
#pragma unroll
    for (int z = 0; z < N; z++) v[z] = (T)0;
#pragma unroll
    for (int ii = 0; ii < 3; ii++) {
        const int xl = X - ii;
        if (xl < 0 || xl >= L::sx) continue;
        T* src = tiles + (ii * NACC + f) * OT::TS + (xl * OT::TY + Y) * OT::TZ + z0;
#pragma unroll
        for (int z = 0; z < N; z++) {
            v[z] += src[z];
            src[z] = (T)0;
        }
    }
    flush_column(dst, v, N);
}

template <class T, class L>
__device__ __forceinline__ void flush_offset_tiles(const StepArgs<T>& a, T* tiles, const int32_t* nbr, int nf, int tid, int nthreads)
{
    constexpr int TX = L::sx + 2, TY = L::sy + 2;
    static_assert(L::sz + 2 - L::sz == 2, "z columns split 4 + 2");
    for (int q = tid; q < nf * TX * TY * 2; q += nthreads) {
        const int half = q & 1, col = q >> 1;
        const int f = col / (TX * TY), ab = col % (TX * TY), ta = ab / TY, tb = ab % TY;
        const int ax = ta >= L::sx, ay = tb >= L::sy;
        const int slot = nbr[ax * 4 + ay * 2 + half];
        if ((uint32_t)slot >= a.b_cap) {
            check_failed(a.st, 5);
            continue;
        }
        T* dst = a.acc + ((size_t)slot * NACC + f) * L::nodes + L::element(ta - ax * L::sx, tb - ay * L::sy, 0);
        if (half)
            flush_offset_column<T, 2>(dst, tiles, f, ta, tb, L::sz);
        else
            flush_offset_column<T, L::sz>(dst, tiles, f, ta, tb, 0);
    }
}

// CHUNK: particles staged per copy (the tile of particles); the scatter CTA is the consumer threads
// (cell x stencil x-offset) plus one producer warp
// NBUF: staging buffers (1: the next chunk's copy overlaps the tile accumulation and flush of the current
// one; 2: it overlaps the whole chunk)
template <class T, int CHUNK, int NBUF>
struct ScatterShape {
    using L = typename LayoutOf<T>::type;
    static constexpr int NCONS = 3 * L::nodes;
    static constexpr int NT = NCONS + 32;
    static constexpr int VEC = 16 / (int)sizeof(T); // elements per 16 bytes: copy granularity
    static constexpr int WIN = CHUNK + CHUNK / 8 + 8; // payload window per field, >= the span of CHUNK particles
    static constexpr size_t buf_bytes = sizeof(T) * Pay<T>::N * WIN;
    static constexpr size_t dyn_bytes = NBUF * buf_bytes;
    static constexpr int MIN_CTAS = sizeof(T) == 4 ? 2 : 1;
    static_assert(CHUNK % 32 == 0 && (WIN * sizeof(T)) % 16 == 0 && (NBUF == 1 || NBUF == 2), "copy alignment, buffers");
};

enum : uint32_t { ITEM_LAST = 1, ITEM_DONE = 2, ITEM_BAD = 4 };

struct ScatterItem {
    uint32_t q0, q1; // sorted particle range of the chunk
    uint32_t base; // payload position of element 0 of the staged window
    uint32_t flags;
    int32_t nf; // accumulator fields in use (4 without damage)
    int32_t nbr[8]; // grid slots of the group's block and its +1 neighbours
};

constexpr uint64_t WAIT_LIMIT_NS = 2000000000ull; // 2 s: far beyond any copy; only a broken pipeline waits this long

// the producer: claims groups, cuts them into chunks and issues one bulk copy per payload field and chunk
template <class T, int CHUNK, int NBUF>
__device__ void scatter_producer(const StepArgs<T>& a, unsigned char* dyn, uint64_t* full, uint64_t* empty, ScatterItem* item)
{
    using S = ScatterShape<T, CHUNK, NBUF>;
    constexpr int WIN = S::WIN, VEC = S::VEC;
    const uint32_t G = a.st->n_items;
    uint32_t ph_empty = 3u; // parity bit per buffer; a fresh barrier counts as released
    uint32_t issues0 = 0, issues1 = 0;
    int b = 0;
    bool stop = false;
    while (!stop) {
        const uint32_t g = atomicAdd(&a.st->work_p2g, 1u);
        uint32_t qs = 0, qe = 0, flags = 0;
        int nf = 4;
        int32_t nbr[8];
        if (g < G) {
            const uint4 it = a.item[g];
            qs = it.x;
            qe = it.y;
            nf = a.scenes[a.kl.scene(a.kl.at(a.keys_sorted, qs))].damage ? NACC : 4;
#pragma unroll
            for (int d = 0; d < 8; d++) {
                nbr[d] = a.i_slot[(size_t)g * 8 + d];
                if (nbr[d] < 0) flags |= ITEM_BAD; // the lookup failed and raised FLAG_CAPACITY
                else if ((uint32_t)nbr[d] >= a.b_cap) {
                    check_failed(a.st, 4);
                    flags |= ITEM_BAD;
                }
            }
            if (qe <= qs || qe > a.n_total) {
                check_failed(a.st, 1);
                flags |= ITEM_BAD;
                qe = qs + 1 <= a.n_total ? qs + 1 : qs; // keep the pipeline moving with an in-bounds chunk
            }
        }
        else
            flags = ITEM_DONE;
        uint32_t q0 = qs;
        do {
            if (!mbar_wait(&empty[b], (ph_empty >> b) & 1u, WAIT_LIMIT_NS)) {
                raise_flag(a.st, FLAG_TIMEOUT);
                stop = true;
                break;
            }
            ph_empty ^= 1u << b;
            ScatterItem& it = item[b];
            if (b) issues1++;
            else issues0++;
            if (flags & ITEM_DONE) {
                it.flags = ITEM_DONE;
                mbar_arrive(&full[b]);
                stop = true;
                break;
            }
            const uint32_t q1 = min(q0 + (uint32_t)CHUNK, qe);
            const uint64_t p0 = pay_pos(q0) & ~(uint64_t)(VEC - 1);
            const uint64_t p1 = (pay_pos(q1 - 1) + VEC) & ~(uint64_t)(VEC - 1);
            uint32_t bytes = (uint32_t)(p1 - p0) * (uint32_t)sizeof(T);
            uint64_t src0 = p0;
            if (p1 > (uint64_t)a.pstride || bytes > (uint32_t)(WIN * sizeof(T))) { // never expected: record it, copy 16 in-bounds bytes
                check_failed(a.st, 2);
                flags |= ITEM_BAD;
                bytes = 16;
                src0 = 0;
            }
            it.q0 = q0;
            it.q1 = q1;
            it.base = (uint32_t)p0;
            it.flags = flags | (q1 == qe ? ITEM_LAST : 0u);
            it.nf = nf;
#pragma unroll
            for (int d = 0; d < 8; d++) it.nbr[d] = nbr[d];
            T* dst = reinterpret_cast<T*>(dyn + b * S::buf_bytes);
            fence_async_smem();
            mbar_arrive_expect_tx(&full[b], bytes * Pay<T>::N);
            for (int f = 0; f < Pay<T>::N; f++) bulk_load(dst + f * WIN, a.pay + f * a.pstride + src0, bytes, &full[b]);
            b = NBUF == 2 ? b ^ 1 : 0;
            q0 = q1;
        } while (q0 < qe);
    }
    // leave no copy in flight behind: wait (bounded) for the last phase issued on each buffer
    if (issues0) mbar_wait(&full[0], (issues0 - 1) & 1u, WAIT_LIMIT_NS);
    if (issues1) mbar_wait(&full[1], (issues1 - 1) & 1u, WAIT_LIMIT_NS);
}

template <class T, int CHUNK, int NBUF, int MIN_CTAS = ScatterShape<T, CHUNK, NBUF>::MIN_CTAS>
__global__ void __launch_bounds__(ScatterShape<T, CHUNK, NBUF>::NT, MIN_CTAS) k_scatter(StepArgs<T> a)
{
    using L = typename LayoutOf<T>::type;
    using S = ScatterShape<T, CHUNK, NBUF>;
    constexpr int NCONS = S::NCONS, WIN = S::WIN, NC = L::nodes;
    constexpr int TX = L::sx + 2, TY = L::sy + 2, TZ = L::sz + 2, TN = TX * TY * TZ;
    extern __shared__ __align__(128) unsigned char scat_dyn[];
    __shared__ T tile[NACC * TN];
    __shared__ __align__(8) uint64_t full[2], empty[2];
    __shared__ ScatterItem item[2];
    __shared__ int16_t cfirst[2][NC], clast[2][NC];
    __shared__ uint32_t ctag[2][NC];
    __shared__ int32_t s_nbr[8]; // the grid slots of the group being flushed (the item is released before the flush)
    __shared__ int s_stop;
    if (aborted_cta(a.st)) return;
    const int tid = threadIdx.x;
    if (tid == 0) {
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        mbar_init(&empty[0], NCONS / 32); // one arrival per consumer warp
        mbar_init(&empty[1], NCONS / 32);
        mbar_init_fence();
        s_stop = 0;
    }
    for (int q = tid; q < NACC * TN; q += S::NT) tile[q] = (T)0;
    for (int q = tid; q < 2 * NC; q += S::NT) (&ctag[0][0])[q] = 0xffffffffu;
    __syncthreads();
    if (tid >= NCONS) { // the producer warp (one lane works); no CTA-wide barrier follows this point
        if (tid == NCONS) scatter_producer<T, CHUNK, NBUF>(a, scat_dyn, full, empty, item);
        return;
    }
    // consumer role: cell c, stencil x-offset ii
    const int ii = tid / NC, c = tid % NC;
    const int cx = c >> (L::zbits + L::ybits), cy = (c >> L::zbits) & (L::sy - 1), cz = c & (L::sz - 1);
    uint32_t ph_full = 0; // parity bit per buffer
    int b = 0;
    for (uint32_t seq = 0;; seq++) {
        const bool ready = mbar_wait(&full[b], (ph_full >> b) & 1u, WAIT_LIMIT_NS);
        ph_full ^= 1u << b;
        const T* buf = reinterpret_cast<const T*>(scat_dyn + b * S::buf_bytes);
        const ScatterItem& it = item[b];
        uint32_t fl = ITEM_DONE;
        uint32_t q0 = 0, base = 0;
        if (!ready) {
            s_stop = 1;
            raise_flag(a.st, FLAG_TIMEOUT);
        }
        else {
            fl = it.flags;
            q0 = it.q0;
            base = it.base;
            if (!(fl & (ITEM_DONE | ITEM_BAD)) && (it.q1 <= q0 || it.q1 - q0 > (uint32_t)CHUNK || pay_pos(it.q1 - 1) - base >= (uint64_t)WIN)) {
                check_failed(a.st, 6); // an item that does not fit its window: skip it
                fl |= ITEM_BAD;
            }
            if (!(fl & (ITEM_DONE | ITEM_BAD))) {
                // runs of equal cells (particles are sorted by cell inside a block)
                const uint32_t q1 = it.q1;
                const T* cellv = buf + Pay<T>::CELL * WIN;
                for (uint32_t q = q0 + tid; q < q1; q += NCONS) {
                    const int e = (int)cellv[pay_pos(q) - base];
                    if ((unsigned)e >= (unsigned)NC) continue; // 255 marks a particle whose key disagreed
                    const int ep = q > q0 ? (int)cellv[pay_pos(q - 1) - base] : -1;
                    if (ep > e) check_failed(a.st, 3); // cells must ascend inside a block: the staged data is not what was written
                    if (q == q0 || ep != e) {
                        cfirst[b][e] = (int16_t)(q - q0);
                        ctag[b][e] = seq;
                    }
                    if (q + 1 == q1 || (int)cellv[pay_pos(q + 1) - base] != e) clast[b][e] = (int16_t)(q + 1 - q0);
                }
            }
        }
        bar_sync(1, NCONS);
        if (s_stop || (fl & ITEM_DONE)) break;
        const int nf = it.nf;
        const bool damage = nf == NACC;
        if ((fl & ITEM_LAST) && tid < 8) s_nbr[tid] = it.nbr[tid]; // read before this warp releases the item
        // per (cell, stencil x-offset): register accumulators of the thread's 9 nodes
        NodeAcc<T> acc;
        acc.zero();
        // decided once: after the release below, faster warps may already mark the next chunk
        const bool mine = !(fl & ITEM_BAD) && ctag[b][c] == seq;
        if (mine) {
            const uint32_t qa = q0 + cfirst[b][c], qb = q0 + clast[b][c];
            if (damage)
                for (uint32_t q = qa; q < qb; q++) accumulate_particle<T, WIN, true>(acc, buf + (pay_pos(q) - base), ii);
            else
                for (uint32_t q = qa; q < qb; q++) accumulate_particle<T, WIN, false>(acc, buf + (pay_pos(q) - base), ii);
        }
        // the chunk's payload is no longer needed: release the buffer (and the item) to the producer
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(&empty[b]);
        if (mine) add_to_tile<T, L>(acc, tile, cx, cy, cz, ii, nf);
        if (fl & ITEM_LAST) {
            bar_sync(1, NCONS); // every chunk of the group is in the tile
            if (!(fl & ITEM_BAD)) flush_tile<T, L>(a, tile, s_nbr, nf, tid, NCONS);
        }
        b = NBUF == 2 ? b ^ 1 : 0;
    }
}

// The fused P2G: one kernel per substep with the same arithmetic, the stress evaluated in the kernel. Per
// group, phase 1 (thread per particle) loads the particle state through the sorted order and stages its
// payload in shared memory (bank-staggered at q + q/8); phases 2 and 3 are those of k_scatter. No payload
// round trip through HBM, at the price of the state loads' latency inside the kernel: the autotuner times
// both forms on the workload.
// CH: particles staged per chunk (a whole block at 8 per cell by default; half of it lets more CTAs fit)
template <class T, int CH = (int)P2G_CHUNK<T>>
struct FusedShape {
    using L = typename LayoutOf<T>::type;
    static constexpr int NT = 3 * L::nodes; // cells x stencil x-offsets
    static constexpr int CHUNK = CH;
    static constexpr int CPAD = CHUNK + CHUNK / 8;
    static constexpr size_t dyn_bytes = sizeof(T) * Pay<T>::CELL * CPAD; // every field but the cell
};

// Elements [lo, hi] of one array, prefetched into L2 (widened to 16-byte boundaries, kept inside [base, end)).
template <class E>
__device__ __forceinline__ void prefetch_l2_range(const E* arr, int64_t lo, int64_t hi, const void* base, const void* end)
{
    uintptr_t b0 = (uintptr_t)(arr + lo) & ~(uintptr_t)15, b1 = ((uintptr_t)(arr + hi + 1) + 15) & ~(uintptr_t)15;
    const uintptr_t lo_lim = ((uintptr_t)base + 15) & ~(uintptr_t)15, hi_lim = (uintptr_t)end & ~(uintptr_t)15;
    b0 = b0 < lo_lim ? lo_lim : b0;
    b1 = b1 > hi_lim ? hi_lim : b1;
    if (b1 > b0) bulk_prefetch_l2((const void*)b0, (uint32_t)(b1 - b0));
}

// MINB: CTAs per SM the register budget is cut for (more CTAs hide more load latency; fewer registers may spill)
template <class T, int MODELS, int MINB, int CH = FusedShape<T>::CHUNK>
__global__ void __launch_bounds__(FusedShape<T, CH>::NT, MINB) k_p2g_fused(StepArgs<T> a)
{
    using L = typename LayoutOf<T>::type;
    using S = FusedShape<T, CH>;
    constexpr int NT = S::NT, CHUNK = S::CHUNK, CPAD = S::CPAD, NC = L::nodes;
    extern __shared__ __align__(16) unsigned char fused_dyn[];
    T* pay = reinterpret_cast<T*>(fused_dyn);
    __shared__ T tile[OffsetTiles<L>::ELEMS]; // one node tile per stencil x-offset
    __shared__ uint8_t cellof[CHUNK];
    __shared__ uint32_t s_piece[NT];
    // the set-up of the current group (buffer b) and of the next one (b ^ 1): group, scene, a bad neighbour slot,
    // the grid slots of the block and its +1 neighbours, the block origin, the sorted range
    __shared__ int s_g[2], s_scene[2], s_bad[2];
    __shared__ int32_t s_nbr[2][8];
    __shared__ int s_org[2][3];
    __shared__ uint32_t s_se[2][2];
    __shared__ __align__(16) uint4 s_next; // the item claimed ahead
    if (aborted_cta(a.st)) return;
    const uint32_t G = a.st->n_items;
    const int tid = threadIdx.x;
    // Items (groups or pieces of them) are claimed one ahead: thread 0 claims the next item at the start of one and copies its
    // range into shared memory while the accumulation runs; around the flush lanes 0-7 load its block's neighbours (lane 0
    // also the key of its first particle) and write them into the other buffer before the last barrier, so no barrier waits
    // on a claim alone. A group's neighbour entries are hash positions; the set-up translates them into grid slots and writes
    // those for G2P.
    auto setup_store = [&](int bb, int gn, uint32_t st, uint32_t en, int32_t hpos) { // lanes 0-7 of warp 0
        const uint64_t key0 = tid == 0 ? a.kl.at(a.keys_sorted, st) : 0ull;
        const int32_t slot = nbr_slot(a, hpos);
        a.i_slot[(size_t)gn * 8 + tid] = slot;
        const unsigned badm = __ballot_sync(0xffu, slot < 0 || (uint32_t)slot >= a.b_cap); // a failed lookup raised FLAG_CAPACITY
        s_nbr[bb][tid] = slot;
        if (tid == 0) {
            uint32_t bi, bj, bk;
            L::block_of_page(a.kl.page(key0), bi, bj, bk);
            s_g[bb] = gn;
            s_bad[bb] = badm != 0;
            s_scene[bb] = (int)a.kl.scene(key0);
            s_org[bb][0] = (int)(bi * L::sx);
            s_org[bb][1] = (int)(bj * L::sy);
            s_org[bb][2] = (int)(bk * L::sz);
            s_se[bb][0] = st;
            s_se[bb][1] = en;
        }
    };
    const int ii = tid / NC, c = tid % NC;
    for (int q = tid; q < OffsetTiles<L>::ELEMS; q += NT) tile[q] = (T)0;
    uint32_t fallbacks = 0;
    // the first item is the CTA's own number (claims count from the grid's size)
    if (tid < 8) {
        const int g0 = blockIdx.x;
        if (g0 < (int)G) {
            const uint4 it = a.item[g0];
            setup_store(0, g0, it.x, it.y, a.g_nbr[(size_t)it.z * 8 + tid]);
        }
        else if (tid == 0)
            s_g[0] = g0;
    }
    __syncthreads();
    int bcur = 0;
    for (;;) {
        const int g = s_g[bcur];
        if (g >= (int)G) break;
        // the next item, claimed now (its set-up is loaded around this item's flush)
        int claimed = 0;
        if (tid == 0) claimed = (int)(gridDim.x + atomicAdd(&a.st->work_p2g, 1u));
        const uint32_t start = s_se[bcur][0], end = s_se[bcur][1];
        const bool bad = s_bad[bcur] != 0;
        const SceneParams<T>& sp = a.scenes[s_scene[bcur]];
        const int nf = sp.damage ? NACC : 4;
        // The state of the item one round of claims ahead (whichever CTA takes it) is prefetched into L2 while this
        // group runs, so that its phase 1 reads L2: the lanes of warp 1 take one array each (state fields P_X .. P_D
        // and the particle ids). Its storage range is that of its first and last sorted particles (storage keeps the
        // previous substep's sorted order; a range that does not look like one group is skipped). The loads are
        // spread over the group so that none of them is waited for.
        constexpr int NPF = P_D + 2;
        const int gpf = g + (int)gridDim.x, pfl = tid - 32;
        const bool pf = (a.opts & OPT_PREFETCH) && pfl >= 0 && pfl < NPF && gpf < (int)G;
        uint32_t pf_a = 0, pf_b = 0, pf_j0 = 0, pf_j1 = 0;
        if (pf) {
            const uint4 it = a.item[gpf];
            pf_a = it.x;
            pf_b = it.y;
        }
        for (uint32_t c0 = start; c0 < end && !bad; c0 += CHUNK) {
            const int cnt = (int)min((uint32_t)CHUNK, end - c0);
            // ---- phase 1: per particle
            // the storage slots of all the thread's particles first (one latency for all), then one particle at a time
            constexpr int PER = (CHUNK + NT - 1) / NT;
            uint32_t js[PER];
#pragma unroll
            for (int k = 0; k < PER; k++) js[k] = tid + k * NT < cnt ? a.vals_sorted[c0 + tid + k * NT] : 0u;
#pragma unroll
            for (int k = 0; k < PER; k++) {
                const int q = tid + k * NT;
                if (q >= cnt) break;
                int b[3];
                particle_payload<T, MODELS>(a.pin, js[k], sp, pay + (q + (q >> 3)), CPAD, b, fallbacks);
                const int l0 = b[0] - s_org[bcur][0], l1 = b[1] - s_org[bcur][1], l2 = b[2] - s_org[bcur][2];
                const bool inside = l0 >= 0 && l0 < L::sx && l1 >= 0 && l1 < L::sy && l2 >= 0 && l2 < L::sz;
                if (!inside) raise_flag(a.st, FLAG_CAPACITY); // keys and positions disagree: abort the substep
                cellof[q] = inside ? (uint8_t)L::element(l0, l1, l2) : (uint8_t)0xff;
            }
            __syncthreads();
            if (tid == 0 && c0 == start && claimed < (int)G) cp_async<16>(&s_next, a.item + claimed);
            // ---- phases 2 and 3. Particles of one cell are contiguous and the cells ascend (sorted by cell inside
            // the block): the cell's range by two binary searches over the chunk's cells, no pass or barrier of its
            // own (a position that disagreed with its key has raised FLAG_CAPACITY; the searches stay in [0, cnt])
            auto cell_lower = [&](int v) {
                int lo = 0, hi = cnt;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (cellof[mid] < v) lo = mid + 1;
                    else hi = mid;
                }
                return lo;
            };
            int qa = cell_lower(c), qb = cell_lower(c + 1);
            s_piece[tid] = split_cells<T>(c, qa, qb); // (read back after the accumulation: it holds no register through it)
            NodeAcc<T> acc;
            acc.zero();
            if (nf == NACC)
                for (int q = qa; q < qb; q++) accumulate_particle<T, CPAD, true>(acc, pay + (q + (q >> 3)), ii);
            else
                for (int q = qa; q < qb; q++) accumulate_particle<T, CPAD, false>(acc, pay + (q + (q >> 3)), ii);
            const uint32_t piece = s_piece[tid], parts = piece >> 20; // (parts: the same for the whole warp)
            if (parts) {
                const int cell = piece & 0xff;
                add_pieces_to_offset_tile<T, L>(acc, tile, cell & (NC - 1), ii, nf, cell < NC, (piece >> 8) & 0xfff, (int)parts);
            }
            else
                add_to_offset_tile<T, L>(acc, tile, c, ii, nf); // all lanes (an empty cell adds zeros)
            __syncthreads();
        }
        int gn = (int)G;
        uint4 nit = make_uint4(0, 0, 0, 0);
        int32_t n_hpos = -1;
        if (tid < 32) {
            if (tid == 0) {
                if (bad && claimed < (int)G) s_next = a.item[claimed];
                cp_async_wait_all();
            }
            __syncwarp();
            gn = __shfl_sync(0xffffffffu, claimed, 0);
            if (tid < 8 && gn < (int)G) {
                nit = s_next;
                n_hpos = a.g_nbr[(size_t)nit.z * 8 + tid];
            }
        }
        if (pf && pf_b > pf_a && pf_b <= a.n_total) {
            pf_j0 = a.vals_sorted[pf_a];
            pf_j1 = a.vals_sorted[pf_b - 1];
        }
        if (!bad) flush_offset_tiles<T, L>(a, tile, s_nbr[bcur], nf, tid, NT);
        if (pf && pf_j1 >= pf_j0 && pf_j1 - pf_j0 < 2 * (pf_b - pf_a) + 64) {
            const Pool<T>& P = a.pin;
            if (pfl < NPF - 1)
                prefetch_l2_range(P.f + (int64_t)pfl * P.stride, pf_j0, pf_j1, P.f, P.f + (int64_t)P_NF * P.stride);
            else
                prefetch_l2_range(P.pid, pf_j0, pf_j1, P.pid, P.pid + P.stride);
        }
        // the next group's set-up into the other buffer (the flush above read this one)
        if (tid < 8) {
            if (gn < (int)G)
                setup_store(bcur ^ 1, gn, nit.x, nit.y, n_hpos);
            else if (tid == 0)
                s_g[bcur ^ 1] = gn;
        }
        __syncthreads();
        bcur ^= 1;
    }
    if (fallbacks) atomicAdd(&a.st->fallback, fallbacks);
}

// ---------------------------------------------------------------------------------------------------
// Warp-specialised fused P2G (the same arithmetic as k_p2g_fused). Producer warps load each chunk's particle
// state, evaluate V0 tau and stage the payload in one of NSTAGE shared-memory buffers; consumer warps (thread per
// (cell, stencil x-offset)) accumulate the previous buffer meanwhile, so the state loads' latency and the
// accumulation overlap inside the CTA instead of alternating behind CTA-wide barriers. Hand-offs are mbarriers:
// full[s] completes when every producer thread has written buffer s, empty[s] when every consumer warp has read
// it. A group's node tiles are double-buffered: the consumer warps meet on one mbarrier before the flush of a
// group, while the next group's additions go to the other tile buffer. Every wait is bounded (2 s) and raises
// FLAG_TIMEOUT. Groups are dealt to CTAs round-robin (blockIdx, + gridDim, ...), so every producer thread knows
// the sequence of chunks without exchanging it.
// ---------------------------------------------------------------------------------------------------
template <class T>
struct WsShape {
    using L = typename LayoutOf<T>::type;
    static constexpr int NCONS = 3 * L::nodes; // consumers: cells x stencil x-offsets
    static constexpr int NPROD = sizeof(T) == 4 ? 128 : 64;
    static constexpr int NT = NCONS + NPROD;
    static constexpr int CHUNK = sizeof(T) == 4 ? 256 : 128;
    static constexpr int CPAD = CHUNK + CHUNK / 8;
    static constexpr int NSTAGE = 2;
    static constexpr size_t pay_bytes = sizeof(T) * Pay<T>::CELL * CPAD;
    static constexpr size_t stage_bytes = pay_bytes + CHUNK; // payload fields, then the cells
    static constexpr size_t dyn_bytes = NSTAGE * stage_bytes;
    static_assert(pay_bytes % 16 == 0 && NCONS % 32 == 0 && NPROD % 32 == 0, "whole warps, aligned buffers");
};

struct WsItem {
    uint32_t c0; // first sorted particle of the chunk
    int32_t cnt, flags, scene, nf;
    int32_t nbr[8];
};

template <class T, int MODELS>
__global__ void __launch_bounds__(WsShape<T>::NT, 2) k_p2g_ws(StepArgs<T> a)
{
    using L = typename LayoutOf<T>::type;
    using S = WsShape<T>;
    using OT = OffsetTiles<L>;
    constexpr int NCONS = S::NCONS, NPROD = S::NPROD, CHUNK = S::CHUNK, CPAD = S::CPAD, NST = S::NSTAGE, NC = L::nodes;
    extern __shared__ __align__(16) unsigned char ws_dyn[];
    __shared__ T tiles[2][OT::ELEMS]; // one set of per-offset node tiles per group parity
    __shared__ __align__(8) uint64_t full[NST], empty[NST], flushed;
    __shared__ WsItem item[NST];
    __shared__ int32_t s_nbr[2][8];
    if (aborted_cta(a.st)) return;
    const int tid = threadIdx.x;
    if (tid == 0) {
        for (int s = 0; s < NST; s++) {
            mbar_init(&full[s], NPROD);
            mbar_init(&empty[s], NCONS / 32);
        }
        mbar_init(&flushed, NCONS / 32);
        mbar_init_fence();
    }
    for (int q = tid; q < 2 * OT::ELEMS; q += S::NT) (&tiles[0][0])[q] = (T)0;
    __syncthreads(); // the last CTA-wide barrier: the roles never meet again
    const uint32_t G = a.st->n_items;
    if (tid >= NCONS) {
        // ---------------- producers
        const int pt = tid - NCONS;
        uint32_t fallbacks = 0, k = 0;
        bool stop = false;
        for (uint32_t g = blockIdx.x; g < G && !stop; g += gridDim.x) {
            const uint4 wit = a.item[g];
            const uint32_t start = wit.x, end = wit.y;
            const uint64_t key0 = a.kl.at(a.keys_sorted, start);
            uint32_t bi, bj, bk;
            L::block_of_page(a.kl.page(key0), bi, bj, bk);
            const int scene = (int)a.kl.scene(key0);
            const int org0 = (int)(bi * L::sx), org1 = (int)(bj * L::sy), org2 = (int)(bk * L::sz);
            const SceneParams<T>& sp = a.scenes[scene];
            int bad = (end <= start || end > a.n_total) ? 1 : 0;
            if (bad) check_failed(a.st, 1);
            for (uint32_t c0 = start; c0 < end || (bad && c0 == start); c0 += CHUNK) {
                const int s = k % NST;
                if (!mbar_wait(&empty[s], ((k / NST) & 1u) ^ 1u, WAIT_LIMIT_NS)) {
                    raise_flag(a.st, FLAG_TIMEOUT);
                    stop = true;
                    break;
                }
                const int cnt = bad ? 0 : (int)min((uint32_t)CHUNK, end - c0);
                const bool last = bad || c0 + CHUNK >= end;
                WsItem& it = item[s];
                if (pt < 32) { // the first producer warp fills the item; a failed slot lookup raised FLAG_CAPACITY
                    int slot = 0;
                    if (pt < 8) {
                        slot = a.i_slot[(size_t)g * 8 + pt];
                        it.nbr[pt] = slot;
                    }
                    const bool nbad = __ballot_sync(0xffffffffu, pt < 8 && (slot < 0 || (uint32_t)slot >= a.b_cap)) != 0;
                    if (pt == 0) {
                        it.c0 = c0;
                        it.cnt = cnt;
                        it.scene = scene;
                        it.nf = sp.damage ? NACC : 4;
                        it.flags = (last ? ITEM_LAST : 0) | ((bad || nbad) ? ITEM_BAD : 0);
                    }
                }
                T* pay = reinterpret_cast<T*>(ws_dyn + s * S::stage_bytes);
                uint8_t* cellof = ws_dyn + s * S::stage_bytes + S::pay_bytes;
                constexpr int PER = (CHUNK + NPROD - 1) / NPROD;
                uint32_t js[PER];
#pragma unroll
                for (int r = 0; r < PER; r++) js[r] = pt + r * NPROD < cnt ? a.vals_sorted[c0 + pt + r * NPROD] : 0u;
#pragma unroll
                for (int r = 0; r < PER; r++) {
                    const int q = pt + r * NPROD;
                    if (q >= cnt) break;
                    int b[3];
                    particle_payload<T, MODELS>(a.pin, js[r], sp, pay + (q + (q >> 3)), CPAD, b, fallbacks);
                    const int l0 = b[0] - org0, l1 = b[1] - org1, l2 = b[2] - org2;
                    const bool inside = l0 >= 0 && l0 < L::sx && l1 >= 0 && l1 < L::sy && l2 >= 0 && l2 < L::sz;
                    if (!inside) raise_flag(a.st, FLAG_CAPACITY); // keys and positions disagree: abort the substep
                    cellof[q] = inside ? (uint8_t)L::element(l0, l1, l2) : (uint8_t)0xff;
                }
                mbar_arrive(&full[s]);
                k++;
                if (bad) break;
            }
        }
        if (!stop) { // the end marker
            const int s = k % NST;
            if (mbar_wait(&empty[s], ((k / NST) & 1u) ^ 1u, WAIT_LIMIT_NS)) {
                if (pt == 0) item[s].flags = ITEM_DONE;
                mbar_arrive(&full[s]);
            }
            else
                raise_flag(a.st, FLAG_TIMEOUT);
        }
        if (fallbacks) atomicAdd(&a.st->fallback, fallbacks);
        return;
    }
    // ---------------- consumers: cell c, stencil x-offset ii
    const int ii = tid / NC, c = tid % NC, lane = tid & 31;
    int tb = 0; // tile buffer of the current group
    uint32_t gseq = 0; // groups flushed (parity of the flush barrier)
    for (uint32_t k = 0;; k++) {
        const int s = k % NST;
        const bool ok = __all_sync(0xffffffffu, mbar_wait(&full[s], (k / NST) & 1u, WAIT_LIMIT_NS));
        if (!ok) {
            if (lane == 0) raise_flag(a.st, FLAG_TIMEOUT);
            break;
        }
        const WsItem& it = item[s];
        const int fl = it.flags;
        if (fl & ITEM_DONE) break;
        const int cnt = it.cnt, nf = it.nf;
        const T* pay = reinterpret_cast<const T*>(ws_dyn + s * S::stage_bytes);
        const uint8_t* cellof = ws_dyn + s * S::stage_bytes + S::pay_bytes;
        if ((fl & ITEM_LAST) && tid < 8) s_nbr[tb][tid] = it.nbr[tid]; // read before this warp releases the buffer
        NodeAcc<T> acc;
        acc.zero();
        const bool use = !(fl & ITEM_BAD);
        if (use) {
            auto cell_lower = [&](int v) {
                int lo = 0, hi = cnt;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (cellof[mid] < v) lo = mid + 1;
                    else hi = mid;
                }
                return lo;
            };
            const int qa = cell_lower(c), qb = cell_lower(c + 1);
            if (nf == NACC)
                for (int q = qa; q < qb; q++) accumulate_particle<T, CPAD, true>(acc, pay + (q + (q >> 3)), ii);
            else
                for (int q = qa; q < qb; q++) accumulate_particle<T, CPAD, false>(acc, pay + (q + (q >> 3)), ii);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]); // the buffer is free for the producers
        if (use) add_to_offset_tile<T, L>(acc, tiles[tb], c, ii, nf); // all lanes (an empty cell adds zeros)
        if (fl & ITEM_LAST) {
            // every consumer warp has added the group: flush its tiles (the next group fills the other tile buffer)
            __syncwarp();
            if (lane == 0) mbar_arrive(&flushed);
            const bool fok = __all_sync(0xffffffffu, mbar_wait(&flushed, gseq & 1u, WAIT_LIMIT_NS));
            gseq++;
            if (!fok) {
                if (lane == 0) raise_flag(a.st, FLAG_TIMEOUT);
                break;
            }
            if (use) flush_offset_tiles<T, L>(a, tiles[tb], s_nbr[tb], nf, tid, NCONS);
            else
                for (int q = tid; q < OT::ELEMS; q += NCONS) tiles[tb][q] = (T)0; // a bad group's partial sums are dropped
            tb ^= 1;
        }
    }
}

// ---------------------------------------------------------------------------------------------------
// grid update
// ---------------------------------------------------------------------------------------------------
constexpr int GRID_NT = 256; // threads per CTA of the grid update

template <class T>
__global__ void __launch_bounds__(GRID_NT) k_grid(StepArgs<T> a)
{
    using L = typename LayoutOf<T>::type;
    // GV consecutive nodes of one block per thread: every field moves as one 16-byte access; TPB threads cover
    // one block (16 in both precisions), so a warp spans 32 / TPB blocks, which may belong to different scenes
    constexpr int GV = (int)(16 / sizeof(T));
    constexpr int TPB = L::nodes / GV;
    static_assert(L::nodes % GV == 0, "a block holds whole vectors");
    static_assert(32 % TPB == 0 && GRID_NT % TPB == 0, "a warp holds whole blocks");
    __shared__ double s_mass[GRID_NT / TPB];
    __shared__ int s_msc[GRID_NT / TPB];
    if (aborted_cta(a.st)) return;
    const uint32_t B = min(a.st->n_blocks, a.b_cap);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.st->max_blocks_seen = max(a.st->max_blocks_seen, B);
        a.st->max_groups_seen = max(a.st->max_groups_seen, a.st->n_groups);
    }
    const uint32_t total = B * (L::nodes / GV);
    // every thread of the CTA runs the same iterations (the loop holds barriers)
    for (uint32_t base = blockIdx.x * GRID_NT; base < total; base += gridDim.x * GRID_NT) {
        const uint32_t t = base + threadIdx.x;
        double gm = 0; // grid mass of the thread's nodes, accumulated in FP64 from the first add
        int scene = -1;
        if (t < total) {
            const uint32_t b = t / (L::nodes / GV), e0 = (t % (L::nodes / GV)) * GV;
            const uint64_t hk = a.b_key[b];
            scene = (int)(hk >> 40);
            const SceneParams<T>& sp = a.scenes[scene];
            Vec16<T>* A = reinterpret_cast<Vec16<T>*>(a.acc + (size_t)b * NACC * L::nodes + e0);
            constexpr int FS = L::nodes / GV; // field stride in vectors
            const Vec16<T> m = A[0], P0 = A[FS], P1 = A[2 * FS], P2 = A[3 * FS], pf = A[4 * FS], pfm = A[5 * FS];
            Vec16<T> zero;
#pragma unroll
            for (int k = 0; k < GV; k++) zero.v[k] = (T)0;
#pragma unroll
            for (int q = 0; q < NACC; q++) A[q * FS] = zero;
            Vec16<T> o0, o1, o2, o3;
            uint32_t bi, bj, bk;
            L::block_of_page(hk & ((1ULL << 40) - 1), bi, bj, bk);
            const T dt = sp.dt;
#pragma unroll
            for (int k = 0; k < GV; k++) {
                const T mk = m.v[k];
                gm += (double)mk;
                if (mk != (T)0) {
                    const int e = (int)e0 + k;
                    const int lx = e >> (L::zbits + L::ybits), ly = (e >> L::zbits) & (L::sy - 1), lz = e & (L::sz - 1);
                    const T xi[3] = { (T)(bi * L::sx + lx) * sp.dx, (T)(bj * L::sy + ly) * sp.dx, (T)(bk * L::sz + lz) * sp.dx };
                    // P = m v + dt f: v + g dt + f dt / m (MpmSimulationBase.cpp:1204-1210)
                    T vi[3] = { P0.v[k] / mk + sp.gravity[0] * dt, P1.v[k] / mk + sp.gravity[1] * dt, P2.v[k] / mk + sp.gravity[2] * dt };
                    collide(sp, (T)sp.time, xi, vi);
                    o0.v[k] = vi[0];
                    o1.v[k] = vi[1];
                    o2.v[k] = vi[2];
                    o3.v[k] = pfm.v[k] != (T)0 ? pf.v[k] / pfm.v[k] : (T)0;
                }
                else
                    o0.v[k] = o1.v[k] = o2.v[k] = o3.v[k] = (T)0;
            }
            Vec16<T>* V = reinterpret_cast<Vec16<T>*>(a.vel + (size_t)b * NVEL * L::nodes + e0);
            V[0] = o0;
            V[FS] = o1;
            V[2 * FS] = o2;
            V[3 * FS] = o3;
        }
        // grid mass per scene (MpmSimulationDataAnalysis.h:130-151, FP64): the TPB threads of one block (one scene)
        // sum in a segmented shuffle, then thread 0 combines the CTA's block sums, one atomic per run of blocks of
        // one scene (a single scene would otherwise send every block's atomic to the same address). Threads past
        // the last block form whole segments with scene -1 (total and base are multiples of TPB).
        double s = gm;
        for (int o = TPB / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, TPB);
        if (threadIdx.x % TPB == 0) {
            s_mass[threadIdx.x / TPB] = s;
            s_msc[threadIdx.x / TPB] = scene;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double run = 0;
            int rsc = -1;
            for (int w = 0; w < GRID_NT / TPB; w++) {
                if (s_msc[w] != rsc) {
                    if (rsc >= 0 && run != 0.0) atomicAdd(&a.grid_mass[rsc], run);
                    rsc = s_msc[w];
                    run = 0;
                }
                run += s_mass[w];
            }
            if (rsc >= 0 && run != 0.0) atomicAdd(&a.grid_mass[rsc], run);
        }
        __syncthreads();
    }
    // the sort's counters and the hash table are used only up to P2G: clear them for the next substep
    for (uint32_t h = blockIdx.x * blockDim.x + threadIdx.x; h < a.sort_zero_n; h += gridDim.x * blockDim.x) a.sort_zero[h] = 0;
    for (uint32_t h = blockIdx.x * blockDim.x + threadIdx.x; h <= a.h_mask; h += gridDim.x * blockDim.x) a.h_keys[h] = HASH_EMPTY;
}

// ---------------------------------------------------------------------------------------------------
// G2P
// ---------------------------------------------------------------------------------------------------
// NT threads per CTA; RESIDENT: threads per SM the register budget is cut for
// G2P's staged particle state: x, F, m, V0, d, sigma_c (fields G2P_SF) and the pid, per thread and buffer
enum { GS_X = 0, GS_F = 3, GS_M = 12, GS_V0 = 13, GS_D = 14, GS_SC = 15, G2P_SF = 16 };
constexpr size_t G2P_HALO = 8 * 1024; // dynamic shared memory of the variants that stage the 8 blocks' velocities
template <class T, int NT>
struct G2pStage {
    // double-buffered per-thread slots, field-major so a warp's accesses are consecutive words; off where the
    // buffers would not fit the 48 KB of static shared memory (FP64 at 256 threads)
    static constexpr bool ON = 2 * NT * (G2P_SF * sizeof(T) + 4) <= 40 * 1024;
    static constexpr int NS = ON ? 2 * G2P_SF * NT : 1, NP = ON ? 2 * NT : 1;
};

// infinity or NaN; FP64 looks at the exponent bits, as a comparison would occupy the FP64 pipe
__device__ __forceinline__ bool nonfinite(float x) { return !isfinite(x); }
__device__ __forceinline__ bool nonfinite(double x) { return (__double2hiint(x) & 0x7ff00000) == 0x7ff00000; }

// Sums of a particle's 27 nodes. Separable: the stencil weight is wx_i wy_j wz_k, so sums over k, then j, then i give
//   pv = sum w v,  M_rc = sum w v_r delta_c,  Gv_rc = sum v_r (grad w)_c dx,
// and with damage the Laplacian (below) and pw = sum w (phase field).
// Along z the sums come from the middle node v1 and the differences e0 = v1 - v0, e1 = v2 - v1 of the line's three nodes,
// staged beside the velocities: as sum w = 1, sum dw = 0 and w1 + 2 w2 = f (the fractional position),
//   sum w v = v1 - w0 e0 + w2 e1,   sum dw v = -dw0 e0 + dw2 e1,   sum k w v = f v1 + 2 w2 e1,
// six operations a component instead of eight, and the gradients are sums of differences that are already taken. FP32 runs
// on pairs (velocity lanes (x, y) and (z, phase field)), FP64 on scalars without the phase field where there is none (DMG).
// tv, te: the particle's corner in the staged tiles, Z1 / Z2 nodes per line.
template <class T>
struct Gathered {
    T pv[3], M[9], Gv[9], lap, pw;
};
template <class T, class L, bool DMG>
__device__ __forceinline__ void gather(const Quad<T>* tv, const Quad<T>* te, const T (&w)[3][3], const T (&dw)[3][3], T fz, Gathered<T>& o)
{
    constexpr int TY = L::sy + 2, Z1 = L::sz, Z2 = L::sz + 1;
#pragma unroll
    for (int r = 0; r < 3; r++) o.pv[r] = 0;
#pragma unroll
    for (int r = 0; r < 9; r++) o.M[r] = o.Gv[r] = 0;
    o.lap = o.pw = 0;
    const T nw0 = -w[2][0], w2 = w[2][2], nd0 = -dw[2][0], d2 = dw[2][2], kw2 = (T)2 * w2;
#pragma unroll
    for (int ii = 0; ii < 3; ii++) {
        // per x-offset: S = sum wy s, U = sum dwy s, Tz = sum wy t, K = sum wy u, J = sum j wy s; lA, lB, lC of the phase field
        T Si[3], Ui[3], Ti[3], Ki[3], Ji[3], lA, lB, lC;
        if constexpr (sizeof(T) == 4) {
            using PT = typename PairOf<T>::type;
            const PT Z = pmake<PT>((T)0, (T)0);
            const PT NW0 = pmake<PT>(nw0, nw0), W2 = pmake<PT>(w2, w2), ND0 = pmake<PT>(nd0, nd0), D2 = pmake<PT>(d2, d2), KW2 = pmake<PT>(kw2, kw2),
                     FZ = pmake<PT>(fz, fz);
            // (S_x, S_y) (S_z, lA) (U_x, U_y) (U_z, lB) (T_x, T_y) (T_z, lC) (K_x, K_y) (K_z, -) (J_x, J_y) (J_z, -)
            PT S01 = Z, S2A = Z, U01 = Z, U2B = Z, T01 = Z, T2C = Z, K01 = Z, J01 = Z;
            T K2 = 0, J2 = 0;
#pragma unroll
            for (int jj = 0; jj < 3; jj++) {
                const Quad<T> v1 = tv[(ii * TY + jj) * Z1], e0 = te[(ii * TY + jj) * Z2], e1 = te[(ii * TY + jj) * Z2 + 1];
                const PT v01 = pmake<PT>(v1.x, v1.y), v2f = pmake<PT>(v1.z, v1.w), a01 = pmake<PT>(e0.x, e0.y), a2f = pmake<PT>(e0.z, e0.w),
                         b01 = pmake<PT>(e1.x, e1.y), b2f = pmake<PT>(e1.z, e1.w);
                // (s_x, s_y) (s_z, pz) (t_x, t_y) (t_z, p1) (u_x, u_y) u_z
                const PT s01 = pfma(W2, b01, pfma(NW0, a01, v01)), s2z = pfma(W2, b2f, pfma(NW0, a2f, v2f));
                const PT t01 = pfma(D2, b01, pmul(ND0, a01));
                PT t2p = pfma(pmake<PT>(d2, (T)1), b2f, pmul(pmake<PT>(nd0, (T)-1), a2f));
                t2p.y = (T)3 * v1.w + t2p.y;
                const PT u01 = pfma(KW2, b01, pmul(FZ, v01));
                const T u2 = kw2 * e1.z + fz * v1.z;
                const T wj = w[1][jj], dwj = dw[1][jj];
                const PT WJ = pmake<PT>(wj, wj);
                S01 = pfma(WJ, s01, S01);
                S2A = pfma(WJ, s2z, S2A);
                U01 = pfma(pmake<PT>(dwj, dwj), s01, U01);
                U2B = pfma(pmake<PT>(dwj, (T)1), s2z, U2B);
                T01 = pfma(WJ, t01, T01);
                T2C = pfma(WJ, t2p, T2C);
                K01 = pfma(WJ, u01, K01);
                K2 = wj * u2 + K2;
                if (jj) {
                    const T jw = (T)jj * wj;
                    J01 = pfma(pmake<PT>(jw, jw), s01, J01);
                    J2 = jw * s2z.x + J2;
                }
            }
            Si[0] = S01.x, Si[1] = S01.y, Si[2] = S2A.x;
            Ui[0] = U01.x, Ui[1] = U01.y, Ui[2] = U2B.x;
            Ti[0] = T01.x, Ti[1] = T01.y, Ti[2] = T2C.x;
            Ki[0] = K01.x, Ki[1] = K01.y, Ki[2] = K2;
            Ji[0] = J01.x, Ji[1] = J01.y, Ji[2] = J2;
            lA = S2A.y, lB = U2B.y, lC = T2C.y;
        }
        else {
            lA = lB = lC = 0;
#pragma unroll
            for (int jj = 0; jj < 3; jj++) {
                const Quad<T> v1 = tv[(ii * TY + jj) * Z1], e0 = te[(ii * TY + jj) * Z2], e1 = te[(ii * TY + jj) * Z2 + 1];
                const T v[3] = { v1.x, v1.y, v1.z }, a[3] = { e0.x, e0.y, e0.z }, b[3] = { e1.x, e1.y, e1.z };
                const T wj = w[1][jj], dwj = dw[1][jj], jw = (T)jj * wj;
#pragma unroll
                for (int r = 0; r < 3; r++) {
                    const T sr = w2 * b[r] + (nw0 * a[r] + v[r]), tr = d2 * b[r] + nd0 * a[r], ur = kw2 * b[r] + fz * v[r];
                    Si[r] = jj ? wj * sr + Si[r] : wj * sr;
                    Ui[r] = jj ? dwj * sr + Ui[r] : dwj * sr;
                    Ti[r] = jj ? wj * tr + Ti[r] : wj * tr;
                    Ki[r] = jj ? wj * ur + Ki[r] : wj * ur;
                    if (jj) Ji[r] = jj > 1 ? jw * sr + Ji[r] : jw * sr;
                }
                if (DMG) {
                    const T ps = w2 * e1.w + (nw0 * e0.w + v1.w), p1 = (T)3 * v1.w + (e1.w - e0.w);
                    lA = wj * ps + lA;
                    lB += ps;
                    lC = wj * p1 + lC;
                }
            }
        }
        const T wi = w[0][ii], dwi = dw[0][ii];
#pragma unroll
        for (int r = 0; r < 3; r++) {
            o.pv[r] += wi * Si[r];
            if (ii) o.M[3 * r] += ((T)ii * wi) * Si[r];
            o.M[3 * r + 1] += wi * Ji[r];
            o.M[3 * r + 2] += wi * Ki[r];
            o.Gv[3 * r] += dwi * Si[r];
            o.Gv[3 * r + 1] += wi * Ui[r];
            o.Gv[3 * r + 2] += wi * Ti[r];
        }
        // the reference's 3D Laplacian weights every term with d2w(i) = (1,-2,1)(i) (MpmGrid.h:607-613):
        // sum_jk pf * d2w_i (wy_j wz_k + wx_i wz_k + wx_i wy_j)
        if (DMG) {
            o.lap += (ii == 1 ? (T)-2 : (T)1) * (lA + wi * (lB + lC));
            o.pw += wi * lA; // sum w times the node field (the damage change of an implicit solve)
        }
    }
}

// BULK: the 8 neighbouring blocks' velocities reach shared memory by bulk asynchronous copies (one 4-field block of
// NVEL * nodes values per copy, completing on an mbarrier) and the node tile is built from there; otherwise each
// thread loads its tile nodes from global memory. The copies land in dynamic shared memory (G2P_HALO bytes): beside the tiles and
// the staged state, FP32 at 256 threads and FP64 at 128 would pass the 48 KB a kernel's static shared memory may have.
// DRIVE: the damage the batch's scenes can have: none, on the Borden model only, any (the drive of the QR-stable model brings a
// QR factorisation and a polar decomposition into the kernel)
enum { DRIVE_NONE = 0, DRIVE_BORDEN = 1, DRIVE_ANY = 2 };
template <class T, int NT, int RESIDENT, bool BULK = false, int DRIVE = DRIVE_ANY>
__global__ void __launch_bounds__(NT, RESIDENT / NT) k_g2p(StepArgs<T> a)
{
    constexpr bool QR = DRIVE == DRIVE_ANY;
    using L = typename LayoutOf<T>::type;
    using GS = G2pStage<T, NT>;
    constexpr int BLK = NVEL * L::nodes; // values of one block's velocity fields (1 KB in both precisions)
    static_assert(8 * BLK * sizeof(T) == G2P_HALO, "eight blocks");
    extern __shared__ __align__(128) unsigned char g2p_dyn[];
    T* s_halo = reinterpret_cast<T*>(g2p_dyn); // (BULK)
    __shared__ __align__(8) uint64_t s_hbar;
    uint32_t hphase = 0;
    // the grid velocities around the group's block as one dense node tile (the block plus 2 nodes on the
    // + side of every axis, the reach of the quadratic stencil): every stencil read is a fixed offset
    constexpr int TY = L::sy + 2, TZ = L::sz + 2, TN = (L::sx + 2) * TY * TZ;
    static_assert(NVEL == 4, "one Quad per tile node");
    // node-major (the 4 fields of a node in one access): the nodes that can be the middle of a z line, and the z differences
    constexpr int Z1 = L::sz, Z2 = L::sz + 1, COLS = (L::sx + 2) * TY;
    static_assert(TZ == 6, "five columns of six nodes per warp");
    __shared__ Quad<T> tv[COLS * Z1], te[COLS * Z2];
    __shared__ Material<T> s_mat[MAX_MATERIALS]; // the group's scene's materials
    __shared__ T s_st[GS::NS]; // staged state of the thread's current and next particle
    __shared__ uint32_t s_pid[GS::NP];
    __shared__ int s_g, s_last, s_nbr[8], s_scene, s_org[3];
    __shared__ uint16_t s_map[TN]; // tile node -> (neighbour block 0-7) << 8 | element in that block
    static_assert(sizeof(tv) + sizeof(te) + sizeof(s_mat) + sizeof(s_st) + sizeof(s_pid) + sizeof(s_map) + 512 <= 48 * 1024,
        "static shared memory of a kernel (512 B: the words above and the arrays' alignment)");
    if (aborted_cta(a.st)) return;
    if (BULK && threadIdx.x == 0) {
        mbar_init(&s_hbar, 1);
        mbar_init_fence();
    }
    for (int node = threadIdx.x; node < TN; node += NT) {
        const int tx = node / (TY * TZ), ty = (node / TZ) % TY, tz = node % TZ;
        const int ax = tx >= L::sx, ay = ty >= L::sy, az = tz >= L::sz;
        s_map[node] = (uint16_t)(((ax * 4 + ay * 2 + az) << 8) | L::element(tx - ax * L::sx, ty - ay * L::sy, tz - az * L::sz));
    }
    const uint32_t G = a.st->n_items;
    const KeyLayout kl = a.kl;
    for (bool first = true;; first = false) {
        int g = blockIdx.x; // the first item is the CTA's own number (claims count from the grid's size)
        if (!first) {
            if (threadIdx.x == 0) s_g = (int)(gridDim.x + atomicAdd(&a.st->work_g2p, 1u));
            __syncthreads();
            g = s_g;
        }
        if (g >= (int)G) break;
        const uint4 it = a.item[g];
        const uint32_t start = it.x, end = it.y;
        if (threadIdx.x < 8) {
            s_nbr[threadIdx.x] = a.i_slot[(size_t)g * 8 + threadIdx.x];
            if (threadIdx.x == 0) {
                uint64_t key0 = a.kl.at(a.keys_sorted, start);
                uint32_t bi, bj, bk;
                L::block_of_page(kl.page(key0), bi, bj, bk);
                s_scene = (int)kl.scene(key0);
                s_org[0] = (int)(bi * L::sx);
                s_org[1] = (int)(bj * L::sy);
                s_org[2] = (int)(bk * L::sz);
            }
        }
        __syncthreads();
        const SceneParams<T>& sp = a.scenes[s_scene];
        const bool damage = DRIVE != DRIVE_NONE && sp.damage != 0;
        const Pool<T>& P = a.pin;
        const Pool<T>& Q = a.pout;
        const uint32_t i0 = start + threadIdx.x;
        uint32_t j_cur = i0 < end ? a.vals_sorted[i0] : 0u; // storage slot of the thread's current particle
        // asynchronous copy of one particle's state into buffer bf of the thread's slots
        auto stage = [&](int bf, uint32_t j) {
            T* d = s_st + bf * G2P_SF * NT + threadIdx.x;
            const T* src = P.f + j;
            const int64_t ps = P.stride;
#pragma unroll
            for (int c = 0; c < 3; c++) cp_async<sizeof(T)>(d + (GS_X + c) * NT, src + (P_X + c) * ps);
#pragma unroll
            for (int c = 0; c < 9; c++) cp_async<sizeof(T)>(d + (GS_F + c) * NT, src + (P_F + c) * ps);
            cp_async<sizeof(T)>(d + GS_M * NT, src + P_M * ps);
            cp_async<sizeof(T)>(d + GS_V0 * NT, src + P_V0 * ps);
            if (damage) {
                cp_async<sizeof(T)>(d + GS_D * NT, src + P_D * ps);
                cp_async<sizeof(T)>(d + GS_SC * NT, src + P_SC * ps);
            }
            cp_async<4>(s_pid + bf * NT + threadIdx.x, P.pid + j);
        };
        // stage the tile from the 8 neighbouring blocks (s_map was built before the first barrier)
        if constexpr (BULK) {
            if (threadIdx.x == 0) { // every thread is past the previous group's reads of s_halo (the barrier above)
                uint32_t nvalid = 0;
                for (int b = 0; b < 8; b++) nvalid += (s_nbr[b] >= 0 && (uint32_t)s_nbr[b] < a.b_cap) ? 1u : 0u;
                fence_async_smem();
                mbar_arrive_expect_tx(&s_hbar, nvalid * (uint32_t)(BLK * sizeof(T)));
                for (int b = 0; b < 8; b++) {
                    const int slot = s_nbr[b];
                    if (slot >= 0 && (uint32_t)slot < a.b_cap) bulk_load(s_halo + b * BLK, a.vel + (size_t)slot * BLK, (uint32_t)(BLK * sizeof(T)), &s_hbar);
                }
            }
            if (!mbar_wait(&s_hbar, hphase, WAIT_LIMIT_NS)) raise_flag(a.st, FLAG_TIMEOUT);
            hphase ^= 1u;
        }
        // a warp takes five z columns of six nodes; a node's upper neighbour is the next lane's
        for (int n0 = (threadIdx.x >> 5) * 30; n0 < TN; n0 += (NT / 32) * 30) {
            const int lane = threadIdx.x & 31, node = n0 + lane;
            const bool in = lane < 30 && node < TN;
            const int m = in ? s_map[node] : 0, slot = s_nbr[m >> 8];
            const bool ok = in && slot >= 0 && (uint32_t)slot < a.b_cap;
            const T* src = BULK ? s_halo + (m >> 8) * BLK + (m & 0xff) : a.vel + (size_t)(ok ? slot : 0) * NVEL * L::nodes + (m & 0xff);
            Quad<T> qv, ev;
            qv.x = ok ? src[0] : (T)0;
            qv.y = ok ? src[L::nodes] : (T)0;
            qv.z = ok ? src[2 * L::nodes] : (T)0;
            qv.w = ok ? src[3 * L::nodes] : (T)0;
            ev.x = __shfl_down_sync(0xffffffffu, qv.x, 1) - qv.x;
            ev.y = __shfl_down_sync(0xffffffffu, qv.y, 1) - qv.y;
            ev.z = __shfl_down_sync(0xffffffffu, qv.z, 1) - qv.z;
            ev.w = __shfl_down_sync(0xffffffffu, qv.w, 1) - qv.w;
            if (in) {
                const int col = node / TZ, z = node - col * TZ;
                if (z >= 1 && z <= Z1) tv[col * Z1 + z - 1] = qv;
                if (z < Z2) te[col * Z2 + z] = ev;
            }
        }
        {
            constexpr int MW = (int)(sizeof(Material<T>) / 4);
            const uint32_t* ms = reinterpret_cast<const uint32_t*>(sp.materials);
            uint32_t* md = reinterpret_cast<uint32_t*>(s_mat);
            for (int k = threadIdx.x; k < MAX_MATERIALS * MW; k += NT) md[k] = ms[k];
        }
        if (GS::ON && i0 < end) stage(0, j_cur);
        __syncthreads();
        const T dx = sp.dx, inv_dx = sp.inv_dx, dt = sp.dt;
        const T caD = sp.apic_a * dx * sp.D_inv, cbD = sp.apic_b * dx * sp.D_inv, gdt = dt * inv_dx;
        const T dx2 = dx * dx, half_cfl2 = dx2 * (T)0.25 * (sp.cfl * sp.cfl);
        // scene constants in registers: read through sp inside the loop they would be re-read after every store
        const int key_cells = sp.domain_cells - 3, n_mat = sp.n_materials;
        const bool implicit = DRIVE != DRIVE_NONE && sp.implicit != 0;
        uint32_t flags = 0;
        // storage slots run one particle ahead of the state: with staging the next particle's state is copied
        // while this one computes; without, its slot is known when its loads issue (one latency, not two)
        uint32_t j_nxt = i0 + (GS::ON ? NT : 0) < end ? a.vals_sorted[i0 + (GS::ON ? NT : 0)] : 0u;
        int bf = 0;
        for (uint32_t i = i0; i < end; i += NT, bf ^= 1) {
            T x[3], F[9], pm, pV0, dd = 0, sc = 0;
            uint32_t pid, j;
            // staged: x now, the rest of the state from shared memory where it is used (it stays valid for the
            // whole iteration), so it holds no registers through the gather
            const T* dsl = s_st + bf * G2P_SF * NT + threadIdx.x;
            if constexpr (GS::ON) {
                j = j_cur;
                cp_async_wait_all(); // this particle's state (the thread's own copies)
#pragma unroll
                for (int c = 0; c < 3; c++) x[c] = dsl[(GS_X + c) * NT];
                if (i + NT < end) stage(bf ^ 1, j_nxt); // the other buffer was read in the previous iteration
                j_cur = j_nxt;
                if (i + 2 * NT < end) j_nxt = a.vals_sorted[i + 2 * NT];
            }
            else {
                j = j_nxt;
                if (i + NT < end) j_nxt = a.vals_sorted[i + NT];
                // every particle load is issued here, so one memory latency covers them all
#pragma unroll
                for (int c = 0; c < 3; c++) x[c] = P.f[(P_X + c) * P.stride + j];
#pragma unroll
                for (int c = 0; c < 9; c++) F[c] = P.f[(P_F + c) * P.stride + j];
                pid = P.pid[j];
                pm = P.f[P_M * P.stride + j];
                pV0 = P.f[P_V0 * P.stride + j];
                if (damage) {
                    dd = P.f[P_D * P.stride + j];
                    sc = P.f[P_SC * P.stride + j];
                }
            }
            int b[3], l[3];
            T w[3][3], dw[3][3], fr[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                T xs = mul_rn(x[c], inv_dx);
                b[c] = int_floor(sub_rn(xs, (T)0.5));
                bspline_w(xs, b[c], w[c], dw[c]);
                fr[c] = xs - (T)b[c];
                l[c] = b[c] - s_org[c];
            }
            if (l[0] < 0 || l[0] >= L::sx || l[1] < 0 || l[1] >= L::sy || l[2] < 0 || l[2] >= L::sz) {
                flags |= FLAG_CAPACITY; // a particle outside its group's block: keys and positions disagree
                continue;
            }
            // the APIC moment sum w v (x_i - x_p)^T = dx (M - pv fr^T) because x_i - x_p = (delta - fr) dx
            Gathered<T> gt;
            {
                const int col = l[0] * TY + l[1];
                const Quad<T>*pv0 = tv + col * Z1 + l[2], *pe0 = te + col * Z2 + l[2];
                if ((sizeof(T) == 4 && DRIVE != DRIVE_NONE) || damage) // FP32 carries the phase field in the fourth lane anyway (zero without damage)
                    gather<T, L, true>(pv0, pe0, w, dw, fr[2], gt);
                else
                    gather<T, L, false>(pv0, pe0, w, dw, fr[2], gt);
            }
            T (&pv)[3] = gt.pv, (&M)[9] = gt.M, (&Gv)[9] = gt.Gv, &lap = gt.lap, &pw = gt.pw;
            lap *= inv_dx * inv_dx;
            T Bm[9]; // the moment over dx; the factors dx and 4 / dx^2 are in caD and cbD, dt / dx in gdt
#pragma unroll
            for (int r = 0; r < 3; r++)
#pragma unroll
                for (int c = 0; c < 3; c++) Bm[3 * r + c] = M[3 * r + c] - fr[c] * pv[r];
            // finish the transfer first so the gather accumulators die before the damage update
            {
                T Fn[9], A[9];
                bool bad = false;
#pragma unroll
                for (int r = 0; r < 3; r++)
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        const T cn = caD * Bm[3 * r + c] + cbD * Bm[3 * c + r];
                        Q.f[(P_C + 3 * r + c) * Q.stride + i] = cn;
                        bad = bad || nonfinite(cn);
                        A[3 * r + c] = (r == c ? (T)1 : (T)0) + gdt * Gv[3 * r + c];
                    }
                if constexpr (GS::ON) {
#pragma unroll
                    for (int c = 0; c < 9; c++) F[c] = dsl[(GS_F + c) * NT];
                }
                mul3(A, F, Fn);
#pragma unroll
                for (int c = 0; c < 9; c++) {
                    bad = bad || nonfinite(Fn[c]);
                    Q.f[(P_F + c) * Q.stride + i] = Fn[c];
                }
                T xn[3], inc2 = 0;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    T inc = dt * pv[c];
                    inc2 += inc * inc;
                    xn[c] = x[c] + inc;
                    Q.f[(P_X + c) * Q.stride + i] = xn[c];
                    Q.f[(P_V + c) * Q.stride + i] = pv[c];
                }
                if (inc2 > dx2) flags |= FLAG_CFL;
                if (inc2 > half_cfl2) flags |= FLAG_CFL_HALF;
                if (bad || nonfinite(inc2)) flags |= FLAG_NONFINITE;
                // key of the next substep
                int nb[3];
                bool in_dom = true;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    nb[c] = base_node(xn[c], inv_dx);
                    in_dom = in_dom && nb[c] >= 0 && nb[c] < key_cells;
                }
                if (!in_dom) {
                    flags |= FLAG_OUT_OF_DOMAIN;
                    nb[0] = nb[1] = nb[2] = 0;
                }
                // the engine's keys carry no particle index (ib = 0), so a particle that stays in its cell gets
                // exactly the key it was sorted by (k_keys and this kernel share base_node): the incremental
                // sort's stayer test compares the two
                kl.put(a.keys_next, i, ((uint64_t)s_scene << (kl.cp + kl.ib)) | ((L::offset(nb[0], nb[1], nb[2]) >> L::data_bits) << kl.ib));
            }
            if constexpr (GS::ON) {
                pm = dsl[GS_M * NT];
                pV0 = dsl[GS_V0 * NT];
                pid = s_pid[bf * NT + threadIdx.x];
                if (damage) {
                    dd = dsl[GS_D * NT];
                    sc = dsl[GS_SC * NT];
                }
            }
            Q.f[P_M * Q.stride + i] = pm;
            Q.f[P_V0 * Q.stride + i] = pV0;
            Q.pid[i] = pid;
            if (implicit) Q.f[P_MDT * Q.stride + i] = P.f[P_MDT * P.stride + j]; // the implicit damage solve's history travels with the particle
            if (damage) {
                // AnisoMPM damage with the F of the start of the substep (AnisoFractureSimulation.h:210-283)
                const uint32_t mat = pid >> L::index_bits;
                const Material<T>& mt = s_mat[mat < (uint32_t)n_mat ? mat : 0];
                if (mt.damage && (mt.model == MODEL_NEOHOOKEAN_BORDEN || mt.model == MODEL_QR_STABLE_NEOHOOKEAN)) {
                    if (implicit) {
                        // damageG2P (AnisoFractureSimulation.h:578-610): the grid holds the solve's change of the
                        // nodal phase field; damage never decreases and stays <= 1
                        const T nd = dd + pw;
                        dd = nd > dd ? nd : dd;
                        dd = dd < (T)1 ? dd : (T)1;
                        // the next substep's solve folds the drive of the new F into the history: computed here,
                        // where the explicit update would evaluate the drive of the old F
                        T Fn[9];
#pragma unroll
                        for (int c = 0; c < 9; c++) Fn[c] = Q.f[(P_F + c) * Q.stride + i];
                        bool fb = false;
                        Q.f[P_DRV * Q.stride + i] = damage_drive<T, QR>(mt, Fn, sc, fb);
                        if (fb) atomicAdd(&a.st->fallback, 1u);
                    }
                    else {
                        bool fb = false;
                        dd = damage_update<T, QR>(mt, F, dd, lap, sc, dt, fb);
                        if (fb) atomicAdd(&a.st->fallback, 1u);
                    }
                    if (nonfinite(dd)) flags |= FLAG_NONFINITE;
                }
                Q.f[P_D * Q.stride + i] = dd;
                Q.f[P_SC * Q.stride + i] = sc;
            }
        }
        if (flags) raise_flag(a.st, flags);
        __syncthreads();
    }
    // The last CTA to finish ends the substep: the scenes' clocks, the substep count and the work counters, unless a
    // particle raised an aborting flag (every CTA's flags precede its arrival). As a kernel of its own this was a
    // launch for a few words (3.5 us).
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(&a.st->g2p_done, 1u) + 1 == gridDim.x;
        __threadfence();
    }
    __syncthreads();
    if (!s_last) return;
    const bool ab = aborted(a.st);
    if (!ab)
        for (int s = threadIdx.x; s < a.n_scenes; s += NT) a.scenes[s].time += (double)a.scenes[s].dt;
    if (threadIdx.x == 0 && !ab) {
        DevStatus* st = a.st;
        st->step += 1;
        st->n_groups = 0;
        st->n_items = 0;
        st->n_blocks = 0;
        st->work_p2g = 0;
        st->work_g2p = 0;
        st->g2p_done = 0;
    }
}

// ---------------------------------------------------------------------------------------------------
// Implicit damage solve (AnisoFractureSimulation::solveDamageSystem, AnisoFractureSimulation.h:437-626), run
// between the grid update and G2P for scenes that ask for it. Unknowns: the nodal phase field x on the nodes
// that damageable particles reach. With per-particle vol = V0 det F, the damage drive history
// D~ = max(D~, zeta <phi - 1>) (updateDTilde, :285-340), c_p = vol (1 + dt/eta (D~ + 1)) and
// e_p = vol dt/eta l0^2:
//   rhs_i = sum_p (dt D~/eta + pf_i) vol w_ip          (pf: the normalised nodal damage of this substep)
//   (A x)_i = diag_i x_i + sum_p (e_p sum_j x_j grad w_jp) . grad w_ip,   diag_i = sum_p c_p w_ip
// solved by Jacobi-preconditioned conjugate gradients from x = 0 as ConjugateGradient::solve does (stop when
// sqrt(r.z) <= min(sqrt(r0.z0), 1e-6), at most 100 iterations). Dot products are per scene, so every scene of a
// batch runs the iterations it would run alone. G2P then adds sum_i w_ip (x_i - pf_i) to the damage.
// ---------------------------------------------------------------------------------------------------
enum { CG_SA = 0, CG_SV, CG_DIAG, CG_X, CG_R, CG_Z, CG_P, CG_AP, CG_NF }; // node vectors
enum { DS_F = 0, DS_E = 3, DS_NF = 4 }; // particle scratch fields in the payload buffer: fractional position, e_p
constexpr int CG_MAX_ITERATIONS = 100;

template <class T>
__device__ __forceinline__ T* cgv(const StepArgs<T>& a, int f, uint32_t slot) { return a.cg + ((size_t)f * a.b_cap + slot) * LayoutOf<T>::type::nodes; }

// The damage drive of every particle of the implicit scenes from its current F, in storage order (the scene from
// the particle's current key): fills the cache P_DRV after a state write made it stale; G2P keeps it afterwards.
template <class T>
__global__ void k_dmg_drive(StepArgs<T> a, const uint64_t* keys)
{
    using L = typename LayoutOf<T>::type;
    const Pool<T>& P = a.pin;
    uint32_t fallbacks = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n_total; i += gridDim.x * blockDim.x) {
        const SceneParams<T>& sp = a.scenes[a.kl.scene(a.kl.at(keys, i))];
        if (!sp.implicit) continue;
        const uint32_t mat = P.pid[i] >> L::index_bits;
        const Material<T>& mt = sp.materials[mat < (uint32_t)sp.n_materials ? mat : 0];
        T drive = 0;
        if (mt.damage && (mt.model == MODEL_NEOHOOKEAN_BORDEN || mt.model == MODEL_QR_STABLE_NEOHOOKEAN)) {
            T F[9];
#pragma unroll
            for (int e = 0; e < 9; e++) F[e] = P.f[(P_F + e) * P.stride + i];
            bool fb = false;
            drive = damage_drive(mt, F, P.f[P_SC * P.stride + i], fb);
            if (fb) fallbacks++;
        }
        P.f[P_DRV * P.stride + i] = drive;
    }
    if (fallbacks) atomicAdd(&a.st->fallback, fallbacks);
}

// node tile of a group (its block plus 2 nodes on the + side): index of node (lx, ly, lz)
template <class L>
__device__ __forceinline__ int tile_index(int lx, int ly, int lz) { return (lx * (L::sy + 2) + ly) * (L::sz + 2) + lz; }

// The per-offset tiles of the fused P2G (OffsetTiles) for NF node vectors of the implicit solve: get(n, f) is
// field f of the thread's node n = 3 jj + kk. Every lane of the warp must call it.
template <class L, int NF, class T, class Get>
__device__ __forceinline__ void add_to_offset_tile_cg(T* tiles, int cx, int cy, int cz, int ii, Get get)
{
    using OT = OffsetTiles<L>;
    T* base = tiles + ii * NF * OT::TS + (cx * OT::TY + cy) * OT::TZ + cz;
#pragma unroll
    for (int jj = 0; jj < 3; jj++)
#pragma unroll
        for (int kk = 0; kk < 3; kk++) {
            T* t = base + jj * OT::TZ + kk;
#pragma unroll
            for (int f = 0; f < NF; f++) t[f * OT::TS] += get(jj * 3 + kk, f);
            __syncwarp();
        }
}

// sum the offsets' tiles per node of the block + halo into node vectors f_of[f] of the 8 neighbouring blocks
// (scalar atomics, zeros skipped), clearing the tiles
template <class T, class L, int NF>
__device__ void flush_offset_tiles_cg(const StepArgs<T>& a, T* tiles, const int32_t* nbr, const int* f_of, int tid, int nthreads)
{
    using OT = OffsetTiles<L>;
    constexpr int TX = L::sx + 2, TY = OT::TY, TZ = OT::TZ, TN = TX * TY * TZ;
    for (int q = tid; q < NF * TN; q += nthreads) {
        const int f = q / TN, node = q % TN;
        const int tx = node / (TY * TZ), ty = (node / TZ) % TY, tz = node % TZ;
        T v = (T)0;
#pragma unroll
        for (int ii = 0; ii < 3; ii++) {
            const int xl = tx - ii;
            if (xl < 0 || xl >= L::sx) continue;
            T* src = tiles + (ii * NF + f) * OT::TS + (xl * TY + ty) * TZ + tz;
            v += *src;
            *src = (T)0;
        }
        if (v == (T)0) continue;
        const int ax = tx >= L::sx, ay = ty >= L::sy, az = tz >= L::sz;
        const int slot = nbr[ax * 4 + ay * 2 + az];
        if (slot < 0 || (uint32_t)slot >= a.b_cap) {
            check_failed(a.st, 7);
            continue;
        }
        atomicAdd(cgv(a, f_of[f], slot) + L::element(tx - ax * L::sx, ty - ay * L::sy, tz - az * L::sz), v);
    }
}

// The items of a damage-solve kernel, dealt to the CTAs in rounds (they are of about equal size). The set-up of the next item
// (its range, the grid slots of its blocks, its scene and whether the kernel has work there) is a chain of four dependent
// reads: threads 0-7 advance it by one link at each next_* call while the CTA works on the current item.
struct DmgItem {
    uint32_t start, end;
    int32_t nbr[8];
    int scene; // -1: nothing to do (a scene without the solve, or finished); -2: no further items
};
template <class T>
struct DmgNext {
    uint4 it;
    int32_t slot;
    int scene;
    uint32_t g;
    __device__ __forceinline__ void range(const StepArgs<T>& a, uint32_t gg, uint32_t G) // threads 0-7
    {
        g = gg;
        it = g < G ? a.item[g] : make_uint4(0, 0, 0, 0);
        slot = g < G ? a.i_slot[(size_t)g * 8 + threadIdx.x] : -1;
    }
    __device__ __forceinline__ void key(const StepArgs<T>& a, uint32_t G) { scene = g < G ? (int)a.kl.scene(a.kl.at(a.keys_sorted, it.x)) : -2; }
    __device__ __forceinline__ void store(const StepArgs<T>& a, DmgItem& d, bool need_unfinished) const
    {
        d.nbr[threadIdx.x] = slot;
        if (threadIdx.x) return;
        d.start = it.x;
        d.end = it.y;
        d.scene = scene < 0 ? scene : ((!a.scenes[scene].implicit || (need_unfinished && a.cgs[scene].done)) ? -1 : scene);
    }
};

// threads and particle chunk of the damage solve's group kernels: one thread per (in-block cell, stencil x-offset);
// a chunk's per-particle values are staged in shared memory for the per-cell sums
template <class T>
struct DmgShape {
    using L = typename LayoutOf<T>::type;
    static constexpr int NT = 3 * L::nodes;
    static constexpr int CHUNK = 512;
    static constexpr int NS = 6; // staged values per particle
    // CTAs per SM the registers are cut for. These kernels wait on memory (loads 5.5 of 13 cycles per issued instruction in
    // k_dmg_rhs), and in FP32 4 / 5 / 6 CTAs cost 79 / 64 / 56 registers with 0 / 8 / 12 bytes of spill (7: 184): per substep
    // 3,407,872 particles 1057 / 1013 / 995 us, 425,984 215.8 / 208.5 / 209.7. FP64 waits on its pipe: 956 / - / 955.
    static constexpr int MINB = sizeof(T) == 4 ? 6 : 4;
};

// v[i] by selects (an index that varies at run time puts the array into local memory)
template <class T>
__device__ __forceinline__ T pick3(const T (&v)[3], int i)
{
    return i == 0 ? v[0] : (i == 1 ? v[1] : v[2]);
}

// cell ranges of a staged chunk: particles of one cell are contiguous (sorted by cell inside the block)
template <int NC>
__device__ __forceinline__ void chunk_cells(const uint8_t* cellof, int cnt, int16_t* cfirst, int16_t* clast, int tid, int nt)
{
    for (int q = tid; q < cnt; q += nt) {
        const int e = cellof[q];
        if (q == 0 || cellof[q - 1] != e) cfirst[e] = (int16_t)q;
        if (q == cnt - 1 || cellof[q + 1] != e) clast[e] = (int16_t)(q + 1);
    }
}

// Per particle of an implicit scene the D~ history folded with the drive of its F (cached in P_DRV) and its coefficients,
// then the right-hand side parts and the preconditioner's diagonal. Per chunk: the particles' values staged in shared memory
// (phase 1, which also leaves the fractional position and e_p for the operator), then one thread per (in-block cell, x-offset) sums the 9 (y, z) nodes over its cell's
// particles in registers (phase 2) and adds them to the group's shared node tile; the tile goes to the node
// vectors CG_SA, CG_SV, CG_DIAG.
template <class T>
__global__ void __launch_bounds__(DmgShape<T>::NT, DmgShape<T>::MINB) k_dmg_rhs(StepArgs<T> a)
{
    using L = typename LayoutOf<T>::type;
    using D = DmgShape<T>;
    constexpr int NC = L::nodes, NT = D::NT, CHUNK = D::CHUNK;
    constexpr int TE = 3 * 3 * OffsetTiles<L>::TS; // per-offset tiles of the 3 node vectors
    __shared__ T tile[TE];
    __shared__ T st[D::NS][CHUNK]; // fr x3, vol D~ dt/eta, vol, c
    __shared__ uint8_t cellof[CHUNK];
    __shared__ int16_t cfirst[NC], clast[NC];
    __shared__ DmgItem s_item[2];
    if (aborted_cta(a.st)) return;
    const uint32_t G = a.st->n_items;
    const KeyLayout kl = a.kl;
    const Pool<T>& P = a.pin;
    const int64_t S = a.pstride;
    const int tid = threadIdx.x, ii = tid / NC, c = tid % NC;
    const int cx = c >> (L::zbits + L::ybits), cy = (c >> L::zbits) & (L::sy - 1), cz = c & (L::sz - 1);
    if (blockIdx.x == 0) // the sums the node passes accumulate
        for (int s = tid; s < a.n_scenes; s += NT) a.cgs[s].zr = a.cgs[s].zr_new = a.cgs[s].pAp = 0;
    for (int q = tid; q < TE; q += NT) tile[q] = (T)0;
    const int f_of[3] = { CG_SA, CG_SV, CG_DIAG };
    DmgNext<T> nx;
    if (tid < 8) {
        nx.range(a, blockIdx.x, G);
        nx.key(a, G);
        nx.store(a, s_item[0], false);
    }
    __syncthreads();
    for (uint32_t g = blockIdx.x, cur = 0; g < G; g += gridDim.x, cur ^= 1) {
        const DmgItem& item = s_item[cur];
        const int sc = item.scene;
        const uint32_t start = item.start, end = sc >= 0 ? item.end : item.start;
        if (tid < 8) nx.range(a, g + gridDim.x, G);
        const SceneParams<T>& sp = a.scenes[sc >= 0 ? sc : 0];
        bool any = false;
        for (uint32_t c0 = start; c0 < end; c0 += CHUNK) {
            const int cnt = (int)min((uint32_t)CHUNK, end - c0);
            if (tid < NC) {
                cfirst[tid] = 0;
                clast[tid] = 0;
            }
            for (int q = tid; q < cnt; q += NT) {
                const uint32_t j = a.vals_sorted[c0 + q];
                // every state load of the particle at once (one latency), ahead of the material test
                T x[3], F[9];
#pragma unroll
                for (int e = 0; e < 3; e++) x[e] = P.f[(P_X + e) * P.stride + j];
#pragma unroll
                for (int e = 0; e < 9; e++) F[e] = P.f[(P_F + e) * P.stride + j];
                const T V0 = P.f[P_V0 * P.stride + j], drive = P.f[P_DRV * P.stride + j];
                T hist = P.f[P_MDT * P.stride + j];
                const uint32_t mat = P.pid[j] >> L::index_bits;
                const Material<T>& mt = sp.materials[mat < (uint32_t)sp.n_materials ? mat : 0];
                T* y = a.pay + pay_pos(c0 + q);
#pragma unroll
                for (int e = 0; e < 3; e++) {
                    const T xs = mul_rn(x[e], sp.inv_dx), fr = xs - (T)int_floor(sub_rn(xs, (T)0.5));
                    st[e][q] = fr;
                    y[(DS_F + e) * S] = fr;
                }
                T av = 0, vol = 0, cc = 0, ev = 0;
                if (mt.damage && (mt.model == MODEL_NEOHOOKEAN_BORDEN || mt.model == MODEL_QR_STABLE_NEOHOOKEAN)) {
                    vol = V0 * det3(F);
                    hist = drive > hist ? drive : hist;
                    P.f[P_MDT * P.stride + j] = hist;
                    const T dt = sp.dt;
                    av = ((dt * hist) / mt.eta) * vol;
                    cc = vol * ((T)1 + ((dt / mt.eta) * (hist + (T)1)));
                    ev = vol * (dt / mt.eta) * mt.l0 * mt.l0;
                }
                st[3][q] = av;
                st[4][q] = vol;
                st[5][q] = cc;
                y[DS_E * S] = ev;
                cellof[q] = (uint8_t)((kl.at(a.keys_sorted, c0 + q) >> kl.ib) & (NC - 1));
            }
            __syncthreads();
            chunk_cells<NC>(cellof, cnt, cfirst, clast, tid, NT);
            __syncthreads();
            T acc[9][3];
#pragma unroll
            for (int n = 0; n < 9; n++) acc[n][0] = acc[n][1] = acc[n][2] = (T)0;
            const int qa = cfirst[c], qb = clast[c];
            for (int q = qa; q < qb; q++) {
                const T cc = st[5][q];
                if (cc == (T)0) continue; // not damageable
                const T av = st[3][q], vol = st[4][q];
                T w[3][3], dw[3][3];
#pragma unroll
                for (int e = 0; e < 3; e++) bspline_w(st[e][q], 0, w[e], dw[e]);
                const T wx = pick3(w[0], ii);
#pragma unroll
                for (int j = 0; j < 3; j++)
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        const T wijk = wx * w[1][j] * w[2][k];
                        acc[j * 3 + k][0] += wijk * av;
                        acc[j * 3 + k][1] += wijk * vol;
                        acc[j * 3 + k][2] += wijk * cc;
                    }
            }
            add_to_offset_tile_cg<L, 3>(tile, cx, cy, cz, ii, [&](int n, int f) { return acc[n][f]; }); // all lanes
            any = true;
            __syncthreads();
        }
        if (tid < 8) nx.key(a, G);
        if (any) flush_offset_tiles_cg<T, L, 3>(a, tile, item.nbr, f_of, tid, NT);
        if (tid < 8) nx.store(a, s_item[cur ^ 1], false);
        __syncthreads();
    }
}

// The operator's particle part for the search direction p. Per chunk: per particle gc = e_p / dx^2 sum_j p_j
// grad w_jp (gradients per unit cell; phase 1, from p staged on the group's tile), staged with the fractional
// position; then per (cell, x-offset) thread the sums gc . grad w over its cell's particles for its 9 nodes
// (phase 2) into the tile, which goes to A p (CG_AP). The particles' share of p . A p is sum gc . (sum_j p_j grad w_jp): it is
// summed here, so no pass over the nodes stands between the operator and the step length.
template <class T>
__global__ void __launch_bounds__(DmgShape<T>::NT, DmgShape<T>::MINB) k_dmg_apply(StepArgs<T> a)
{
    using L = typename LayoutOf<T>::type;
    using D = DmgShape<T>;
    constexpr int NC = L::nodes, NT = D::NT, CHUNK = D::CHUNK, TY = L::sy + 2, TZ = L::sz + 2, TN = (L::sx + 2) * TY * TZ;
    constexpr int TE = 3 * OffsetTiles<L>::TS; // per-offset tiles of A p
    __shared__ T tile[TE];
    __shared__ T ptile[TN];
    __shared__ T st[D::NS][CHUNK]; // fr x3, gc x3
    __shared__ uint8_t cellof[CHUNK];
    __shared__ int16_t cfirst[NC], clast[NC];
    __shared__ DmgItem s_item[2];
    __shared__ int s_last;
    __shared__ uint16_t s_map[TN]; // tile node -> (neighbour block 0-7) << 8 | element in that block
    if (aborted_cta(a.st)) return;
    const uint32_t G = a.st->n_items;
    const KeyLayout kl = a.kl;
    const int64_t S = a.pstride;
    const int tid = threadIdx.x, ii = tid / NC, c = tid % NC;
    const int cx = c >> (L::zbits + L::ybits), cy = (c >> L::zbits) & (L::sy - 1), cz = c & (L::sz - 1);
    for (int q = tid; q < TE; q += NT) tile[q] = (T)0;
    for (int q = tid; q < TN; q += NT) {
        const int tx = q / (TY * TZ), ty = (q / TZ) % TY, tz = q % TZ;
        const int ax = tx >= L::sx, ay = ty >= L::sy, az = tz >= L::sz;
        s_map[q] = (uint16_t)(((ax * 4 + ay * 2 + az) << 8) | L::element(tx - ax * L::sx, ty - ay * L::sy, tz - az * L::sz));
    }
    const int f_of[1] = { CG_AP };
    __shared__ double s_en[NT / 32];
    double energy = 0; // of the items of scene esc
    int esc = -1;
    auto add_energy = [&]() { // every thread of the CTA
        double v = energy;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        __syncthreads();
        if ((tid & 31) == 0) s_en[tid >> 5] = v;
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < NT / 32; w++) v += s_en[w];
            if (esc >= 0 && v != 0.0) atomicAdd(&a.cgs[esc].pAp, v);
        }
        energy = 0;
    };
    DmgNext<T> nx;
    if (tid < 8) {
        nx.range(a, blockIdx.x, G);
        nx.key(a, G);
        nx.store(a, s_item[0], true);
    }
    __syncthreads();
    for (uint32_t g = blockIdx.x, cur = 0; g < G; g += gridDim.x, cur ^= 1) {
        const DmgItem& item = s_item[cur];
        const int sc = item.scene;
        if (tid < 8) nx.range(a, g + gridDim.x, G);
        if (sc < 0) { // the whole CTA
            if (tid < 8) {
                nx.key(a, G);
                nx.store(a, s_item[cur ^ 1], true);
            }
            __syncthreads();
            continue;
        }
        const uint32_t start = item.start, end = item.end;
        if (sc != esc) {
            if (esc >= 0) add_energy();
            esc = sc;
        }
        for (int q = tid; q < TN; q += NT) {
            const int m = s_map[q], slot = item.nbr[m >> 8];
            ptile[q] = (slot >= 0 && (uint32_t)slot < a.b_cap) ? cgv(a, CG_P, slot)[m & 0xff] : (T)0;
        }
        __syncthreads();
        const T inv_dx = a.scenes[sc].inv_dx;
        for (uint32_t c0 = start; c0 < end; c0 += CHUNK) {
            const int cnt = (int)min((uint32_t)CHUNK, end - c0);
            if (tid < NC) {
                cfirst[tid] = 0;
                clast[tid] = 0;
            }
            for (int q = tid; q < cnt; q += NT) {
                const T* y = a.pay + pay_pos(c0 + q);
                const T ev = y[DS_E * S];
                const int e = (int)((kl.at(a.keys_sorted, c0 + q) >> kl.ib) & (NC - 1));
                cellof[q] = (uint8_t)e;
                T fr[3], w[3][3], dw[3][3];
#pragma unroll
                for (int f = 0; f < 3; f++) {
                    fr[f] = y[(DS_F + f) * S];
                    st[f][q] = fr[f];
                    bspline_w(fr[f], 0, w[f], dw[f]);
                }
                T g0 = 0, g1 = 0, g2 = 0;
                if (ev != (T)0) {
                    const int lx = e >> (L::zbits + L::ybits), ly = (e >> L::zbits) & (L::sy - 1), lz = e & (L::sz - 1);
                    const T* pt = ptile + tile_index<L>(lx, ly, lz);
                    // separable sums of p against the gradient weights: over z, then y, then x
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        T sA = 0, sB = 0, sC = 0;
#pragma unroll
                        for (int j = 0; j < 3; j++) {
                            T zA = 0, zD = 0;
#pragma unroll
                            for (int k = 0; k < 3; k++) {
                                const T pj = pt[(i * TY + j) * TZ + k];
                                zA += w[2][k] * pj;
                                zD += dw[2][k] * pj;
                            }
                            sA += w[1][j] * zA;
                            sB += dw[1][j] * zA;
                            sC += w[1][j] * zD;
                        }
                        g0 += dw[0][i] * sA;
                        g1 += w[0][i] * sB;
                        g2 += w[0][i] * sC;
                    }
                    const T sgc = ev * inv_dx * inv_dx; // both gradients carry 1/dx
                    energy += gradient_share(sgc, g0, g1, g2);
                    g0 *= sgc;
                    g1 *= sgc;
                    g2 *= sgc;
                }
                st[3][q] = g0;
                st[4][q] = g1;
                st[5][q] = g2;
            }
            __syncthreads();
            chunk_cells<NC>(cellof, cnt, cfirst, clast, tid, NT);
            __syncthreads();
            T acc[9];
#pragma unroll
            for (int n = 0; n < 9; n++) acc[n] = (T)0;
            const int qa = cfirst[c], qb = clast[c];
            for (int q = qa; q < qb; q++) {
                const T g0 = st[3][q], g1 = st[4][q], g2 = st[5][q];
                if (g0 == (T)0 && g1 == (T)0 && g2 == (T)0) continue;
                T w[3][3], dw[3][3];
#pragma unroll
                for (int e = 0; e < 3; e++) bspline_w(st[e][q], 0, w[e], dw[e]);
                const T wx = pick3(w[0], ii), a0 = g0 * pick3(dw[0], ii), a1 = g1 * wx, a2 = g2 * wx;
#pragma unroll
                for (int j = 0; j < 3; j++)
#pragma unroll
                    for (int k = 0; k < 3; k++) acc[j * 3 + k] += (a0 * w[1][j] + a1 * dw[1][j]) * w[2][k] + a2 * (w[1][j] * dw[2][k]);
            }
            add_to_offset_tile_cg<L, 1>(tile, cx, cy, cz, ii, [&](int n, int) { return acc[n]; }); // all lanes
            __syncthreads();
        }
        if (tid < 8) nx.key(a, G);
        flush_offset_tiles_cg<T, L, 1>(a, tile, item.nbr, f_of, tid, NT);
        if (tid < 8) nx.store(a, s_item[cur ^ 1], true);
        __syncthreads();
    }
    add_energy();
    // the step lengths, once per scene, by the CTA that finishes last (its counter wraps to zero): a division in every thread
    // of the node pass would be an FP64 division
    if (tid == 0) {
        __threadfence();
        s_last = atomicInc(&a.st->cg_done, gridDim.x - 1) == gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (s_last)
        for (int s = tid; s < a.n_scenes; s += NT)
            if (a.scenes[s].implicit && !a.cgs[s].done) a.cgs[s].alpha = a.cgs[s].zr / __ldcg(&a.cgs[s].pAp);
}

// Per-scene sums of a node pass: a warp's nodes are of one block (and so of one scene). A warp keeps its sum while the scene
// stays; the CTA adds its warps' sums with one atomic per run of warps of one scene (an atomic per warp to the one address
// of a scene took longer than the pass).
constexpr int CG_NT = 256;
struct SceneSum {
    double sum = 0;
    int scene = -1;
    __device__ __forceinline__ void add(double v, int sc, CgScalars* cgs, double CgScalars::* to) // whole warps
    {
        const int s0 = __shfl_sync(0xffffffffu, sc, 0);
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (s0 < 0) return;
        if (s0 != scene && scene >= 0) {
            if ((threadIdx.x & 31) == 0 && sum != 0.0) atomicAdd(&(cgs[scene].*to), sum);
            sum = 0;
        }
        scene = s0;
        sum += v; // (lane 0's is the warp's)
    }
    __device__ __forceinline__ void finish(CgScalars* cgs, double CgScalars::* to, double* s_v, int* s_s) // whole CTAs
    {
        if ((threadIdx.x & 31) == 0) {
            s_v[threadIdx.x >> 5] = sum;
            s_s[threadIdx.x >> 5] = scene;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double run = 0;
            int rsc = -1;
            for (int w = 0; w <= CG_NT / 32; w++) {
                const int sc = w < CG_NT / 32 ? s_s[w] : -1;
                if (sc != rsc) {
                    if (rsc >= 0 && run != 0.0) atomicAdd(&(cgs[rsc].*to), run);
                    rsc = sc;
                    run = 0;
                }
                if (w < CG_NT / 32) run += s_v[w];
            }
        }
        __syncthreads();
    }
};

// Node passes of the solve. CG_INIT: r = rhs, z = r / diag, p = z, with r.z and the diagonal's share of p.Ap. CG_STEP: the
// operator's diagonal added, x, r and z moved along p, r.z, A p cleared. CG_DIR: p = z + beta p and the diagonal's share of
// p.Ap. CG_END: the grid's phase field becomes x - pf, the vectors are cleared for the next solve. The last CTA of CG_INIT and
// CG_STEP does the scenes' bookkeeping (per scene: tolerance; iteration count, beta and whether it is done) and, after a step,
// sets the condition of the loop that runs the further iterations: some scene unfinished, and never more than
// CG_MAX_ITERATIONS + 1 passes (each scene stops itself at CG_MAX_ITERATIONS, so the loop always ends).
// An iteration is three kernels (direction, operator, step). With the operator's product, its dot product, the step, the
// direction and the bookkeeping in one kernel each it was five, and the first iteration a pass of the conditional loop.
enum { CG_INIT = 0, CG_STEP, CG_DIR, CG_END };
template <class T, int STAGE>
__global__ void __launch_bounds__(CG_NT) k_cg_nodes(StepArgs<T> a, cudaGraphConditionalHandle loop, int has_loop)
{
    using L = typename LayoutOf<T>::type;
    __shared__ double s_v[CG_NT / 32];
    __shared__ int s_s[CG_NT / 32], s_last;
    __shared__ uint32_t s_active;
    if (aborted_cta(a.st)) { // by an earlier kernel: every CTA leaves, and the loop ends
        if (STAGE == CG_STEP && has_loop && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(loop, 0u);
        return;
    }
    const uint32_t B = min(a.st->n_blocks, a.b_cap);
    const uint32_t total = B * L::nodes;
    SceneSum zr, pAp;
    for (uint32_t t = blockIdx.x * CG_NT + threadIdx.x; t < ((total + 31) & ~31u); t += gridDim.x * CG_NT) {
        double acc = 0, dsum = 0;
        int scene = -1;
        if (t < total) {
            const uint32_t b = t / L::nodes, e = t % L::nodes;
            T* dg = cgv(a, CG_DIAG, b) + e;
            T* x = cgv(a, CG_X, b) + e;
            T* r = cgv(a, CG_R, b) + e;
            T* z = cgv(a, CG_Z, b) + e;
            T* p = cgv(a, CG_P, b) + e;
            T* Ap = cgv(a, CG_AP, b) + e;
            T* sa = cgv(a, CG_SA, b) + e;
            T* sv = cgv(a, CG_SV, b) + e;
            T* pf = a.vel + (size_t)b * NVEL * L::nodes + 3 * L::nodes + e;
            // every load of the node at once, ahead of the scene's test
            T diag, xv = 0, rv = 0, zv = 0, pv = 0, apv = 0, sav = 0, svv = 0, pfv = 0;
            diag = *dg;
            if (STAGE == CG_INIT) sav = *sa, svv = *sv;
            if (STAGE == CG_INIT || STAGE == CG_END) pfv = *pf;
            if (STAGE == CG_STEP) rv = *r, apv = *Ap;
            if (STAGE == CG_STEP || STAGE == CG_END) xv = *x;
            if (STAGE == CG_STEP || STAGE == CG_DIR) pv = *p;
            if (STAGE == CG_DIR) zv = *z;
            const int sc = (int)(a.b_key[b] >> 40);
            const CgScalars& cs = a.cgs[sc];
            if (a.scenes[sc].implicit && (STAGE == CG_INIT || STAGE == CG_END || !cs.done)) {
                scene = sc;
                const bool on = diag > (T)0;
                if (STAGE == CG_INIT) {
                    const T rhs = on ? sav + pfv * svv : (T)0;
                    const T zz = on ? rhs / diag : (T)0;
                    *x = 0;
                    *r = rhs;
                    *z = zz;
                    *p = zz;
                    *Ap = 0;
                    acc = (double)rhs * (double)zz;
                    dsum = on ? diagonal_share(diag, zz) : 0.0;
                }
                else if (STAGE == CG_STEP) {
                    const T alpha = (T)cs.alpha;
                    const T ap = on ? apv + diag * pv : (T)0;
                    const T rn = rv - ap * alpha, zn = on ? rn / diag : (T)0;
                    *x = xv + pv * alpha;
                    *r = rn;
                    *z = zn;
                    *Ap = 0;
                    acc = (double)zn * (double)rn;
                }
                else if (STAGE == CG_DIR) {
                    const T pn = zv + (T)cs.beta * pv;
                    *p = pn;
                    dsum = on ? diagonal_share(diag, pn) : 0.0;
                }
                else {
                    *pf = on ? xv - pfv : (T)0;
                    // the solve's vectors start from zero next time
                    *sa = 0;
                    *sv = 0;
                    *dg = 0;
                    *Ap = 0;
                }
            }
        }
        if (STAGE == CG_INIT) zr.add(acc, scene, a.cgs, &CgScalars::zr);
        if (STAGE == CG_STEP) zr.add(acc, scene, a.cgs, &CgScalars::zr_new);
        if (STAGE == CG_INIT || STAGE == CG_DIR) pAp.add(dsum, scene, a.cgs, &CgScalars::pAp);
    }
    if (STAGE == CG_INIT) zr.finish(a.cgs, &CgScalars::zr, s_v, s_s);
    if (STAGE == CG_STEP) zr.finish(a.cgs, &CgScalars::zr_new, s_v, s_s);
    if (STAGE == CG_INIT || STAGE == CG_DIR) pAp.finish(a.cgs, &CgScalars::pAp, s_v, s_s);
    if (STAGE != CG_INIT && STAGE != CG_STEP) return;
    // the bookkeeping, by the CTA that finishes last (its counter wraps to zero)
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicInc(&a.st->cg_done, gridDim.x - 1) == gridDim.x - 1;
        s_active = 0;
        __threadfence();
    }
    __syncthreads();
    if (!s_last) return;
    for (int s = threadIdx.x; s < a.n_scenes; s += CG_NT) {
        CgScalars& cs = a.cgs[s];
        if (!a.scenes[s].implicit) {
            cs.done = 1;
            continue;
        }
        if (STAGE == CG_INIT) {
            const double res = sqrt(__ldcg(&cs.zr));
            cs.tol = res < 1e-6 ? res : 1e-6;
            cs.iter = 0;
            cs.done = res <= cs.tol;
        }
        else if (!cs.done) {
            const double zn = __ldcg(&cs.zr_new);
            cs.beta = zn / cs.zr;
            cs.zr = zn;
            cs.iter++;
            cs.done = sqrt(zn) <= cs.tol || cs.iter >= CG_MAX_ITERATIONS;
            cs.pAp = 0;
        }
        cs.zr_new = 0;
        if (!cs.done) atomicAdd(&s_active, 1u);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (STAGE == CG_INIT)
            a.st->cg_loops = 0;
        else {
            const uint32_t loops = ++a.st->cg_loops;
            if (has_loop) cudaGraphSetConditional(loop, (s_active > 0 && loops <= (uint32_t)CG_MAX_ITERATIONS) ? 1u : 0u);
        }
    }
}

// ---------------------------------------------------------------------------------------------------
// host <-> device field transfer (caller order <-> storage order via the original index)
// ---------------------------------------------------------------------------------------------------
// Storage slot of every particle of a scene in the caller's order (inv[orig] = slot), for the row transfers.
template <class T>
__global__ void k_inv(Pool<T> p, int64_t first, int64_t n, uint32_t* inv)
{
    using L = typename LayoutOf<T>::type;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t orig = p.pid[first + i] & ((1u << L::index_bits) - 1);
        if (orig < (uint64_t)n) inv[orig] = (uint32_t)(first + i);
    }
}

// Field groups of a row transfer: rows of W = sum nc values in the caller's order, fields f0[k] .. f0[k]+nc[k]-1.
struct RowFields {
    int f0[8], nc[8], count, W;
};
constexpr int IO_ROWS = 128; // rows per CTA (one per thread)

// Rows of a scene between the particle pool and row-major buffers (host memory mapped into the device, or a
// staging buffer). A CTA moves IO_ROWS consecutive rows: pool <-> shared memory per row (thread per row, slot from
// inv), shared memory <-> buffer as one contiguous run of IO_ROWS * W values (coalesced, whole lines over the
// host link). MODE: ROWS_IMPORT (in -> pool), ROWS_EXPORT (pool -> out), ROWS_EXCHANGE (pool -> out, then in ->
// pool, row by row: a CTA reads its rows out of the pool before it overwrites them, and CTAs own disjoint rows,
// so out receives the state from before the call; with many CTAs in flight both directions of the link are busy
// at once).
enum { ROWS_IMPORT = 0, ROWS_EXPORT = 1, ROWS_EXCHANGE = 2 };
template <class T, class O, int MODE>
__global__ void __launch_bounds__(IO_ROWS) k_rows(Pool<T> p, const uint32_t* inv, int64_t n, RowFields rf, const O* in, O* out)
{
    extern __shared__ __align__(16) unsigned char rows_dyn[];
    const int W = rf.W;
    O* sm_o = reinterpret_cast<O*>(rows_dyn); // rows leaving the pool
    O* sm_i = MODE == ROWS_EXCHANGE ? sm_o + IO_ROWS * W : sm_o; // rows entering it
    for (int64_t base = (int64_t)blockIdx.x * IO_ROWS; base < n; base += (int64_t)gridDim.x * IO_ROWS) {
        const int rows = (int)min((int64_t)IO_ROWS, n - base);
        const uint32_t slot = threadIdx.x < rows ? inv[base + threadIdx.x] : 0u;
        if (MODE != ROWS_IMPORT) {
            if (threadIdx.x < rows) {
                O* r = sm_o + threadIdx.x * W;
                int c0 = 0;
                for (int k = 0; k < rf.count; k++) {
                    for (int c = 0; c < rf.nc[k]; c++) r[c0 + c] = (O)p.f[(int64_t)(rf.f0[k] + c) * p.stride + slot];
                    c0 += rf.nc[k];
                }
            }
            __syncthreads();
        }
        {
            O* run_o = MODE != ROWS_IMPORT ? out + base * W : nullptr;
            const O* run_i = MODE != ROWS_EXPORT ? in + base * W : nullptr;
            for (int q = threadIdx.x; q < rows * W; q += IO_ROWS) {
                if (MODE != ROWS_IMPORT) run_o[q] = sm_o[q];
                if (MODE != ROWS_EXPORT) sm_i[q] = run_i[q];
            }
            __syncthreads();
        }
        if (MODE != ROWS_EXPORT) {
            if (threadIdx.x < rows) {
                const O* r = sm_i + threadIdx.x * W;
                int c0 = 0;
                for (int k = 0; k < rf.count; k++) {
                    for (int c = 0; c < rf.nc[k]; c++) p.f[(int64_t)(rf.f0[k] + c) * p.stride + slot] = (T)r[c0 + c];
                    c0 += rf.nc[k];
                }
            }
            __syncthreads();
        }
    }
}

// FP64-accumulated particle reductions of one scene: mass, momentum (3), kinetic energy, max speed
template <class T>
__global__ void k_reduce(Pool<T> p, int64_t first, int64_t n, double* out)
{
    double M = 0, px = 0, py = 0, pz = 0, ke = 0, vmax = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t s = first + i;
        double m = p.f[P_M * p.stride + s];
        double vx = p.f[(P_V + 0) * p.stride + s], vy = p.f[(P_V + 1) * p.stride + s], vz = p.f[(P_V + 2) * p.stride + s];
        M += m;
        px += m * vx;
        py += m * vy;
        pz += m * vz;
        double s2 = vx * vx + vy * vy + vz * vz;
        ke += 0.5 * m * s2;
        vmax = fmax(vmax, sqrt(s2));
    }
    for (int o = 16; o > 0; o >>= 1) {
        M += __shfl_down_sync(0xffffffffu, M, o);
        px += __shfl_down_sync(0xffffffffu, px, o);
        py += __shfl_down_sync(0xffffffffu, py, o);
        pz += __shfl_down_sync(0xffffffffu, pz, o);
        ke += __shfl_down_sync(0xffffffffu, ke, o);
        vmax = fmax(vmax, __shfl_down_sync(0xffffffffu, vmax, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(out + 0, M);
        atomicAdd(out + 1, px);
        atomicAdd(out + 2, py);
        atomicAdd(out + 3, pz);
        atomicAdd(out + 4, ke);
        // speeds are non-negative: their IEEE bit patterns order like unsigned integers
        atomicMax((unsigned long long*)(out + 5), (unsigned long long)__double_as_longlong(vmax));
    }
}

template <class T>
__global__ void k_iota_pid(uint32_t* pid, const uint8_t* mat, int64_t first, int64_t n)
{
    using L = typename LayoutOf<T>::type;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        pid[first + i] = (uint32_t)i | ((uint32_t)(mat ? mat[i] : 0) << L::index_bits);
}

template <class T>
__global__ void k_iota(uint32_t* v, uint32_t n)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) v[i] = i;
}

} // namespace zr
