// pool_tiled.cu -- the pool's tiled schedule: per-tile node gathers and per-(tile, node)
// force partials.
//
// In the other schedules every tet writes its four corner forces to node-major slots
// (64 B per tet) and the node pass reads them back (64 B per tet): half of a step's
// HBM traffic.  Here a block takes one element tile (up to 128 consecutive tets of one
// mesh) and:
//   1. gathers the displacements (and compensations) of the tile's distinct nodes once
//      into shared memory -- about 90 nodes for the 512 corners of a Kuhn box mesh;
//   2. evaluates each tet from its corners there, with the arithmetic of every other
//      schedule (tet_element_f32_eval), its corner forces into shared memory;
//   3. sums, for each distinct node, the corner forces of the tile's tets that name
//      it, in ascending tet order, and writes that one partial to the node's run of
//      the per-(tile, node) CSR;
// and the node pass sums a node's partials in ascending tile order (the other
// schedules' node kernel over this CSR).  Per tet, the slot traffic falls from 128 B to
// twice 16 B per (tile, node) pair -- about 22 B.
//
// A node's force is then (partial of its first tile) + (partial of the next) + ...,
// each partial summed in tet order: the same terms as the other schedules' single
// ascending run, associated per tile.  Tiles are aligned to their mesh's first tet, so
// the association, and with it every bit of a mesh's result, does not depend on where
// the mesh sits in the pool or what else is there; it differs from the other
// schedules' in rounding only.
//
// The tables are built on the device for each work list: per tile, its corners are
// sorted by (node, corner) in shared memory (a bitonic sort of 512 keys), which gives
// the distinct nodes in ascending order, each corner's place in that list and, per
// node, its corners in ascending order.
#include <algorithm>
#include <mutex>

#include <cub/block/block_scan.cuh>

#include "common.cuh"
#include "pool.hpp"
#include "tet_f32.cuh"

namespace fs {
namespace {

constexpr int kTiledTile = 128;              // tets per tile
constexpr int kTiledCorners = 4 * kTiledTile;  // 512

// The tile's corners, sorted: key = node << 9 | corner (corner = 4 x tet-in-tile + c);
// slots past the tile's corners hold ~0 and sort last.  All 128 threads call it.
__device__ __forceinline__ void sort_tile_corners(const PoolDevice& d, const PoolTile& tl,
                                                  unsigned long long* key) {
    const int corners = 4 * (int)(tl.end - tl.begin);
    for (int i = threadIdx.x; i < kTiledCorners; i += kTiledTile) {
        unsigned long long k = ~0ull;
        if (i < corners) {
            const uint4 id = d.index[tl.begin + (i >> 2)];
            const uint32_t c = i & 3;
            const uint32_t node = c == 0 ? id.x : (c == 1 ? id.y : (c == 2 ? id.z : id.w));
            k = ((unsigned long long)node << 9) | (unsigned long long)i;
        }
        key[i] = k;
    }
    __syncthreads();
    for (int size = 2; size <= kTiledCorners; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = threadIdx.x; i < kTiledCorners; i += kTiledTile) {
                const int j = i ^ stride;
                if (j > i) {
                    const unsigned long long a = key[i], b = key[j];
                    const bool up = (i & size) == 0;
                    if ((a > b) == up) {
                        key[i] = b;
                        key[j] = a;
                    }
                }
            }
            __syncthreads();
        }
}

// The sorted position i starts a new node (and is a real corner).
__device__ __forceinline__ bool starts_node(const unsigned long long* key, int i) {
    if (key[i] == ~0ull) return false;
    return i == 0 || (key[i] >> 9) != (key[i - 1] >> 9);
}

using TileScan = cub::BlockScan<int, kTiledTile>;

// Each thread takes four consecutive sorted positions; returns the thread's exclusive
// prefix of node starts, and the tile's total in `total`.
__device__ __forceinline__ int scan_node_starts(const unsigned long long* key, int (&flag)[4], int& total,
                                                typename TileScan::TempStorage& tmp) {
    int mine = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        flag[q] = starts_node(key, 4 * threadIdx.x + q) ? 1 : 0;
        mine += flag[q];
    }
    int before = 0;
    TileScan(tmp).ExclusiveSum(mine, before, total);
    return before;
}

// A tile's lists are padded to a multiple of 8 entries, so each starts on a 16-byte
// boundary (for the staged pass's asynchronous copies).
constexpr int kTablePad = 8;

// Pass 1: per tile, its corners sorted; the distinct-node count (and its padded
// span), and the two tables that need no global offset: the sorted corners (inv) and
// each tet's corner places in the tile's node list (lidx).
__global__ void __launch_bounds__(kTiledTile) pool_tile_count(PoolDevice d, uint32_t* count, uint32_t* span,
                                                               ushort4* lidx, uint16_t* inv) {
    __shared__ unsigned long long key[kTiledCorners];
    __shared__ uint16_t local[kTiledCorners];  // by corner: its node's place in the list
    __shared__ typename TileScan::TempStorage tmp;
    const PoolTile tl = d.etiles[blockIdx.x];
    sort_tile_corners(d, tl, key);
    int flag[4], total = 0;
    int at = scan_node_starts(key, flag, total, tmp) - 1;  // the node of position 4 x thread - 1
    const long long c0 = 4 * tl.begin;  // the tile's corners in the per-corner arrays
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int i = 4 * threadIdx.x + q;
        const unsigned long long k = key[i];
        if (k == ~0ull) continue;
        if (flag[q]) ++at;
        const int corner = (int)(k & 511ull);
        // stored as the corner's place in the element pass's force buffer, corner c of
        // tet i at c x 128 + i
        inv[c0 + i] = (uint16_t)((corner & 3) * kTiledTile + (corner >> 2));
        local[corner] = (uint16_t)at;
    }
    if (threadIdx.x == 0) {
        count[blockIdx.x] = (uint32_t)total;
        span[blockIdx.x] = (uint32_t)((total + kTablePad - 1) / kTablePad * kTablePad);
    }
    __syncthreads();
    const long long t = tl.begin + threadIdx.x;
    if (t < tl.end) {
        const int c = 4 * threadIdx.x;
        lidx[t] = make_ushort4(local[c], local[c + 1], local[c + 2], local[c + 3]);
    }
}

// Pass 2, after the scan of the spans into `off`: the node list and, per node, the
// start of its corners in the sorted list -- from the corner places alone, without a
// second sort: a node's start is the number of the tile's corners whose nodes come
// before it in the list.  Padding entries name node `dump`, one past every mesh's
// nodes, so that the partials' CSR counts them under a node no tile reads.
__global__ void __launch_bounds__(kTiledTile) pool_tile_fill(PoolDevice d, const uint32_t* off, const uint32_t* count,
                                                              uint32_t* node_tab, uint16_t* inv_start,
                                                              uint32_t dump) {
    __shared__ int hist[kTiledCorners];
    __shared__ typename TileScan::TempStorage tmp;
    const PoolTile tl = d.etiles[blockIdx.x];
    const uint32_t base = off[blockIdx.x];
    const int total = (int)count[blockIdx.x];
    for (int j = threadIdx.x; j < kTiledCorners; j += kTiledTile) hist[j] = 0;
    __syncthreads();
    const long long t = tl.begin + threadIdx.x;
    if (t < tl.end) {
        const ushort4 l = d.lidx[t];
        const uint4 id = d.index[t];
        atomicAdd(&hist[l.x], 1);
        atomicAdd(&hist[l.y], 1);
        atomicAdd(&hist[l.z], 1);
        atomicAdd(&hist[l.w], 1);
        // every corner of a node writes the same id
        node_tab[base + l.x] = id.x;
        node_tab[base + l.y] = id.y;
        node_tab[base + l.z] = id.z;
        node_tab[base + l.w] = id.w;
    }
    __syncthreads();
    // exclusive scan of the per-node corner counts: four consecutive nodes a thread
    int v[4], mine = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        v[q] = hist[4 * threadIdx.x + q];
        mine += v[q];
    }
    int before = 0, all = 0;
    TileScan(tmp).ExclusiveSum(mine, before, all);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int j = 4 * threadIdx.x + q;
        if (j < total) inv_start[base + j] = (uint16_t)before;
        before += v[q];
    }
    const int padded = (total + kTablePad - 1) / kTablePad * kTablePad;
    if ((int)threadIdx.x < padded - total) {
        node_tab[base + total + threadIdx.x] = dump;
        inv_start[base + total + threadIdx.x] = 0;
    }
}

// L2 prefetch, one line a thread, of the rows the tiled pass reads for a tile's tets:
// Dm^-1 (9 rows of 4 B a tet), the volume and the plastic state (7 rows) on threads 0-67,
// the corner places and the sorted corners (8 B a tet each) on threads 68-83.  A line
// starts inside its row's range.
__device__ __forceinline__ void prefetch_tiled_rows(const PoolDevice& d, long long begin, long long end) {
    const int n = (int)(end - begin);
    int row = threadIdx.x >> 2, line = threadIdx.x & 3;
    if (row < 17) {
        if (line * 32 >= n) return;
        const float* rowp = row < 9 ? d.rest_inv + (size_t)row * d.tet_cap
                                    : (row == 9 ? d.rest_vol : d.plastic + (size_t)(row - 10) * d.tet_cap);
        prefetch_l2(rowp + begin + line * 32);
    } else if (row < 21) {
        line += 4 * ((row - 17) & 1);
        if (line * 16 >= n) return;
        if (row < 19)
            prefetch_l2(d.lidx + begin + line * 16);
        else
            prefetch_l2(d.inv + 4 * (begin + line * 16));
    }
}

// A tet's own rows, loaded into registers before the tile's corners arrive (so their
// latency runs alongside the wait), handed to tet_element_f32_eval as its `Rows`.
struct RegRows {
    float dm[9], v, pl[7];
    __device__ __forceinline__ float inv(int k, long long) const { return dm[k]; }
    __device__ __forceinline__ float vol(long long) const { return v; }
    __device__ __forceinline__ float plastic(int i, long long) const { return pl[i]; }
};

// ---- the staged form: a persistent block walks its tiles, and while it computes one,
// the next one's node gather and tables are already on their way into the other of two
// shared-memory stages (cp.async, per thread, completed by wait_group and a barrier).

// One stage for tiles of up to `kcap` distinct nodes (a multiple of 8): the nodes'
// displacement and compensation, the tile's corner starts and partial slots (padded
// lists, copied whole), its corners sorted by node.
struct TiledStage {
    float4* su;
    float4* sc;
    uint32_t* slot;
    uint16_t* start;
    uint16_t* inv;
    __device__ __forceinline__ TiledStage(unsigned char* p, int kcap) {
        su = reinterpret_cast<float4*>(p);
        sc = su + kcap;
        slot = reinterpret_cast<uint32_t*>(sc + kcap);
        start = reinterpret_cast<uint16_t*>(slot + kcap);
        inv = start + kcap;
    }
    __host__ __device__ static size_t bytes(int kcap) {
        return (size_t)kcap * 32 + (size_t)kcap * 4 + (size_t)kcap * 2 + (size_t)kTiledCorners * 2;
    }
};

// What a block needs of a tile: from the work list and the tables in one go, all loads
// of it independent but the mesh's step.
struct TiledInfo {
    long long begin;
    uint32_t base;
    int n, k, mesh, part;
    __device__ __forceinline__ void load(const PoolDevice& d, int g) {
        const PoolTile tl = d.etiles[g];
        begin = tl.begin;
        n = (int)(tl.end - tl.begin);
        mesh = tl.mesh;
        part = tl.part;
        base = d.tab_off[g];
        k = (int)d.tab_count[g];
    }
    __device__ __forceinline__ bool live(const PoolDevice& d, int sub) const {
        const PoolMesh& m = d.meshes[mesh];
        return m.step + sub < m.target;
    }
};

// Queue the copies of a tile's gather and tables into `st` (every thread its share);
// `node` is this thread's entry of the tile's node list.
__device__ __forceinline__ void tiled_fill(const PoolDevice& d, const TiledInfo& t, uint32_t node, const TiledStage& st) {
    const int kp = (t.k + kTablePad - 1) / kTablePad * kTablePad;
    for (int j = threadIdx.x; j < t.k; j += kTiledTile) {
        const uint32_t n = j < kTiledTile ? node : d.node_tab[t.base + j];
        cp_async16(st.su + j, d.disp + n);
        cp_async16(st.sc + j, d.disp_c + n);
    }
    // the padded lists from their 16-byte aligned starts: 4 slots, or 8 starts, a copy
    for (int q = threadIdx.x; q < kp / 4; q += kTiledTile) cp_async16(st.slot + 4 * q, d.part_slot + t.base + 4 * q);
    for (int q = threadIdx.x; q < kp / 8; q += kTiledTile)
        cp_async16(st.start + 8 * q, d.inv_start + t.base + 8 * q);
    // the sorted corners: four of them (8 bytes) per tet
    if ((int)threadIdx.x < t.n) cp_async8(st.inv + 4 * threadIdx.x, d.inv + 4 * (t.begin + threadIdx.x));
}

// The loop is ordered so that no load is waited for where it is issued: a tile's record
// and its node ids are read two tiles ahead, during the node sums; its gather and tables
// go out one tile ahead, before the evaluation; its tets' own rows are read into
// registers during the node sums of the tile before, where few others are needed.  Two
// barriers a tile: one that ends the wait for the gather (and the last tile's node sums,
// whose stage is then refilled), one between the corner forces and the node sums.  The
// tile's energy sums are left per warp and added up after the next barrier.  The pass is
// bound by latency, issue and the L1 and shared-memory pipe together (each of the two 65 %
// busy on 982,014 tets, 8 blocks of 64 registers an SM; 6, 7 and 9 blocks: 516, 494 and 500 us
// for 458).  256 meshes, 10.99 M
// tets: 491 us with the record, ids and rows read where they were used and four barriers,
// 458 us so; 128 threads, each with its tet's 18 values, are more warps than two tets a
// thread would leave.
__global__ void __launch_bounds__(kTiledTile, 1024 / kTiledTile) pool_elements_tiled_ring(PoolDevice d, int sub,
                                                                                          int kcap) {
    extern __shared__ __align__(16) unsigned char tiled_smem[];
    __shared__ float4 sf[kTiledCorners];  // corner c of tet i at c x 128 + i
    __shared__ double warp_sums[2][2][kTiledTile / 32];
    __shared__ TiledInfo info[2];
    __shared__ int is_live[2];
    const int G = (int)gridDim.x;
    int g = blockIdx.x;
    if (g >= d.n_etiles) return;
    const TiledStage st0(tiled_smem, kcap), st1(tiled_smem + TiledStage::bytes(kcap), kcap);
    // this tet's rows and corner places in its tile
    RegRows rr;
    ushort4 l = make_ushort4(0, 0, 0, 0);
    const auto load_rows = [&](long long begin, int n, bool live) {
        if (live && (int)threadIdx.x < n) {
            const long long t = begin + threadIdx.x;
            l = d.lidx[t];
#pragma unroll
            for (int q = 0; q < 9; ++q) rr.dm[q] = d.rest_inv[(size_t)q * d.tet_cap + t];
            rr.v = d.rest_vol[t];
#pragma unroll
            for (int i = 0; i < 7; ++i) rr.pl[i] = d.plastic[(size_t)i * d.tet_cap + t];
        }
    };
    // a finished tile's account: its warps' sums in warp order
    const auto close_tile = [&](int which) {
        if (threadIdx.x == 0 && is_live[which]) {
            double diss = 0.0, energy = 0.0;
#pragma unroll
            for (int w = 0; w < kTiledTile / 32; ++w) {
                diss += warp_sums[which][0][w];
                energy += warp_sums[which][1][w];
            }
            account_add(&d.e_diss[info[which].part], diss);
            d.e_strain[info[which].part] = energy;
        }
    };
    TiledInfo next;  // the tile after the one in hand: its record, this thread's node of it, its mesh live
    uint32_t node = 0;
    bool next_live;
    {
        TiledInfo first;
        first.load(d, g);
        const bool live = first.live(d, sub);
        if ((int)threadIdx.x < first.k) node = d.node_tab[first.base + threadIdx.x];
        if (threadIdx.x == 0) {
            info[0] = first;
            is_live[0] = live ? 1 : 0;
        }
        if (live) tiled_fill(d, first, node, st0);  // a frozen mesh's tile reads nothing
        cp_async_commit();
        load_rows(first.begin, first.n, live);
        next.load(d, g + G < d.n_etiles ? g + G : g);
        next_live = next.live(d, sub);
        if ((int)threadIdx.x < next.k) node = d.node_tab[next.base + threadIdx.x];
    }
    for (int it = 0;; ++it) {
        const int b = it & 1;
        const TiledStage& cur = b ? st1 : st0;
        cp_async_wait_all();
        __syncthreads();
        if (it > 0) close_tile(b ^ 1);
        const bool more = g + G < d.n_etiles;
        if (more) {
            if (next_live) tiled_fill(d, next, node, b ? st0 : st1);
            cp_async_commit();
            if (threadIdx.x == 0) {
                info[b ^ 1] = next;
                is_live[b ^ 1] = next_live ? 1 : 0;
            }
        }
        const int after = g + 2 * G;
        if (after < d.n_etiles) {
            const PoolTile nx = d.etiles[after];
            prefetch_tiled_rows(d, nx.begin, nx.end);
        }
        const bool live = is_live[b] != 0;
        double diss = 0.0, energy = 0.0;
        if (live && (int)threadIdx.x < info[b].n) {
            const float4 un[4] = {cur.su[l.x], cur.su[l.y], cur.su[l.z], cur.su[l.w]};
            const float4 cn[4] = {cur.sc[l.x], cur.sc[l.y], cur.sc[l.z], cur.sc[l.w]};
            const TetElementRefs r{d.index,     d.slot, d.rest_inv, d.rest_vol, d.plastic,
                                   d.plastic_c, d.disp, d.disp_c,   d.slots,    d.tet_cap};
            float4 fc[4];
            tet_element_f32_eval<true, RegRows>(r, rr, info[b].begin + threadIdx.x, d.meshes[info[b].mesh].mat, un, cn,
                                                diss, energy, fc);
            sf[threadIdx.x] = fc[0];
            sf[kTiledTile + threadIdx.x] = fc[1];
            sf[2 * kTiledTile + threadIdx.x] = fc[2];
            sf[3 * kTiledTile + threadIdx.x] = fc[3];
        }
        __syncthreads();
        if (more) {
            load_rows(info[b ^ 1].begin, info[b ^ 1].n, is_live[b ^ 1] != 0);
            next.load(d, after < d.n_etiles ? after : g);
        }
        if (live) {
            const int k = info[b].k, corners = 4 * info[b].n;
            for (int j = threadIdx.x; j < k; j += kTiledTile) {
                const int s = cur.start[j], e = j + 1 < k ? cur.start[j + 1] : corners;
                float4 f = sf[cur.inv[s]];
                for (int q = s + 1; q < e; ++q) {
                    const float4 h = sf[cur.inv[q]];
                    f.x += h.x;
                    f.y += h.y;
                    f.z += h.z;
                }
                d.slots[cur.slot[j]] = make_float4(f.x, f.y, f.z, 0.0f);
            }
        }
        warp_sum2(diss, energy);
        if ((threadIdx.x & 31) == 0) {
            warp_sums[b][0][threadIdx.x >> 5] = diss;
            warp_sums[b][1][threadIdx.x >> 5] = energy;
        }
        if (!more) {
            __syncthreads();
            close_tile(b);
            break;
        }
        next_live = next.live(d, sub);
        if ((int)threadIdx.x < next.k) node = d.node_tab[next.base + threadIdx.x];
        g += G;
    }
}

}  // namespace

void launch_pool_tiled_element_pass(const PoolDevice& d, int sub, cudaStream_t stream) {
    if (!d.n_etiles || d.tab_kcap <= 0) return;  // no tables: nothing to step
    // a persistent grid of as many blocks as fit with two stages of kcap nodes.  The
    // kernel's dynamic shared-memory ceiling only ever grows (under a lock), so a pool
    // with smaller stages, in this thread or another, never lowers it under a launch.
    static std::mutex lock;
    static size_t ceiling = 0;
    const size_t dyn = 2 * TiledStage::bytes(d.tab_kcap);
    int per_sm = 0;
    {
        std::lock_guard<std::mutex> hold(lock);
        if (dyn > ceiling) {
            cudaFuncSetAttribute(pool_elements_tiled_ring, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
            ceiling = dyn;
        }
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pool_elements_tiled_ring, kTiledTile, dyn);
    }
    const int grid = std::min(d.n_etiles, std::max(per_sm, 1) * sm_count());
    pool_elements_tiled_ring<<<grid, kTiledTile, dyn, stream>>>(d, sub, d.tab_kcap);
}

void launch_pool_tile_count(const PoolDevice& d, uint32_t* count, uint32_t* span, ushort4* lidx, uint16_t* inv,
                            cudaStream_t stream) {
    if (d.n_etiles) pool_tile_count<<<d.n_etiles, kTiledTile, 0, stream>>>(d, count, span, lidx, inv);
}

void launch_pool_tile_fill(const PoolDevice& d, const uint32_t* off, const uint32_t* count, uint32_t* node_tab,
                           uint16_t* inv_start, uint32_t dump, cudaStream_t stream) {
    if (d.n_etiles)
        pool_tile_fill<<<d.n_etiles, kTiledTile, 0, stream>>>(d, off, count, node_tab, inv_start, dump);
}

}  // namespace fs
