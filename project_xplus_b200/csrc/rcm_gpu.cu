// rcm_gpu.cu -- reverse Cuthill-McKee and the symmetric permutation on the GPU, bit-identical
// to rcm_order / permute_symmetric (rcm.cpp), which the oracle restates (sell_rcm_oracle.py).
//
// The host order is sequential: components by lowest unplaced index; start node the component's
// minimum-(degree, index) node refined by the George-Liu pseudo-peripheral search; Cuthill-McKee
// BFS appending each node's unvisited neighbours sorted by (degree, index); reversed.
// The GPU computes the same order level by level.  When the nodes of level L sit at queue
// positions [lb, le), the host gives each node u of level L + 1 to the first node of level L
// (lowest position) adjacent to it, and lists level L + 1 parent by parent, each parent's
// children by (degree, index).  So the ordering's BFS (k_bfs, one persistent cooperative launch)
// does, per level:
//   count   children of p = {u in adj(p) : claim[u] == p}, kept in shared memory
//   write   exclusive scan of the counts in frontier order gives every parent its offset; it
//           writes its children sorted by (degree, index) there, and every child, now that it
//           has a position, claims its neighbours: claim[w] = min(claim[w], position)
// with a bounded grid barrier after each.  Positions only grow, so a claim never takes a node
// that is already in the queue, and the claim array is also the mark of what has been reached.
// The pseudo-peripheral search needs the level sets alone, in no order: its BFS (k_levels) appends
// what it reaches through a counter, one grid barrier per level.  A node with more than
// kMaxChildren claimed children, or a row with a repeated column, sends the whole ordering to the
// host function instead (same result, host speed).  Where a node has more neighbours than that, the
// first search is the ordering's BFS, so that such a graph learns it there and not after every
// search (60^2 and 300^2 meshes with a node of 100 leaves: 3.4 -> 2.1 and 29.2 -> 22.4 ms; the same
// 300^2 mesh with 62 leaves, which the GPU orders, pays 12.2 instead of 11.1).
//
// What bounds both is the chain of dependent L2 round trips and barriers of a level (order, row
// pointers, columns, claims): a level of a 2D mesh of n nodes has about sqrt(n) of them.  Eight
// lanes take a node, so that a row's columns, and their claims, come in one round trip each.
// One BFS for both purposes, a thread per node and three barriers per level, with serial sums over
// the CTAs between them, took rcm_device + permute_symmetric_device of a permuted 500^2 mesh 66.8 ms;
// this takes 31.1, most of the rest the host's copies and structure checks.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <vector>

#include "common.hpp"
#include "device_common.cuh"

namespace xplus {

void rcm_order(int n, const int* row_ptr, const int* col_idx, int* perm);  // rcm.cpp

namespace {

using namespace dev;

constexpr int kFree = 0x7F7F7F7F;  // claim of a node no frontier node has claimed (memset 0x7F)
constexpr int kMaxChildren = 64;
constexpr int kBfsThreads = 512;

constexpr int kLanes = 8;  // lanes per node
constexpr int kGroups = kBfsThreads / kLanes;

struct BfsArgs {
    const int* rp;
    const int* ci;
    const int* deg;
    int* claim;         // kFree; -1: ordered by an earlier component; else reached (position of the claimant)
    int* order;         // BFS order
    int* cnt;           // children of each frontier node (frontier-relative), where they are counted twice
    int* block_sum;     // per CTA
    int* out;           // {visited, levels, first position of the last level, too many children}
    int* tail;          // k_levels: nodes appended by a level, three levels in turn
    int root;
    unsigned* bar;
    int* err;
    long long timeout_ns;
};

// What the host reads, and the claims of this BFS taken back.  Every CTA calls it after a barrier.
__device__ __forceinline__ void finish_bfs(const BfsArgs& a, int visited, int levels, int last_b) {
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < visited; q += gridDim.x * blockDim.x)
        a.claim[a.order[q]] = kFree;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.out[0] = visited;
        a.out[1] = levels;
        a.out[2] = last_b;
    }
}

// Level sets alone: the order of the nodes within a level is whatever the appends make it.
__global__ void __launch_bounds__(kBfsThreads, 1) k_levels(BfsArgs a) {
    __shared__ int s_flag;
    GridBarrier bar{a.bar, a.err, a.timeout_ns, 0u, -1};
    const int lane = threadIdx.x & 31, l = threadIdx.x & (kLanes - 1);
    // consecutive warps of a frontier on different SMs
    const int warp = static_cast<int>((threadIdx.x >> 5) * gridDim.x + blockIdx.x);
    const int warps = static_cast<int>(gridDim.x * (blockDim.x >> 5));
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.order[0] = a.root;
        a.claim[a.root] = 0;
    }
    if (!bar.sync(&s_flag)) return;
    int lb = 0, le = 1, levels = 0, last_b = 0;
    while (le > lb) {
        int* tail = a.tail + levels % 3;
        // the next level's counter: its last reading (two levels ago) is a barrier behind
        if (blockIdx.x == 0 && threadIdx.x == 0) a.tail[(levels + 1) % 3] = 0;
        ++levels;
        last_b = lb;
        const int fs = le - lb;
        for (int q0 = warp * (32 / kLanes); q0 < fs; q0 += warps * (32 / kLanes)) {
            const int q = q0 + lane / kLanes;
            int k = 0, e = 0;
            if (q < fs) {
                const int x = a.order[lb + q];
                k = a.rp[x] + l;
                e = a.rp[x + 1];
            }
            while (__any_sync(0xffffffffu, k < e)) {
                int u = 0;
                bool own = false;
                if (k < e) {
                    u = a.ci[k];
                    // a stale kFree only leads to the exchange, which decides
                    own = a.claim[u] == kFree && atomicCAS(&a.claim[u], kFree, 0) == kFree;
                }
                const unsigned got = __ballot_sync(0xffffffffu, own);
                if (got) {
                    const int first = __ffs(got) - 1;
                    int base = 0;
                    if (lane == first) base = atomicAdd(tail, __popc(got));
                    base = __shfl_sync(0xffffffffu, base, first);
                    if (own) a.order[le + base + __popc(got & ((1u << lane) - 1u))] = u;
                }
                k += kLanes;
            }
        }
        if (!bar.sync(&s_flag)) return;
        lb = le;
        le += ld_volatile_int(tail);
    }
    finish_bfs(a, le, levels, last_b);
}

// The children of frontier node x at position p, as (degree, index) keys, in the group's slots:
// returns how many there are (those beyond kMaxChildren are counted, not kept).
__device__ __forceinline__ int gather_children(const BfsArgs& a, int x, int p, unsigned gmask, int l,
                                               unsigned long long* kid) {
    int m = 0;
    const int e = a.rp[x + 1];
    for (int k0 = a.rp[x]; k0 < e; k0 += kLanes) {
        const int k = k0 + l;
        const int u = k < e ? a.ci[k] : -1;
        const bool own = u >= 0 && u != x && a.claim[u] == p;
        const unsigned got = (__ballot_sync(gmask, own) & gmask) >> (threadIdx.x & 24);
        const int at = m + __popc(got & ((1u << l) - 1u));
        if (own && at < kMaxChildren)
            kid[at] = (static_cast<unsigned long long>(a.deg[u]) << 32) | static_cast<unsigned>(u);
        m += __popc(got);
    }
    __syncwarp(gmask);
    return m;
}

// Cuthill-McKee order from the root.
__global__ void __launch_bounds__(kBfsThreads, 1) k_bfs(BfsArgs a) {
    __shared__ int s_flag;
    __shared__ int s_warp[kBfsThreads / 32];
    __shared__ int s_cnt[kGroups];
    __shared__ unsigned long long s_kid[kGroups][kMaxChildren];
    GridBarrier bar{a.bar, a.err, a.timeout_ns, 0u, -1};
    const int lane = threadIdx.x & 31, l = threadIdx.x & (kLanes - 1), g = threadIdx.x / kLanes;
    const unsigned gmask = 0xFFu << (threadIdx.x & 24);
    unsigned long long* kid = s_kid[g];
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0) {
            a.order[0] = a.root;
            a.claim[a.root] = -1;
        }
        for (int k = a.rp[a.root] + threadIdx.x; k < a.rp[a.root + 1]; k += blockDim.x)
            if (a.ci[k] != a.root) atomicMin(&a.claim[a.ci[k]], 0);
    }
    if (!bar.sync(&s_flag)) return;
    int lb = 0, le = 1, levels = 0, last_b = 0;
    while (le > lb) {
        ++levels;
        last_b = lb;
        const int fs = le - lb;
        // count, over contiguous frontier chunks per CTA; a chunk of one node per group keeps its children
        const int chunk = (fs + gridDim.x - 1) / gridDim.x;
        const int c0 = min(fs, static_cast<int>(blockIdx.x) * chunk), c1 = min(fs, c0 + chunk);
        const bool held = chunk <= kGroups;
        int mine = 0, m = 0;
        for (int q = c0 + g; q < c1; q += kGroups) {
            m = gather_children(a, a.order[lb + q], lb + q, gmask, l, kid);
            if (l == 0) {
                if (m > kMaxChildren) atomicExch(a.out + 3, 1);
                if (!held) a.cnt[q] = m;
                mine += m;
            }
        }
        __syncwarp();
        mine = __reduce_add_sync(0xffffffffu, mine);
        if (lane == 0) s_warp[threadIdx.x >> 5] = mine;
        __syncthreads();
        if (threadIdx.x == 0) {
            int t = 0;
#pragma unroll
            for (int w = 0; w < kBfsThreads / 32; ++w) t += s_warp[w];
            a.block_sum[blockIdx.x] = t;
        }
        if (!bar.sync(&s_flag)) return;
        if (ld_volatile_int(a.out + 3) != 0) return;  // every block sees it: the host takes over
        int run = 0, total = 0;
        for (int b = lane; b < static_cast<int>(gridDim.x); b += 32) {
            const int v = a.block_sum[b];
            total += v;
            if (b < static_cast<int>(blockIdx.x)) run += v;
        }
        run = __reduce_add_sync(0xffffffffu, run);
        total = __reduce_add_sync(0xffffffffu, total);
        // write
        for (int t0 = c0; t0 < c1; t0 += kGroups) {
            const int q = t0 + g;
            if (!held) m = q < c1 ? a.cnt[q] : 0;
            if (l == 0) s_cnt[g] = q < c1 ? m : 0;
            __syncthreads();
            int off = 0, tile = 0;
            for (int i = lane; i < kGroups; i += 32) tile += s_cnt[i];
            tile = __reduce_add_sync(0xffffffffu, tile);
            for (int i = l; i < g; i += kLanes) off += s_cnt[i];
            __syncwarp();
            off = __reduce_add_sync(gmask, off) + run;
            if (q < c1 && m > 0) {
                if (!held) gather_children(a, a.order[lb + q], lb + q, gmask, l, kid);
                for (int j = 0; j < m; ++j) {
                    const unsigned long long key = kid[j];
                    int rank = 0;
                    for (int i = l; i < m; i += kLanes) rank += kid[i] < key;
                    __syncwarp(gmask);
                    const int pos = le + off + __reduce_add_sync(gmask, rank);
                    const int u = static_cast<int>(key & 0xFFFFFFFFu);
                    if (l == 0) a.order[pos] = u;
                    const int e = a.rp[u + 1];
                    for (int k = a.rp[u] + l; k < e; k += kLanes) {
                        const int w = a.ci[k];
                        if (a.claim[w] > pos) atomicMin(&a.claim[w], pos);
                    }
                    __syncwarp(gmask);
                }
            }
            run += tile;
            __syncthreads();
        }
        if (!bar.sync(&s_flag)) return;
        lb = le;
        le += total;
    }
    finish_bfs(a, le, levels, last_b);
}

constexpr int kRepeated = 1, kWide = 2;  // a row with a repeated column; a node of more than kMaxChildren neighbours
__global__ void k_degree(const int* __restrict__ rp, const int* __restrict__ ci, int n, int* __restrict__ deg,
                         int* __restrict__ flags) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int d = 0;
    for (int k = rp[i]; k < rp[i + 1]; ++k) {
        const int u = ci[k];
        if (u == i) continue;
        ++d;
        for (int q = rp[i]; q < k; ++q)
            if (ci[q] == u) atomicOr(flags, kRepeated);
    }
    if (d > kMaxChildren) atomicOr(flags, kWide);
    deg[i] = d;
}

// minimum (degree, index) over order[b, e) into *best (the caller sets it to ULLONG_MAX)
__global__ void k_argmin(const int* __restrict__ order, int b, int e, const int* __restrict__ deg,
                         unsigned long long* __restrict__ best) {
    const int q = b + blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= e) return;
    const int v = order[q];
    atomicMin(best, (static_cast<unsigned long long>(deg[v]) << 32) | static_cast<unsigned>(v));
}

__global__ void k_place(const int* __restrict__ order, int count, int* __restrict__ claim, int* __restrict__ result,
                        int pos) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= count) return;
    claim[order[q]] = -1;
    result[pos + q] = order[q];
}

__global__ void k_first_unplaced(const int* __restrict__ claim, int from, int n, int* __restrict__ first) {
    const int i = from + blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && claim[i] == kFree) atomicMin(first, i);
}

__global__ void k_reverse(const int* __restrict__ result, int n, int* __restrict__ perm) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) perm[i] = result[n - 1 - i];
}

void ck(cudaError_t e, const char* what) {
    if (e != cudaSuccess) {
        cudaGetLastError();
        throw Error(XPLUS_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
    }
}

struct Tmp {
    std::vector<void*> p;
    template <typename T>
    T* get(size_t count) {
        void* q = nullptr;
        const cudaError_t e = cudaMalloc(&q, std::max<size_t>(count * sizeof(T), 256));
        if (e != cudaSuccess) {
            cudaGetLastError();
            throw Error(XPLUS_ERR_NOMEM, std::string("cudaMalloc: ") + cudaGetErrorString(e));
        }
        p.push_back(q);
        return static_cast<T*>(q);
    }
    ~Tmp() {
        for (void* q : p) cudaFree(q);
    }
};

}  // namespace

// Reverse Cuthill-McKee of the device CSR (d_rp, d_ci; n rows) into d_perm (perm[new] = old).
// Returns false, with nothing written, when the graph needs the host ordering (a node with more
// than kMaxChildren children claimed at once, or a repeated column); the caller runs it then.
bool rcm_device(int n, const int* d_rp, const int* d_ci, int* d_perm, cudaStream_t st) {
    Tmp tmp;
    int* deg = tmp.get<int>(static_cast<size_t>(n));
    int* claim = tmp.get<int>(static_cast<size_t>(n));
    int* order = tmp.get<int>(static_cast<size_t>(n));
    int* result = tmp.get<int>(static_cast<size_t>(n));
    int* cnt = tmp.get<int>(static_cast<size_t>(n));
    int* small = tmp.get<int>(8);  // {flags, first unplaced}
    unsigned long long* best = tmp.get<unsigned long long>(1);
    int dev = 0, sms = 0, per_sm = 0;
    ck(cudaGetDevice(&dev), "cudaGetDevice");
    ck(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "attr");
    for (const auto kernel : {k_bfs, k_levels}) {
        ck(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBfsThreads, 0), "occupancy");
        require(per_sm > 0, XPLUS_ERR_CUDA, "rcm: the BFS kernel cannot be resident");
    }
    const int grid = sms;  // one block per SM, co-resident
    int* block_sum = tmp.get<int>(static_cast<size_t>(grid));
    int* ctl = tmp.get<int>(9);  // what a BFS starts from zeroed: out[4], tail[3], barrier counter, error flag
    const int tb = 256;
    ck(cudaMemsetAsync(small, 0, 8 * sizeof(int), st), "memset");
    k_degree<<<(n + tb - 1) / tb, tb, 0, st>>>(d_rp, d_ci, n, deg, small);
    ck(cudaGetLastError(), "rcm degree");
    int flags = 0;
    ck(cudaMemcpyAsync(&flags, small, sizeof(int), cudaMemcpyDeviceToHost, st), "D2H");
    ck(cudaStreamSynchronize(st), "sync");
    if (flags & kRepeated) return false;
    ck(cudaMemsetAsync(claim, 0x7F, static_cast<size_t>(n) * sizeof(int), st), "memset");
    // one BFS from root over the unplaced nodes: {visited, levels, last level begin}
    auto bfs = [&](void (*kernel)(BfsArgs), int root, int (&res)[3]) -> bool {
        BfsArgs a{};
        a.rp = d_rp;
        a.ci = d_ci;
        a.deg = deg;
        a.claim = claim;
        a.order = order;
        a.cnt = cnt;
        a.block_sum = block_sum;
        a.out = ctl;
        a.tail = ctl + 4;
        a.root = root;
        a.bar = reinterpret_cast<unsigned*>(ctl + 7);
        a.err = ctl + 8;
        a.timeout_ns = 2000000000LL;
        ck(cudaMemsetAsync(ctl, 0, 9 * sizeof(int), st), "memset");
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(kBfsThreads);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        ck(cudaLaunchKernelEx(&cfg, kernel, a), "rcm BFS launch");
        int h_out[9];
        ck(cudaMemcpyAsync(h_out, ctl, sizeof(h_out), cudaMemcpyDeviceToHost, st), "D2H");
        ck(cudaStreamSynchronize(st), "sync");
        require(h_out[8] == 0, XPLUS_ERR_CUDA, "rcm: a grid barrier timed out");
        if (h_out[3]) return false;
        res[0] = h_out[0];
        res[1] = h_out[1];
        res[2] = h_out[2];
        return true;
    };
    auto argmin = [&](int b, int e) {
        const unsigned long long init = ~0ull;
        ck(cudaMemcpyAsync(best, &init, sizeof(init), cudaMemcpyHostToDevice, st), "H2D");
        k_argmin<<<(e - b + tb - 1) / tb, tb, 0, st>>>(order, b, e, deg, best);
        ck(cudaGetLastError(), "rcm argmin");
        unsigned long long h = 0;
        ck(cudaMemcpyAsync(&h, best, sizeof(h), cudaMemcpyDeviceToHost, st), "D2H");
        ck(cudaStreamSynchronize(st), "sync");
        return static_cast<int>(h & 0xFFFFFFFFull);
    };
    int pos = 0, seed = 0;
    while (pos < n) {
        // the lowest unplaced node
        const int big = INT_MAX;
        ck(cudaMemcpyAsync(small + 1, &big, sizeof(int), cudaMemcpyHostToDevice, st), "H2D");
        k_first_unplaced<<<(n - seed + tb - 1) / tb, tb, 0, st>>>(claim, seed, n, small + 1);
        ck(cudaGetLastError(), "rcm seed");
        ck(cudaMemcpyAsync(&seed, small + 1, sizeof(int), cudaMemcpyDeviceToHost, st), "D2H");
        ck(cudaStreamSynchronize(st), "sync");
        int r[3];
        if (!bfs(flags & kWide ? k_bfs : k_levels, seed, r)) return false;
        int v = argmin(0, r[0]);  // the component's minimum-(degree, index) node
        if (!bfs(k_levels, v, r)) return false;
        int ecc = r[1], last_b = r[2], last_e = r[0];
        while (true) {  // George-Liu pseudo-peripheral node
            const int u = argmin(last_b, last_e);
            int r2[3];
            if (!bfs(k_levels, u, r2)) return false;
            if (r2[1] > ecc) {
                v = u;
                ecc = r2[1];
                last_b = r2[2];
                last_e = r2[0];
            } else {
                break;
            }
        }
        if (!bfs(k_bfs, v, r)) return false;  // Cuthill-McKee from v
        k_place<<<(r[0] + tb - 1) / tb, tb, 0, st>>>(order, r[0], claim, result, pos);
        ck(cudaGetLastError(), "rcm place");
        pos += r[0];
    }
    k_reverse<<<(n + tb - 1) / tb, tb, 0, st>>>(result, n, d_perm);
    ck(cudaGetLastError(), "rcm reverse");
    ck(cudaStreamSynchronize(st), "sync");
    return true;
}

namespace {

__global__ void k_inverse_perm(const int* __restrict__ perm, int n, int* __restrict__ iperm, int* __restrict__ bad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int p = perm[i];
    if (p < 0 || p >= n || atomicExch(&iperm[p], i) != -1) atomicOr(bad, 1);
}

__global__ void k_perm_lengths(const int* __restrict__ rp, const int* __restrict__ perm, int n, int* __restrict__ len) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) len[i] = rp[perm[i] + 1] - rp[perm[i]];
}

// out[0] = 0, out[i + 1] = out[i] + len[i]: one CTA, each thread a contiguous chunk
__global__ void __launch_bounds__(1024) k_scan_int(const int* __restrict__ len, int n, int* __restrict__ out) {
    __shared__ int s_sum[1024];
    const int t = threadIdx.x;
    const int per = (n + blockDim.x - 1) / blockDim.x;
    const int b = min(n, t * per), e = min(n, b + per);
    int acc = 0;
    for (int i = b; i < e; ++i) acc += len[i];
    s_sum[t] = acc;
    __syncthreads();
    for (int o = 1; o < static_cast<int>(blockDim.x); o <<= 1) {
        const int v = t >= o ? s_sum[t - o] : 0;
        __syncthreads();
        s_sum[t] += v;
        __syncthreads();
    }
    int run = t > 0 ? s_sum[t - 1] : 0;
    if (t == 0) out[0] = 0;
    for (int i = b; i < e; ++i) {
        run += len[i];
        out[i + 1] = run;
    }
}

// new row i = old row perm[i], columns renumbered by iperm and stably sorted ascending (the
// host's stable_sort of (column, value) pairs)
__global__ void k_perm_fill(const int* __restrict__ rp, const int* __restrict__ ci, const double* __restrict__ v,
                            const int* __restrict__ perm, const int* __restrict__ iperm, const int* __restrict__ orp,
                            int n, int* __restrict__ oci, double* __restrict__ ov) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int old = perm[i];
    const int o0 = orp[i];
    int m = 0;
    for (int k = rp[old]; k < rp[old + 1]; ++k, ++m) {
        const int c = iperm[ci[k]];
        const double x = v[k];
        int j = o0 + m;  // insertion: shift only strictly greater columns (stable)
        while (j > o0 && oci[j - 1] > c) {
            oci[j] = oci[j - 1];
            ov[j] = ov[j - 1];
            --j;
        }
        oci[j] = c;
        ov[j] = x;
    }
}

}  // namespace

void permute_symmetric_device(int n, const int* d_rp, const int* d_ci, const double* d_v, const int* d_perm,
                              int* d_orp, int* d_oci, double* d_ov, cudaStream_t st) {
    Tmp tmp;
    int* iperm = tmp.get<int>(static_cast<size_t>(n));
    int* len = tmp.get<int>(static_cast<size_t>(n));
    int* bad = tmp.get<int>(1);
    const int tb = 256;
    ck(cudaMemsetAsync(iperm, 0xFF, static_cast<size_t>(n) * sizeof(int), st), "memset");
    ck(cudaMemsetAsync(bad, 0, sizeof(int), st), "memset");
    k_inverse_perm<<<(n + tb - 1) / tb, tb, 0, st>>>(d_perm, n, iperm, bad);
    ck(cudaGetLastError(), "inverse permutation");
    int h_bad = 0;
    ck(cudaMemcpyAsync(&h_bad, bad, sizeof(int), cudaMemcpyDeviceToHost, st), "D2H");
    ck(cudaStreamSynchronize(st), "sync");
    require(h_bad == 0, XPLUS_ERR_ARG, "perm is not a permutation");
    k_perm_lengths<<<(n + tb - 1) / tb, tb, 0, st>>>(d_rp, d_perm, n, len);
    k_scan_int<<<1, 1024, 0, st>>>(len, n, d_orp);
    k_perm_fill<<<(n + tb - 1) / tb, tb, 0, st>>>(d_rp, d_ci, d_v, d_perm, iperm, d_orp, n, d_oci, d_ov);
    ck(cudaGetLastError(), "permute");
    ck(cudaStreamSynchronize(st), "sync");
}

}  // namespace xplus

using namespace xplus;

namespace {

// the device CSR's structure, checked before anything is indexed (XPLUS_ERR_DATA)
void check_device_csr(int n, const int* d_rp, const int* d_ci, cudaStream_t st) {
    require(n > 0 && d_rp && d_ci, XPLUS_ERR_ARG, "invalid argument");
    int dev = 0;
    ck(cudaGetDevice(&dev), "cudaGetDevice");
    require_device_memory(d_rp, dev, "d_row_ptr");
    require_device_memory(d_ci, dev, "d_col_idx");
    std::vector<int> rp(static_cast<size_t>(n) + 1);
    ck(cudaMemcpyAsync(rp.data(), d_rp, rp.size() * sizeof(int), cudaMemcpyDeviceToHost, st), "D2H");
    ck(cudaStreamSynchronize(st), "sync");
    require(rp[0] == 0, XPLUS_ERR_DATA, "row_ptr[0] must be 0");
    for (int i = 0; i < n; ++i) require(rp[static_cast<size_t>(i)] <= rp[static_cast<size_t>(i) + 1], XPLUS_ERR_DATA, "row_ptr must be nondecreasing");
    std::vector<int> ci(static_cast<size_t>(rp[static_cast<size_t>(n)]));
    if (!ci.empty()) {
        ck(cudaMemcpyAsync(ci.data(), d_ci, ci.size() * sizeof(int), cudaMemcpyDeviceToHost, st), "D2H");
        ck(cudaStreamSynchronize(st), "sync");
        for (int c : ci) require(c >= 0 && c < n, XPLUS_ERR_DATA, "col_idx out of range");
    }
}

}  // namespace

extern "C" {

int xplus_rcm_device(int n, const int* d_row_ptr, const int* d_col_idx, int* d_perm, int* used_gpu, void* stream) {
    return guarded([&] {
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        check_device_csr(n, d_row_ptr, d_col_idx, st);
        int dev = 0;
        ck(cudaGetDevice(&dev), "cudaGetDevice");
        require_device_memory(d_perm, dev, "d_perm");
        const bool on_gpu = rcm_device(n, d_row_ptr, d_col_idx, d_perm, st);
        if (!on_gpu) {
            // the host ordering (same result): a node with many children at once, or a repeated column
            std::vector<int> rp(static_cast<size_t>(n) + 1), perm(static_cast<size_t>(n));
            ck(cudaMemcpy(rp.data(), d_row_ptr, rp.size() * sizeof(int), cudaMemcpyDeviceToHost), "D2H");
            std::vector<int> ci(static_cast<size_t>(rp[static_cast<size_t>(n)]));
            ck(cudaMemcpy(ci.data(), d_col_idx, ci.size() * sizeof(int), cudaMemcpyDeviceToHost), "D2H");
            rcm_order(n, rp.data(), ci.data(), perm.data());
            ck(cudaMemcpy(d_perm, perm.data(), perm.size() * sizeof(int), cudaMemcpyHostToDevice), "H2D");
        }
        if (used_gpu) *used_gpu = on_gpu ? 1 : 0;
    });
}

int xplus_permute_symmetric_device(int n, const int* d_row_ptr, const int* d_col_idx, const double* d_values,
                                   const int* d_perm, int* d_out_row_ptr, int* d_out_col_idx, double* d_out_values,
                                   void* stream) {
    return guarded([&] {
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        check_device_csr(n, d_row_ptr, d_col_idx, st);
        int dev = 0;
        ck(cudaGetDevice(&dev), "cudaGetDevice");
        for (const void* p : {static_cast<const void*>(d_values), static_cast<const void*>(d_perm),
                              static_cast<const void*>(d_out_row_ptr), static_cast<const void*>(d_out_col_idx),
                              static_cast<const void*>(d_out_values)})
            require_device_memory(p, dev, "device array");
        permute_symmetric_device(n, d_row_ptr, d_col_idx, d_values, d_perm, d_out_row_ptr, d_out_col_idx, d_out_values,
                                 st);
    });
}

}  // extern "C"
