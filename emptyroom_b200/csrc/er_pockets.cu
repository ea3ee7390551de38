// er_pockets.cu -- pocket blocking on the GPU (er_block_pockets*) and the
// hard-sphere accessibility grid (er_accessibility).
//
// FindAndBlockPockets (src/pocketblocking.cc:126-391) labels 6-connected
// segments of accessible points (E < 15 T) with a serial flood fill in scan
// order, links segments across the three periodic faces, and calls a segment
// a POCKET unless a walk over those links returns to it in another unit cell.
// Here:
//   1. tiles     label of every accessible point = smallest point of its
//                component inside its 4 x 8 x 32-point tile (runs along k by
//                warp ballots, then union-find over the runs in shared memory)
//   2. faces     lock-free union-find across the tile faces; a root is always
//                linked to a smaller root, so every component ends rooted at
//                its smallest linear index
//   3. links     (from = root at N-1, to = root at 0, direction) over the
//                periodic faces, deduplicated in a device hash set
//   4. classify  on the host: weighted union-find over the (few) links; a
//                component is a CHANNEL iff some link contradicts the unit-cell
//                offsets (a cycle with non-zero net translation, self-links
//                included) -- the same verdict as the reference's DFS, which
//                checks every link of the component against a spanning walk
//   5. block     every point walks to its root and meets a channel's or not:
//                pocket points -> 1e13 (host double grid) or mask = 1 (device),
//                and the pocket roots are counted
// The reference numbers segments in the order its flood fill meets them, by
// smallest index: roots ranked in index order (compress and number), needed
// only when the caller asks for the numbers.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "er_ctx.h"
#include "er_host.h"
#include "er_nvtx.h"

namespace er {

__device__ __forceinline__ int cc_find(const int* lab, int x) {
    int y = lab[x];
    while (y != x) {
        x = y;
        y = lab[x];
    }
    return x;
}

// The same walk reading through L2 (labels change under concurrent unions).
// Labels only ever decrease along a chain, so the walk ends.
__device__ __forceinline__ int cc_find_l2(const int* lab, int x) {
    int y = __ldcg(lab + x);
    while (y != x) {
        x = y;
        y = __ldcg(lab + x);
    }
    return x;
}

// Links the roots of a and b (larger root under smaller). Every failed CAS
// means another thread has just linked that root to a smaller label, so a
// strictly decreases and the loop ends.
__device__ __forceinline__ void cc_unite(int* lab, int a, int b) {
    for (;;) {
        a = cc_find_l2(lab, a);
        b = cc_find_l2(lab, b);
        if (a == b) return;
        if (a < b) {
            const int t = a; a = b; b = t;
        }
        const int old = atomicCAS(&lab[a], a, b);
        if (old == a) return;
        a = old;
    }
}

// Tiled labelling: a CTA labels one tile of kTI x kTJ x kTK points (k fastest,
// so a warp's row is 32 consecutive points). A row's accessible points come as
// one ballot word; each starts at the first point of its run, which joins the
// neighbours along k without an atomic, and two neighbouring rows need one
// union per stretch in which both are accessible. Then each accessible point's
// label is written as the global index of its tile-local root. Local indices
// order like global ones inside a tile, and a tile-local root is the smallest
// index of its local component, so every label is <= its point and roots point
// to themselves: a valid state for cc_unite. The unions across tile faces
// follow in cc_union_faces, after every tile has written (a face union into a
// tile that had not yet written could be overwritten).
// On a 129^3 grid 18 us against 80 with a union per neighbouring pair of points
// (and 6 for a pass that wrote the first labels), the face unions 17 against
// 57; the device mask of that grid takes 93 us a call against 247, which
// numbered every segment and waited for the host four times.
constexpr int kTK = 32, kTJ = 8, kTI = 4, kTile = kTK * kTJ * kTI, kTRows = kTI * kTJ;
static_assert(kTK == 32 && kTJ == 8, "a warp per row of points, 256 threads per layer");

__device__ __forceinline__ int cc_find_s(const int* sl, int x) {
    int y = sl[x];
    while (y != x) {
        x = y;
        y = sl[x];
    }
    return x;
}

__device__ __forceinline__ void cc_unite_s(int* sl, int a, int b) {
    for (;;) {
        a = cc_find_s(sl, a);
        b = cc_find_s(sl, b);
        if (a == b) return;
        if (a < b) {
            const int t = a; a = b; b = t;
        }
        const int old = atomicCAS(&sl[a], a, b);
        if (old == a) return;
        a = old;
    }
}

template <typename G>
__global__ void __launch_bounds__(256) cc_label_tiles(const G* __restrict__ E, double thr, int nx,
                                                      int ny, int nz, int* __restrict__ lab) {
    __shared__ int sl[kTile];
    __shared__ unsigned open[kTRows];  // accessible points of each row
    const int tk = (nz + kTK - 1) / kTK, tj = (ny + kTJ - 1) / kTJ;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int k = (int)(blockIdx.x % tk) * kTK + lane;
    const int j0 = (int)((blockIdx.x / tk) % tj) * kTJ;
    const int i0 = (int)(blockIdx.x / (tk * tj)) * kTI;
    // rows w, w + 8, ... of the tile: all kTI loads in flight together
    G e[kTI];
    bool in[kTI];
#pragma unroll
    for (int u = 0; u < kTI; ++u) {
        const int i = i0 + u, j = j0 + w;
        in[u] = i < nx && j < ny && k < nz;
        if (in[u]) e[u] = E[(int64_t)k + (int64_t)j * nz + (int64_t)i * ny * nz];
    }
#pragma unroll
    for (int u = 0; u < kTI; ++u) {
        const int row = u * kTJ + w;
        const bool acc = in[u] && !((double)e[u] >= thr);  // src/pocketblocking.cc:138
        const unsigned b = __ballot_sync(0xffffffffu, acc);
        const unsigned gaps = ~b & ((1u << lane) - 1u);  // blocked points below this one
        sl[row * kTK + lane] = acc ? row * kTK + (gaps ? 32 - __clz(gaps) : 0) : -1;
        if (lane == 0) open[row] = b;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kTI; ++u) {
        const int row = u * kTJ + w, q = row * kTK + lane;
        const unsigned bit = 1u << lane;
        if (w > 0) {
            const unsigned both = open[row] & open[row - 1];
            if (both & ~(both << 1) & bit) cc_unite_s(sl, q, q - kTK);
        }
        if (u > 0) {
            const unsigned both = open[row] & open[row - kTJ];
            if (both & ~(both << 1) & bit) cc_unite_s(sl, q, q - kTK * kTJ);
        }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kTI; ++u) {
        if (!in[u]) continue;
        const int q = (u * kTJ + w) * kTK + lane;
        int l = -1;
        if (sl[q] >= 0) {
            const int r = cc_find_s(sl, q);
            l = (int)((int64_t)(k - lane + r % kTK) + (int64_t)(j0 + (r / kTK) % kTJ) * nz +
                      (int64_t)(i0 + r / (kTK * kTJ)) * ny * nz);
        }
        lab[(int64_t)k + (int64_t)(j0 + w) * nz + (int64_t)(i0 + u) * ny * nz] = l;
    }
}

// Unions across the lower faces of the tiles (global union-find), one thread
// per face point. Two neighbours along a face that are accessible on both
// sides, inside one tile on each, are joined there already: only the first of
// such a stretch unites.
__global__ void __launch_bounds__(256) cc_union_faces(int* __restrict__ lab, int nx, int ny,
                                                      int nz) {
    const int64_t syz = (int64_t)ny * nz;
    const int64_t fi = (int64_t)((nx - 1) / kTI) * syz;             // i = kTI, 2 kTI, ...
    const int64_t fj = (int64_t)((ny - 1) / kTJ) * nx * nz;         // j = kTJ, ...
    const int64_t fk = (int64_t)((nz - 1) / kTK) * nx * ny;         // k = kTK, ...
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < fi + fj + fk;
         q += (int64_t)gridDim.x * blockDim.x) {
        // fewer than 2^31 points: 32-bit quotients
        int64_t p, across, along;  // the point, its neighbour's and its stretch's offsets
        bool first;                // the stretch cannot have begun before this point
        if (q < fi) {
            const unsigned i = (unsigned)q / (unsigned)syz, r = (unsigned)q % (unsigned)syz;
            p = (int64_t)(i + 1) * kTI * syz + r;
            across = syz;
            along = 1;
            first = r % (unsigned)nz % kTK == 0;
        } else if (q < fi + fj) {
            const unsigned t = (unsigned)(q - fi), k = t % (unsigned)nz, ij = t / (unsigned)nz;
            const int64_t i = ij % (unsigned)nx, j = (int64_t)(ij / (unsigned)nx + 1) * kTJ;
            p = k + j * nz + i * syz;
            across = nz;
            along = 1;
            first = k % kTK == 0;
        } else {
            const unsigned t = (unsigned)(q - fi - fj), j = t % (unsigned)ny, ik = t / (unsigned)ny;
            const int64_t i = ik % (unsigned)nx, k = (int64_t)(ik / (unsigned)nx + 1) * kTK;
            p = k + j * nz + i * syz;
            across = 1;
            along = nz;
            first = j % kTJ == 0;
        }
        if (__ldcg(lab + p) < 0 || __ldcg(lab + p - across) < 0) continue;
        if (!first && __ldcg(lab + p - along) >= 0 && __ldcg(lab + p - along - across) >= 0)
            continue;
        cc_unite(lab, (int)p, (int)(p - across));
    }
}

__global__ void cc_compress(int* __restrict__ lab, int64_t n) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n;
         p += (int64_t)gridDim.x * blockDim.x) {
        if (lab[p] >= 0) lab[p] = cc_find(lab, (int)p);
    }
}

constexpr int kScanItems = 4096;  // points per scan block (1024 threads x 4)

// Number of roots in each block of kScanItems points.
__global__ void __launch_bounds__(1024) cc_root_counts(const int* __restrict__ lab, int64_t n,
                                                       int* __restrict__ counts) {
    const int64_t base = (int64_t)blockIdx.x * kScanItems;
    int c = 0;
    for (int q = threadIdx.x; q < kScanItems; q += 1024) {
        const int64_t p = base + q;
        if (p < n && lab[p] == (int)p) ++c;
    }
    __shared__ int s[32];
    int v = c;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        int w = s[threadIdx.x];
        for (int o = 16; o > 0; o >>= 1) w += __shfl_down_sync(0xffffffffu, w, o);
        if (threadIdx.x == 0) counts[blockIdx.x] = w;
    }
}

// Exclusive scan of n ints by one CTA (contiguous chunks); out[n] = total.
__global__ void __launch_bounds__(1024) cc_scan_small(const int* __restrict__ in,
                                                      int* __restrict__ out, int n) {
    __shared__ int sums[1024];
    const int t = threadIdx.x;
    const int per = (n + 1023) / 1024;
    const int lo = min(n, t * per), hi = min(n, lo + per);
    int s = 0;
    for (int i = lo; i < hi; ++i) s += in[i];
    sums[t] = s;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const int v = t >= o ? sums[t - o] : 0;
        __syncthreads();
        sums[t] += v;
        __syncthreads();
    }
    int run = sums[t] - s;
    for (int i = lo; i < hi; ++i) {
        const int v = in[i];
        out[i] = run;
        run += v;
    }
    if (t == 1023) out[n] = sums[1023];
}

// rank[p] = number of roots below p, for every root p (thread q owns points
// base + 4q .. base + 4q + 3, so ranks follow the linear index).
__global__ void __launch_bounds__(1024) cc_root_ranks(const int* __restrict__ lab, int64_t n,
                                                      const int* __restrict__ block_off,
                                                      int* __restrict__ rank) {
    __shared__ int wsum[32];
    const int64_t base = (int64_t)blockIdx.x * kScanItems + 4 * threadIdx.x;
    int f[4], c = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int64_t p = base + u;
        f[u] = (p < n && lab[p] == (int)p) ? 1 : 0;
        c += f[u];
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = c;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    if (w == 0) {
        int t = wsum[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        wsum[lane] = t;
    }
    __syncthreads();
    int run = block_off[blockIdx.x] + (w ? wsum[w - 1] : 0) + x - c;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        if (f[u]) rank[base + u] = run;
        run += f[u];
    }
}

__global__ void cc_segments(const int* __restrict__ lab, const int* __restrict__ rank, int64_t n,
                            int* __restrict__ seg) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n;
         p += (int64_t)gridDim.x * blockDim.x) {
        const int l = lab[p];
        seg[p] = l >= 0 ? rank[l] : -1;
    }
}

__host__ __device__ __forceinline__ uint64_t mix64(uint64_t x) {
    x ^= x >> 33;
    x *= 0xff51afd7ed558ccdull;
    x ^= x >> 33;
    x *= 0xc4ceb9fe1a85ec53ull;
    x ^= x >> 33;
    return x;
}

// Counters at the head of PocketScratch::misc; the whole block starts as ~0,
// so each counts from -1.
struct PocketCounters {
    int links, pockets;
};
constexpr size_t kCounterBytes = 256;

__host__ __device__ inline unsigned long long link_key(int from, int to, int dir) {
    return ((unsigned long long)from << 33) | ((unsigned long long)to << 2) |
           (unsigned long long)dir;
}

// Face links of src/pocketblocking.cc:277-321 between component roots, inserted
// once each into an open-addressing set; new keys are appended to `list`. A
// link that the lane before has too is left to it.
__global__ void __launch_bounds__(256) cc_face_links(const int* __restrict__ lab, int nx, int ny,
                                                     int nz, unsigned long long* __restrict__ table,
                                                     int table_mask,
                                                     unsigned long long* __restrict__ list,
                                                     int list_cap, PocketCounters* cnt) {
    const int64_t fx = (int64_t)ny * nz, fy = (int64_t)nx * nz, fz = (int64_t)nx * ny;
    const int64_t total = fx + fy + fz;
    const int64_t syz = (int64_t)ny * nz;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t q0 = blockIdx.x * (int64_t)blockDim.x; q0 < total; q0 += stride) {
        const int64_t q = q0 + threadIdx.x;
        unsigned long long key = ~0ull;
        if (q < total) {
            int64_t a, b;
            int dir;
            if (q < fx) {  // i = 0 face against i = N_x - 1
                a = q;
                b = a + (int64_t)(nx - 1) * syz;
                dir = 1;
            } else if (q < fx + fy) {  // j = 0 face against j = N_y - 1
                const unsigned r = (unsigned)(q - fx);
                a = r % (unsigned)nz + r / (unsigned)nz * syz;
                b = a + (int64_t)(ny - 1) * nz;
                dir = 2;
            } else {  // k = 0 face against k = N_z - 1
                const unsigned r = (unsigned)(q - fx - fy);
                a = (int64_t)(r % (unsigned)ny) * nz + r / (unsigned)ny * syz;
                b = a + (nz - 1);
                dir = 3;
            }
            if (lab[a] >= 0 && lab[b] >= 0)
                key = link_key(cc_find(lab, (int)b), cc_find(lab, (int)a), dir);
        }
        const unsigned long long before = __shfl_up_sync(0xffffffffu, key, 1);
        if (key == ~0ull || ((threadIdx.x & 31) && before == key)) continue;
        unsigned h = (unsigned)(mix64(key) & (uint64_t)table_mask);
        for (int probe = 0; probe <= table_mask; ++probe) {
            const unsigned long long old = atomicCAS(&table[h], ~0ull, key);
            if (old == ~0ull) {
                const int at = atomicAdd(&cnt->links, 1) + 1;
                if (at < list_cap) list[at] = key;
                break;
            }
            if (old == key) break;
            h = (h + 1) & (unsigned)table_mask;
        }
    }
}

// The channel roots, by value where they are few (a grid's channels usually are
// one or two): copying them up and marking their labels took 2 of 75 us of a 64^3
// mask's call.
// Otherwise n is 0 and the roots are marked.
struct Channels {
    int n = 0;
    int root[16];
};

// Channel roots r become -2 - r: the walk to a root ends at any negative label.
__global__ void cc_mark_channels(const int* __restrict__ roots, int n, int* __restrict__ lab) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) lab[roots[t]] = -2 - roots[t];
}

// Walks every point to its root. FP64 grid: pocket points become 1e13
// (src/pocketblocking.cc:373-382); mask: 1 on pocket points, else 0. Counts
// the pockets (roots that no channel marking reached).
template <bool MASK>
__global__ void __launch_bounds__(256) cc_block(const int* __restrict__ lab, int64_t n,
                                                const __grid_constant__ Channels ch,
                                                double* __restrict__ E,
                                                uint8_t* __restrict__ mask, PocketCounters* cnt) {
    int roots = 0;
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n;
         p += (int64_t)gridDim.x * blockDim.x) {
        int x = (int)p, l = lab[p];
        while (l >= 0 && l != x) {
            x = l;
            l = lab[x];
        }
        for (int k = 0; k < ch.n; ++k)
            if (l == ch.root[k]) l = -1;
        roots += l == (int)p;
        if (MASK) mask[p] = l >= 0;
        else if (l >= 0) E[p] = 1e13;
    }
    roots = __reduce_add_sync(0xffffffffu, roots);
    __shared__ int warp_roots[8];
    if ((threadIdx.x & 31) == 0) warp_roots[threadIdx.x >> 5] = roots;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int k = 0; k < 8; ++k) t += warp_roots[k];
        if (t) atomicAdd(&cnt->pockets, t);
    }
}

// Host: weighted union-find over the links, in any order; the roots of components
// that have a link which contradicts the unit-cell offsets. The roots get their
// numbers from a hash set as they come: sorting them (and the links) took most of
// the call where a grid has thousands of links (device mask of a checkerboard of
// 97^3 points 2481 -> 400 us, of 97^3 points 30 % open at random 455 -> 155).
static std::vector<int> channel_roots(const std::vector<unsigned long long>& links) {
    unsigned slots = 64;
    while (slots < 4 * links.size()) slots <<= 1;
    std::vector<int> slot(slots, -1);
    std::vector<int> roots, ends;  // every root that has a link; the links' two, in turn
    ends.reserve(2 * links.size());
    auto number = [&](int root) {
        unsigned h = (unsigned)(mix64((unsigned)root) & (slots - 1));
        while (slot[h] >= 0 && roots[slot[h]] != root) h = (h + 1) & (slots - 1);
        if (slot[h] < 0) {
            slot[h] = (int)roots.size();
            roots.push_back(root);
        }
        return slot[h];
    };
    for (unsigned long long key : links) {
        ends.push_back(number((int)(key >> 33)));
        ends.push_back(number((int)((key >> 2) & 0x7fffffffull)));
    }
    const int n = (int)roots.size();
    std::vector<int> parent(n);
    std::vector<int> ox(n, 0), oy(n, 0), oz(n, 0);  // offset to parent
    std::vector<unsigned char> bad(n, 0);
    for (int s = 0; s < n; ++s) parent[s] = s;
    auto find = [&](int s, int& x, int& y, int& z) {
        // returns the root and the offset of s relative to it; compresses
        int r = s;
        x = y = z = 0;
        while (parent[r] != r) {
            x += ox[r]; y += oy[r]; z += oz[r];
            r = parent[r];
        }
        int c = s, cx = x, cy = y, cz = z;
        while (parent[c] != c) {
            const int nxt = parent[c];
            const int tx = ox[c], ty = oy[c], tz = oz[c];
            parent[c] = r; ox[c] = cx; oy[c] = cy; oz[c] = cz;
            cx -= tx; cy -= ty; cz -= tz;
            c = nxt;
        }
        return r;
    };
    for (size_t k = 0; k < links.size(); ++k) {
        const int dir = (int)(links[k] & 3ull), from = ends[2 * k], to = ends[2 * k + 1];
        // uc(to) - uc(from) = e_dir (src/pocketblocking.cc:62-83)
        const int ex = dir == 1, ey = dir == 2, ez = dir == 3;
        int fx, fy, fz, tx, ty, tz;
        const int rf = find(from, fx, fy, fz);
        const int rt = find(to, tx, ty, tz);
        if (rf == rt) {
            if (tx - fx != ex || ty - fy != ey || tz - fz != ez) bad[rf] = 1;
        } else {
            parent[rt] = rf;
            ox[rt] = fx + ex - tx;
            oy[rt] = fy + ey - ty;
            oz[rt] = fz + ez - tz;
            bad[rf] |= bad[rt];
        }
    }
    std::vector<int> out;
    for (int s = 0; s < n; ++s) {
        int x, y, z;
        if (bad[find(s, x, y, z)]) out.push_back(roots[s]);
    }
    return out;
}

// Sizes of the face-link set and of the scratch that holds it: the counters,
// the list of links and the hash table, in this order.
struct LinkLayout {
    int64_t faces, slots;
    size_t list_at, table_at, bytes;
    LinkLayout(int nx, int ny, int nz) {
        faces = (int64_t)ny * nz + (int64_t)nx * nz + (int64_t)nx * ny;
        slots = 1024;
        while (slots < 2 * faces) slots <<= 1;
        list_at = kCounterBytes;
        table_at = list_at + (size_t)faces * sizeof(unsigned long long);
        bytes = table_at + (size_t)slots * sizeof(unsigned long long);
    }
};
// Links copied back with their count, before it is known (the others follow).
constexpr int64_t kFirstLinks = 2048;

// Labels the grid E (device) and finds the channels, whose roots go to ch or are
// marked in ps.lab, on stream st, which it synchronises once (twice past
// kFirstLinks links). With `numbers` the segment of every point goes to ps.seg.
template <typename G>
static int label_and_classify(er_ctx* ctx, PocketScratch& ps, cudaStream_t st, const G* E,
                              double thr, int nx, int ny, int nz, bool numbers, Channels& ch) {
    const int64_t n = (int64_t)nx * ny * nz;
    const LinkLayout L(nx, ny, nz);
    const int64_t tiles = (int64_t)((nz + kTK - 1) / kTK) * ((ny + kTJ - 1) / kTJ) *
                          ((nx + kTI - 1) / kTI);
    if (tiles > INT32_MAX) return set_error(ctx, ER_ERR_LIMIT, "pockets: grid too large");
    int* lab = (int*)ps.lab.ptr;
    char* misc = (char*)ps.misc.ptr;
    PocketCounters* cnt = (PocketCounters*)misc;
    unsigned long long* list = (unsigned long long*)(misc + L.list_at);
    unsigned long long* table = (unsigned long long*)(misc + L.table_at);
    ER_CUDA(ctx, cudaMemsetAsync(misc, 0xff, L.bytes, st));
    cc_label_tiles<G><<<(unsigned)tiles, 256, 0, st>>>(E, thr, nx, ny, nz, lab);
    const int64_t inner = (int64_t)((nx - 1) / kTI) * ny * nz +
                          (int64_t)((ny - 1) / kTJ) * nx * nz + (int64_t)((nz - 1) / kTK) * nx * ny;
    auto blocks = [&](int64_t threads) {
        return (int)std::max<int64_t>(
            1, std::min<int64_t>((threads + 255) / 256, (int64_t)ctx->num_sms * 32));
    };
    if (inner > 0) cc_union_faces<<<blocks(inner), 256, 0, st>>>(lab, nx, ny, nz);
    cc_face_links<<<blocks(L.faces), 256, 0, st>>>(lab, nx, ny, nz, table, (int)(L.slots - 1), list,
                                                   (int)L.faces, cnt);
    ER_CUDA(ctx, cudaGetLastError());
    const int64_t first = std::min(L.faces, kFirstLinks);
    const size_t head = L.list_at + (size_t)first * sizeof(unsigned long long);
    ER_CUDA(ctx, cudaMemcpyAsync(ps.host.ptr, misc, head, cudaMemcpyDeviceToHost, st));
    if (numbers) {
        const int nblk = (int)((n + kScanItems - 1) / kScanItems);
        int* rank = (int*)ps.grid.ptr;
        int* bcount = rank + n;
        int* boff = bcount + nblk;
        cc_compress<<<blocks(n), 256, 0, st>>>(lab, n);
        cc_root_counts<<<nblk, 1024, 0, st>>>(lab, n, bcount);
        cc_scan_small<<<1, 1024, 0, st>>>(bcount, boff, nblk);
        cc_root_ranks<<<nblk, 1024, 0, st>>>(lab, n, boff, rank);
        cc_segments<<<blocks(n), 256, 0, st>>>(lab, rank, n, (int*)ps.seg.ptr);
        ER_CUDA(ctx, cudaGetLastError());
    }
    ER_CUDA(ctx, cudaStreamSynchronize(st));
    const char* h = (const char*)ps.host.ptr;
    const int nl = ((const PocketCounters*)h)->links + 1;
    const unsigned long long* hl = (const unsigned long long*)(h + L.list_at);
    std::vector<unsigned long long> links(hl, hl + std::min<int64_t>(nl, first));
    if (nl > first) {
        links.resize(nl);
        ER_CUDA(ctx, cudaMemcpyAsync(links.data() + first, list + first,
                                     (size_t)(nl - first) * sizeof(unsigned long long),
                                     cudaMemcpyDeviceToHost, st));
        ER_CUDA(ctx, cudaStreamSynchronize(st));
    }
    const std::vector<int> channels = channel_roots(links);
    if (channels.size() <= sizeof(ch.root) / sizeof(int)) {
        ch.n = (int)channels.size();
        std::copy(channels.begin(), channels.end(), ch.root);
    } else {
        const size_t bytes = channels.size() * sizeof(int);
        if (ps.host.ensure(bytes) != ER_OK || ps.flags.ensure_on(bytes, ctx->pool, st) != ER_OK)
            return set_error(ctx, ER_ERR_NOMEM, "pockets: channel list allocation");
        memcpy(ps.host.ptr, channels.data(), bytes);  // nothing on st uses it any more
        ER_CUDA(ctx, cudaMemcpyAsync(ps.flags.ptr, ps.host.ptr, bytes, cudaMemcpyHostToDevice, st));
        cc_mark_channels<<<(unsigned)((channels.size() + 255) / 256), 256, 0, st>>>(
            (const int*)ps.flags.ptr, (int)channels.size(), lab);
        ER_CUDA(ctx, cudaGetLastError());
    }
    return ER_OK;
}

static int ensure_pocket_scratch(er_ctx* ctx, PocketScratch& ps, cudaStream_t st, int nx, int ny,
                                 int nz, bool numbers) {
    const int64_t n = (int64_t)nx * ny * nz;
    const LinkLayout L(nx, ny, nz);
    const size_t nblk = (size_t)((n + kScanItems - 1) / kScanItems);
    const size_t host = L.list_at + (size_t)std::min(L.faces, kFirstLinks) * sizeof(uint64_t);
    cudaMemPool_t pool = ctx->pool;
    if (ps.lab.ensure_on(n * sizeof(int), pool, st) || ps.misc.ensure_on(L.bytes, pool, st) ||
        (numbers && (ps.seg.ensure_on(n * sizeof(int), pool, st) ||
                     ps.grid.ensure_on((n + 2 * nblk + 1) * sizeof(int), pool, st))))
        return set_error(ctx, ER_ERR_NOMEM, "pockets: device scratch allocation failed");
    if (ps.host.ensure(host)) return set_error(ctx, ER_ERR_NOMEM, "pockets: pinned staging failed");
    return ER_OK;
}

static int block_grid(er_ctx* ctx, int64_t n) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, ctx->num_sms * 16));
}

static int check_dims(er_ctx* ctx, int nx, int ny, int nz, double T) {
    if (nx < 2 || ny < 2 || nz < 2) return set_error(ctx, ER_ERR_INVALID, "pockets: dims >= 2");
    if ((int64_t)nx * ny * nz >= (int64_t)INT32_MAX)
        return set_error(ctx, ER_ERR_LIMIT, "pockets: grid must have < 2^31 points");
    if (!std::isfinite(T)) return set_error(ctx, ER_ERR_INVALID, "pockets: temperature");
    return ER_OK;
}

}  // namespace er

using namespace er;

extern "C" int er_block_pockets(er_ctx* ctx, double* grid, int nx, int ny, int nz,
                                double temperature, int* n_pockets, int* segments_out) {
    er::NvtxRange nvtx("er_block_pockets");
    if (!ctx || !grid || !n_pockets) return ER_ERR_INVALID;
    int stt = check_dims(ctx, nx, ny, nz, temperature);
    if (stt != ER_OK) return stt;
    ER_CUDA(ctx, cudaSetDevice(ctx->device));
    const int64_t n = (int64_t)nx * ny * nz;
    PocketScratch& ps = ctx->pocket;
    cudaStream_t st = ctx->stream;
    if ((stt = ensure_pocket_scratch(ctx, ps, st, nx, ny, nz, segments_out != nullptr)) != ER_OK)
        return stt;
    if (ps.mask.ensure_on(n * sizeof(double), ctx->pool, st) != ER_OK)
        return set_error(ctx, ER_ERR_NOMEM, "pockets: grid allocation failed");
    double* dE = (double*)ps.mask.ptr;
    ER_CUDA(ctx, cudaMemcpyAsync(dE, grid, n * sizeof(double), cudaMemcpyHostToDevice, st));
    Channels ch;
    if ((stt = label_and_classify(ctx, ps, st, dE, 15.0 * temperature, nx, ny, nz,
                                  segments_out != nullptr, ch)) != ER_OK)
        return stt;
    PocketCounters* cnt = (PocketCounters*)ps.misc.ptr;
    cc_block<false><<<block_grid(ctx, n), 256, 0, st>>>((const int*)ps.lab.ptr, n, ch, dE,
                                                        nullptr, cnt);
    ER_CUDA(ctx, cudaGetLastError());
    int np = 0;
    ER_CUDA(ctx, cudaMemcpyAsync(&np, &cnt->pockets, sizeof(int), cudaMemcpyDeviceToHost, st));
    ER_CUDA(ctx, cudaMemcpyAsync(grid, dE, n * sizeof(double), cudaMemcpyDeviceToHost, st));
    if (segments_out)
        ER_CUDA(ctx, cudaMemcpyAsync(segments_out, ps.seg.ptr, n * sizeof(int),
                                     cudaMemcpyDeviceToHost, st));
    ER_CUDA(ctx, cudaStreamSynchronize(st));
    ++np;  // counted from -1
    *n_pockets = np;
    return ER_OK;
}

namespace er {

int block_pockets_device_on(er_ctx* ctx, PocketScratch& ps, cudaStream_t st, const float* grid,
                            int nx, int ny, int nz, double temperature, uint8_t* mask_out,
                            int* n_pockets) {
    int stt = check_dims(ctx, nx, ny, nz, temperature);
    if (stt != ER_OK) return stt;
    const int64_t n = (int64_t)nx * ny * nz;
    if ((stt = ensure_pocket_scratch(ctx, ps, st, nx, ny, nz, false)) != ER_OK) return stt;
    Channels ch;
    if ((stt = label_and_classify(ctx, ps, st, grid, 15.0 * temperature, nx, ny, nz, false, ch)) !=
        ER_OK)
        return stt;
    PocketCounters* cnt = (PocketCounters*)ps.misc.ptr;
    cc_block<true><<<block_grid(ctx, n), 256, 0, st>>>((const int*)ps.lab.ptr, n, ch, nullptr,
                                                       mask_out, cnt);
    ER_CUDA(ctx, cudaGetLastError());
    int np = 0;
    ER_CUDA(ctx, cudaMemcpyAsync(&np, &cnt->pockets, sizeof(int), cudaMemcpyDeviceToHost, st));
    ER_CUDA(ctx, cudaStreamSynchronize(st));
    ++np;  // counted from -1
    *n_pockets = np;
    return ER_OK;
}

}  // namespace er

extern "C" int er_block_pockets_device(er_ctx* ctx, const float* grid, int nx, int ny, int nz,
                                       double temperature, uint8_t* pocket_mask_out,
                                       int* n_pockets) {
    er::NvtxRange nvtx("er_block_pockets_device");
    if (!ctx || !grid || !pocket_mask_out || !n_pockets) return ER_ERR_INVALID;
    ER_CUDA(ctx, cudaSetDevice(ctx->device));
    return block_pockets_device_on(ctx, ctx->pocket, ctx->stream, grid, nx, ny, nz, temperature,
                                   pocket_mask_out, n_pockets);
}

// ------------------------------------------------------------------ accessibility
// ComputeGridSheetAccessibleOrNot (src/computegridsheet.h:101-165): a point is
// inaccessible (0) when some atom image within +-1 cells has r^2 < sigma_mix^2.
// Image positions and r^2 follow the reference's FP64 expressions without
// contraction, so the mask is bit-exact.
namespace er {

struct AccParams {
    double t[9];
    double reach[3];  // 1 / (distance between opposite faces), per axis; inf for a flat cell
    int n[3];
};

__device__ __forceinline__ void acc_cart(const double* t, double xf, double yf, double zf,
                                         double& x, double& y, double& z) {
    x = __dadd_rn(__dadd_rn(__dmul_rn(t[0], xf), __dmul_rn(t[1], yf)), __dmul_rn(t[2], zf));
    y = __dadd_rn(__dadd_rn(__dmul_rn(t[3], xf), __dmul_rn(t[4], yf)), __dmul_rn(t[5], zf));
    z = __dadd_rn(__dadd_rn(__dmul_rn(t[6], xf), __dmul_rn(t[7], yf)), __dmul_rn(t[8], zf));
}

// Marks the points that an atom's images cover; blocks y share the atom's boxes.
// An image covers points whose fractional distance along axis d is at most
// sigma / width_d, so only the lattice box of that half-width (a thousandth of a
// spacing wider, far above the rounding of its FP64 bounds) is tested, with the
// reference's own expressions; the other points cannot pass the test. Every
// covered point is written by whichever images cover it, all with the same 0.
// The lanes of a warp form the boxes of the 27 images at once, and the few that
// reach the cell are then taken in turn. Testing every point against every image
// took 2.3 ms on a 65 x 63 x 64 grid of a 424-atom cell, 3e9 tests; this makes
// 2.4e6 in 17 us (a block per image, most of which miss the cell, 23 us; a loop
// over the 27 images in one block, where each miss costs its latency, 46 us).
constexpr int kAccAxis = 1024;  // axis values held on chip (longer boxes divide per point)
constexpr int kAccThreads = 128;

__device__ __forceinline__ void mark_image(const AccParams& P, const double4& at, int m,
                                           const int* l, const int* n, double* axis,
                                           uint8_t* __restrict__ out) {
    const double q[3] = {__dadd_rn(at.x, (double)(m / 9 - 1)),
                         __dadd_rn(at.y, (double)((m / 3) % 3 - 1)),
                         __dadd_rn(at.z, (double)(m % 3 - 1))};
    double ix, iy, iz;
    acc_cart(P.t, q[0], q[1], q[2], ix, iy, iz);  // src/computegridsheet.h:134-140
    const bool table = (int64_t)n[0] + n[1] + n[2] <= kAccAxis;
    if (table) {
        __syncthreads();  // the table of the image before is no longer read
        for (int e = threadIdx.x; e < n[0] + n[1] + n[2]; e += blockDim.x) {
            const int d = e < n[0] ? 0 : e < n[0] + n[1] ? 1 : 2;
            const int k = e - (d > 0 ? n[0] : 0) - (d > 1 ? n[1] : 0);
            axis[e] = __ddiv_rn((double)(l[d] + k), (double)(P.n[d] - 1));
        }
        __syncthreads();
    }
    const int64_t total = (int64_t)n[0] * n[1] * n[2];
    for (int64_t c = blockIdx.y * (int64_t)blockDim.x + threadIdx.x; c < total;
         c += (int64_t)gridDim.y * blockDim.x) {
        int i, j, k;
        if (total <= INT32_MAX) {
            const unsigned u = (unsigned)c, row = u / (unsigned)n[2];
            k = (int)(u - row * (unsigned)n[2]);
            i = (int)(row / (unsigned)n[1]);
            j = (int)(row - (unsigned)i * (unsigned)n[1]);
        } else {
            const int64_t row = c / n[2];
            k = (int)(c - row * n[2]);
            i = (int)(row / n[1]);
            j = (int)(row - (int64_t)i * n[1]);
        }
        double xf, yf, zf, x, y, z;
        if (table) {
            xf = axis[i];
            yf = axis[n[0] + j];
            zf = axis[n[0] + n[1] + k];
        } else {
            xf = __ddiv_rn((double)(l[0] + i), (double)(P.n[0] - 1));
            yf = __ddiv_rn((double)(l[1] + j), (double)(P.n[1] - 1));
            zf = __ddiv_rn((double)(l[2] + k), (double)(P.n[2] - 1));
        }
        acc_cart(P.t, xf, yf, zf, x, y, z);
        const double dx = __dsub_rn(x, ix), dy = __dsub_rn(y, iy), dz = __dsub_rn(z, iz);
        const double r2 =
            __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
        if (r2 < at.w)  // src/computegridsheet.h:148
            out[(size_t)(l[2] + k) + (size_t)(l[1] + j) * P.n[2] +
                (size_t)(l[0] + i) * P.n[1] * P.n[2]] = 0;
    }
}

__global__ void __launch_bounds__(kAccThreads)
    acc_mark_kernel(const double4* __restrict__ atoms, const __grid_constant__ AccParams P,
                    uint8_t* __restrict__ out) {
    __shared__ double axis[kAccAxis];
    const double4 at = atoms[blockIdx.x];
    const double s = sqrt(at.w);
    if (!(s > 0.0)) return;  // r^2 < 0 holds nowhere
    const int lane = threadIdx.x & 31;
    int lo[3] = {0, 0, 0}, len[3] = {0, 0, 0};  // of image `lane`
    bool any = lane < 27;
    if (any) {
        const double q[3] = {__dadd_rn(at.x, (double)(lane / 9 - 1)),
                             __dadd_rn(at.y, (double)((lane / 3) % 3 - 1)),
                             __dadd_rn(at.z, (double)(lane % 3 - 1))};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double nm1 = (double)(P.n[d] - 1), w = s * P.reach[d];
            const double a = fmax(ceil((q[d] - w) * nm1 - 1e-3), 0.0);
            const double b = fmin(floor((q[d] + w) * nm1 + 1e-3), nm1);
            any = any && a <= b;
            lo[d] = any ? (int)a : 0;
            len[d] = any ? (int)b - (int)a + 1 : 0;
        }
    }
    // the same in every warp of the block
    for (unsigned left = __ballot_sync(0xffffffffu, any); left; left &= left - 1) {
        const int m = __ffs(left) - 1;
        int l[3], n[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            l[d] = __shfl_sync(0xffffffffu, lo[d], m);
            n[d] = __shfl_sync(0xffffffffu, len[d], m);
        }
        mark_image(P, at, m, l, n, axis, out);
    }
}

// The same from the points' side, for spheres that overlap many times over (below):
// every point tests the images until one covers it.
__global__ void acc_images_kernel(const double4* __restrict__ atoms, int n,
                                  const __grid_constant__ AccParams P, double4* __restrict__ img) {
    const int total = 27 * n;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < total; q += gridDim.x * blockDim.x) {
        const int a = q / 27, m = q % 27;
        const double4 at = atoms[a];
        double x, y, z;
        // src/computegridsheet.h:134-140
        acc_cart(P.t, __dadd_rn(at.x, (double)(m / 9 - 1)),
                 __dadd_rn(at.y, (double)((m / 3) % 3 - 1)), __dadd_rn(at.z, (double)(m % 3 - 1)),
                 x, y, z);
        img[q] = make_double4(x, y, z, at.w);
    }
}

__global__ void __launch_bounds__(256)
    acc_points_kernel(const double4* __restrict__ img, int nimg,
                      const __grid_constant__ AccParams P, uint8_t* __restrict__ out) {
    __shared__ double4 tile[512];
    const int64_t n = (int64_t)P.n[0] * P.n[1] * P.n[2];
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    double x = 0, y = 0, z = 0;
    bool open = p < n;
    if (open) {
        const int k = (int)(p % P.n[2]), j = (int)((p / P.n[2]) % P.n[1]),
                  i = (int)(p / ((int64_t)P.n[1] * P.n[2]));
        acc_cart(P.t, __ddiv_rn((double)i, (double)(P.n[0] - 1)),
                 __ddiv_rn((double)j, (double)(P.n[1] - 1)),
                 __ddiv_rn((double)k, (double)(P.n[2] - 1)), x, y, z);
    }
    for (int base = 0; base < nimg; base += 512) {
        const int cnt = min(512, nimg - base);
        if (!__syncthreads_or(open)) break;  // (also: the tile before is no longer read)
        for (int q = threadIdx.x; q < cnt; q += blockDim.x) tile[q] = img[base + q];
        __syncthreads();
        for (int q = 0; open && q < cnt; ++q) {
            const double4 w = tile[q];
            const double dx = __dsub_rn(x, w.x), dy = __dsub_rn(y, w.y), dz = __dsub_rn(z, w.z);
            const double r2 =
                __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
            open = !(r2 < w.w);  // src/computegridsheet.h:148
        }
    }
    if (p < n) out[p] = open ? 1 : 0;
}

// Marking takes c tests a point, c = the boxes that lie over it (27 images: at most
// 3 along an axis); a point takes some multiple of 27 n / c images until one covers
// it. So c^2 / n decides, at 18 (grids of few points, whose blocks are too few to
// hide a point's chain of tests, 48; fewer than 16 atoms, whose chains are short and
// whose boxes are few for the GPU, 8). Measured boxes / points, us a call: 424 atoms
// in 25.8 A, sigma 3.5 A (c^2 / n = 0.17), 65^3 71 / 1793; 259 in 12 A, 3.7 A (14),
// 33^3 50 / 112, 65^3 130 / 197, 129^3 697 / 777; 150 in 10 A, 3.7 A (25) 51 / 76, 128
// / 118, 709 / 480; 76 in 8 A, 3.7 A (48) 55 / 56, 133 / 85, 689 / 333; 76 in 8 A, 7 A
// (2183) 131 / 34, 529 / 61, 3547 / 214; 4 in 6 A, 3 A (4) 43 / 43, 65 / 72, 261 / 275,
// 3.7 A (14) 48 / 37, 84 / 60, 331 / 224.
static bool acc_from_points(const FwRecord& f, const double* reach, int64_t points) {
    double c = f.n_atoms;
    for (int d = 0; d < 3; ++d) c *= std::min(2.0 * f.sig_mean * reach[d], 3.0);
    const double line = f.n_atoms < 16 ? 8.0 : points < 100000 ? 48.0 : 18.0;
    return c * c > line * f.n_atoms && f.n_atoms <= INT32_MAX / 27;
}

}  // namespace er

extern "C" int er_accessibility(er_ctx* ctx, int fw_id, int nx, int ny, int nz, uint8_t* out) {
    if (!ctx || !out) return ER_ERR_INVALID;
    if (int st = er::check_grid_dims(ctx, nx, ny, nz, "accessibility")) return st;
    ER_CUDA(ctx, cudaSetDevice(ctx->device));
    const er::FwRecord* f = er::find_fw(ctx, fw_id);
    if (!f) return er::set_error(ctx, ER_ERR_NOT_FOUND, "accessibility: unknown framework id");
    const int64_t n = (int64_t)nx * ny * nz;
    cudaStream_t st = ctx->stream;
    if (ctx->pocket.seg.ensure_on((size_t)n, ctx->pool, st))
        return er::set_error(ctx, ER_ERR_NOMEM, "accessibility: scratch allocation failed");
    uint8_t* mask = (uint8_t*)ctx->pocket.seg.ptr;
    er::AccParams P;
    for (int k = 0; k < 9; ++k) P.t[k] = f->t[k];
    double w[3];
    er::perpendicular_widths(f->t, w);
    for (int d = 0; d < 3; ++d) P.reach[d] = w[d] > 0.0 ? 1.0 / w[d] : INFINITY;
    P.n[0] = nx; P.n[1] = ny; P.n[2] = nz;
    if (er::acc_from_points(*f, P.reach, n)) {
        const int nimg = 27 * f->n_atoms;
        if (ctx->pocket.lab.ensure_on((size_t)nimg * sizeof(double4), ctx->pool, st))
            return er::set_error(ctx, ER_ERR_NOMEM, "accessibility: scratch allocation failed");
        double4* img = (double4*)ctx->pocket.lab.ptr;
        er::acc_images_kernel<<<std::max(1, std::min((nimg + 255) / 256, ctx->num_sms * 8)), 256, 0,
                                st>>>(f->dev.atom_frac, f->n_atoms, P, img);
        er::acc_points_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(img, nimg, P, mask);
        ER_CUDA(ctx, cudaGetLastError());
    } else {
        ER_CUDA(ctx, cudaMemsetAsync(mask, 1, (size_t)n, st));
        if (f->n_atoms > 0) {
            // sixteen blocks per SM: few atoms share their boxes among more blocks
            const unsigned parts =
                (unsigned)std::max(1, std::min(64, 16 * ctx->num_sms / f->n_atoms));
            er::acc_mark_kernel<<<dim3((unsigned)f->n_atoms, parts), er::kAccThreads, 0, st>>>(
                f->dev.atom_frac, P, mask);
            ER_CUDA(ctx, cudaGetLastError());
        }
    }
    ER_CUDA(ctx, cudaMemcpyAsync(out, ctx->pocket.seg.ptr, (size_t)n, cudaMemcpyDeviceToHost, st));
    ER_CUDA(ctx, cudaStreamSynchronize(st));
    return ER_OK;
}
