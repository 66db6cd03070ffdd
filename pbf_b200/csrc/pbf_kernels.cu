// PBF substep kernels for sm_100a.
//
// Data layout in HBM (all particle arrays in cell-sorted slot order, float4 with
// xyz in .x/.y/.z so that a neighbour gather is one 16-byte load):
//   x, v, x_old        float4[n]
//   xl                 float4[n]  positions with lambda in .w (output of the lambda pass)
//   perm               int[n]     slot -> original particle id
//   cell, ticket, tmp  int[n]     hash key, arrival ticket, unsorted cell fill
//   cell_start         int[ncells + 2]: start of each cell, then the out-of-grid bin, then n
//   nbr                int[max_nbr][stride]  slot-major neighbour list (coalesced per slot)
//   ncnt               int[n]
//
// Reference kernels replaced (kernels/cudaPBFSolver.cu): updateParticles :4-13,
// calculateParticlesGid :31-40, calculatePrefixSum :42-89, addBlockSum :91-96,
// setGrid :99-111, countingSort :112-122, buildNeighborhood :124-154; the
// neighbour-sum passes (lambda, dp, curl, vorticity) are in pbf_pairs.cu.
#include <algorithm>

#include "pbf_kernels.h"
#include "pbf_launch.cuh"
#include "pbf_packed.cuh"

namespace pbf {

// ---------------------------------------------------------------------------
// a1 + a2: predict, bound, hash, histogram (one arrival ticket per particle)
// ---------------------------------------------------------------------------
template <bool PREDICT, int U>
__global__ void __launch_bounds__(256, 8) k_hash(KParams p, const float4* __restrict__ x, const float4* __restrict__ v,
                                              int* __restrict__ cell, int* __restrict__ ticket, int* __restrict__ cnt,
                                              int* __restrict__ err) {
    // Each warp takes U rounds of 32 consecutive slots; the loads, and then the
    // histogram atomics, of all rounds are in flight together.
    const int lane = threadIdx.x & 31;
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int key[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const long long i = (w * U + u) * 32 + lane;
        key[u] = -1;
        if (i < p.n) {
            const SceneView sc = scene_of(p, (int)i);
            f3 xi = make3(x[i]);
            if (PREDICT) {
                f3 vi = make3(v[i]);
                predict(p, sc, xi, vi);
            }
            if (!(isfinite(xi.x) && isfinite(xi.y) && isfinite(xi.z))) atomicOr(err, DEVERR_NONFINITE);
            key[u] = cell_key(p, sc, xi);
        }
    }
    // Run-aggregated histogram: slots are in cell order from the previous substep,
    // so equal keys come in runs; one atomic per run of equal keys in the warp.
    // (The ticket is only an arrival order; k_reorder makes the order stable.)
    int base[U], leader[U], rank[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int prev = __shfl_up_sync(0xffffffffu, key[u], 1);
        const unsigned starts = __ballot_sync(0xffffffffu, lane == 0 || prev != key[u]);
        const unsigned upto = starts & (0xffffffffu >> (31 - lane));  // run starts at or below this lane
        leader[u] = 31 - __clz(upto);
        const unsigned above = starts & ~(0xffffffffu >> (31 - lane));
        const int end = above ? __ffs(above) - 1 : 32;  // first run start above this lane
        rank[u] = lane - leader[u];
        base[u] = 0;
        if (key[u] >= 0 && lane == leader[u]) base[u] = atomicAdd(&cnt[key[u]], end - leader[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int b = __shfl_sync(0xffffffffu, base[u], leader[u]);
        const long long i = (w * U + u) * 32 + lane;
        if (i < p.n) {
            cell[i] = key[u];
            ticket[i] = b + rank[u];
        }
    }
}

// ---------------------------------------------------------------------------
// a3 + a4: exclusive scan of the cell counts with decoupled look-back; writes
// cell_start[0..m) and cell_start[m] = total, and clears the counts for the next
// substep. Status words: (epoch << 34) | (flag << 32) | value, flag 1 = tile
// aggregate, 2 = inclusive prefix. Tiles are numbered in launch order by an atomic
// ticket, so every predecessor is already running and the wait always ends; the
// wait is bounded anyway and reports DEVERR_SCAN_TIMEOUT.
//
// The workspace is the status words, then the ticket counter. With KEEP (the
// solver's own workspace, zeroed once, its scans all of one size) tickets go on from
// run to run and the epoch is a ticket's run, which invalidates the words of the run
// before, so a substep needs no memset; other callers' workspaces are cleared before
// the launch.
// KEEP also writes the cleared counts only where there were any: most cells of a
// large grid are empty, and the pass is bound by its bytes (65.6 M keys, 4.7 M
// particles: 194 us -> 144 us with 524 MB instead of 786).
// ---------------------------------------------------------------------------
constexpr long long SCAN_SPIN_LIMIT = 1ll << 22;
// What the pass waits for is the chain of prefixes, so a tile publishes its aggregate
// before it scans its items, one atomic gives tile and epoch, and the words are
// relaxed accesses (5 M counts: 13.2 us -> 9.9; 65.6 M keys: 148 -> 131; 25,000: 4.4
// -> 3.3). More words per poll cost more than the hops they save (65.6 M keys, two and
// four per lane: 138 and 162 us), a window of the whole block more again (302).
// Tiles of 8,192 counts, or of 16,384 above 2^22 counts, where half as many tiles
// make a shorter chain (65.6 M keys, mostly empty: 131 us against 165 with 8,192 and
// 191 with 4,096; 5 M counts: 9.9 against 13.2 and 13.5). The solver's own scan takes
// 4,096 up to 2^19 counts, where 8,192 leave most SMs idle (1.02 M keys: 5.8 us with
// 8,192, 7.3 with 4,096).
constexpr int SCAN_THREADS = 256;
constexpr int SCAN_SMALL_MAX = 1 << 19;
constexpr int SCAN_LARGE_MIN = (1 << 22) + 1;
static int scan_tile(int m) { return m >= SCAN_LARGE_MIN ? 16384 : 8192; }
constexpr unsigned SCAN_EPOCHS = 1u << 30;

// Status words carry their value with them and order nothing else: relaxed accesses.
__device__ __forceinline__ void st_status(unsigned long long* a, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(a), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_status(const unsigned long long* a) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(a) : "memory");
    return v;
}

// Sum of all tiles before `tile`, by one whole warp: windows of 32 predecessors, the
// nearest on lane 0. A window is polled until the words up to its nearest inclusive
// prefix (or all of them) are there. False, with the sum so far, when spin_limit
// polls of a window did not suffice.
__device__ __forceinline__ bool look_back(const unsigned long long* status, int tile, unsigned long long ep,
                                          long long spin_limit, int& excl) {
    const int lane = threadIdx.x & 31;
    excl = 0;
    for (int pos = tile - 1; pos >= 0; pos -= 32) {
        for (long long spins = 0;; ++spins) {
            const unsigned long long w =
                pos >= lane ? ld_status(&status[pos - lane]) : ep | (2ull << 32);  // before tile 0: an empty prefix
            const unsigned flag = (w & ~0x3ffffffffull) == ep ? (unsigned)(w >> 32) & 3u : 0u;
            const unsigned there = __ballot_sync(0xffffffffu, flag != 0u), prefix = __ballot_sync(0xffffffffu, flag == 2u);
            const int last = prefix ? __ffs(prefix) - 1 : 31;  // lanes up to here count
            const bool wait = (~there & (0xffffffffu >> (31 - last))) != 0u;
            if (wait && spins < spin_limit) {
                __nanosleep(32);
                continue;
            }
            excl += __reduce_add_sync(0xffffffffu, flag != 0u && lane <= last ? (int)(unsigned)w : 0);
            if (wait) return false;
            if (prefix) return true;
            break;
        }
    }
    return true;
}

// VEC: cnt and out are 16-byte aligned; each lane moves four consecutive counts
// per access (int4), rounds of 128 per warp instead of 32.
// silent_tile >= 0 (the failure-injection test only): that tile publishes no
// status, so its successors' look-back waits run out after spin_limit polls.
template <bool VEC, bool KEEP, int ITEMS>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan(int* __restrict__ cnt, int* __restrict__ out, int m,
                                                       unsigned long long* __restrict__ status, int tiles,
                                                       int* __restrict__ err, int* host_err, int silent_tile,
                                                       long long spin_limit, int* __restrict__ zero, int nzero) {
    static_assert(VEC || !KEEP, "the solver's arrays are aligned");
    constexpr int TILE = SCAN_THREADS * ITEMS, WARPS = SCAN_THREADS / 32;
    __shared__ int s_tile;
    __shared__ unsigned s_epoch;
    __shared__ int s_warp[WARPS];
    __shared__ int s_excl;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0) {
        const unsigned long long ticket = atomicAdd(status + tiles, 1ull);
        // (without KEEP the counter starts from zero)
        const unsigned long long e = !KEEP ? 0ull : ticket >> 32 ? ticket / (unsigned)tiles : (unsigned)ticket / (unsigned)tiles;
        const int tile = (int)(ticket - e * (unsigned)tiles);
        s_tile = tile;
        s_epoch = (unsigned)(e % SCAN_EPOCHS);
    }
    __syncthreads();
    const int tile = s_tile;
    if (KEEP && tile == 0)  // words of the caller to be cleared along the way
        for (int i = t; i < nzero; i += SCAN_THREADS) zero[i] = 0;
    const unsigned long long ep = (unsigned long long)s_epoch << 34;

    // Warp w owns elements [tile * TILE + w * 32 ITEMS, + 32 ITEMS) in rounds of consecutive
    // elements (coalesced: 32 counts per round, or 128 as int4 when VEC); each
    // round is scanned across the warp and carried into the next.
    const long long wbase = (long long)tile * TILE + (long long)warp * (32 * ITEMS);
    int item[ITEMS];
    int sum = 0;
    unsigned filled = 0u;  // rounds (int4 groups) of this lane that hold a count
    if (VEC) {
#pragma unroll
        for (int r = 0; r < ITEMS / 4; ++r) {
            const long long i0 = wbase + r * 128 + lane * 4;
            if (i0 + 3 < m) {
                const int4 q = *reinterpret_cast<const int4*>(cnt + i0);
                item[4 * r] = q.x; item[4 * r + 1] = q.y; item[4 * r + 2] = q.z; item[4 * r + 3] = q.w;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) item[4 * r + e] = i0 + e < m ? cnt[i0 + e] : 0;
            }
        }
#pragma unroll
        for (int r = 0; r < ITEMS / 4; ++r) {
            const int tot = item[4 * r] + item[4 * r + 1] + item[4 * r + 2] + item[4 * r + 3];
            if (KEEP) filled |= tot != 0 ? 1u << r : 0u;
            sum += tot;
        }
    } else {
#pragma unroll
        for (int q = 0; q < ITEMS; ++q) {
            const long long idx = wbase + q * 32 + lane;
            item[q] = idx < m ? cnt[idx] : 0;
            sum += item[q];
        }
    }
    // the tile's aggregate first, for the tiles that wait for it
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) s_warp[warp] = sum;  // the warp's total
    __syncthreads();
    // every thread: the sum of the warps before its own, and of all
    int before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
        const int v = s_warp[w];
        before += w < warp ? v : 0;
        total += v;
    }
    const bool publish = tile != silent_tile;
    if (t == 0 && publish) st_status(&status[tile], ep | ((tile == 0 ? 2ull : 1ull) << 32) | (unsigned)total);
    // exclusive prefixes within the warp's range, round by round
    int carry = 0;
    if (VEC) {
#pragma unroll
        for (int r = 0; r < ITEMS / 4; ++r) {
            const int a0 = item[4 * r], a1 = a0 + item[4 * r + 1], a2 = a1 + item[4 * r + 2];
            const int tot = a2 + item[4 * r + 3];
            int incl = tot;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const int ex = carry + incl - tot;
            carry += __shfl_sync(0xffffffffu, incl, 31);
            item[4 * r] = ex;
            item[4 * r + 1] = ex + a0;
            item[4 * r + 2] = ex + a1;
            item[4 * r + 3] = ex + a2;
        }
    } else {
#pragma unroll
        for (int q = 0; q < ITEMS; ++q) {
            int incl = item[q];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const int excl_q = carry + incl - item[q];
            carry += __shfl_sync(0xffffffffu, incl, 31);
            item[q] = excl_q;
        }
    }
    if (warp == 0) {
        int e;
        const bool ok = look_back(status, tile, ep, spin_limit, e);
        if (lane == 0) {
            s_excl = e;
            if (!ok) {
                atomicOr(err, DEVERR_SCAN_TIMEOUT);
                if (host_err) *(volatile int*)host_err = DEVERR_SCAN_TIMEOUT;
            }
        }
    }
    __syncthreads();
    const int excl = s_excl;
    if (t == 0 && publish && tile > 0)
        st_status(&status[tile], ep | (2ull << 32) | (unsigned)(excl + total));
    const int off = excl + before;
    if (VEC) {
#pragma unroll
        for (int r = 0; r < ITEMS / 4; ++r) {
            const long long i0 = wbase + r * 128 + lane * 4;
            if (i0 + 3 < m) {
                *reinterpret_cast<int4*>(out + i0) =
                    make_int4(off + item[4 * r], off + item[4 * r + 1], off + item[4 * r + 2], off + item[4 * r + 3]);
                // (most cells of a large grid are empty: those need no write)
                if (KEEP && (filled >> r & 1u)) *reinterpret_cast<int4*>(cnt + i0) = make_int4(0, 0, 0, 0);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (i0 + e < m) {
                        out[i0 + e] = off + item[4 * r + e];
                        if (KEEP) cnt[i0 + e] = 0;
                    }
            }
        }
    } else {
#pragma unroll
        for (int q = 0; q < ITEMS; ++q) {
            const long long idx = wbase + q * 32 + lane;
            if (idx < m) out[idx] = off + item[q];
        }
    }
    if (tile == tiles - 1 && t == 0) out[m] = excl + total;  // the grand total
}

// ---------------------------------------------------------------------------
// a5: scatter by ticket (unordered within a cell), then a stable rank within the
// cell and the reorder of the particle state into slot order (a6).
// ---------------------------------------------------------------------------
// Each thread takes U slots 256 apart within its block's tile of 256 U (the
// loads of all U in flight together).
template <int U>
__global__ void __launch_bounds__(256) k_scatter(int n, const int* __restrict__ cell, const int* __restrict__ ticket,
                                                 const int* __restrict__ cell_start, int* __restrict__ tmp,
                                                 int* __restrict__ err) {
    pdl_wait();
    const long long i0 = (long long)blockIdx.x * blockDim.x * U + threadIdx.x;
    int c[U], t[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const long long i = i0 + (long long)u * blockDim.x;
        c[u] = i < n ? cell[i] : 0;
        t[u] = i < n ? ticket[i] : 0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const long long i = i0 + (long long)u * blockDim.x;
        if (i >= n) break;
        const int dst = cell_start[c[u]] + t[u];
        if (dst < 0 || dst >= n) {  // counts and tickets disagree: report, never write out of bounds
            atomicOr(err, DEVERR_BAD_INDEX);
            continue;
        }
        tmp[dst] = (int)i;
    }
}

template <bool PREDICT>
__global__ void __launch_bounds__(256, 8) k_reorder(KParams p, const float4* __restrict__ x, const float4* __restrict__ v,
                                                 const int* __restrict__ perm, const int* __restrict__ cell,
                                                 const int* __restrict__ cell_start, const int* __restrict__ tmp,
                                                 float4* __restrict__ xp, float4* __restrict__ vp,
                                                 float4* __restrict__ xold, int* __restrict__ perm_out,
                                                 int* __restrict__ cell_sorted, const float* __restrict__ lam_in,
                                                 float* __restrict__ lam_out, int* __restrict__ err) {
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const int c = cell[i];
    const int s = cell_start[c], e = min(cell_start[c + 1], p.n);
    if (s < 0 || s >= e) {
        atomicOr(err, DEVERR_BAD_INDEX);
        return;
    }
    const SceneView sc = scene_of(p, i);
    const bool desc = p.cell_order == 1 && c != sc.cell_base + sc.ncells;  // out-of-grid bin stays ascending
    int q = 0;
    for (int k = s; k < e; ++k) {
        const int o = tmp[k];
        q += desc ? (o > i) : (o < i);
    }
    const int dst = s + q;  // < e <= n
    const float4 x4 = x[i];
    f3 xi = make3(x4);
    f3 vi = make3(v[i]);
    if (PREDICT) predict(p, sc, xi, vi);
    xp[dst] = make_float4(xi.x, xi.y, xi.z, 0.0f);
    if (vp) vp[dst] = make_float4(vi.x, vi.y, vi.z, 0.0f);
    xold[dst] = make_float4(x4.x, x4.y, x4.z, 0.0f);
    perm_out[dst] = perm[i];
    cell_sorted[dst] = c;
    if (lam_out) lam_out[dst] = lam_in[i];
}

// ---------------------------------------------------------------------------
// a7: 27-cell neighbour search (a (2R+1)^3 stencil when cells are smaller than
// h). The stencil is visited dz-major, dy, then the dx cells of a row, which are
// one contiguous slot range because keys are x-fastest; within a cell, slot
// order. For R = 1 this is the reference order (buildNeiborhood cu:133-136)
// applied to the sorted slots. Rows and row ends that lie farther than h from the
// particle are skipped: a row (dy, dz) is visited only where the distance from the
// particle to its y and z slabs leaves room within h, and only over the x cells
// within the remaining half-width. The clipping is conservative (clip_margin), so every
// candidate it drops fails the r^2 <= h^2 test and the lists do not change. Cell 0
// of an axis reaches one cell below the grid, because cell_dims truncates.
// ---------------------------------------------------------------------------
// Above the rounding of the keys and of the cell edges they are compared with: 4 x 2^-24
// of the distance from the grid's corner, whose coordinates are in KParams::clip.
__device__ __forceinline__ float clip_margin(const KParams& p, const f3& x) {
    return p.clip + 1e-6f * (fabsf(x.x) + fabsf(x.y) + fabsf(x.z));
}

// Where cell t (or a slab of cells) starts along an axis with origin g.
__device__ __forceinline__ float cell_from(const KParams& p, float g, int t) {
    return g + (float)(t == 0 ? -1 : t) * p.cell;
}

// Stencil radius RR as a constant (1: cells of h, 2: cells of h/2; 0: any radius,
// read from p.radius). Places in a list are 32-bit offsets from its first entry, in
// units of 32 ints (the stride between entries is a multiple of that).
//
// For RR > 0 the pass is bound by instructions (a lane of a warp of 32 walks its
// own rows, about 20 of 32 lanes are active), so they are what is saved: the
// distances to the cells beside the particle's own are squared once per particle
// and a row's range is a few compares; candidates go two or four per step, a step
// without branches (predicated stores); the particle itself is left out by splitting
// its own row's range, and the cap is tested per row. 262,144 particles, cells of
// h/2: 67.8 us -> 52.6 (57.1 with the entries counted and multiplied by the stride,
// 53.6 with byte offsets); cells of h: 79 -> 64.
//
// Candidates per step: rows hold 3-4 in cells of h/2, where four per step only add
// instructions (64 scenes, 1.3 M particles: 225 us with two, 240 with four), and 10 or more
// in cells of h (262,144 particles: 76 us with two, 64 with four, 67 with six).
template <int RR>
__device__ __forceinline__ void neighbors_one(const KParams& p, int k, const float4* __restrict__ x,
                                              const int* __restrict__ cell_start, int* __restrict__ nbr,
                                              int* __restrict__ ncnt) {
    if (k >= p.n) return;
    const SceneView sc = scene_of(p, k);
    const f3 xk = make3(x[k]);
    int d[3];
    cell_dims(p, sc, xk, d);
    const int nx = sc.dims[0], ny = sc.dims[1], nz = sc.dims[2];
    const int cap = p.max_nbr;
    const float m = clip_margin(p, xk);
    const float hm2 = (p.h + m) * (p.h + m);
    // entry i of the list is i step units after entry 0
    const unsigned step = (unsigned)p.stride / 32, last = (unsigned)cap * step;
    unsigned o = 0;  // of the next entry
    int* __restrict__ list = nbr + k;
    auto at = [&](unsigned i) { return list + (size_t)i * 32; };
    const float h2 = p.h2;
    // candidates [s, e) in slot order, two or four at a time: |r|^2 as dot_fma gives
    // it, packed. The last step of a range may read slots after it (the position
    // array has SEARCH_SLACK slots more than there are particles) and drops them.
    auto r2_pair = [&](const float4& a0, const float4& a1) {
        const float2 rx = make_float2(xk.x - a0.x, xk.x - a1.x), ry = make_float2(xk.y - a0.y, xk.y - a1.y),
                     rz = make_float2(xk.z - a0.z, xk.z - a1.z);
        return vfma(rz, rz, vfma(ry, ry, vmul(rx, rx)));
    };
    auto scan = [&](int s, int e) {
        const float4* q = x + s;
        if constexpr (RR == 1) {
            for (int j = s; j < e; j += 4, q += 4) {
                const float4 a0 = q[0], a1 = q[1], a2 = q[2], a3 = q[3];
                const float2 d01 = r2_pair(a0, a1), d23 = r2_pair(a2, a3);
                const int left = e - j;
                if (d01.x <= h2) {
                    *at(o) = j;
                    o += step;
                }
                if (d01.y <= h2 && left > 1) {
                    *at(o) = j + 1;
                    o += step;
                }
                if (d23.x <= h2 && left > 2) {
                    *at(o) = j + 2;
                    o += step;
                }
                if (d23.y <= h2 && left > 3) {
                    *at(o) = j + 3;
                    o += step;
                }
            }
        } else {
            for (int j = s; j < e; j += 2, q += 2) {
                const float4 a0 = q[0], a1 = q[1];
                const float2 d01 = r2_pair(a0, a1);
                if (d01.x <= h2) {
                    *at(o) = j;
                    o += step;
                }
                if (d01.y <= h2 && j + 1 < e) {
                    *at(o) = j + 1;
                    o += step;
                }
            }
        }
    };
    // the same near the cap. In cells of h a row may hold more candidates than the cap, and
    // all of them come here: four at a time there too (60,000 particles with about 1,000
    // candidates each: 107 us one at a time, 62; in cells of h/2 the registers it takes
    // cost every scene more, 1 M particles 167 us against 176).
    auto scan_capped = [&](int s, int e) {
        if constexpr (RR == 1) {
            for (int j = s; j < e && o < last; j += 4) {
                const float4 a0 = x[j], a1 = x[j + 1], a2 = x[j + 2], a3 = x[j + 3];
                const float2 d01 = r2_pair(a0, a1), d23 = r2_pair(a2, a3);
                const int left = e - j;
                if (d01.x <= h2) {
                    *at(o) = j;
                    o += step;
                }
                if (d01.y <= h2 && left > 1 && o < last) {
                    *at(o) = j + 1;
                    o += step;
                }
                if (d23.x <= h2 && left > 2 && o < last) {
                    *at(o) = j + 2;
                    o += step;
                }
                if (d23.y <= h2 && left > 3 && o < last) {
                    *at(o) = j + 3;
                    o += step;
                }
            }
        } else {
            for (int j = s; j < e && o < last; ++j) {
                const float4 a0 = x[j];
                const f3 r = {xk.x - a0.x, xk.y - a0.y, xk.z - a0.z};
                if (dot_fma(r, r) <= h2) {
                    *at(o) = j;
                    o += step;
                }
            }
        }
    };
    auto scan_row = [&](int s, int e) {
        if (o + (unsigned)min(e - s, cap + 1) * step <= last) scan(s, e);
        else scan_capped(s, e);
    };
    if (RR > 0) {
        // squared distance, less the margin, from q to the cell (slab of cells) i
        // below or above its own cell `cell`
        auto below = [&](float q, float g, int cell, int i) {
            const float e = fmaxf(q - (g + (float)(cell - i + 1) * p.cell) - m, 0.0f);
            return e * e;
        };
        auto above = [&](float q, float g, int cell, int i) {
            const float e = fmaxf(cell_from(p, g, cell + i) - q - m, 0.0f);
            return e * e;
        };
        constexpr int W = RR > 0 ? 2 * RR + 1 : 1, R1 = RR > 0 ? RR : 1;
        // +inf for rows and cells outside the grid
        float ey2[W], xl2[R1], xr2[R1];
        ey2[RR] = d[1] >= 0 && d[1] < ny ? 0.0f : INFINITY;
#pragma unroll
        for (int u = 1; u <= RR; ++u) {
            const int yl = d[1] - u, yh = d[1] + u;
            ey2[RR - u] = yl >= 0 && yl < ny ? below(xk.y, sc.gmin[1], d[1], u) : INFINITY;
            ey2[RR + u] = yh >= 0 && yh < ny ? above(xk.y, sc.gmin[1], d[1], u) : INFINITY;
            xl2[u - 1] = d[0] - u >= 0 ? below(xk.x, sc.gmin[0], d[0], u) : INFINITY;
            xr2[u - 1] = d[0] + u < nx ? above(xk.x, sc.gmin[0], d[0], u) : INFINITY;
        }
        // (a particle outside the grid along x takes all the cells of a row that its
        // stencil reaches)
        const bool in_x = d[0] >= 0 && d[0] < nx;
        const int x0 = max(d[0] - RR, 0), x1 = min(d[0] + RR, nx - 1);
        for (int dz = -RR; dz <= RR && o < last && x0 <= x1; ++dz) {
            const int z = d[2] + dz;
            if (z < 0 || z >= nz) continue;
            const float ez2 = dz == 0 ? 0.0f : dz < 0 ? below(xk.z, sc.gmin[2], d[2], -dz) : above(xk.z, sc.gmin[2], d[2], dz);
            const float hz = hm2 - ez2;
            if (!(hz >= 0.0f)) continue;
            const int* plane = cell_start + (sc.cell_base + (d[1] + z * ny) * nx + d[0]);
            int s[W], e[W];
#pragma unroll
            for (int i = 0; i < W; ++i) {
                const float rem = hz - ey2[i];
                s[i] = e[i] = 0;
                if (rem >= 0.0f) {
                    const int* row = plane + (i - RR) * nx;
                    int a = 0, b = 1;
                    if (in_x) {
#pragma unroll
                        for (int u = 0; u < RR; ++u) {
                            a -= xl2[u] <= rem ? 1 : 0;
                            b += xr2[u] <= rem ? 1 : 0;
                        }
                    } else {
                        a = x0 - d[0];
                        b = x1 + 1 - d[0];
                    }
                    s[i] = row[a];
                    e[i] = row[b];
                }
            }
#pragma unroll
            for (int i = 0; i < W; ++i) {
                if (i == RR && dz == 0 && k >= s[i] && k < e[i]) {
                    scan_row(s[i], k);
                    scan_row(k + 1, e[i]);
                } else {
                    scan_row(s[i], e[i]);
                }
            }
        }
    } else {
        const int R = p.radius;
        const int x0 = max(d[0] - R, 0), x1 = min(d[0] + R, nx - 1);
        for (int dz = -R; dz <= R && o < last && x0 <= x1; ++dz) {
            const int z = d[2] + dz;
            if (z < 0 || z >= nz) continue;
            // distance from the particle to the z slab of this plane of cells
            const float gz = dz > 0 ? cell_from(p, sc.gmin[2], z) - xk.z
                                    : xk.z - (sc.gmin[2] + (float)(z + 1) * p.cell);
            const float ez = dz == 0 ? 0.0f : fmaxf(gz - m, 0.0f);
            if (ez * ez > hm2) continue;
            for (int dy = -R; dy <= R && o < last; ++dy) {
                const int y = d[1] + dy;
                if (y < 0 || y >= ny) continue;
                const float gy = dy > 0 ? cell_from(p, sc.gmin[1], y) - xk.y
                                        : xk.y - (sc.gmin[1] + (float)(y + 1) * p.cell);
                const float ey = dy == 0 ? 0.0f : fmaxf(gy - m, 0.0f);
                const float rem = hm2 - ez * ez - ey * ey;
                if (!(rem >= 0.0f)) continue;
                // the half-width only bounds the candidates (the margin m of at least
                // 1e-3 h is far above the approximate root's relative error of 2^-22)
                float w;
                asm("sqrt.approx.f32 %0, %1;" : "=f"(w) : "f"(rem));
                w += m;
                const int xa = max(x0, (int)floorf((xk.x - w - sc.gmin[0]) * p.inv_cell));
                const int xb = min(x1, (int)((xk.x + w - sc.gmin[0]) * p.inv_cell));
                if (xa > xb) continue;
                const int row = sc.cell_base + y * nx + z * nx * ny;
                const int s = cell_start[row + xa], e = cell_start[row + xb + 1];
                if (k >= s && k < e) {
                    scan_row(s, k);
                    scan_row(k + 1, e);
                } else {
                    scan_row(s, e);
                }
            }
        }
    }
    int c = (int)(o / step);
    ncnt[k] = c;
    for (; (c & (p.pad - 1)) != 0; ++c, o += step) *at(o) = p.pad_slot;
}

// nvb tiles of blockDim.x slots; the grid strides over them (a grid of nvb
// blocks is the ordinary one-block-per-tile launch)
template <int RR>
__global__ void __launch_bounds__(256) k_neighbors(KParams p, int nvb, const float4* __restrict__ x,
                                                   const int* __restrict__ cell_start, int* __restrict__ nbr,
                                                   int* __restrict__ ncnt) {
    pdl_wait();
    for (int vb = blockIdx.x; vb < nvb; vb += gridDim.x)
        neighbors_one<RR>(p, vb * blockDim.x + threadIdx.x, x, cell_start, nbr, ncnt);
}

// The same search for small scenes, where one thread's walk over its 9 or 25 rows
// is what the pass takes (21 us for 4,080 particles): WIDE threads share a
// particle. In each round they take the next WIDE rows, one each, keep their hits as a
// bit per candidate, and after a prefix sum over the team write them at their place in
// the list, so the list is that of neighbors_one. 4,096 particles: 20.0 us -> 8.1.
// A list that is full ends the rounds: in clouds with more neighbours than the cap the
// rows were walked to the end when each thread had a run of them (30,000 particles with
// 300 neighbours, 63 kept: 114 us, one thread per particle 68, in rounds 68; without such
// clouds 4,080 particles 8.1 both ways, 39,304 19.9 and 20.4).
constexpr int SEARCH_WIDE = 8;
constexpr int SEARCH_WIDE_THREADS = 128;

template <int RR>
__global__ void __launch_bounds__(SEARCH_WIDE_THREADS) k_neighbors_wide(KParams p, const float4* __restrict__ x,
                                                                        const int* __restrict__ cell_start,
                                                                        int* __restrict__ nbr,
                                                                        int* __restrict__ ncnt) {
    pdl_wait();
    constexpr int W = 2 * RR + 1, ROWS = W * W, MR = (ROWS + SEARCH_WIDE - 1) / SEARCH_WIDE;
    const int t = threadIdx.x & (SEARCH_WIDE - 1);
    const int team = (blockIdx.x * SEARCH_WIDE_THREADS + threadIdx.x) / SEARCH_WIDE;
    const bool on = team < p.n;
    const int k = on ? team : p.n - 1;  // (every thread of the warp stays for the shuffles)
    const SceneView sc = scene_of(p, k);
    const f3 xk = make3(x[k]);
    int d[3];
    cell_dims(p, sc, xk, d);
    const int nx = sc.dims[0], ny = sc.dims[1], nz = sc.dims[2];
    const float m = clip_margin(p, xk);
    const float hm2 = (p.h + m) * (p.h + m);
    // squared distance, less the margin, to the slab of cells i away (i < 0: below)
    auto slab2 = [&](float q, float g, int cell, int i) {
        const float gap = i > 0 ? cell_from(p, g, cell + i) - q : q - (g + (float)(cell + i + 1) * p.cell);
        const float e = i == 0 ? 0.0f : fmaxf(gap - m, 0.0f);
        return e * e;
    };
    float xl2[RR], xr2[RR];
#pragma unroll
    for (int u = 1; u <= RR; ++u) {
        xl2[u - 1] = slab2(xk.x, sc.gmin[0], d[0], -u);
        xr2[u - 1] = slab2(xk.x, sc.gmin[0], d[0], u);
    }
    const int x0 = max(d[0] - RR, 0), x1 = min(d[0] + RR, nx - 1);
    const bool in_x = d[0] >= 0 && d[0] < nx;
    auto row_range = [&](int r, int& s, int& e) {
        const int y = d[1] + r % W - RR, z = d[2] + r / W - RR;
        s = e = 0;
        if (!on || r >= ROWS || x0 > x1 || y < 0 || y >= ny || z < 0 || z >= nz) return;
        const float rem = hm2 - slab2(xk.z, sc.gmin[2], d[2], z - d[2]) - slab2(xk.y, sc.gmin[1], d[1], y - d[1]);
        if (!(rem >= 0.0f)) return;
        int a = x0, b = x1 + 1;
        if (in_x) {
            a = d[0];
            b = d[0] + 1;
#pragma unroll
            for (int u = 0; u < RR; ++u) {
                a -= xl2[u] <= rem ? 1 : 0;
                b += xr2[u] <= rem ? 1 : 0;
            }
            a = max(a, 0);
            b = min(b, nx);
        }
        const int* row = cell_start + (sc.cell_base + (y + z * ny) * nx);
        s = row[a];
        e = row[b];
    };
    auto near = [&](int j) {
        const float4 q = x[j];
        const f3 r = {xk.x - q.x, xk.y - q.y, xk.z - q.z};
        return dot_fma(r, r) <= p.h2 && j != k;
    };
    const int cap = p.max_nbr;
    int s[MR], e[MR];
#pragma unroll
    for (int i = 0; i < MR; ++i) row_range(i * SEARCH_WIDE + t, s[i], e[i]);
    int total = 0;
#pragma unroll
    for (int i = 0; i < MR; ++i) {
        unsigned hit = 0u;
        int c = 0;
        if (total >= cap) e[i] = s[i];
        if (e[i] - s[i] <= 32) {
#pragma unroll 4
            for (int j = s[i]; j < e[i]; ++j) hit |= (near(j) ? 1u : 0u) << (j - s[i]);
            c = __popc(hit);
        } else {  // (a row of more than 32 candidates is walked again below)
            for (int j = s[i]; j < e[i]; ++j) c += near(j) ? 1 : 0;
        }
        int incl = c;
#pragma unroll
        for (int o = 1; o < SEARCH_WIDE; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o, SEARCH_WIDE);
            if (t >= o) incl += v;
        }
        int at = total + incl - c;
        if (e[i] - s[i] <= 32) {
            for (unsigned h = hit; h; h &= h - 1, ++at)
                if (at < cap) nbr[(size_t)at * p.stride + k] = s[i] + __ffs(h) - 1;
        } else {
            for (int j = s[i]; j < e[i]; ++j)
                if (near(j)) {
                    if (at < cap) nbr[(size_t)at * p.stride + k] = j;
                    ++at;
                }
        }
        total += __shfl_sync(0xffffffffu, incl, SEARCH_WIDE - 1, SEARCH_WIDE);
    }
    total = min(total, cap);
    if (on) {
        if (t == 0) ncnt[k] = total;
        const int end = (total + p.pad - 1) / p.pad * p.pad;
        for (int q = total + t; q < end; q += SEARCH_WIDE) nbr[(size_t)q * p.stride + k] = p.pad_slot;
    }
}

// Copies features and total lambda of the given slots (training rows).
__global__ void k_gather_rows(const int* __restrict__ slots, int count, int n, const float* __restrict__ feat,
                              const float* __restrict__ lam_acc, float* __restrict__ out_feat,
                              float* __restrict__ out_target, int* __restrict__ err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const int s = slots[i];
    if (s < 0 || s >= n) {
        atomicOr(err, DEVERR_BAD_INDEX);
        return;
    }
#pragma unroll
    for (int c = 0; c < 12; ++c) out_feat[(size_t)i * 12 + c] = feat[(size_t)s * 12 + c];
    out_target[i] = lam_acc[s];
}

// Adds the substep's corrections to the running total and counts the substep as
// a fallback when the adaptive loop needed more than the configured count.
__global__ void k_count_fallback(const int* __restrict__ iters, int first, int configured, int* __restrict__ fallback,
                                 long long* __restrict__ total) {
    const int used = first + *iters;
    if (used > configured) *fallback += 1;
    *total += used;
}

// v = (x - x_old) / dt as its own pass (adaptive iteration counts)
__global__ void __launch_bounds__(256) k_velocity(KParams p, const float4* __restrict__ x,
                                                  const float4* __restrict__ xold, float4* __restrict__ v) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= p.n) return;
    const float4 xn = x[k], xo = xold[k];
    v[k] = make_float4(__fdiv_rn(xn.x - xo.x, p.dt), __fdiv_rn(xn.y - xo.y, p.dt), __fdiv_rn(xn.z - xo.z, p.dt), 0.0f);
}

// ---------------------------------------------------------------------------
// a18: one-sided density error over the neighbour list, accumulated in FP64:
// e_k = max(rho_k / rho0 - 1, 0); writes max (as ordered bits) and sum.
// When tol >= 0 it also raises *done once max <= tol (adaptive iterations).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_density_error(KParams p, const float4* __restrict__ x,
                                                       const int* __restrict__ nbr, const int* __restrict__ ncnt,
                                                       unsigned long long* __restrict__ max_bits,
                                                       double* __restrict__ sum, const int* __restrict__ skip) {
    if (skip && *skip) return;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    double e = 0.0;
    if (k < p.n) {
        const float4 xk = x[k];
        const int cnt = ncnt[k];
        double rho = 0.0;
        const double h2 = (double)p.h * (double)p.h;
        for (int q = 0; q < cnt; ++q) {
            const int j = nbr[(size_t)q * p.stride + k];
            const float4 xj = x[j];
            const double rx = (double)xk.x - (double)xj.x, ry = (double)xk.y - (double)xj.y,
                         rz = (double)xk.z - (double)xj.z;
            const double r2 = rx * rx + ry * ry + rz * rz;
            if (r2 <= h2) {
                const double t = h2 - r2;
                rho += p.poly6_c64 * t * t * t;
            }
        }
        e = fmax(rho / (double)p.rho0 - 1.0, 0.0);
    }
    __shared__ double s_max[8], s_sum[8];
    double m = e, s = e;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        s += __shfl_xor_sync(0xffffffffu, s, o);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { s_max[warp] = m; s_sum[warp] = s; }
    __syncthreads();
    if (threadIdx.x == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        for (int w = 1; w < nw; ++w) { m = fmax(m, s_max[w]); s += s_sum[w]; }
        atomicMax(max_bits, (unsigned long long)__double_as_longlong(m));  // m >= 0: bits order as values
        atomicAdd(sum, s);
    }
}

// ---------------------------------------------------------------------------
// layout kernels
// ---------------------------------------------------------------------------
// Upload: AoS to the float4 state in particle order, the total lambda cleared, and
// the first substep's grid hash (a1 + a2) of the state while it is in registers
// (later substeps get theirs from the vorticity pass before them). One pass of 24 B
// read and 48 B written per particle, instead of a conversion, a clear and a hash
// that reads the state again (with the single clear before it and the one-pass
// download, a frame of 4,080 particles and two substeps went from 252 to 234 us).
__global__ void __launch_bounds__(256, 6) k_upload(KParams p, const float* __restrict__ pos,
                                                   const float* __restrict__ vel, float4* __restrict__ x,
                                                   float4* __restrict__ v, int* __restrict__ perm,
                                                   float* __restrict__ lam_acc, int* __restrict__ cell,
                                                   int* __restrict__ ticket, int* __restrict__ cnt,
                                                   int* __restrict__ err) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int key = -1;
    if (i < p.n) {
        f3 xi = {pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]};
        f3 vi = {vel[3 * i], vel[3 * i + 1], vel[3 * i + 2]};
        bool fine = isfinite(xi.x) && isfinite(xi.y) && isfinite(xi.z) && isfinite(vi.x) && isfinite(vi.y) &&
                    isfinite(vi.z);
        x[i] = make_float4(xi.x, xi.y, xi.z, 0.0f);
        v[i] = make_float4(vi.x, vi.y, vi.z, 0.0f);
        perm[i] = (int)i;
        lam_acc[i] = 0.0f;
        const SceneView sc = scene_of(p, (int)i);
        predict(p, sc, xi, vi);
        fine = fine && isfinite(xi.x) && isfinite(xi.y) && isfinite(xi.z);
        if (!fine) atomicOr(err, DEVERR_NONFINITE);
        key = cell_key(p, sc, xi);
    }
    const int tk = warp_histogram(key, cnt);
    if (key >= 0) {
        cell[i] = key;
        ticket[i] = tk;
    }
}

// The state in slot order: AoS x and v, the loaded index of each slot, the key
// of the cell the slot was sorted into and its rank within that cell (any
// output may be null).
__global__ void k_sorted_state(int n, const float4* __restrict__ x, const float4* __restrict__ v,
                               const int* __restrict__ perm, const int* __restrict__ cell_sorted,
                               const int* __restrict__ cell_start, float* __restrict__ pos, float* __restrict__ vel,
                               int* __restrict__ ids, int* __restrict__ key, int* __restrict__ rank) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    if (pos) {
        const float4 q = x[k];
        pos[3 * k] = q.x;
        pos[3 * k + 1] = q.y;
        pos[3 * k + 2] = q.z;
    }
    if (vel) {
        const float4 q = v[k];
        vel[3 * k] = q.x;
        vel[3 * k + 1] = q.y;
        vel[3 * k + 2] = q.z;
    }
    if (ids) ids[k] = perm[k];
    const int c = cell_sorted[k];
    if (key) key[k] = c;
    if (rank) rank[k] = k - cell_start[c];
}

// slot order -> original order, AoS xyz: a to out and, when both are given, a2 to
// out2 in the same pass over perm
__global__ void __launch_bounds__(256) k_to_aos(int n, const float4* __restrict__ a, const float4* __restrict__ a2,
                                                const int* __restrict__ perm, float* __restrict__ out,
                                                float* __restrict__ out2, int* __restrict__ err) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const long long o = perm[k];
    if (o < 0 || o >= n) {
        atomicOr(err, DEVERR_BAD_INDEX);
        return;
    }
    const float4 q = a[k];
    out[3 * o] = q.x;
    out[3 * o + 1] = q.y;
    out[3 * o + 2] = q.z;
    if (out2) {
        const float4 r = a2[k];
        out2[3 * o] = r.x;
        out2[3 * o + 1] = r.y;
        out2[3 * o + 2] = r.z;
    }
}

__global__ void k_fill_pad(float4* x, float4* q, float4* v, float4* vw) {
    *x = *q = make_float4(PAD_POSITION, PAD_POSITION, PAD_POSITION, 0.0f);
    *v = *vw = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

__global__ void k_copy4(int n, const float4* __restrict__ a, float4* __restrict__ b) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) b[k] = a[k];
}

// ---------------------------------------------------------------------------
// FP32 throughput probe: every thread runs 8 independent chains of fused
// multiply-adds (scalar FFMA, or packed fma.rn.f32x2 with two lanes each), long
// enough that launch and tail are negligible. The result is stored only under a
// condition the chains never meet, so nothing is optimised away and nothing is
// written. FLOPs = 2 per multiply-add lane.
// ---------------------------------------------------------------------------
template <bool PACKED>
__global__ void __launch_bounds__(256) k_fma_peak(int iters, float seed, float* __restrict__ sink) {
    const float b = 0.999999f, c = 1e-7f;
    if (PACKED) {
        float2 a[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = make_float2(seed + (float)(threadIdx.x + i), seed - (float)i);
        for (int it = 0; it < iters; ++it) {
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = vfma(a[i], bc<float2>(b), bc<float2>(c));
        }
        float t = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) t += a[i].x + a[i].y;
        if (t == -1.0f) sink[threadIdx.x] = t;
    } else {
        float a[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = seed + (float)(threadIdx.x + i);
        for (int it = 0; it < iters; ++it) {
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = __fmaf_rn(a[i], b, c);
        }
        float t = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) t += a[i];
        if (t == -1.0f) sink[threadIdx.x] = t;
    }
}

// Best of three timed launches of each form (CUDA events), after a warm-up launch.
int measure_fp32_peak(double* scalar_tflops, double* packed_tflops) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return -1;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    float* sink = nullptr;
    if (cudaMalloc(&sink, 256 * sizeof(float)) != cudaSuccess) return -1;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    const int blocks = sms * 8, threads = 256, iters = 1 << 14;
    double best[2] = {0.0, 0.0};
    for (int form = 0; form < 2; ++form) {
        const double lanes = form ? 2.0 : 1.0;
        const double flops = 2.0 * 8.0 * lanes * iters * (double)blocks * threads;
        for (int rep = 0; rep < 4; ++rep) {
            cudaEventRecord(a, 0);
            if (form) k_fma_peak<true><<<blocks, threads>>>(iters, 1.0f, sink);
            else k_fma_peak<false><<<blocks, threads>>>(iters, 1.0f, sink);
            cudaEventRecord(b, 0);
            cudaEventSynchronize(b);
            float ms = 0.0f;
            cudaEventElapsedTime(&ms, a, b);
            if (rep > 0 && ms > 0.0f) best[form] = std::max(best[form], flops / (ms * 1e-3) / 1e12);
        }
    }
    const cudaError_t e = cudaGetLastError();
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(sink);
    if (e != cudaSuccess) return -1;
    *scalar_tflops = best[0];
    *packed_tflops = best[1];
    return 0;
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static inline int blocks_for(int n, int bs) { return (n + bs - 1) / bs; }
static inline bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }
void launch_hash(const KParams& p, bool predict_on, const float4* x, const float4* v, int* cell, int* ticket, int* cnt,
                 int* err, cudaStream_t st) {
    // four rounds per warp once there are enough particles to fill the device
    // with them (about 1 M); below that, one round keeps more blocks resident
    if (p.n >= (1 << 20)) {
        const int b = blocks_for(p.n, 256 * 4);
        if (predict_on) k_hash<true, 4><<<b, 256, 0, st>>>(p, x, v, cell, ticket, cnt, err);
        else k_hash<false, 4><<<b, 256, 0, st>>>(p, x, v, cell, ticket, cnt, err);
    } else {
        const int b = blocks_for(p.n, 256);
        if (predict_on) k_hash<true, 1><<<b, 256, 0, st>>>(p, x, v, cell, ticket, cnt, err);
        else k_hash<false, 1><<<b, 256, 0, st>>>(p, x, v, cell, ticket, cnt, err);
    }
}

// tile count in 64-bit arithmetic (m + tile - 1 would overflow an int near INT_MAX)
static int tiles_of(int m, int tile) { return (int)(((long long)m + tile - 1) / tile); }

size_t scan_status_bytes(int m) { return (size_t)tiles_of(m, scan_tile(m)) * sizeof(unsigned long long) + 16; }

template <bool VEC>
static void launch_scan_cleared(int* cnt, int* out, int m, void* ws, int* err, int* host_err, cudaStream_t st,
                                int silent_tile = -1, long long spin_limit = SCAN_SPIN_LIMIT) {
    unsigned long long* status = (unsigned long long*)ws;
    const int tiles = tiles_of(m, scan_tile(m));
    if (scan_tile(m) == 16384)
        k_scan<VEC, false, 64><<<tiles, SCAN_THREADS, 0, st>>>(cnt, out, m, status, tiles, err, host_err, silent_tile,
                                                                spin_limit, nullptr, 0);
    else
        k_scan<VEC, false, 32><<<tiles, SCAN_THREADS, 0, st>>>(cnt, out, m, status, tiles, err, host_err, silent_tile,
                                                                spin_limit, nullptr, 0);
}

static int keep_tile(int m) { return m <= SCAN_SMALL_MAX ? 4096 : scan_tile(m); }
size_t scan_keep_bytes(int m) { return (size_t)tiles_of(m, keep_tile(m)) * sizeof(unsigned long long) + 16; }

void launch_scan(int* cnt, int* out, int m, void* ws, int* zero, int nzero, int* err, cudaStream_t st) {
    unsigned long long* status = (unsigned long long*)ws;
    const int tile = keep_tile(m), tiles = tiles_of(m, tile);
    auto go = [&](auto kernel) {
        kernel<<<tiles, SCAN_THREADS, 0, st>>>(cnt, out, m, status, tiles, err, nullptr, -1, SCAN_SPIN_LIMIT, zero, nzero);
    };
    if (tile == 4096) go(k_scan<true, true, 16>);
    else if (tile == 8192) go(k_scan<true, true, 32>);
    else go(k_scan<true, true, 64>);
}

void launch_scan_const(const int* in, int* out, int m, void* ws, size_t clear_bytes, int* err, int* host_err,
                       cudaStream_t st) {
    cudaMemsetAsync(ws, 0, clear_bytes, st);
    if (aligned16(in) && aligned16(out))
        launch_scan_cleared<true>(const_cast<int*>(in), out, m, ws, err, host_err, st);
    else
        launch_scan_cleared<false>(const_cast<int*>(in), out, m, ws, err, host_err, st);
}

void launch_scan_silent_tile(const int* in, int* out, int m, void* ws, int* err, int silent_tile,
                             long long spin_limit, cudaStream_t st) {
    cudaMemsetAsync(ws, 0, scan_status_bytes(m), st);
    launch_scan_cleared<false>(const_cast<int*>(in), out, m, ws, err, nullptr, st, silent_tile, spin_limit);
}

void launch_scatter(bool pdl, int n, const int* cell, const int* ticket, const int* cell_start, int* tmp, int* err,
                    cudaStream_t st) {
    if (n >= (1 << 20))
        launch(pdl, k_scatter<4>, blocks_for(n, 256 * 4), 256, 0, st, n, cell, ticket, cell_start, tmp, err);
    else
        launch(pdl, k_scatter<1>, blocks_for(n, 256), 256, 0, st, n, cell, ticket, cell_start, tmp, err);
}

void launch_reorder(const KParams& p, bool predict_on, const float4* x, const float4* v, const int* perm,
                    const int* cell, const int* cell_start, const int* tmp, float4* xp, float4* vp, float4* xold,
                    int* perm_out, int* cell_sorted, const float* lam_in, float* lam_out, int* err, cudaStream_t st) {
    const int b = blocks_for(p.n, 256);
    if (predict_on)
        launch(p.pdl, k_reorder<true>, b, 256, 0, st, p, x, v, perm, cell, cell_start, tmp, xp, vp, xold, perm_out, cell_sorted,
                                           lam_in, lam_out, err);
    else
        launch(p.pdl, k_reorder<false>, b, 256, 0, st, p, x, v, perm, cell, cell_start, tmp, xp, vp, xold, perm_out, cell_sorted,
                                            lam_in, lam_out, err);
}

// Grid over nvb tiles: nvb blocks, or with p.persistent the blocks resident at
// once (SMs x blocks per SM), each striding over the tiles.
template <typename K> static int resident_grid(const KParams& p, K kernel, int nvb) {
    if (!p.persistent) return nvb;
    int dev = 0, sms = 1, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, p.block, 0) != cudaSuccess || per_sm <= 0)
        per_sm = 1;
    const long long g = (long long)per_sm * (sms > 0 ? sms : 1);
    return (int)(g < nvb ? g : nvb);
}

// Particles up to which SEARCH_WIDE threads share one: its time grows with the
// particles, one thread's walk takes the same until the device is full. Cells of h/2,
// shared against not: 18.2 / 20.6 us at 32,768 particles, 20.4 / 20.5 at 39,304, 22.9 /
// 21.1 at 46,656; cells of h: 14.1 / 14.9 at 13,824, 17.6 / 15.2 at 21,952.
constexpr int SEARCH_WIDE_MAX_N[3] = {0, 16384, 40960};  // by stencil radius

void launch_neighbors(const KParams& p, const float4* x, const int* cell_start, int* nbr, int* ncnt, cudaStream_t st) {
    if (p.radius <= 2 && p.n <= SEARCH_WIDE_MAX_N[p.radius] && !p.persistent) {
        const int b = blocks_for(p.n, SEARCH_WIDE_THREADS / SEARCH_WIDE);
        if (p.radius == 1) launch(p.pdl, k_neighbors_wide<1>, b, SEARCH_WIDE_THREADS, 0, st, p, x, cell_start, nbr, ncnt);
        else launch(p.pdl, k_neighbors_wide<2>, b, SEARCH_WIDE_THREADS, 0, st, p, x, cell_start, nbr, ncnt);
        return;
    }
    const int b = blocks_for(p.n, p.block);
    auto go = [&](auto k) { launch(p.pdl, k, resident_grid(p, k, b), p.block, 0, st, p, b, x, cell_start, nbr, ncnt); };
    if (p.radius == 1) go(k_neighbors<1>);
    else if (p.radius == 2) go(k_neighbors<2>);
    else go(k_neighbors<0>);
}

void launch_gather_rows(const int* slots, int count, int n, const float* feat, const float* lam_acc, float* out_feat,
                        float* out_target, int* err, cudaStream_t st) {
    if (count > 0)
        k_gather_rows<<<blocks_for(count, 256), 256, 0, st>>>(slots, count, n, feat, lam_acc, out_feat, out_target,
                                                               err);
}

void launch_count_fallback(const int* iters, int first, int configured, int* fallback, long long* total,
                           cudaStream_t st) {
    k_count_fallback<<<1, 1, 0, st>>>(iters, first, configured, fallback, total);
}

void launch_velocity(const KParams& p, const float4* x, const float4* xold, float4* v, cudaStream_t st) {
    k_velocity<<<blocks_for(p.n, 256), 256, 0, st>>>(p, x, xold, v);
}

void launch_density_error(const KParams& p, const float4* x, const int* nbr, const int* ncnt,
                          unsigned long long* max_bits, double* sum, const int* skip, cudaStream_t st) {
    k_density_error<<<blocks_for(p.n, 256), 256, 0, st>>>(p, x, nbr, ncnt, max_bits, sum, skip);
}

void launch_upload(const KParams& p, const float* pos, const float* vel, float4* x, float4* v, int* perm,
                   float* lam_acc, int* cell, int* ticket, int* cnt, int* err, cudaStream_t st) {
    k_upload<<<blocks_for(p.n, 256), 256, 0, st>>>(p, pos, vel, x, v, perm, lam_acc, cell, ticket, cnt, err);
}

void launch_to_aos(int n, const float4* a, const float4* a2, const int* perm, float* out, float* out2, int* err,
                   cudaStream_t st) {
    k_to_aos<<<blocks_for(n, 256), 256, 0, st>>>(n, a, a2, perm, out, out2, err);
}

void launch_sorted_state(int n, const float4* x, const float4* v, const int* perm, const int* cell_sorted,
                         const int* cell_start, float* pos, float* vel, int* ids, int* key, int* rank,
                         cudaStream_t st) {
    k_sorted_state<<<blocks_for(n, 256), 256, 0, st>>>(n, x, v, perm, cell_sorted, cell_start, pos, vel, ids, key,
                                                       rank);
}

void launch_fill_pad(float4* x, float4* q, float4* v, float4* vw, cudaStream_t st) {
    k_fill_pad<<<1, 1, 0, st>>>(x, q, v, vw);
}

void launch_copy4(int n, const float4* a, float4* b, cudaStream_t st) {
    k_copy4<<<blocks_for(n, 256), 256, 0, st>>>(n, a, b);
}

}  // namespace pbf
