// List rebuild path of the GB300 DEM engine: Morton keys, stable LSB radix
// sort, particle reorder, cell ranges, Verlet lists, wall mesh tree and wall lists.
//
// Reference counterparts (gpudem): dk_morton_key / update_pList_withSort
// (BoundingBox.cu:1007, :664), radixSortUint32 / CUB SortPairs
// (BoundingBox.cu:33, :1235), d_swap_ps (BoundingBox.cu:928), d_update_pList
// (BoundingBox.cu:1266), k_update_neighborlist_endsort (BoundingBox.cu:1106),
// buildBVH (BVH.cu:741), k_update_neighborlist_wall (BVH.cu:493).
//
// Every kernel that decides list membership uses the reference's FP64
// arithmetic in the same operation order; this file is compiled with
// -fmad=false so no multiply-add is contracted.
#include <cuda_runtime.h>
#include <stdint.h>

#include "gdem_internal.cuh"

namespace gdem {

// ===================================================================== radix sort
// Stable least-significant-digit radix sort of (key, value) pairs with 8-bit
// digits.  One pass = upsweep (per-tile digit histograms, digit-major table),
// scan (per-digit exclusive scan over tiles), downsweep (stable scatter).  The
// scatter ranks equal digits inside a tile with __match_any_sync, so the
// permutation is the unique stable one — the same that radixSortUint32
// (BoundingBox.cu:33-104) and CUB's SortPairs produce.  No kernel waits on
// another block.
constexpr int RS_THREADS = 256;
constexpr int RS_ROUNDS = 8;
constexpr int RS_TILE = RS_THREADS * RS_ROUNDS;

int rs_blocks_for(int n) { return n <= 0 ? 1 : (n + RS_TILE - 1) / RS_TILE; }

__global__ void __launch_bounds__(RS_THREADS) k_rs_upsweep(const uint32_t* __restrict__ keys, int n,
                                                           int shift, uint32_t* __restrict__ hist,
                                                           int nblocks, const Ctl* ctl, int gated) {
    if (gated && ctl->refresh == 0u) return;
    __shared__ uint32_t cnt[256];
    cnt[threadIdx.x] = 0;
    __syncthreads();
    const int base = blockIdx.x * RS_TILE;
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; r++) {
        const int i = base + r * RS_THREADS + threadIdx.x;
        if (i < n) atomicAdd(&cnt[(keys[i] >> shift) & 0xFFu], 1u);
    }
    __syncthreads();
    hist[threadIdx.x * nblocks + blockIdx.x] = cnt[threadIdx.x];
}

// one block per digit: exclusive scan of that digit's tile counts
__global__ void __launch_bounds__(1024) k_rs_scan(uint32_t* __restrict__ hist, int nblocks,
                                                  uint32_t* __restrict__ tot, const Ctl* ctl, int gated) {
    if (gated && ctl->refresh == 0u) return;
    __shared__ uint32_t warp_sums[32];
    __shared__ uint32_t carry;
    uint32_t* row = hist + (size_t)blockIdx.x * nblocks;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < nblocks; base += blockDim.x) {
        const int i = base + threadIdx.x;
        const uint32_t x = i < nblocks ? row[i] : 0u;
        uint32_t incl = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) warp_sums[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            const int nw = blockDim.x >> 5;
            uint32_t s = lane < nw ? warp_sums[lane] : 0u;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
                if (lane >= o) s += y;
            }
            if (lane < nw) warp_sums[lane] = s;  // inclusive warp prefix
        }
        __syncthreads();
        const uint32_t warp_excl = warp ? warp_sums[warp - 1] : 0u;
        const uint32_t c = carry;
        if (i < nblocks) row[i] = c + warp_excl + incl - x;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = c + warp_excl + incl;
        __syncthreads();
    }
    if (threadIdx.x == 0) tot[blockIdx.x] = carry;
}

// SMALL: few tiles (nblocks <= RS_SMALL_TILES); the tile counts are then
// read unscanned and each block sums what it needs itself, with no scan
// kernel in between.
constexpr int RS_SMALL_TILES = 32;

template <bool SMALL>
__global__ void __launch_bounds__(RS_THREADS) k_rs_downsweep(
    const uint32_t* __restrict__ kin, const int* __restrict__ vin, uint32_t* __restrict__ kout,
    int* __restrict__ vout, int n, int shift, const uint32_t* __restrict__ hist,
    const uint32_t* __restrict__ tot, int nblocks, const Ctl* ctl, int gated) {
    if (gated && ctl->refresh == 0u) return;
    constexpr int NW = RS_THREADS / 32;
    __shared__ uint32_t base[256];
    __shared__ uint32_t wcnt[NW][256];
    __shared__ uint32_t scan_tmp[256];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    // digit base = exclusive prefix of the digit totals + this tile's offset
    uint32_t total, mine;
    if (SMALL) {
        total = 0u;
        mine = 0u;
        for (int b = 0; b < nblocks; b++) {
            const uint32_t c = hist[t * nblocks + b];
            if (b < (int)blockIdx.x) mine += c;
            total += c;
        }
    } else {
        total = tot[t];
        mine = hist[t * nblocks + blockIdx.x];
    }
    scan_tmp[t] = total;
    __syncthreads();
    for (int o = 1; o < 256; o <<= 1) {
        const uint32_t y = t >= o ? scan_tmp[t - o] : 0u;
        __syncthreads();
        scan_tmp[t] += y;
        __syncthreads();
    }
    base[t] = scan_tmp[t] - total + mine;
#pragma unroll
    for (int w = 0; w < NW; w++) wcnt[w][t] = 0;
    __syncthreads();
    const unsigned lt_mask = (1u << lane) - 1u;
    const int tile = blockIdx.x * RS_TILE;
    for (int r = 0; r < RS_ROUNDS; r++) {
        const int i = tile + r * RS_THREADS + t;
        const bool valid = i < n;
        uint32_t key = 0;
        int val = 0;
        uint32_t d = 256u;  // invalid lanes get a digit of their own
        if (valid) {
            key = kin[i];
            val = vin[i];
            d = (key >> shift) & 0xFFu;
        }
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const uint32_t wrank = __popc(peers & lt_mask);
        if (valid && (peers & lt_mask) == 0u) wcnt[warp][d] = __popc(peers);
        __syncthreads();
        // per digit: exclusive prefix over warps, then advance the base
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < NW; w++) {
            const uint32_t c = wcnt[w][t];
            wcnt[w][t] = run;
            run += c;
        }
        __syncthreads();
        if (valid) {
            const uint32_t dst = base[d] + wcnt[warp][d] + wrank;
            kout[dst] = key;
            vout[dst] = val;
        }
        __syncthreads();
        base[t] += run;
#pragma unroll
        for (int w = 0; w < NW; w++) wcnt[w][t] = 0;
        __syncthreads();
    }
}

// The same stable sort of up to kSortSmall pairs in one launch, by one CTA: a
// bitonic network over key << 32 | position in shared memory (equal keys keep
// their order by position).  Strides up to 32 stay within the 64 elements that a
// warp holds, so 27 of the 78 stages of 4,096 elements wait for the whole CTA.
// A sort this small is bound by launches and latency: beside the step of 2,000
// spheres the mesh tree of 300 triangles took 41 us with the eight launches of the
// radix passes and 25 with this one, the list rebuild of 100 spheres 148 and 113.

__global__ void __launch_bounds__(1024) k_sort_small(uint32_t* __restrict__ keys, int* __restrict__ vals, int n,
                                                     int padded, const Ctl* ctl, int gated) {
    __shared__ unsigned long long a[kSortSmall];
    if (gated && ctl->refresh == 0u) return;
    const int t = threadIdx.x;
    int val[kSortSmall / 1024];
    for (int i = t; i < padded; i += 1024)
        a[i] = i < n ? (unsigned long long)keys[i] << 32 | (unsigned)i : ~0ull;
    __syncthreads();
    for (int k = 2; k <= padded; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int p = t; p < padded >> 1; p += 1024) {
                const int lo = 2 * p - (p & (j - 1)), hi = lo + j;
                const unsigned long long x = a[lo], y = a[hi];
                if ((x > y) == ((lo & k) == 0)) {
                    a[lo] = y;
                    a[hi] = x;
                }
            }
            // the next stage's stride is j / 2, or k when this one ends a merge
            if (j >= 64 || (j == 1 && k >= 64)) __syncthreads();
            else __syncwarp();
        }
    __syncthreads();
    // the payloads move through registers: they are sorted in place
#pragma unroll
    for (int u = 0; u < kSortSmall / 1024; u++) {
        const int i = t + u * 1024;
        val[u] = i < n ? vals[(unsigned)a[i]] : 0;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kSortSmall / 1024; u++) {
        const int i = t + u * 1024;
        if (i < n) {
            keys[i] = (uint32_t)(a[i] >> 32);
            vals[i] = val[u];
        }
    }
}

static void rs_passes(uint32_t* k0, int* v0, uint32_t* k1, int* v1, uint32_t* hist, uint32_t* tot,
                      int n, int nblocks, int first_pass, int npasses, cudaStream_t st,
                      const Ctl* ctl, int gated) {
    if (n <= kSortSmall && first_pass == 0 && npasses == 4) {
        int padded = 64;
        while (padded < n) padded *= 2;
        if (n > 0) k_sort_small<<<1, 1024, 0, st>>>(k0, v0, n, padded, ctl, gated);
        return;
    }
    uint32_t* ks[2] = {k0, k1};
    int* vs[2] = {v0, v1};
    for (int p = 0; p < npasses; p++) {
        const int shift = 8 * (first_pass + p);
        const int a = p & 1;
        k_rs_upsweep<<<nblocks, RS_THREADS, 0, st>>>(ks[a], n, shift, hist, nblocks, ctl, gated);
        if (nblocks <= RS_SMALL_TILES) {
            k_rs_downsweep<true><<<nblocks, RS_THREADS, 0, st>>>(ks[a], vs[a], ks[a ^ 1], vs[a ^ 1], n, shift,
                                                                 hist, tot, nblocks, ctl, gated);
        } else {
            k_rs_scan<<<256, 1024, 0, st>>>(hist, nblocks, tot, ctl, gated);
            k_rs_downsweep<false><<<nblocks, RS_THREADS, 0, st>>>(ks[a], vs[a], ks[a ^ 1], vs[a ^ 1], n, shift,
                                                                  hist, tot, nblocks, ctl, gated);
        }
    }
}

void radix_sort_pairs(uint32_t* keys0, int* vals0, uint32_t* keys1, int* vals1, uint32_t* hist,
                      uint32_t* tot, int n, int nblocks, int first_pass, int npasses,
                      cudaStream_t st) {
    rs_passes(keys0, vals0, keys1, vals1, hist, tot, n, nblocks, first_pass, npasses, st, nullptr, 0);
}

// ===================================================================== keys
// Morton key of every particle from its ghost-offset cell coordinates
// (update_pList_withSort, BoundingBox.cu:680-690).  Inactive particles get an
// all-ones key so they sort behind every cell; a particle leaving the box this
// step (status 2) is still keyed, like the reference CPU loop still lists it.
template <class T>
__global__ void k_keys(View<T> v, int gated) {
    const Ctl* ctl = v.ctl;
    if (gated && ctl->refresh == 0u) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= v.n) return;
    const SBank<T> S = v.S[ctl->s];
    uint32_t key = kNoKey;
    if (S.rot[i].w != 0) {
        const double4_32a p = load_pos(S, i);
        const int cx = cell_x(v, p.x);
        const int cy = cell_coord(p.y, v.miny, v.invdy);
        const int cz = cell_coord(p.z, v.minz, v.invdz);
        key = morton3((uint32_t)cx, (uint32_t)cy, (uint32_t)cz);
    }
    v.keys[0][i] = key;
    v.vals[0][i] = i;
}

// Deactivate particles that left the box at the last step (status 2 -> 0);
// runs before a rebuild requested between steps.
template <class T>
__global__ void k_finalize_oob(View<T> v) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= v.n) return;
    const SBank<T> S = v.S[v.ctl->s];
    if (S.rot[i].w == 2) S.rot[i].w = 0;  // (mixed: posh.w is already negative)
}

template <class T>
void launch_finalize_oob(const View<T>& v, cudaStream_t st) {
    k_finalize_oob<T><<<(v.n + kBlock - 1) / kBlock, kBlock, 0, st>>>(v);
}

// ===================================================================== reorder
// Mixed mode: the inverse of the sort permutation, for remapping the history
// keys (storage indices of contact partners) when the particles move.
template <class T>
__global__ void k_inverse_order(View<T> v, int gated) {
    const Ctl* ctl = v.ctl;
    if (gated && ctl->refresh == 0u) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= v.n) return;
    v.inv[v.vals[0][i]] = i;
}

// Gather every per-particle array into sorted order (d_swap_ps,
// BoundingBox.cu:928-1005, but with compact histories: only live slots move).
template <class T>
__global__ void __launch_bounds__(kBlock, 4) k_reorder(View<T> v, int gated) {
    Ctl* ctl = v.ctl;
    if (gated && ctl->refresh == 0u) return;
    const int s = ctl->s, p = ctl->p;
    const int n = v.n;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const int src = v.vals[0][i];
        const SBank<T> A = v.S[s], B = v.S[s ^ 1];
        if (!T::mixed) B.pos[i] = A.pos[src];
        B.vel[i] = A.vel[src];
        B.rot[i] = A.rot[src];
        if (T::mixed) {
            B.posh[i] = A.posh[src];
            B.posl[i] = A.posl[src];
            B.vell[i] = A.vell[src];
            B.rotl[i] = A.rotl[src];
        }
        const PBank<T> P = v.P[p], Q = v.P[p ^ 1];
        Q.mat[i] = P.mat[src];
        Q.pid[i] = P.pid[src];
        // live history slots, four at a time with their loads in flight
        // together (the slot rows are slot-major: slot k of particle i at
        // k * n + i, so a warp's loads of one slot are contiguous)
        using R = typename T::real;
        const int nc = P.nc[src];
        Q.nc[i] = nc;
        for (int k0 = 0; k0 < nc; k0 += 4) {
            int id[4];
            R t[6][4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (k0 + q >= nc) continue;
                const size_t a = (size_t)(k0 + q) * n + src;
                id[q] = P.hid[a];
                t[0][q] = P.hx[a]; t[1][q] = P.hy[a]; t[2][q] = P.hz[a];
                if (T::mixed) { t[3][q] = P.cx[a]; t[4][q] = P.cy[a]; t[5][q] = P.cz[a]; }
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (k0 + q >= nc) continue;
                const size_t b = (size_t)(k0 + q) * n + i;
                Q.hid[b] = T::mixed ? v.inv[id[q]] : id[q];
                Q.hx[b] = t[0][q]; Q.hy[b] = t[1][q]; Q.hz[b] = t[2][q];
                if (T::mixed) { Q.cx[b] = t[3][q]; Q.cy[b] = t[4][q]; Q.cz[b] = t[5][q]; }
            }
        }
        const int ncw = P.ncw[src];
        Q.ncw[i] = ncw;
        for (int k0 = 0; k0 < ncw; k0 += 2) {
            int id[2];
            R t[6][2];
#pragma unroll
            for (int q = 0; q < 2; q++) {
                if (k0 + q >= ncw) continue;
                const size_t a = (size_t)(k0 + q) * n + src;
                id[q] = P.hwid[a];
                t[0][q] = P.hwx[a]; t[1][q] = P.hwy[a]; t[2][q] = P.hwz[a];
                if (T::mixed) { t[3][q] = P.cwx[a]; t[4][q] = P.cwy[a]; t[5][q] = P.cwz[a]; }
            }
#pragma unroll
            for (int q = 0; q < 2; q++) {
                if (k0 + q >= ncw) continue;
                const size_t b = (size_t)(k0 + q) * n + i;
                Q.hwid[b] = id[q];
                Q.hwx[b] = t[0][q]; Q.hwy[b] = t[1][q]; Q.hwz[b] = t[2][q];
                if (T::mixed) { Q.cwx[b] = t[3][q]; Q.cwy[b] = t[4][q]; Q.cwz[b] = t[5][q]; }
            }
        }
    }
    if (last_block(&ctl->done[1])) {
        if (threadIdx.x == 0) {
            ctl->done[1] = 0;
            ctl->s = s ^ 1;
            ctl->p = p ^ 1;
        }
    }
}

// Per-step force/torque outputs follow the particles they belong to.
template <class T>
__global__ void k_reorder_forces(View<T> v, int gated) {
    const Ctl* ctl = v.ctl;
    if (gated && ctl->refresh == 0u) return;
    const int n = v.n;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int src = v.vals[0][i];
    double* f[6] = {v.fx, v.fy, v.fz, v.tx, v.ty, v.tz};
    for (int c = 0; c < 6; c++) v.ftmp[(size_t)c * n + i] = f[c][src];
}
template <class T>
__global__ void k_copy_forces(View<T> v, int gated) {
    const Ctl* ctl = v.ctl;
    if (gated && ctl->refresh == 0u) return;
    const int n = v.n;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double* f[6] = {v.fx, v.fy, v.fz, v.tx, v.ty, v.tz};
    for (int c = 0; c < 6; c++) f[c][i] = v.ftmp[(size_t)c * n + i];
}

// ===================================================================== cells
template <class T>
__global__ void k_cells_clear(View<T> v, int gated) {
    const Ctl* ctl = v.ctl;
    if (gated && ctl->refresh == 0u) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) v.ctl->wall_alloc = 0u;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < v.ncells; c += gridDim.x * blockDim.x) {
        v.cell_start[c] = 0;
        v.cell_end[c] = 0;
    }
}

// Cell ranges from the sorted keys: equal keys are one cell, found by
// comparing neighbours in the sorted order (no atomics; replaces
// dk_build_cellCount + ExclusiveSum + dk_build_pList, BoundingBox.cu:1266).
template <class T>
__global__ void k_cell_ranges(View<T> v, int gated) {
    const Ctl* ctl = v.ctl;
    if (gated && ctl->refresh == 0u) return;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = v.n;
    if (q >= n) return;
    const int jq = v.reorder ? q : v.vals[0][q];
    const uint32_t* key = v.keys[0];
    const uint32_t kq = key[q];
    if (kq == kNoKey) {
        v.nnei[jq] = 0;  // in no cell: an empty Verlet row
        return;
    }
    const int cx = (int)compact10(kq >> 2), cy = (int)compact10(kq >> 1), cz = (int)compact10(kq);
    if (cx >= v.sizex || cy >= v.sizey || cz >= v.sizez) {
        atomicOr(&v.ctl->error, 0x40u);
        v.nnei[jq] = 0;
        return;
    }
    const int cell = (v.sizey * cz + cy) * v.sizex + cx;
    if (q == 0 || key[q - 1] != kq) v.cell_start[cell] = q;
    if (q == n - 1 || key[q + 1] != kq) v.cell_end[cell] = q + 1;
}

// The occupied cells in sorted (Morton) order: the first sorted position of
// every cell inside the grid, compacted by a count per block of kBlock
// positions, one exclusive scan over the blocks and an emit that ranks each
// start within its block.  Neighbouring entries are neighbouring cells, so
// the groups of lanes beside one another in k_cell_walls test much the same
// part of the mesh tree.
template <class T>
__device__ __forceinline__ bool is_cell_start(const View<T>& v, int q) {
    if (q >= v.n) return false;
    const uint32_t* key = v.keys[0];
    const uint32_t kq = key[q];
    if (kq == kNoKey || (q > 0 && key[q - 1] == kq)) return false;
    return (int)compact10(kq >> 2) < v.sizex && (int)compact10(kq >> 1) < v.sizey && (int)compact10(kq) < v.sizez;
}

template <class T>
__global__ void __launch_bounds__(kBlock) k_cell_count(View<T> v, int gated) {
    if (gated && v.ctl->refresh == 0u) return;
    const int c = __syncthreads_count(is_cell_start(v, blockIdx.x * blockDim.x + threadIdx.x));
    if (threadIdx.x == 0) v.cell_bc[blockIdx.x] = c;
}

// Exclusive scan of the nb block counts in place, by one CTA of 1024 threads
// (each a run of consecutive counts); the total goes to ctl->ncell_list.
template <class T>
__global__ void __launch_bounds__(1024) k_cell_scan(View<T> v, int gated, int nb) {
    if (gated && v.ctl->refresh == 0u) return;
    __shared__ int part[1024];
    const int t = threadIdx.x;
    const int per = (nb + 1023) / 1024;
    const int lo = t * per, hi = min(lo + per, nb);
    int sum = 0;
    for (int b = lo; b < hi; b++) sum += v.cell_bc[b];
    part[t] = sum;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const int add = t >= o ? part[t - o] : 0;
        __syncthreads();
        part[t] += add;
        __syncthreads();
    }
    int run = part[t] - sum;  // exclusive prefix of this run
    for (int b = lo; b < hi; b++) {
        const int c = v.cell_bc[b];
        v.cell_bc[b] = run;
        run += c;
    }
    if (t == 1023) v.ctl->ncell_list = (unsigned)part[1023];
}

template <class T>
__global__ void __launch_bounds__(kBlock) k_cell_emit(View<T> v, int gated) {
    if (gated && v.ctl->refresh == 0u) return;
    __shared__ int wbase[kBlock / 32];
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const bool f = is_cell_start(v, q);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned m = __ballot_sync(0xffffffffu, f);
    if (lane == 0) wbase[w] = __popc(m);
    __syncthreads();
    if (f) {
        int off = v.cell_bc[blockIdx.x];
        for (int u = 0; u < w; u++) off += wbase[u];
        v.cell_list[off + __popc(m & ((1u << lane) - 1u))] = q;
    }
}

// ===================================================================== Verlet lists
// FP64 mode: FP32 copy of the positions for the prefilter of k_neighbors.
template <class T>
__global__ void k_posf(View<T> v, int gated) {
    const Ctl* ctl = v.ctl;
    if (gated && ctl->refresh == 0u) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= v.n) return;
    const double4_32a p = v.S[ctl->s].pos[i];
    v.posf[i] = make_float4((float)p.x, (float)p.y, (float)p.z, (float)p.w);
}

// Cell of particle i (FP32 position f).  With reordered storage it is decoded
// from the sorted key, which holds the FP64 cell coordinates; a particle outside
// the box, whose coordinates the key may have wrapped, has them computed.  (The
// FP64 arithmetic, two lanes an SM, was a fifth of k_neighbors on a pour.)
template <class T>
__device__ __forceinline__ int3 cell_of(const View<T>& v, const SBank<T>& S, int i, float4 f) {
    if (v.reorder && f.x >= v.boxf[0] && f.x <= v.boxf[3] && f.y >= v.boxf[1] && f.y <= v.boxf[4] &&
        f.z >= v.boxf[2] && f.z <= v.boxf[5]) {
        const uint32_t k = v.keys[0][i];
        return make_int3((int)compact10(k >> 2), (int)compact10(k >> 1), (int)compact10(k));
    }
    const double4_32a p = load_pos(S, i);
    return make_int3(cell_x(v, p.x), cell_coord(p.y, v.miny, v.invdy), cell_coord(p.z, v.minz, v.invdz));
}

// Scan the 27 cells around a particle's cell, keep every listed j != i with
// |xi - xj|^2 < (ri + rj + skin)^2 (the test of BoundingBox.cu:1136-1144, FP64
// in every mode), order the row by the partner's pId (the reference's index
// space) and record the reference position.  Cells outside the grid hold nobody
// and are skipped.
//
// Most candidates are far from the cutoff, so each is first tested on FP32
// positions: nb_delta bounds how far the FP32 distance can be from the FP64
// one (eight FP32 ulps of the largest box coordinate, more than the two
// roundings of the coordinates), and only a candidate whose FP32 distance is
// within that band of the cutoff takes the FP64 test.  The decision is the
// FP64 test's in every case.
//
// kNbLanes lanes to a particle: they take a cell's candidates side by side (its
// positions are consecutive in memory), three cells along x in flight together,
// and keep those that are listed by ballot; the row is then ranked by pId by
// counting and written slot by slot, 32 consecutive ints at a time.  It is bound
// by the latency of that chain of loads; with a thread per particle the chain was
// a load for every four candidates of the 27 cells.  A thread, 4 and 8 lanes to a
// particle: bed of 30,000 spheres 116, 54 and 51 us, 250,000 346, 286 and 335,
// 1,000,000 1119, 1105 and 1316, a pour of 300,000 (two candidates a cell) 161,
// 161 and 229.
constexpr int kNbBlock = 128;
constexpr int kNbLanes = 4;
constexpr int kNbPer = kNbBlock / kNbLanes;  // particles of a CTA

template <class T, int CAP>
__global__ void __launch_bounds__(kNbBlock) k_neighbors(View<T> v, int gated) {
    constexpr int kStride = CAP + 1;
    extern __shared__ int nb_smem[];
    int* js = nb_smem;                          // [particle][entry]: partners as found
    int* ids = js + kNbPer * kStride;           // their pIds
    int* out = ids + kNbPer * kStride;          // partners by pId
    int* len = out + kNbPer * kStride;          // [particle] row lengths
    Ctl* ctl = v.ctl;
    if (gated && ctl->refresh == 0u) return;
    const int n = v.n;
    const int lane = threadIdx.x & 31, l = threadIdx.x % kNbLanes, slot = threadIdx.x / kNbLanes;
    const unsigned gmask = ((1u << kNbLanes) - 1u) << (lane & ~(kNbLanes - 1)), below = gmask & ((1u << lane) - 1u);
    const int i0 = blockIdx.x * kNbPer, i = i0 + slot;
    const SBank<T> S = v.S[ctl->s];
    const PBank<T> P = v.P[ctl->p];
    const float4* __restrict__ PF = T::mixed ? S.posh : v.posf;
    const int* __restrict__ pidv = P.pid;
    int* const row = js + slot * kStride;
    const bool on = i < n && S.rot[i].w != 0;
    const float4 fi = on ? PF[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int3 cc = on ? cell_of(v, S, i, fi) : make_int3(-4, -4, -4);
    const float delta = v.nb_delta, rfi = fabsf(fi.w) + (float)v.skin;
    int count = 0;
    // the bounds of the three cells along x of cell row k (of nine); a row's are
    // loaded while the row before it is tested
    const auto range = [&](int k, int* b, int* e) {
        const int zz = cc.z + k / 3 - 1, yy = cc.y + k % 3 - 1;
        const bool in = on && zz >= 0 && zz < v.sizez && yy >= 0 && yy < v.sizey;
#pragma unroll
        for (int u = 0; u < 3; u++) {
            int xx = cc.x + u - 1;
            bool ok = in;
            if (v.per_x) {
                // cells 1..nxp wrap around (nxp >= 3: no cell twice)
                if (xx < 1) xx += v.nxp;
                else if (xx > v.nxp) xx -= v.nxp;
            } else {
                ok = ok && xx >= 0 && xx < v.sizex;
            }
            b[u] = e[u] = 0;
            if (ok) {
                const int cell = (v.sizey * zz + yy) * v.sizex + xx;
                b[u] = v.cell_start[cell];
                e[u] = v.cell_end[cell];
            }
        }
    };
    int nb[3], ne[3];
    range(0, nb, ne);
    for (int k = 0; k < 9; k++) {
        int b[3], e[3], most = 0;
#pragma unroll
        for (int u = 0; u < 3; u++) {
            b[u] = nb[u] + l;
            e[u] = ne[u];
            most = max(most, ne[u] - nb[u]);
        }
        if (k < 8) range(k + 1, nb, ne);
        most = __reduce_max_sync(0xffffffffu, most);
        for (int c0 = 0; c0 < most; c0 += kNbLanes) {
            int jj[3];
            float4 fj[3];
#pragma unroll
            for (int u = 0; u < 3; u++) {
                const int q = b[u] + c0;
                jj[u] = q < e[u] ? (v.reorder ? q : v.vals[0][q]) : -1;
                if (jj[u] >= 0) fj[u] = PF[jj[u]];
            }
#pragma unroll
            for (int u = 0; u < 3; u++) {
                const int j = jj[u];
                bool inside = false;
                if (j >= 0 && j != i) {
                    const float ex = image_dxf(v, fi.x - fj[u].x), ey = fi.y - fj[u].y, ez = fi.z - fj[u].z;
                    const float dsqf = ex * ex + ey * ey + ez * ez;
                    const float Rf = rfi + fabsf(fj[u].w);
                    const float Rhi = Rf + delta, Rlo = Rf - delta;
                    if (!(dsqf > Rhi * Rhi * 1.0000039f)) {  // (1 + 2^-18): else surely outside
                        inside = Rlo > 0.f && dsqf < Rlo * Rlo * 0.9999962f;  // surely inside
                        if (!inside) {
                            const double4_32a pi = load_pos(S, i), pj = load_pos(S, j);
                            const double dx = image_dx(v, pi.x - pj.x);
                            const double dy = pi.y - pj.y;
                            const double dz = pi.z - pj.z;
                            const double distsq = dx * dx + dy * dy + dz * dz;
                            const double R = pi.w + pj.w + v.skin;
                            inside = distsq < R * R;
                        }
                    }
                }
                const unsigned hit = __ballot_sync(0xffffffffu, inside) & gmask;
                const int at = count + __popc(hit & below);
                if (inside && at < CAP) row[at] = j;
                count += __popc(hit);
            }
        }
    }
    __syncwarp();
    if (on && count > v.nei_cap && l == 0) atomicOr(&ctl->error, 0x1u);
    // the row by pId: an entry's place is the number of smaller pIds
    const int cs = count < CAP ? count : CAP;
    int* const id = ids + slot * kStride;
    for (int a = l; a < cs; a += kNbLanes) id[a] = pidv[row[a]];
    __syncwarp();
    for (int a = l; a < cs; a += kNbLanes) {
        const int key = id[a];
        int place = 0;
        for (int f = 0; f < cs; f++) place += id[f] < key ? 1 : 0;
        out[slot * kStride + place] = row[a];
    }
    const int m = cs < v.nei_cap ? cs : v.nei_cap;
    if (l == 0) {
        len[slot] = m;
        if (i < n) v.nnei[i] = m;
        if (on) {
            if constexpr (T::mixed) {
                v.refh[i] = make_float4(fi.x, fi.y, fi.z, 0.f);
            } else {
                const double4_32a pi = S.pos[i];
                v.ref[i] = make_double4_32a(pi.x, pi.y, pi.z, 0.0);
            }
        }
    }
    __syncthreads();
    const int p = threadIdx.x % kNbPer, pm = len[p];
    for (int k = threadIdx.x / kNbPer; k < pm; k += kNbLanes) v.nei[(size_t)k * n + i0 + p] = out[p * kStride + k];
    const int wmax = __reduce_max_sync(0xffffffffu, count);
    if (lane == 0 && wmax > 0) atomicMax(&ctl->max_nei, wmax);
}

template <class T, int CAP>
static void launch_neighbors(const View<T>& v, int gated, cudaStream_t st) {
    constexpr int bytes = (3 * kNbPer * (CAP + 1) + kNbPer) * (int)sizeof(int);
    // per device; beyond the default for the widest rows only
    if (bytes > 48 * 1024) cudaFuncSetAttribute(k_neighbors<T, CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    k_neighbors<T, CAP><<<(v.n + kNbPer - 1) / kNbPer, kNbBlock, bytes, st>>>(v, gated);
}

// ===================================================================== wall lists
// Mesh tree traversal with an explicit stack; a triangle joins the list when
// its AABB and its closest feature are within r + skin (BVH.cu:493-540, with
// sphereAABBOverlapNeighbor and dist_triangle_neighbor).  The set does not
// depend on the tree shape: an ancestor's box contains its leaves' boxes, so
// the box test never rejects an ancestor of a leaf that passes.  Rows are
// sorted by triangle index, as BVH.cu:538 does.

// children of mesh tree node (L, k), L > 0, pushed right first
__device__ __forceinline__ bool seg_push(unsigned* stack, int& sp, int L, int k, int ntri) {
    if (sp + 2 > kBvhStack) return false;
    const int below = (ntri + (1 << (L - 1)) - 1) >> (L - 1);
    const unsigned lv = (unsigned)(L - 1) << kSegShift;
    if (2 * k + 1 < below) stack[sp++] = lv | (unsigned)(2 * k + 1);
    stack[sp++] = lv | (unsigned)(2 * k);
    return true;
}
// Wall candidates of every occupied cell: the mesh tree's FP32 boxes (rounded
// outwards) traversed with the cell's box grown by v.cw_reach (every particle's
// cutoff r + skin, the mixed rows' widening, a margin) and rounded outwards too,
// every triangle whose box overlaps it, ascending.  An ancestor's box contains
// its leaves', and every rounding widens a box, so no leaf that a particle's own
// tree test (sphere against the triangle's box) would pass is left out.  A
// periodic x also takes the cell's box one period away where it reaches over an
// x face.  A cell with more than kCellWalls candidates (or kCellNodes nodes at
// some level of the tree), or one that finds the buffer full, is marked -1 and
// its particles traverse the tree themselves.
//
// kCwLanes lanes to a cell, level by level: the nodes that overlap the cell at
// one level are a list in shared memory, and the lanes test their children, one
// each, into the list of the level below; the triangles that remain are ranked
// by counting.  It is bound by the latency of the box loads, one per level here;
// a thread per cell with a stack paid it per node.  Rebuild of a bed of 30,000
// spheres 118 -> 17 us, of 250,000 143 -> 24, of a pour of 300,000 (200,000
// cells) 104 -> 51.  Beyond a million cells the chip is full and the lanes cost
// more than they hide: a channel of ten million spheres 1,010 -> 1,710, in a
// rebuild of 10 ms.  The cell's box is formed in FP32 with a margin for its
// rounding; in FP64 (64 cycles a warp instruction) a rebuild of a million spheres
// on a lattice over the chute took 997 us, now 932.
constexpr int kCellWalls = 96;
constexpr int kCellNodes = 128;
constexpr int kCwLanes = 8;
constexpr int kCwBlock = 128;

template <class T>
__global__ void __launch_bounds__(kCwBlock) k_cell_walls(View<T> v, int gated) {
    constexpr int kGroups = kCwBlock / kCwLanes;
    __shared__ int nodes_s[kGroups][2][kCellNodes], tris_s[kGroups][kCellWalls];
    Ctl* ctl = v.ctl;
    if (gated && ctl->refresh == 0u) return;
    const int lane = threadIdx.x & 31, l = threadIdx.x % kCwLanes, group = threadIdx.x / kCwLanes;
    const unsigned gmask = ((1u << kCwLanes) - 1u) << (lane & ~(kCwLanes - 1)), below = gmask & ((1u << lane) - 1u);
    const int cells = (int)ctl->ncell_list;
    const int first = lane & ~(kCwLanes - 1);
    // the cell's grown box, one bound a lane (lanes 0..2 the lower ones, 3..5 the
    // upper)
    const int axis = l % 3;
    const bool upper = l >= 3;
    const float w = axis == 0 ? v.cellw[0] : (axis == 1 ? v.cellw[1] : v.cellw[2]);
    const float reach = v.cw_reach + (T::mixed ? v.wall_delta : 0.f);
    const float edge = (axis == 0 ? v.boxf[0] : (axis == 1 ? v.boxf[1] : v.boxf[2])) + (upper ? reach : -reach);
    // whole warps take turns: the launch has a bounded number of them
    for (int c0 = blockIdx.x * kGroups + (threadIdx.x & ~31) / kCwLanes; c0 < cells; c0 += gridDim.x * kGroups) {
        const int c_idx = c0 + lane / kCwLanes;
        const bool on = c_idx < cells;
        const int q = v.cell_list[on ? c_idx : cells - 1];
        if (v.ntri == 0) {
            if (on && l == 0) v.cw_cnt[q] = 0;
            continue;
        }
        const uint32_t kq = v.keys[0][q];
        const int cc = (int)compact10(axis == 0 ? kq >> 2 : (axis == 1 ? kq >> 1 : kq)) - (upper ? 0 : 1);
        const float bound = fmaf((float)cc, w, edge);
        bool past_lo = false, past_hi = false;  // periodic x: over a face
        if (v.per_x) {
            past_lo = (__ballot_sync(0xffffffffu, l == 0 && bound < v.perf[0]) & gmask) != 0u;
            past_hi = (__ballot_sync(0xffffffffu, l == 3 && bound > v.perf[1]) & gmask) != 0u;
        }
        const bool twice = past_lo || past_hi;
        const int nimg = __any_sync(0xffffffffu, twice) ? 2 : 1;
        // the highest level with more than kCwLanes nodes below it is the first tested
        int top = v.seg_top;
        while (top > 0 && ((v.ntri + (1 << (top - 1)) - 1) >> (top - 1)) <= kCwLanes) top--;
        int* found = tris_s[group];
        int count = 0;
        bool full = false;
        for (int img = 0; img < nimg; img++) {
            const bool here = on && (img == 0 || twice);
            const float f = img == 1 && axis == 0 ? bound + (past_hi ? -v.Lxh : v.Lxh) : bound;
            float flo[3], fhi[3];
#pragma unroll
            for (int a = 0; a < 3; a++) {
                flo[a] = __shfl_sync(0xffffffffu, f, first + a);
                fhi[a] = __shfl_sync(0xffffffffu, f, first + 3 + a);
            }
            int m = 0;  // nodes of the level above that overlap (all lanes of the group alike)
            for (int L = top; L >= 0; L--) {
                const int nodes = (v.ntri + (1 << L) - 1) >> L;
                const int cands = !here || full ? 0 : (L == top ? nodes : 2 * m);
                const int most = __reduce_max_sync(0xffffffffu, cands);
                if (most == 0) break;  // none of the warp's cells reaches further down
                const int* src = nodes_s[group][L & 1];
                int* dst = L == 0 ? found : nodes_s[group][(L & 1) ^ 1];
                int got = L == 0 ? count : 0;
                for (int k0 = 0; k0 < most; k0 += kCwLanes) {
                    const int k = k0 + l;
                    int node = -1;
                    if (k < cands) node = L == top ? k : 2 * src[k >> 1] + (k & 1);
                    bool in = false;
                    if (node >= 0 && node < nodes) {
                        const SegBoxF B = v.segf[v.seg_off[L] + node];
                        in = !(B.lo[0] > fhi[0] || B.hi[0] < flo[0] || B.lo[1] > fhi[1] || B.hi[1] < flo[1] ||
                               B.lo[2] > fhi[2] || B.hi[2] < flo[2]);
                    }
                    const unsigned hit = __ballot_sync(0xffffffffu, in) & gmask;
                    const int at = got + __popc(hit & below);
                    got += __popc(hit);
                    if (in && at < (L == 0 ? kCellWalls : kCellNodes)) dst[at] = L == 0 ? v.seg_tri[node] : node;
                }
                if (got > (L == 0 ? kCellWalls : kCellNodes)) full = true;
                __syncwarp();
                m = full ? 0 : got;
                if (L == 0 && !full) count = got;
            }
        }
        if (full) count = 0;
        // a triangle met at both images counts once
        int drop = 0;
        if (nimg == 2) {
            for (int e = l; e < count; e += kCwLanes)
                for (int f = 0; f < e; f++)
                    if (found[f] == found[e]) {
                        drop |= 1 << (e / kCwLanes);
                        break;
                    }
            __syncwarp();
            for (int e = l; e < count; e += kCwLanes)
                if ((drop >> (e / kCwLanes)) & 1) found[e] = 0x7fffffff;
            __syncwarp();
        }
        int kept = 0;
        for (int e = l; e < count; e += kCwLanes) kept += found[e] != 0x7fffffff ? 1 : 0;
#pragma unroll
        for (int o = kCwLanes / 2; o > 0; o >>= 1) kept += __shfl_xor_sync(0xffffffffu, kept, o);
        int base = 0;
        if (on && l == 0 && kept > 0) base = (int)atomicAdd(&ctl->wall_alloc, (unsigned)kept);
        base = __shfl_sync(0xffffffffu, base, lane & ~(kCwLanes - 1));
        if (base + kept > v.cw_cap) full = true;
        if (on && l == 0) {
            v.cw_base[q] = base;
            v.cw_cnt[q] = full ? -1 : kept;
        }
        // ascending: a triangle's place is the number of smaller ones
        for (int e = l; on && !full && e < count; e += kCwLanes) {
            const int t = found[e];
            if (t == 0x7fffffff) continue;
            int place = 0;
            for (int f = 0; f < count; f++) place += found[f] < t ? 1 : 0;
            v.cw_list[base + place] = t;
        }
        __syncwarp();  // the lists are the next cells'
    }
}

// The cell wall candidates of particle i's cell (first sorted position q0 and
// count), or count -1 when its particles traverse the tree themselves.
template <class T>
__device__ __forceinline__ int cell_walls_of(const View<T>& v, int3 c, int& base) {
    const int cx = c.x, cy = c.y, cz = c.z;
    if (cx < 0 || cx >= v.sizex || cy < 0 || cy >= v.sizey || cz < 0 || cz >= v.sizez) return -1;
    const int cell = (v.sizey * cz + cy) * v.sizex + cx;
    if (v.cell_end[cell] <= v.cell_start[cell]) return -1;
    const int q0 = v.cell_start[cell];
    base = v.cw_base[q0];
    return v.cw_cnt[q0];
}

template <class T, int CAP>
__global__ void __launch_bounds__(kBlock) k_wall_lists(View<T> v, int gated) {
    Ctl* ctl = v.ctl;
    if (gated && ctl->refresh == 0u) return;
    const int n = v.n;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int s = ctl->s;
    int count = 0;
    if (i < n) {
        const SBank<T> S = v.S[s];
        if (S.rot[i].w == 0 || v.ntri == 0) {
            v.nneiw[i] = 0;
        } else if constexpr (T::mixed) {
            // FP32 traversal of the FP32 tree (boxes rounded outwards) and the
            // FP32 closest feature, with the cutoff widened by their error
            // bounds: the rows hold every triangle within r + skin (and maybe
            // a few more, which the step's exact overlap turns away), so the
            // contacts are those of the FP64 rows
            const float4 h = S.posh[i], l = S.posl[i];
            const float3 pl = make_float3(l.x, l.y, l.z);
            const float R = fabsf(h.w) + l.w + (float)v.skin + v.nb_delta + v.wall_delta;
            const float Rsq = R * R;
            int cand[CAP];
            bool overflow = false;
            int cbase = 0;
            const int ccnt = cell_walls_of(v, cell_of(v, S, i, h), cbase);
            if (ccnt >= 0) {
                // the cell's candidates, ascending: the row comes out sorted
                for (int k = 0; k < ccnt; k++) {
                    const int t = v.cw_list[cbase + k];
                    float3 qh = make_float3(h.x, h.y, h.z), ql = pl;
                    if (v.per_x) {
                        const float d = qh.x - v.trif[t].v0h[0];
                        if (d > v.halfLxf || d < -v.halfLxf) {
                            qh.x = d > 0.f ? qh.x - v.Lxh : qh.x + v.Lxh;
                            ql.x = 0.f;  // the period's low part is within the margin
                        }
                    }
                    const FeatureF f = closest_feature_f(qh, ql, Rsq, v.trif[t]);
                    if (!(f.dist < R)) continue;
                    if (count >= CAP) {
                        overflow = true;
                        break;
                    }
                    cand[count++] = t;
                }
            }
            unsigned stack[kBvhStack];
            const int nimg = ccnt >= 0 ? 0 : (v.per_x && (h.x + R > v.perf[1] || h.x - R < v.perf[0]) ? 2 : 1);
            for (int img = 0; img < nimg; img++) {
                float3 ph = make_float3(h.x, h.y, h.z);
                if (img == 1) ph.x = h.x + R > v.perf[1] ? h.x - v.Lxh : h.x + v.Lxh;
                int sp = 0;
                stack[sp++] = (unsigned)v.seg_top << kSegShift;
                while (sp > 0) {
                    const unsigned e = stack[--sp];
                    const int L = (int)(e >> kSegShift), nk = (int)(e & ((1u << kSegShift) - 1u));
                    const SegBoxF N = v.segf[v.seg_off[L] + nk];
                    const float dx = fmaxf(fmaxf(N.lo[0] - ph.x, ph.x - N.hi[0]), 0.f);
                    const float dy = fmaxf(fmaxf(N.lo[1] - ph.y, ph.y - N.hi[1]), 0.f);
                    const float dz = fmaxf(fmaxf(N.lo[2] - ph.z, ph.z - N.hi[2]), 0.f);
                    if (!(dx * dx + dy * dy + dz * dz <= Rsq)) continue;
                    if (L == 0) {
                        const int t = v.seg_tri[nk];
                        float3 qh = ph, ql = pl;
                        if (img == 1) ql.x = 0.f;  // the period's low part is within the margin
                        const FeatureF f = closest_feature_f(qh, ql, Rsq, v.trif[t]);
                        if (f.dist < R) {
                            if (count >= CAP) {
                                overflow = true;
                                continue;
                            }
                            int k = count;
                            while (k > 0 && cand[k - 1] > t) {
                                cand[k] = cand[k - 1];
                                k--;
                            }
                            cand[k] = t;
                            count++;
                        }
                    } else if (!seg_push(stack, sp, L, nk, v.ntri)) {
                        atomicOr(&ctl->error, 0x10u);
                        break;
                    }
                }
            }
            if (overflow || count > v.wall_cap) atomicOr(&ctl->error, 0x2u);
            const int m = count < v.wall_cap ? count : v.wall_cap;
            for (int k = 0; k < m; k++) v.neiw[(size_t)k * n + i] = cand[k];
            v.nneiw[i] = m;
        } else {
            const double4_32a pi = load_pos(S, i);
            const double py = pi.y, pz = pi.z;
            const double R = pi.w + v.skin;
            const double Rsq = R * R;
            int cand[CAP];
            bool overflow = false;
            int cbase = 0;
            const int ccnt = cell_walls_of(v, cell_of(v, S, i, v.posf[i]), cbase);
            if (ccnt >= 0) {
                // the cell's candidates, ascending, through the same two tests
                // as the traversal below (sphere against the triangle's box,
                // then the closest feature): the same row, already sorted
                for (int k = 0; k < ccnt; k++) {
                    const int t = v.cw_list[cbase + k];
                    const double px = image_x_near(v, pi.x, v.tri[t].v0[0]);
                    const double* bb = v.tri_aabb + 6 * (size_t)t;
                    if (!sphere_aabb(px, py, pz, Rsq, bb, bb + 3)) continue;
                    const Feature f = closest_feature(px, py, pz, Rsq, v.tri[t]);
                    if (!(f.dist < pi.w + v.skin)) continue;
                    if (count >= CAP) {
                        overflow = true;
                        break;
                    }
                    cand[count++] = t;
                }
            }
            unsigned stack[kBvhStack];
            // periodic x: a sphere within R of an x face also queries the mesh
            // at its image one period away (no triangle is found twice: the
            // mesh's triangles are narrower than a quarter period)
            const int nimg = ccnt >= 0 ? 0 : (v.per_x && (pi.x + R > v.maxx || pi.x - R < v.minx) ? 2 : 1);
            for (int img = 0; img < nimg; img++) {
                const double px = img == 0 ? pi.x : (pi.x + R > v.maxx ? pi.x - v.Lx : pi.x + v.Lx);
                int sp = 0;
                stack[sp++] = (unsigned)v.seg_top << kSegShift;
                while (sp > 0) {
                    const unsigned e = stack[--sp];
                    const int L = (int)(e >> kSegShift), nk = (int)(e & ((1u << kSegShift) - 1u));
                    const SegBox& B = v.seg[v.seg_off[L] + nk];
                    if (!sphere_aabb(px, py, pz, Rsq, B.lo, B.hi)) continue;
                    if (L == 0) {
                        const int t = v.seg_tri[nk];
                        const Feature f = closest_feature(px, py, pz, Rsq, v.tri[t]);
                        if (f.dist < pi.w + v.skin) {
                            if (count >= CAP) {
                                overflow = true;
                                continue;
                            }
                            int k = count;
                            while (k > 0 && cand[k - 1] > t) {
                                cand[k] = cand[k - 1];
                                k--;
                            }
                            cand[k] = t;
                            count++;
                        }
                    } else if (!seg_push(stack, sp, L, nk, v.ntri)) {
                        atomicOr(&ctl->error, 0x10u);
                        break;
                    }
                }
            }
            if (overflow || count > v.wall_cap) atomicOr(&ctl->error, 0x2u);
            const int m = count < v.wall_cap ? count : v.wall_cap;
            for (int k = 0; k < m; k++) v.neiw[(size_t)k * n + i] = cand[k];
            v.nneiw[i] = m;
        }
    }
    int wmax = count;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) wmax = max(wmax, __shfl_xor_sync(0xffffffffu, wmax, o));
    if ((threadIdx.x & 31) == 0 && wmax > 0) atomicMax(&ctl->max_wall, wmax);
    // the last block closes the rebuild: clear the request, count it
    if (last_block(&ctl->done[2])) {
        if (threadIdx.x == 0) {
            ctl->done[2] = 0;
            ctl->refresh = 0u;
            ctl->rebuilds += 1ull;
            ctl->lists_valid = 1;
            ctl->irefresh = 1u;  // new list rows (and storage order): new inner rows
        }
    }
}

// ===================================================================== inner rows
// Mixed mode: the partners of each list row within r_i + r_j + inner skin,
// in row order (so in partner-pId order), the wall-row triangles within
// r_i + inner skin (in row order), and the high-part positions they were taken
// at.  Both tests run in FP32, the pairs' on the high parts with the list
// prefilter's error bound added to the cutoff, the walls' closest feature with
// its own as well, so they keep all that is within the cutoff in exact
// arithmetic.  A pair left out is more than the inner skin
// apart, and it cannot touch before some particle has moved half the inner
// skin, when the step asks for new rows (ctl->irefresh); every list rebuild
// asks too.  Gated on that request in every launch mode.
constexpr int kInnerKeys = 8;
// row entries in flight per thread: 4 measured 180 us on the 1M bed, 8 and 16
// (more registers, fewer resident warps) 207 and 277 us
constexpr int kInnerUnroll = 4;

template <class T>
__global__ void __launch_bounds__(kBlock) k_inner(View<T> v) {
    Ctl* ctl = v.ctl;
    if (ctl->irefresh == 0u) return;
    const int n = v.n;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const float skin = ctl->inner_next;
    if constexpr (T::mixed) {
        if (i < n) {
            const SBank<T> S = v.S[ctl->s];
            const float4 hi = S.posh[i];
            int m = 0;
            if (hi.w > 0.f) {
                const int nn = v.nnei[i];
                const float cut = skin + v.nb_delta;
                const bool hints = v.row_mask != 0xFFFFFFFFu;
                const PBank<T> P = v.P[ctl->p];
                // the first kInnerKeys history keys in registers for the
                // slot hints (the rest, rarely used, read when needed)
                const int nc = hints ? P.nc[i] : 0;
                int hk[kInnerKeys];
#pragma unroll
                for (int q = 0; q < kInnerKeys; q++) hk[q] = q < nc ? P.hid[(size_t)q * n + i] : -1;
                // kInnerUnroll row entries at a time, their gathers in flight together
                for (int k0 = 0; k0 < nn; k0 += kInnerUnroll) {
                    int jj[kInnerUnroll];
                    float4 hj[kInnerUnroll];
#pragma unroll
                    for (int u = 0; u < kInnerUnroll; u++) jj[u] = k0 + u < nn ? v.nei[(size_t)(k0 + u) * n + i] : -1;
#pragma unroll
                    for (int u = 0; u < kInnerUnroll; u++)
                        if (jj[u] >= 0) hj[u] = S.posh[jj[u]];
#pragma unroll
                    for (int u = 0; u < kInnerUnroll; u++) {
                        const int j = jj[u];
                        if (j < 0 || !(hj[u].w > 0.f)) continue;  // inactive for good
                        const float dx = image_dxf(v, hi.x - hj[u].x), dy = hi.y - hj[u].y, dz = hi.z - hj[u].z;
                        const float R = hi.w + hj[u].w + cut;
                        if (!(dx * dx + dy * dy + dz * dz < R * R * 1.0000039f)) continue;
                        if (m < v.nei_cap) {
                            // the partner's history slot, if it has one, as a hint
                            int e = j;
                            if (hints) {
                                int q = -1;
#pragma unroll
                                for (int a = 0; a < kInnerKeys; a++)
                                    if (q < 0 && hk[a] == j) q = a;
                                for (int a = kInnerKeys; q < 0 && a < nc && a < 63; a++)
                                    if (P.hid[(size_t)a * n + i] == j) q = a;
                                if (q >= 0) e = j | ((q + 1) << kHintShift);
                            }
                            v.inn[(size_t)m * n + i] = e;
                        }
                        m++;
                    }
                }
            }
            v.ninn[i] = m < v.nei_cap ? m : v.nei_cap;
            int mw = 0;
            if (hi.w > 0.f && v.ntri > 0) {
                // FP32 closest feature with the cutoff widened by its error bound
                const float4 lo = S.posl[i];
                const float R = hi.w + lo.w + skin + v.nb_delta + v.wall_delta;
                const int nw = v.nneiw[i];
                for (int k = 0; k < nw; k++) {
                    const int t = v.neiw[(size_t)k * n + i];
                    float3 ph = make_float3(hi.x, hi.y, hi.z), pl = make_float3(lo.x, lo.y, lo.z);
                    if (v.per_x) {
                        const float d = ph.x - v.trif[t].v0h[0];
                        if (d > v.halfLxf || d < -v.halfLxf) {
                            ph.x = d > 0.f ? ph.x - v.Lxh : ph.x + v.Lxh;
                            pl.x = 0.f;  // within the margin
                        }
                    }
                    const FeatureF f = closest_feature_f(ph, pl, R * R, v.trif[t]);
                    if (f.dist < R) v.innw[(size_t)mw++ * n + i] = t;
                }
            }
            v.ninnw[i] = mw;
            v.refi[i] = make_float4(hi.x, hi.y, hi.z, 0.f);
        }
    }
    if (last_block(&ctl->done[3])) {
        if (threadIdx.x == 0) {
            ctl->done[3] = 0;
            ctl->irefresh = 0u;
            ctl->inner_thresh_sq = 0.25f * skin * skin;
            // Rows that lasted under 5 steps (a list rebuild aside, which ends them
            // early) get a wider skin the next time, rows that lasted over 10 a
            // narrower one: a build interrupts the chain of steps (50 us on a pour of
            // 300,000 spheres, where every third step asked for one: 71 -> 66 us a
            // step, and 104 -> 98 once the spheres pile up); on beds the rows last
            // hundreds of steps and the skin stays.  Results do not depend on it.
            const unsigned long long lasted = ctl->steps - ctl->inner_at;
            const bool own = ctl->inner_builds > 0ull && ctl->inner_lists == ctl->rebuilds;
            ctl->inner_at = ctl->steps;
            ctl->inner_lists = ctl->rebuilds;
            if (v.inner_adapt && own) {
                if (lasted < 5ull) ctl->inner_next = fminf(skin * 1.25f, v.skinf);
                else if (lasted > 10ull) ctl->inner_next = fmaxf(skin / 1.25f, v.inner_skinf);
            }
            ctl->inner_builds += 1ull;
        }
    }
}

// ===================================================================== step chains
__global__ void k_chain_start(Ctl* ctl, int steps, int span, int inner) {
    ctl->remaining = steps;
    ctl->span = span;
    ctl->hold = ctl->refresh != 0u || (inner && ctl->irefresh != 0u) ? 1u : 0u;
}
__global__ void k_chain_any(Ctl* ctl, int inner, cudaGraphConditionalHandle any, cudaGraphConditionalHandle loop) {
    ctl->hold = 0u;
    cudaGraphSetConditional(any, ctl->refresh != 0u || (inner && ctl->irefresh != 0u) ? 1u : 0u);
    cudaGraphSetConditional(loop, ctl->remaining > 0 ? 1u : 0u);
}
__global__ void k_chain_which(Ctl* ctl, int inner, int has_often, cudaGraphConditionalHandle lists,
                              cudaGraphConditionalHandle in, cudaGraphConditionalHandle often) {
    const unsigned r = ctl->refresh;
    cudaGraphSetConditional(lists, r != 0u ? 1u : 0u);
    // a list rebuild makes new inner rows itself
    if (inner) cudaGraphSetConditional(in, r == 0u && ctl->irefresh != 0u ? 1u : 0u);
    if (!has_often) return;
    const unsigned long long lasted = ctl->steps - ctl->asked_at;
    ctl->asked_at = ctl->steps;
    cudaGraphSetConditional(often, ctl->remaining > 0 && lasted <= (unsigned long long)ctl->span ? 1u : 0u);
}
__global__ void k_chain_again(Ctl* ctl, cudaGraphConditionalHandle loop) {
    cudaGraphSetConditional(loop, ctl->remaining > 0 ? 1u : 0u);
}
void launch_chain_start(Ctl* ctl, int steps, int span, int inner, cudaStream_t st) {
    k_chain_start<<<1, 1, 0, st>>>(ctl, steps, span, inner);
}
void launch_chain_any(Ctl* ctl, int inner, cudaGraphConditionalHandle any, cudaGraphConditionalHandle loop,
                      cudaStream_t st) {
    k_chain_any<<<1, 1, 0, st>>>(ctl, inner, any, loop);
}
void launch_chain_which(Ctl* ctl, int inner, int has_often, cudaGraphConditionalHandle lists,
                        cudaGraphConditionalHandle in, cudaGraphConditionalHandle often, cudaStream_t st) {
    k_chain_which<<<1, 1, 0, st>>>(ctl, inner, has_often, lists, in, often);
}
void launch_chain_again(Ctl* ctl, cudaGraphConditionalHandle loop, cudaStream_t st) {
    k_chain_again<<<1, 1, 0, st>>>(ctl, loop);
}

static inline int grid_for(int n) { return (n + kBlock - 1) / kBlock; }

template <class T>
void launch_inner(const View<T>& v, cudaStream_t st) {
    if (T::mixed && v.inner_on) k_inner<T><<<grid_for(v.n), kBlock, 0, st>>>(v);
}
template void launch_inner<FP64>(const View<FP64>&, cudaStream_t);
template void launch_inner<Mixed>(const View<Mixed>&, cudaStream_t);

template <class T>
void launch_rebuild(const View<T>& v, cudaStream_t st, int force) {
    const int gated = force ? 0 : 1;
    const int n = v.n;
    const int g = grid_for(n);
    k_keys<T><<<g, kBlock, 0, st>>>(v, gated);
    rs_passes(v.keys[0], v.vals[0], v.keys[1], v.vals[1], v.rs_hist, v.rs_tot, n, v.rs_blocks, 0, 4, st,
              v.ctl, gated);
    if (v.reorder) {
        if (v.store_forces) {
            k_reorder_forces<T><<<g, kBlock, 0, st>>>(v, gated);
            k_copy_forces<T><<<g, kBlock, 0, st>>>(v, gated);
        }
        if constexpr (T::mixed) k_inverse_order<T><<<g, kBlock, 0, st>>>(v, gated);
        k_reorder<T><<<g, kBlock, 0, st>>>(v, gated);
    }
    const int gc = grid_for(v.ncells) < 4096 ? grid_for(v.ncells) : 4096;
    k_cells_clear<T><<<gc, kBlock, 0, st>>>(v, gated);
    k_cell_ranges<T><<<g, kBlock, 0, st>>>(v, gated);
    k_cell_count<T><<<g, kBlock, 0, st>>>(v, gated);
    k_cell_scan<T><<<1, 1024, 0, st>>>(v, gated, g);
    k_cell_emit<T><<<g, kBlock, 0, st>>>(v, gated);
    if constexpr (!T::mixed) k_posf<T><<<g, kBlock, 0, st>>>(v, gated);
    if (v.nei_cap <= 32)
        launch_neighbors<T, 32>(v, gated, st);
    else if (v.nei_cap <= 64)
        launch_neighbors<T, 64>(v, gated, st);
    else
        launch_neighbors<T, 128>(v, gated, st);
    // a group of lanes per occupied cell, of which there are n at most; a bounded
    // number of CTAs, since most of one per 16 particles would find no cell left
    const int gw = (n + kCwBlock / kCwLanes - 1) / (kCwBlock / kCwLanes);
    k_cell_walls<T><<<gw < 4096 ? gw : 4096, kCwBlock, 0, st>>>(v, gated);
    if (v.wall_cap <= 16)
        k_wall_lists<T, 16><<<g, kBlock, 0, st>>>(v, gated);
    else if (v.wall_cap <= 32)
        k_wall_lists<T, 32><<<g, kBlock, 0, st>>>(v, gated);
    else
        k_wall_lists<T, 64><<<g, kBlock, 0, st>>>(v, gated);
    launch_inner(v, st);
}

template void launch_rebuild<FP64>(const View<FP64>&, cudaStream_t, int);
template void launch_rebuild<Mixed>(const View<Mixed>&, cudaStream_t, int);
template void launch_finalize_oob<FP64>(const View<FP64>&, cudaStream_t);
template void launch_finalize_oob<Mixed>(const View<Mixed>&, cudaStream_t);

// ===================================================================== mesh
// Per-triangle precompute of load_ascii_stl_double (TriangleMesh.cu:560-630)
// from welded vertices (tv = sorted vertex ids, te = edge ids + nShift) and
// the raw third corner (the plane offset uses it, TriangleMesh.cu:607) or,
// when raw3 is null, the plane offsets the loader already computed (dplane),
// plus the centroid Morton key of mortonKeyGen (TriangleMesh.cu:4-21).
__global__ void k_tri_precompute(TriRec* rec, uint32_t* morton, int* idx, const double* vx,
                                 const double* vy, const double* vz, const int* tv, const int* te,
                                 const double* raw3, const double* dplane, int ntri, double gminx, double gminy,
                                 double gminz, double irx, double iry, double irz) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntri) return;
    const int a = tv[3 * t + 0], b = tv[3 * t + 1], c = tv[3 * t + 2];
    TriRec R;
    R.v0[0] = vx[a]; R.v0[1] = vy[a]; R.v0[2] = vz[a];
    R.v1[0] = vx[b]; R.v1[1] = vy[b]; R.v1[2] = vz[b];
    R.v2[0] = vx[c]; R.v2[1] = vy[c]; R.v2[2] = vz[c];
    for (int k = 0; k < 3; k++) {
        R.e01[k] = R.v1[k] - R.v0[k];
        R.e02[k] = R.v2[k] - R.v0[k];
        R.e12[k] = R.v2[k] - R.v1[k];
    }
    const double d00 = R.e01[0] * R.e01[0] + R.e01[1] * R.e01[1] + R.e01[2] * R.e01[2];
    const double d01 = R.e01[0] * R.e02[0] + R.e01[1] * R.e02[1] + R.e01[2] * R.e02[2];
    const double d11 = R.e02[0] * R.e02[0] + R.e02[1] * R.e02[1] + R.e02[2] * R.e02[2];
    const double d22 = R.e12[0] * R.e12[0] + R.e12[1] * R.e12[1] + R.e12[2] * R.e12[2];
    R.d00 = d00;
    R.d01 = d01;
    R.d11 = d11;
    R.d00inv = 1. / d00;
    R.d11inv = 1. / d11;
    R.d22inv = 1. / d22;
    R.denom = 1. / (d00 * d11 - d01 * d01);
    // n = normalize(e01 x e02)
    double nx = R.e01[1] * R.e02[2] - R.e01[2] * R.e02[1];
    double ny = R.e01[2] * R.e02[0] - R.e01[0] * R.e02[2];
    double nz = R.e01[0] * R.e02[1] - R.e01[1] * R.e02[0];
    const double inv = 1. / sqrt(nx * nx + ny * ny + nz * nz);
    nx = inv * nx;
    ny = inv * ny;
    nz = inv * nz;
    R.n[0] = nx;
    R.n[1] = ny;
    R.n[2] = nz;
    if (raw3) {
        const double x = raw3[3 * t + 0], y = raw3[3 * t + 1], z = raw3[3 * t + 2];
        R.d = -nx * x - ny * y - nz * z;
    } else {
        R.d = dplane[t];
    }
    R.i0 = a;
    R.i1 = b;
    R.i2 = c;
    R.e0 = te[3 * t + 0];
    R.e1 = te[3 * t + 1];
    R.e2 = te[3 * t + 2];
    rec[t] = R;
    const double cx = (R.v0[0] + R.v1[0] + R.v2[0]) / 3.0;
    const double cy = (R.v0[1] + R.v1[1] + R.v2[1]) / 3.0;
    const double cz = (R.v0[2] + R.v1[2] + R.v2[2]) / 3.0;
    const uint32_t ix = (uint32_t)((cx - gminx) * irx);
    const uint32_t iy = (uint32_t)((cy - gminy) * iry);
    const uint32_t iz = (uint32_t)((cz - gminz) * irz);
    morton[t] = morton3(ix, iy, iz);
    idx[t] = t;
}

void launch_tri_precompute(TriRec* rec, uint32_t* morton, int* idx, const double* vx,
                           const double* vy, const double* vz, const int* tv, const int* te,
                           const double* raw3, const double* dplane, int ntri, const double* gmin,
                           const double* invrange, cudaStream_t st) {
    if (ntri <= 0) return;
    k_tri_precompute<<<grid_for(ntri), kBlock, 0, st>>>(rec, morton, idx, vx, vy, vz, tv, te, raw3, dplane,
                                                        ntri, gmin[0], gmin[1], gmin[2], invrange[0],
                                                        invrange[1], invrange[2]);
}

// Centroid keys of the triangles from their records (the key formula of
// k_tri_precompute), for rebuilding the tree of a mesh already set.
__global__ void k_tri_keys(const TriRec* rec, uint32_t* morton, int* idx, int ntri, double gminx, double gminy,
                           double gminz, double irx, double iry, double irz) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntri) return;
    const TriRec& R = rec[t];
    const double cx = (R.v0[0] + R.v1[0] + R.v2[0]) / 3.0;
    const double cy = (R.v0[1] + R.v1[1] + R.v2[1]) / 3.0;
    const double cz = (R.v0[2] + R.v1[2] + R.v2[2]) / 3.0;
    const uint32_t ix = (uint32_t)((cx - gminx) * irx);
    const uint32_t iy = (uint32_t)((cy - gminy) * iry);
    const uint32_t iz = (uint32_t)((cz - gminz) * irz);
    morton[t] = morton3(ix, iy, iz);
    idx[t] = t;
}

void launch_tri_keys(const TriRec* rec, uint32_t* morton, int* idx, int ntri, const double* gmin,
                     const double* invrange, cudaStream_t st) {
    if (ntri <= 0) return;
    k_tri_keys<<<grid_for(ntri), kBlock, 0, st>>>(rec, morton, idx, ntri, gmin[0], gmin[1], gmin[2], invrange[0],
                                                  invrange[1], invrange[2]);
}

// ---- mesh tree: built per 256 sorted triangles in shared memory by one CTA
// each, the levels above by the last CTA to finish (atomic counter, no
// waiting).

__host__ __device__ __forceinline__ int seg_count(int n, int level) {
    return (int)(((long long)n + (1ll << level) - 1) >> level);
}
__host__ __device__ __forceinline__ int seg_offset(int n, int level) {
    int off = 0;
    for (int L = 0; L < level; L++) off += seg_count(n, L);
    return off;
}
int seg_levels(int n) {
    int L = 0;
    while (seg_count(n, L) > 1) L++;
    return L + 1;
}
int seg_count_host(int n, int level) { return seg_count(n, level); }
int seg_offset_host(int n, int level) { return seg_offset(n, level); }

// The tree's comparisons and conversions by integer operations (a warp's FP64
// instruction takes 64 cycles, and a tree of a few hundred triangles sits on one
// or two SMs: its step of 2,000 spheres 25.0 -> 22.6 us): a < b of finite values, and x rounded down or up to FP32, which
// outside FP32's normal range is left to the conversion.
__device__ __forceinline__ bool less64(double a, double b) {
    long long x = __double_as_longlong(a), y = __double_as_longlong(b);
    x ^= (x >> 63) & 0x7fffffffffffffffll;
    y ^= (y >> 63) & 0x7fffffffffffffffll;
    return x < y;
}
template <bool UP>
__device__ __forceinline__ float round64(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned e = (hi >> 20) & 0x7ffu;
    if (e - 897u >= 253u) return UP ? __double2float_ru(x) : __double2float_rd(x);
    const unsigned cut = ((__funnelshift_l(lo, hi, 3) - (896u << 23)) & 0x7fffffffu) | (hi & 0x80000000u);
    const bool away = (lo & 0x1fffffffu) != 0u && (UP ? !(hi >> 31) : (bool)(hi >> 31));
    return __uint_as_float(cut + (away ? 1u : 0u));
}

__device__ __forceinline__ SegBox seg_union(const SegBox& a, const SegBox& b) {
    SegBox c;
    for (int k = 0; k < 3; k++) {
        c.lo[k] = less64(a.lo[k], b.lo[k]) ? a.lo[k] : b.lo[k];
        c.hi[k] = less64(b.hi[k], a.hi[k]) ? a.hi[k] : b.hi[k];
    }
    return c;
}

// boxes written by other CTAs: read through L2
__device__ __forceinline__ SegBox seg_load_cg(const SegBox* p) {
    SegBox b;
    for (int k = 0; k < 3; k++) {
        b.lo[k] = __ldcg(&p->lo[k]);
        b.hi[k] = __ldcg(&p->hi[k]);
    }
    return b;
}

constexpr int kSegTile = 256;
constexpr int kSegTileLevels = 9;  // levels 0..8 inside one CTA's 256 leaves

// box and its FP32 copy (rounded outwards)
__device__ __forceinline__ void put_box(SegBox* seg, SegBoxF* segf, int i, const SegBox& b) {
    seg[i] = b;
    SegBoxF f;
    for (int k = 0; k < 3; k++) {
        f.lo[k] = round64<false>(b.lo[k]);
        f.hi[k] = round64<true>(b.hi[k]);
    }
    segf[i] = f;
}

__global__ void __launch_bounds__(kSegTile) k_mesh_tree(const double* aabb, const int* sorted_idx, SegBox* seg,
                                                         SegBoxF* segf, unsigned* done, int n) {
    __shared__ SegBox sb[kSegTile];
    const int tid = threadIdx.x;
    const int l = blockIdx.x * kSegTile + tid;
    if (l < n) {
        const int t = sorted_idx[l];
        SegBox b;
        for (int k = 0; k < 3; k++) {
            b.lo[k] = aabb[6 * t + k];
            b.hi[k] = aabb[6 * t + 3 + k];
        }
        put_box(seg, segf, l, b);
        sb[tid] = b;
    }
    __syncthreads();
    // levels 1..8 of this CTA's leaves
    for (int L = 1; L < kSegTileLevels; L++) {
        const int span = 1 << L;
        const int local = tid * span;             // first leaf (CTA-relative) of node tid at level L
        const int k = (blockIdx.x * kSegTile >> L) + tid;
        const bool live = local < kSegTile && k < seg_count(n, L);
        SegBox c;
        if (live) {
            c = sb[local];
            const int right = local + (span >> 1);
            if (blockIdx.x * kSegTile + right < n) c = seg_union(c, sb[right]);
        }
        __syncthreads();
        if (live) {
            sb[local] = c;
            put_box(seg, segf, seg_offset(n, L) + k, c);
        }
        __syncthreads();
    }
    // the levels above the CTAs, by the last CTA to finish
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (tid == 0) last = atomicAdd(done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    int L = kSegTileLevels;  // the lowest level not built yet
    // through L2 while the level below holds more boxes than one tile
    for (; seg_count(n, L - 1) > kSegTile; L++) {
        const int cnt = seg_count(n, L), below = seg_count(n, L - 1);
        const int ob = seg_offset(n, L - 1), oc = seg_offset(n, L);
        for (int k = tid; k < cnt; k += blockDim.x) {
            SegBox c = seg_load_cg(seg + ob + 2 * k);
            if (2 * k + 1 < below) c = seg_union(c, seg_load_cg(seg + ob + 2 * k + 1));
            put_box(seg, segf, oc + k, c);
        }
        __threadfence();
        __syncthreads();
    }
    // the rest from one tile of the level below, in shared memory: node k of
    // m levels up sits at entry k 2^m of the tile
    const int cb = seg_count(n, L - 1);
    if (cb > 1) {
        if (tid < cb) sb[tid] = seg_load_cg(seg + seg_offset(n, L - 1) + tid);
        __syncthreads();
        for (int m = 1; (cb + (1 << (m - 1)) - 1) >> (m - 1) > 1; m++) {
            const int span = 1 << m;
            const int local = tid * span;
            const bool live = local < cb;
            SegBox c;
            if (live) {
                c = sb[local];
                const int right = local + (span >> 1);
                if (right < cb) c = seg_union(c, sb[right]);
            }
            __syncthreads();
            if (live) {
                sb[local] = c;
                put_box(seg, segf, seg_offset(n, L - 1 + m) + tid, c);
            }
            __syncthreads();
        }
    }
    if (tid == 0) *done = 0u;
}

void launch_bvh_build(const double* aabb, const int* sorted_idx, SegBox* seg, SegBoxF* segf, unsigned* done,
                      int ntri, cudaStream_t st) {
    if (ntri <= 0) return;
    k_mesh_tree<<<(ntri + kSegTile - 1) / kSegTile, kSegTile, 0, st>>>(aabb, sorted_idx, seg, segf, done, ntri);
}

// the segment tree's nodes: every level up to the root, and at least the
// levels one CTA writes
size_t bvh_scratch_bytes(int ntri) {
    if (ntri <= 0) return 0;
    const int levels = seg_levels(ntri) > kSegTileLevels ? seg_levels(ntri) : kSegTileLevels;
    return sizeof(SegBox) * (size_t)seg_offset(ntri, levels);
}

// FP32 copy of the triangles for the mixed-precision step kernel, and the
// low parts of its normal and corner-0 edges.
__global__ void k_trif(const TriRec* tri, TriRecF* out, TriLoF* lo, int ntri) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntri) return;
    const TriRec& T = tri[t];
    TriRecF F;
    TriLoF L;
    for (int k = 0; k < 3; k++) {
        split2(T.v0[k], F.v0h[k], F.v0l[k]);
        split2(T.n[k], F.n[k], L.nl[k]);
        split2(T.e01[k], F.e01[k], L.e01l[k]);
        split2(T.e02[k], F.e02[k], L.e02l[k]);
        F.e12[k] = (float)T.e12[k];
        L.pad[k] = 0.f;
    }
    F.d00 = (float)T.d00; F.d01 = (float)T.d01; F.d11 = (float)T.d11; F.denom = (float)T.denom;
    F.d00inv = (float)T.d00inv; F.d11inv = (float)T.d11inv; F.d22inv = (float)T.d22inv;
    F.i0 = T.i0; F.i1 = T.i1; F.i2 = T.i2; F.e0 = T.e0; F.e1 = T.e1; F.e2 = T.e2;
    F.pad = 0;
    out[t] = F;
    lo[t] = L;
}

void launch_trif(const TriRec* tri, TriRecF* out, TriLoF* lo, int ntri, cudaStream_t st) {
    if (ntri <= 0) return;
    k_trif<<<grid_for(ntri), kBlock, 0, st>>>(tri, out, lo, ntri);
}

// ===================================================================== probes
__global__ void k_dist_triangle(const TriRec* tri, const double* pos, const double* r, const int* t,
                                int m, double* out4, int* hit) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= m) return;
    const double rr = r[q];
    const double rsq = rr * rr;
    const Feature f = closest_feature(pos[3 * q], pos[3 * q + 1], pos[3 * q + 2], rsq, tri[t[q]]);
    out4[4 * q + 0] = f.nx;
    out4[4 * q + 1] = f.ny;
    out4[4 * q + 2] = f.nz;
    out4[4 * q + 3] = f.dist;
    hit[q] = f.dist < 1e9 ? f.hit : -2;
}

void launch_dist_triangle(const TriRec* tri, const double* pos, const double* r, const int* t, int m,
                          double* out4, int* hit, cudaStream_t st) {
    if (m <= 0) return;
    k_dist_triangle<<<grid_for(m), kBlock, 0, st>>>(tri, pos, r, t, m, out4, hit);
}

}  // namespace gdem
