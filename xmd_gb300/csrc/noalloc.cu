// noalloc.cu - a Verlet pair search that allocates no device memory.
//
// Some callers of this library cannot call cudaMalloc at the point where they
// need a pair list: code that runs while a CUDA graph is being captured on its
// stream (an allocation there is not captured and may break the capture),
// hosts whose device memory is owned by a fixed pool or by a framework's
// caching allocator, and tight loops that cannot afford the implicit device
// synchronisation of cudaMalloc / cudaFree.  For them,
// xmd_gpu_verlet_pairs_noalloc() takes device buffers for all inputs and
// outputs and keeps the scratch of its cell list (bucket counts, starts and
// fills, bucket-sorted bead indices, per-bead row counts and offsets) in the
// file-scope array below: about 10 MiB that every GPU which loads the
// library holds until the process exits.
//
// The search itself is the one the engine runs at every Verlet rebuild:
// pairs i < j, not in the same chain with |seq_i - seq_j| < 3
// (legacy_update.cpp:24-26), whose minimum-image distance is below the
// cutoff (legacy_update.cpp:28-29), in (i, j) order.
//
// Eight launches, all over the whole grid: bounds and grid, bucket counts,
// their scan, the bucket sort (with FP32 coordinates beside the indices), row
// counts, their scan, the rows.  Rows are bound by instruction issue: one warp
// takes one bead, in bucket order, and its lanes the candidates of the
// neighbouring buckets 32 at a time, so a bead's latency chain is a few
// rounds instead of one candidate after another.  A candidate is decided in
// FP32 unless its distance lies in the FP32 error band around the cutoff,
// where the FP64 test decides (GB300 runs an FP64 warp instruction over 16
// cycles; FP64 throughout would make the search FP64-bound).  The count keeps
// rows of up to NA_KEEP partners, put in order in registers, so that writing
// them is a copy; a longer row is searched again and put in order by rank in
// shared memory up to NA_ROW partners, beyond that by insertion in global
// memory, O(m^2) for m partners (a periodic box under two cutoffs wide, a
// cluster much denser than a protein).
//
// 30,720 beads at 1e-3 A^-3, cutoff 20 A: 3,200 us -> 96 us (one block for
// the grid took 250 us of it, and one thread per row, twice, 1,500 us each;
// searching every row twice 12 us).
#include <cuda_runtime.h>

#include <climits>
#include <cstdint>
#include <mutex>
#include <stdexcept>
#include <string>

#include "../../include/xmd_gpu.h"
#include "engine.h"

namespace xmdg {
namespace {

constexpr int NA_MAX = XMD_NOALLOC_MAX_BEADS;   // beads, and buckets
static_assert(NA_MAX <= 65536, "kept partners are 16 bits wide");
constexpr int NA_SCAN = 1024;                   // elements per scan block
constexpr int NA_PARTS = NA_MAX / NA_SCAN;
constexpr int NA_ROW = 512;                     // partners of a row ordered in shared memory
constexpr int NA_KEEP = 64;                     // partners of a row that the count keeps for the output
constexpr int NA_WARPS = 8;
constexpr int NA_PACK = 1023;                   // cell coordinates that fit the packed form

struct __align__(16) NaScratch {
    int start[NA_MAX];     // bucket counts, then starts within their scan block
    int row[NA_MAX];       // sort cursors per bucket; then row counts, then row offsets within their scan block
    float4 items[NA_MAX];  // beads in bucket order: FP32 coordinates and the bead's index
    int cell[NA_MAX];      // packed cell coordinates of each bead (or its bucket, when they do not fit)
    uint16_t kept[NA_MAX][NA_KEEP];   // rows of up to NA_KEEP partners, in order (an index is below NA_MAX)
    int start_base[NA_PARTS], row_base[NA_PARTS], part[NA_PARTS];
    unsigned long long lo_key[3], hi_key[3];
    unsigned done[3];
    // grid of the current call
    int per[3], dims[3], nbuckets, direct, packed;
    int far;               // some bead lies so many boxes away that its wrapped FP32 coordinate is off
    double lo[3], inv_edge, box[3], box_inv[3];
    float blo, bhi, L[3];  // FP32 decision band of the squared distance; box lengths
};

// The scratch.  Every call reuses it and leaves its contents behind; each
// call clears what has to start at zero.  Calls that overlap on the GPU (two
// streams, or a second call before the first finishes on another stream)
// race on it.
static __device__ __align__(256) NaScratch g_na_scratch;

// doubles as unsigned integers of the same order
__device__ __forceinline__ unsigned long long na_key_of(double x) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x);
    return (u >> 63) ? ~u : u | 0x8000000000000000ull;
}
__device__ __forceinline__ double na_of_key(unsigned long long k) {
    return __longlong_as_double((long long)((k >> 63) ? k & 0x7fffffffffffffffull : ~k));
}

__device__ __forceinline__ int na_coord(const NaScratch &s, int a, double x) {
    if (s.per[a]) {
        double f = x * s.box_inv[a];
        f -= floor(f);
        int k = (int)(f * s.dims[a]);
        return k < 0 ? 0 : (k >= s.dims[a] ? s.dims[a] - 1 : k);
    }
    int k = (int)floor((x - s.lo[a]) * s.inv_edge);
    return k < 0 ? 0 : k;
}
// bucket of a cell: the cell itself on a grid that is periodic along every
// axis and fits, hashed otherwise
__device__ __forceinline__ int na_bucket(const NaScratch &s, int cx, int cy, int cz) {
    if (s.direct) return (cz * s.dims[1] + cy) * s.dims[0] + cx;
    uint32_t h = (uint32_t)cx * 73856093u ^ (uint32_t)cy * 19349663u ^ (uint32_t)cz * 83492791u;
    h ^= h >> 15;
    return (int)(h & (uint32_t)(s.nbuckets - 1));
}
__device__ __forceinline__ double na_dist(const NaScratch &s, const double *r, int i, int j) {
    double d[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        double x = __dsub_rn(r[3 * j + a], r[3 * i + a]);
        d[a] = __dsub_rn(x, __dmul_rn(s.box[a], rint(__dmul_rn(x, s.box_inv[a]))));
    }
    return __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(d[0], d[0]), __dmul_rn(d[1], d[1])), __dmul_rn(d[2], d[2])));
}
__device__ __forceinline__ float na_image(float d, float L) {
    const float h = 0.5f * L;
    d = d > h ? d - L : d;
    return d < -h ? d + L : d;
}

__global__ void __launch_bounds__(256) k_na_clear(NaScratch *s) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < NA_MAX) {
        s->start[i] = 0;
        s->row[i] = 0;
    }
    if (i == 0) s->far = 0;
    if (i < 3) {
        s->lo_key[i] = ~0ull;
        s->hi_key[i] = 0ull;
        s->done[i] = 0u;
    }
}

// bounds along the open axes; the last block sets the grid and the FP32 band
__global__ void __launch_bounds__(256) k_na_grid(NaScratch *s, const double *__restrict__ r, int n, double c0,
                                                 double c1, double c2, double cutoff) {
    const double cell[3] = {c0, c1, c2};
    const int t = threadIdx.x, lane = t & 31;
    __shared__ int last;
    for (int a = 0; a < 3; ++a) {
        if (cell[a] != 0.0) continue;
        double lo = 1e300, hi = -1e300;
        for (int i = blockIdx.x * 256 + t; i < n; i += gridDim.x * 256) {
            const double x = r[3 * i + a];
            lo = fmin(lo, x);
            hi = fmax(hi, x);
        }
        for (int o = 16; o; o >>= 1) {
            lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (lane == 0) {
            atomicMin(&s->lo_key[a], na_key_of(lo));
            atomicMax(&s->hi_key[a], na_key_of(hi));
        }
    }
    __syncthreads();
    if (t == 0) {
        __threadfence();
        last = atomicAdd(&s->done[0], 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last || t != 0) return;
    __threadfence();
    const double edge = cutoff * (1.0 + 1e-9);
    double ext = cutoff;
    bool direct = true, packed = true;
    long long total = 1;
    for (int a = 0; a < 3; ++a) {
        s->box[a] = cell[a];
        s->box_inv[a] = cell[a] != 0.0 ? 1.0 / cell[a] : 0.0;
        s->per[a] = cell[a] != 0.0;
        s->L[a] = (float)cell[a];
        int dm = 1;
        if (cell[a] != 0.0) {
            const double q = floor(cell[a] / edge);
            dm = q < 1.0 ? 1 : (q > 1e9 ? 1000000000 : (int)q);
            ext = fmax(ext, cell[a]);
            s->lo[a] = 0.0;
        } else {
            direct = false;
            const double lo = na_of_key(*(volatile unsigned long long *)&s->lo_key[a]);
            const double hi = na_of_key(*(volatile unsigned long long *)&s->hi_key[a]);
            s->lo[a] = lo;
            ext = fmax(ext, hi - lo);
            packed = packed && (hi - lo) / edge < (double)(NA_PACK - 1);
        }
        packed = packed && dm <= NA_PACK;
        s->dims[a] = dm;
        total = total > NA_MAX ? total : total * dm;
    }
    s->inv_edge = 1.0 / edge;
    s->direct = direct && total <= NA_MAX;
    s->packed = packed;
    int nb = 1024;
    while (nb < 2 * n && nb < NA_MAX) nb *= 2;
    s->nbuckets = s->direct ? (int)total : nb;
    // FP32 coordinates of magnitude <= ext, each rounded once, give distances
    // within 5e-7 ext (three axes, at most four roundings each, and the
    // squares' three); the band is three times that.  Outside the range in
    // which FP32 squares neither overflow nor vanish, the exact test decides
    // every candidate.
    const double m = 1.5e-6 * ext, a = cutoff - m, b = cutoff + m;
    const bool in_range = ext < 1e15 && cutoff > 1e-12;
    s->blo = in_range && a > 0.0 ? __double2float_rd(a * a) : -1.0f;
    s->bhi = in_range ? __double2float_ru(b * b) : __int_as_float(0x7f800000);
}

__device__ __forceinline__ int na_bucket_of(const NaScratch &s, int v) {
    return s.packed ? na_bucket(s, v & 1023, (v >> 10) & 1023, (v >> 20) & 1023) : v;
}
__global__ void __launch_bounds__(256) k_na_count(NaScratch *s, const double *__restrict__ r, int n) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const int cx = na_coord(*s, 0, r[3 * i]), cy = na_coord(*s, 1, r[3 * i + 1]), cz = na_coord(*s, 2, r[3 * i + 2]);
    const int b = na_bucket(*s, cx, cy, cz);
    s->cell[i] = s->packed ? (cx & 1023) | (cy & 1023) << 10 | (cz & 1023) << 20 : b;
    atomicAdd(&s->start[b], 1);
    bool far = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) far |= fabs(r[3 * i + a] * s->box_inv[a]) > 1e6;
    if (far) s->far = 1;
}

// exclusive scan of v[0..m) within blocks of NA_SCAN elements; the last block
// to finish scans the blocks' totals into base (and writes the grand total)
__global__ void __launch_bounds__(256) k_na_scan(NaScratch *s, int rows, int m, int32_t *count) {
    int *v = rows ? s->row : s->start, *base = rows ? s->row_base : s->start_base;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    __shared__ int ws[8], last;
    const int e = blockIdx.x * NA_SCAN + 4 * t;
    int q[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) q[k] = e + k < m ? v[e + k] : 0;
    const int sum = q[0] + q[1] + q[2] + q[3];
    int x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    int before = x - sum;
    for (int k = 0; k < w; ++k) before += ws[k];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (e + k < m) v[e + k] = before;
        before += q[k];
    }
    if (t == 255) s->part[blockIdx.x] = before;
    __syncthreads();
    if (t == 0) {
        __threadfence();
        last = atomicAdd(&s->done[1 + rows], 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last || w != 0) return;
    __threadfence();
    int run = 0;
    for (int k0 = 0; k0 < (int)gridDim.x; k0 += 32) {
        const int k = k0 + lane;
        const int p = k < (int)gridDim.x ? *(volatile int *)&s->part[k] : 0;
        int y = p;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= o) y += u;
        }
        if (k < (int)gridDim.x) base[k] = run + y - p;
        run += __shfl_sync(0xffffffffu, y, 31);
    }
    if (lane == 0 && count) *count = run;
}

__device__ __forceinline__ int na_start(const NaScratch &s, int b) { return s.start[b] + s.start_base[b / NA_SCAN]; }

// the order inside a bucket is free: each row is ordered by j below
__global__ void __launch_bounds__(256) k_na_sort(NaScratch *s, const double *__restrict__ r, int n) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const int b = na_bucket_of(*s, s->cell[i]);
    const int at = na_start(*s, b) + atomicAdd(&s->row[b], 1);
    float f[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double x = r[3 * i + a];
        f[a] = (float)(s->per[a] ? x - s->box[a] * floor(x * s->box_inv[a]) : x - s->lo[a]);
    }
    s->items[at] = make_float4(f[0], f[1], f[2], __int_as_float(i));
}

// 32 U register entries in ascending order over a warp (bitonic)
template <int U> __device__ __forceinline__ void na_sort(int (&v)[U], int lane) {
#pragma unroll
    for (int k = 2; k <= 32 * U; k <<= 1)
#pragma unroll
        for (int j = k >> 1; j; j >>= 1) {
            if (j >= 32) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int w = u ^ (j >> 5);
                    if (w < u) continue;
                    const int lo = min(v[u], v[w]), hi = max(v[u], v[w]);
                    v[u] = ((u * 32) & k) == 0 ? lo : hi;
                    v[w] = ((u * 32) & k) == 0 ? hi : lo;
                }
            } else {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int o = __shfl_xor_sync(0xffffffffu, v[u], j);
                    const bool up = ((u * 32 + lane) & k) == 0;
                    v[u] = up == ((lane & j) == 0) ? min(v[u], o) : max(v[u], o);
                }
            }
        }
}

// partners j > i, one warp per bead; pass 0 counts (and keeps rows of up to
// NA_KEEP partners in order), pass 1 writes the row in order of j (its m
// smallest partners, m = what fits below cap, so that the output is always
// the (i, j)-ordered prefix of the full list), searching again only for longer
// rows
template <int PASS>
__global__ void __launch_bounds__(NA_WARPS * 32) k_na_rows(NaScratch *s, const double *__restrict__ r,
                                                           const int32_t *__restrict__ chain,
                                                           const int32_t *__restrict__ seq, int n, double cutoff,
                                                           int32_t *pairs, int cap, const int32_t *count) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int slot = blockIdx.x * NA_WARPS + wp;
    if (slot >= n) return;   // warp-uniform exits
    __shared__ int buf[NA_WARPS][PASS ? NA_ROW : NA_KEEP];
    __shared__ int s_queue[NA_WARPS][64];
    const float4 me = s->items[slot];
    const int i = __float_as_int(me.w);
    int base = 0, m = 0, rows = 0;
    if (PASS) {
        base = s->row[i] + s->row_base[i / NA_SCAN];
        rows = (i + 1 < n ? s->row[i + 1] + s->row_base[(i + 1) / NA_SCAN] : *count) - base;
        m = min(rows, max(0, cap - base));
        if (m == 0) return;
        if (rows <= NA_KEEP) {
            int32_t *const out = pairs + 2 * (size_t)base;
            for (int k = lane; k < m; k += 32) {
                out[2 * k] = i;
                out[2 * k + 1] = s->kept[i][k];
            }
            return;
        }
    }
    const bool per = (s->per[0] | s->per[1] | s->per[2]) != 0;
    const float Lx = s->L[0], Ly = s->L[1], Lz = s->L[2];
    const float blo = s->far ? -1.0f : s->blo, bhi = s->far ? __int_as_float(0x7f800000) : s->bhi;
    int cc[3];
    if (s->packed) {
        const int v = s->cell[i];
        cc[0] = v & 1023; cc[1] = (v >> 10) & 1023; cc[2] = (v >> 20) & 1023;
    } else {
        for (int a = 0; a < 3; ++a) cc[a] = na_coord(*s, a, r[3 * i + a]);
    }
    // neighbouring buckets: lane l < 27 takes offsets (l % 3, l / 3 % 3, l / 9) - 1,
    // the first lane of each bucket its range
    int key = -1;
    if (lane < 27) {
        const int off[3] = {lane % 3 - 1, lane / 3 % 3 - 1, lane / 9 - 1};
        bool ok = true;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            int k = cc[a] + off[a];
            if (s->per[a]) {
                const int dm = s->dims[a];
                k = k < 0 ? k + dm : (k >= dm ? k - dm : k);
            } else if (k < 0) {
                ok = false;
            }
            cc[a] = k;
        }
        if (ok) key = na_bucket(*s, cc[0], cc[1], cc[2]);
    }
    const unsigned same = __match_any_sync(FULL, key);
    int q0 = 0, len = 0;
    if (key >= 0 && (same & ((1u << lane) - 1u)) == 0u) {
        q0 = na_start(*s, key);
        len = (key + 1 < s->nbuckets ? na_start(*s, key + 1) : n) - q0;
    }
    int pre = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, pre, o);
        if (lane >= o) pre += y;
    }
    const int total = __shfl_sync(FULL, pre, 31);
    pre -= len;
    q0 -= pre;
    const int ci = chain[i], si = seq[i];
    int32_t *const row = pairs + 2 * (size_t)base;
    const bool long_row = PASS && rows > NA_ROW;
    // candidates within reach with j > i (one in a dozen), 32 of them to a test
    // of the chain distance and, inside the error band, of the FP64 distance
    constexpr int EXACT = 1 << 30;
    int *const queue = s_queue[wp];
    int cnt = 0, kept = 0, qn = 0;
    for (int g0 = 0; g0 < total; g0 += 32) {
        // candidate g lies in the bucket of the last lane that starts at or before it
        const int g = g0 + lane;
        int lo = 0;
#pragma unroll
        for (int h = 16; h; h >>= 1) {
            const int pm = __shfl_sync(FULL, pre, lo + h);
            if (pm <= g) lo += h;
        }
        const int q = __shfl_sync(FULL, q0, lo) + g;
        bool in = false;
        int e = 0;
        if (g < total) {
            const float4 f = s->items[q];
            e = __float_as_int(f.w);
            float dx = f.x - me.x, dy = f.y - me.y, dz = f.z - me.z;
            if (per) {
                dx = na_image(dx, Lx);
                dy = na_image(dy, Ly);
                dz = na_image(dz, Lz);
            }
            const float d2 = dx * dx + dy * dy + dz * dz;
            in = e > i && !(d2 > bhi);
            if (!(d2 < blo)) e |= EXACT;
        }
        const unsigned im = __ballot_sync(FULL, in);
        if (in) queue[qn + __popc(im & ((1u << lane) - 1u))] = e;
        qn += __popc(im);
        const bool last = g0 + 32 >= total;
        while (qn >= 32 || (last && qn)) {
            __syncwarp();
            bool hit = false;
            int j = -1;
            if (lane < qn) {
                const int e2 = queue[lane];
                j = e2 & ~EXACT;
                const int sj = seq[j], df = si > sj ? si - sj : sj - si;
                if (!(chain[j] == ci && df < 3)) hit = !(e2 & EXACT) || na_dist(*s, r, i, j) < cutoff;
            }
            const int left = queue[32 + lane];
            __syncwarp();
            queue[lane] = left;
            __syncwarp();
            qn = max(qn - 32, 0);
            unsigned bm = __ballot_sync(FULL, hit);
            if (!PASS) {
                const int at = cnt + __popc(bm & ((1u << lane) - 1u));
                if (hit && at < NA_KEEP) buf[wp][at] = j;
            }
            if (PASS && !long_row) {
                if (hit) buf[wp][cnt + __popc(bm & ((1u << lane) - 1u))] = j;
            } else if (PASS) {
                // insertion, the row's m smallest kept in order
                for (; bm; bm &= bm - 1) {
                    const int jj = __shfl_sync(FULL, j, __ffs(bm) - 1);
                    if (lane != 0) continue;
                    if (kept == m && jj >= row[2 * (m - 1) + 1]) continue;
                    int y = kept < m ? kept : m - 1;
                    while (y > 0 && row[2 * (y - 1) + 1] > jj) {
                        row[2 * y + 1] = row[2 * (y - 1) + 1];
                        --y;
                    }
                    row[2 * y + 1] = jj;
                    if (kept < m) ++kept;
                }
                continue;
            }
            cnt += __popc(bm);
        }
    }
    if (!PASS) {
        if (lane == 0) s->row[i] = cnt;
        __syncwarp();
        if (cnt <= 32) {
            int v[1] = {lane < cnt ? buf[wp][lane] : INT_MAX};
            na_sort(v, lane);
            if (lane < cnt) s->kept[i][lane] = (uint16_t)v[0];
        } else if (cnt <= NA_KEEP) {
            int v[2] = {buf[wp][lane], lane + 32 < cnt ? buf[wp][lane + 32] : INT_MAX};
            na_sort(v, lane);
            s->kept[i][lane] = (uint16_t)v[0];
            if (lane + 32 < cnt) s->kept[i][lane + 32] = (uint16_t)v[1];
        }
        return;
    }
    __syncwarp();
    if (long_row) {
        for (int k = lane; k < m; k += 32) row[2 * k] = i;
        return;
    }
    // each partner's rank among the row's is its place
    for (int k0 = 0; k0 < cnt; k0 += 32) {
        const int k = k0 + lane, v = k < cnt ? buf[wp][k] : INT_MAX;
        int rank = 0;
        for (int u = 0; u < cnt; ++u) rank += buf[wp][u] < v;
        if (k < cnt && rank < m) {
            row[2 * rank] = i;
            row[2 * rank + 1] = v;
        }
    }
}

// Device address of the scratch, looked up once per device with that device
// current (in host code the symbol names a host-side stand-in, not device
// memory).
void *scratch_address() {
    static std::mutex mu;
    static void *addr[128] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) throw std::runtime_error(std::string("CUDA error ") + cudaGetErrorString(e));
    if (dev < 0 || dev >= 128) throw std::runtime_error("CUDA device ordinal out of range");
    std::lock_guard<std::mutex> lk(mu);
    if (!addr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_na_scratch);
        if (e != cudaSuccess)
            throw std::runtime_error(std::string("CUDA error ") + cudaGetErrorString(e) +
                                     " at cudaGetSymbolAddress(scratch)");
        addr[dev] = p;
    }
    return addr[dev];
}

}  // namespace

int verlet_pairs_noalloc(const double *d_r, const int32_t *d_chain, const int32_t *d_seq, int32_t n,
                         const double cell[3], double cutoff, int32_t *d_pairs, int32_t cap, int32_t *d_count,
                         void *stream) {
    cudaStream_t st = (cudaStream_t)stream;
    auto *s = (NaScratch *)scratch_address();
    if (n == 0) {
        cudaError_t e = cudaMemsetAsync(d_count, 0, sizeof(int32_t), st);
        if (e != cudaSuccess) throw std::runtime_error(std::string("CUDA error ") + cudaGetErrorString(e));
        return XMD_OK;
    }
    const int nb = (n + 255) / 256, nw = (n + NA_WARPS - 1) / NA_WARPS;
    const bool open = cell[0] == 0.0 || cell[1] == 0.0 || cell[2] == 0.0;
    k_na_clear<<<NA_MAX / 256, 256, 0, st>>>(s);
    k_na_grid<<<open ? nb : 1, 256, 0, st>>>(s, d_r, n, cell[0], cell[1], cell[2], cutoff);
    k_na_count<<<nb, 256, 0, st>>>(s, d_r, n);
    k_na_scan<<<NA_PARTS, 256, 0, st>>>(s, 0, NA_MAX, nullptr);
    k_na_sort<<<nb, 256, 0, st>>>(s, d_r, n);
    k_na_rows<0><<<nw, NA_WARPS * 32, 0, st>>>(s, d_r, d_chain, d_seq, n, cutoff, d_pairs, cap, d_count);
    k_na_scan<<<(n + NA_SCAN - 1) / NA_SCAN, 256, 0, st>>>(s, 1, n, d_count);
    k_na_rows<1><<<nw, NA_WARPS * 32, 0, st>>>(s, d_r, d_chain, d_seq, n, cutoff, d_pairs, cap, d_count);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) throw std::runtime_error(std::string("CUDA error ") + cudaGetErrorString(e));
    return XMD_OK;
}

}  // namespace xmdg
