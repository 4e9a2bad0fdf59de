// graph_prep.cu -- per-call preparation of the pairwise stage.
//
// Contigs are put in ascending log-size order (stable, by original index on
// ties), or, for a whole graph, in narrow bands of log size and by their GC
// projection within a band (k_band_keys), so that every tile of the pairwise
// schedule covers a narrow range of sizes and, in the second form, of the
// projection; the size-dependent distance threshold d*(x, y) of the MetaBAT2
// model (cuda/Cuda2.cu:199-240 solved for d) is then nearly constant over a
// tile and one conservative bound per tile filters its pairs.  This file
// builds: the permutation, sorted FP32 rows and log sizes, the per-contig
// FP64 model parts used by the exact stage, the centred BF16 rows with their
// norms and rounding errors for the tensor-core filter, per-block metadata,
// and the d* table.
//
// Every kernel works on a set of one or more contig sets ("segments") laid
// end to end, each from a 256-row boundary on, so a batch of assemblies is
// prepared by the same few launches as one: k_scan (one pass over the rows
// as they come: column means, and for a single set a content hash and the
// log-size range), the sort, k_rows (gather, model parts, reduced-precision
// rows), k_meta.
#include <cub/cub.cuh>

#include <string>

#include <cmath>
#include <cstring>

#include "graph.cuh"

namespace {

__device__ __forceinline__ unsigned long long dkey(double v) {
    unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}

// The segment of prepared row `pos`: its index and itself.
__device__ __forceinline__ uint32_t seg_of(const PrepSet& v, uint64_t pos, PrepSeg& seg) {
    const uint32_t k = v.segs ? v.blk_seg[pos >> 8] : 0u;
    seg = v.segs ? v.segs[k] : v.one;
    return k;
}

// Four consecutive floats at p; rows are 544 bytes, so a row array is 16-byte
// aligned in every row or in none.
__device__ __forceinline__ float4 load4(const float* __restrict__ p, bool aligned) {
    if (aligned) return __ldg(reinterpret_cast<const float4*>(p));
    return make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
}

// Sort keys and values: the value is the prepared-row index of the contig
// before the sort (segment base + original index).  Padding rows (present
// when several segments are sorted together) sort last in their segment.
__global__ void k_keys(PrepSet v, uint64_t rows, unsigned long long* __restrict__ keys, uint32_t* __restrict__ vals) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= rows) return;
    PrepSeg seg;
    seg_of(v, i, seg);
    const uint64_t r = i - seg.base;
    keys[i] = r < seg.n ? dkey(seg.ls[r]) : ~0ull;
    vals[i] = (uint32_t)i;
}

// Order of a whole graph: bands of log size, `inv_h` per unit, and within a
// band the GC projection in 16 bits.  Any order gives the same graph; this one
// makes most tiles provably empty (tile_kept).
__global__ void k_band_keys(const double* __restrict__ ls, const float* __restrict__ proj, uint64_t n, float inv_h,
                            uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float band = fminf(fmaxf(floorf((float)ls[i] * inv_h), 0.f), 65535.f);  // NaN: band 0
    const float p = fminf(fmaxf((proj[i] + 1.f) * 32767.5f, 0.f), 65535.f);
    keys[i] = (uint32_t)band << 16 | (uint32_t)p;
    vals[i] = (uint32_t)i;
}

// The segment index of every value, the key of the second (stable) sort.
__global__ void k_seg_keys(PrepSet v, uint64_t rows, const uint32_t* __restrict__ vals, uint32_t* __restrict__ keys) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i < rows) keys[i] = v.blk_seg[vals[i] >> 8];
}

constexpr int kCols4 = MDET_NTNF / 4;  // 34
constexpr int kScanWarps = 8;

// The GC direction: the unit vector v whose entry is proportional to a
// tetranucleotide's G and C bases less two.  |v . (a - b)| <= ||a - b|| for
// every pair, and GC content is what TNF rows differ in most.
struct GcVector {
    float v[MDET_NTNF];
};
GcVector gc_vector() {
    GcVector g;
    double norm = 0;
    for (int k = 0; k < MDET_NTNF; ++k) {
        int gc = -2;  // C and G are the odd codes
        for (int b = 0; b < 4; ++b) gc += (tn_tables().col_fw[k] >> (2 * b)) & 1;
        g.v[k] = (float)gc;
        norm += gc * gc;
    }
    const double scale = (1.0 - 1e-6) / sqrt(norm);  // rounding leaves the norm below 1
    for (int k = 0; k < MDET_NTNF; ++k) g.v[k] = (float)(g.v[k] * scale);
    return g;
}

// What k_scan finds over a single set: a hash of the contents, and the
// smallest (complemented, so that zeros start both) and largest size key.
struct ScanStat {
    unsigned long long hash, min_inv, max;
    unsigned long long pad;
};

// One pass over the rows in their original order, rpb rows per block, a warp
// per row (four columns a lane, the last eight on lanes 0 to 7): column sums,
// with stat the content hash -- per 16 bytes one 64 x 64 -> 128-bit product of
// the words, each offset by its position, folded and added up -- and the log
// sizes' range, and with proj the row's GC projection.  The sums run in
// float-float (250,000 contigs: 163 us for the FP64 adds of a separate pass
// and 79 us for a separate hash; 66 us here without projections, 76 us with, 136 MB); the last block of a
// segment turns them into means.  rpb is 256, the size of a segment's blocks,
// or 64 up to 65,536 rows, where 256 would leave SMs without a block (us with 64
// and 256: 1,500 contigs 10 and 22, 16,000 20 and 34, 65,000 38 and 40, 100,000 54 and
// 45, 262,000 102 and 85).
__global__ void __launch_bounds__(kScanWarps * 32) k_scan(PrepSet v, uint32_t rpb, double* __restrict__ sums,
                                                          uint32_t* __restrict__ done, float* __restrict__ mu,
                                                          ScanStat* __restrict__ stat, float* __restrict__ proj,
                                                          const __grid_constant__ GcVector gc) {
    __shared__ ff part[kScanWarps][MDET_NTNF];
    __shared__ bool last;
    PrepSeg seg;
    const uint64_t pos0 = (uint64_t)blockIdx.x * rpb;
    const uint32_t k = seg_of(v, pos0, seg);
    const uint32_t r0 = (uint32_t)(pos0 - seg.base);
    if (r0 >= seg.n) return;  // block-uniform
    const uint32_t rows = min(rpb, seg.n - r0);
    const uint32_t t = threadIdx.x, w = t >> 5, lane = t & 31;
    const bool al = ((uintptr_t)seg.tnf & 15) == 0;
    float g[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    if (proj) {
#pragma unroll
        for (int j = 0; j < 4; ++j) g[j] = gc.v[4 * lane + j];
        if (lane < 8) g[4] = gc.v[128 + lane];
    }
    ff acc[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) acc[j] = ff_make(0.f, 0.f);
    unsigned long long h = 0;
#pragma unroll 4
    for (uint32_t r = w; r < rows; r += kScanWarps) {
        const float* row = seg.tnf + (uint64_t)(r0 + r) * MDET_NTNF;
        const float4 x = load4(row + 4 * lane, al);
        const float y = lane < 8 ? __ldg(row + 128 + lane) : 0.f;
        const float e[5] = {x.x, x.y, x.z, x.w, y};
        if (sums) {
#pragma unroll
            for (int j = 0; j < 5; ++j) {
                const ff s2 = two_sum(acc[j].hi, e[j]);
                acc[j].hi = s2.hi;
                acc[j].lo = __fadd_rn(acc[j].lo, s2.lo);
            }
        }
        if (stat) {
            const unsigned long long pos = ((uint64_t)(r0 + r) * 32 + lane + 1) * 0x9E3779B97F4A7C15ull;
            const unsigned long long a =
                ((unsigned long long)__float_as_uint(x.y) << 32 | __float_as_uint(x.x)) + pos;
            const unsigned long long b =
                ((unsigned long long)__float_as_uint(x.w) << 32 | __float_as_uint(x.z)) ^ (pos + 0xBF58476D1CE4E5B9ull);
            h += (a * b) ^ __umul64hi(a, b) ^ (a + (b << 1));
            const unsigned long long c = (pos ^ __float_as_uint(y)) * 0x94D049BB133111EBull;
            h += c ^ (c >> 29);
        }
        if (proj) {
            float d = __fmul_rn(e[0], g[0]);
#pragma unroll
            for (int j = 1; j < 5; ++j) d = __fmaf_rn(e[j], g[j], d);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
            // the rounding bound of tile_kept needs entries of a unit row; any
            // other row (or a NaN) keeps all its tiles
            bool unit = true;
#pragma unroll
            for (int j = 0; j < 5; ++j) unit = unit && fabsf(e[j]) <= 1.0625f;
            unit = __all_sync(0xffffffffu, unit);
            if (lane == 0) proj[r0 + r] = unit ? d : __int_as_float(0x7fc00000);
        }
    }
    if (stat) {
        unsigned long long lo = 0, hi = 0;
        if (t < rows) {
            const double s = seg.ls[r0 + t];
            unsigned long long z = (unsigned long long)__double_as_longlong(s) +
                                   (unsigned long long)(r0 + t + 1) * 0x94D049BB133111EBull;
            z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
            h += z ^ (z >> 31);
            hi = dkey(s);
            lo = ~hi;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            h += __shfl_xor_sync(0xffffffffu, h, o);
            const unsigned long long l2 = __shfl_xor_sync(0xffffffffu, lo, o);
            const unsigned long long h2 = __shfl_xor_sync(0xffffffffu, hi, o);
            lo = lo > l2 ? lo : l2;
            hi = hi > h2 ? hi : h2;
        }
        if (lane == 0) {
            atomicAdd(&stat->hash, h);
            if (hi | lo) {
                atomicMax(&stat->min_inv, lo);
                atomicMax(&stat->max, hi);
            }
        }
    }
    if (!sums) return;
#pragma unroll
    for (int j = 0; j < 4; ++j) part[w][4 * lane + j] = acc[j];
    if (lane < 8) part[w][128 + lane] = acc[4];
    __syncthreads();
    if (t < MDET_NTNF) {
        ff a = part[0][t];
        for (int q = 1; q < kScanWarps; ++q) a = ff_add(a, part[q][t]);
        atomicAdd(&sums[(uint64_t)k * MDET_NTNF + t], ff_to_double(a));
    }
    __threadfence();
    __syncthreads();
    if (t == 0) last = atomicAdd(&done[k], 1u) + 1 == (seg.n + rpb - 1) / rpb;
    __syncthreads();
    if (last && t < MDET_NTNF)
        mu[(uint64_t)k * MDET_NTNF + t] = (float)(__ldcg(&sums[(uint64_t)k * MDET_NTNF + t]) / (double)seg.n);
}

__device__ __forceinline__ double poly(const double* c, int deg, double v) {
    double r = c[deg];
    for (int k = deg - 1; k >= 0; --k) r = fma(r, v, c[k]);
    return r;
}

// round to nearest, ties away, low 13 bits zero: the tensor cores read such
// FP32 containers unchanged
__device__ __forceinline__ float to_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

// The prepared arrays as k_rows writes them.
struct RowsOut {
    uint32_t* perm;  // in: sorted position -> pre-sort row (padding of a single set is filled in)
    uint32_t* inv;
    float* x32;
    double* ls;
    PartsFF* parts;
    uint16_t *xa, *xb;
    float *ta, *tb;
    float *nsq, *err, *nrm;
    const float* mu;
};

__device__ __forceinline__ uint32_t bf16_bits(float v) {
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    return *reinterpret_cast<const uint16_t*>(&h);
}

// Four columns (4q ..) of a reduced-precision row in one of its roles.
template <int TCK>
__device__ __forceinline__ void store4(uint16_t* bf, float* tf, uint64_t row, uint32_t q, const float (&e)[4]) {
    if constexpr (TCK == kTcBf16) {
        uint2 u;
        u.x = bf16_bits(e[0]) | bf16_bits(e[1]) << 16;
        u.y = bf16_bits(e[2]) | bf16_bits(e[3]) << 16;
        *reinterpret_cast<uint2*>(bf + row * MDET_KPAD + 4 * q) = u;
    } else if constexpr (TCK == kTcTf32) {
        *reinterpret_cast<float4*>(tf + row * MDET_KPAD + 4 * q) = make_float4(e[0], e[1], e[2], e[3]);
    }
}

// Blocks [0, pblocks): the model parts, thread per sorted position -- FP64 is
// a narrow unit here (about two lanes a clock), so its work is spread over
// whole warps with eight independent polynomials a thread.  (250,000 contigs:
// 381 us for a gather with nine lanes of each row's warp on one polynomial
// each, 117 us for the reduced-precision rows in a pass of their own; 136 us
// for both here, 436 MB.)
//
// The other blocks: warp per sorted position, four columns a lane.  The
// FP32 row is copied; with TCK the centred reduced-precision copies in both
// GEMM roles, the squared norm of the rounded row and its exact distance to
// the unrounded centred row follow from the registers.  Columns 136/137 fold
// the column term of ||a||^2+||b||^2-2a.b into the GEMM: the A role carries
// 1, 1 and the B role -hi, -lo of ||b~||^2/2 (a two-term split in the row's
// own precision), so a.b' = a.b - ||b~||^2/2 comes out of TMEM.
template <int TCK>
__global__ void __launch_bounds__(256) k_rows(PrepSet v, uint64_t rows, uint32_t pblocks, RowsOut out, ModelSplit ms) {
    if (blockIdx.x < pblocks) {
        const uint64_t s = blockIdx.x * 256ull + threadIdx.x;
        if (s >= rows) return;
        PrepSeg seg;
        seg_of(v, s, seg);
        if (s - seg.base >= seg.n) return;
        const double x = seg.ls[out.perm[s] - seg.base];
        out.ls[s] = x;
        PartsFF p;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            p.f[m] = ff_from_double(poly(ms.F[m], 7, x));
            double r = ms.G[m][6];  // G_m without its constant
#pragma unroll
            for (int k = 5; k >= 1; --k) r = fma(r, x, ms.G[m][k]);
            p.g[m] = ff_from_double(r * x);
        }
        p.ls = ff_from_double(x);
        p.pad[0] = p.pad[1] = 0.f;
        out.parts[s] = p;
        return;
    }
    const uint64_t s = (blockIdx.x - pblocks) * 8ull + (threadIdx.x >> 5);
    const uint32_t lane = threadIdx.x & 31;
    if (s >= rows) return;
    PrepSeg seg;
    const uint32_t k = seg_of(v, s, seg);
    const float inf = __int_as_float(0x7f800000);
    if (s - seg.base >= seg.n) {  // padding: neutral rows that no pair passes with
        if (lane == 0) {
            out.perm[s] = (uint32_t)s;
            out.inv[s] = (uint32_t)s;
        }
        if constexpr (TCK != kTcNone) {
            for (uint32_t q = lane; q < MDET_KPAD / 4; q += 32) {
                const bool tail = q == MDET_NTNF / 4;
                const float ea[4] = {tail ? 1.f : 0.f, tail ? 1.f : 0.f, 0.f, 0.f};
                const float eb[4] = {tail ? -inf : 0.f, 0.f, 0.f, 0.f};
                store4<TCK>(out.xa, out.ta, s, q, ea);
                store4<TCK>(out.xb, out.tb, s, q, eb);
            }
            if (lane == 0) {
                out.nsq[s] = inf;
                out.err[s] = 0.f;
                out.nrm[s] = 0.f;
            }
        }
        return;
    }
    const uint32_t o = out.perm[s];
    if (lane == 0) out.inv[o] = (uint32_t)s;
    const float* src = seg.tnf + (uint64_t)(o - seg.base) * MDET_NTNF;
    const bool al = ((uintptr_t)seg.tnf & 15) == 0;
    // FP32 throughout.  hv^2 is exact in FP32 (8- or 11-bit significands), so
    // a float-float accumulator gives ||x~||^2 exactly to ~2^-44; the rounding
    // error d = hv - (a - mu) is exact per entry up to one FP32 rounding
    // (TwoSum of a - mu; v - hv is exact by Sterbenz), and its sum of squares
    // is inflated before the square root is rounded up, so err stays an upper
    // bound of ||x~ - x||.
    float e2 = 0.f;
    ff q2 = ff_make(0.f, 0.f);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const uint32_t q = lane + 32 * half;
        if (q < kCols4) {
            const float4 x = load4(src + 4 * q, al);
            *reinterpret_cast<float4*>(out.x32 + s * MDET_NTNF + 4 * q) = x;
            if constexpr (TCK != kTcNone) {
                const float4 m = __ldg(reinterpret_cast<const float4*>(out.mu + (uint64_t)k * MDET_NTNF + 4 * q));
                const float a[4] = {x.x, x.y, x.z, x.w}, mm[4] = {m.x, m.y, m.z, m.w};
                float e[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const ff c = two_sum(a[j], -mm[j]);  // c.hi + c.lo == a - mu exactly
                    e[j] = TCK == kTcBf16 ? __bfloat162float(__float2bfloat16_rn(c.hi)) : to_tf32(c.hi);
                    const float d = __fadd_rn(__fsub_rn(c.hi, e[j]), c.lo);
                    e2 = __fmaf_rn(d, d, e2);
                    q2 = ff_add_f(q2, __fmul_rn(e[j], e[j]));
                }
                store4<TCK>(out.xa, out.ta, s, q, e);
                store4<TCK>(out.xb, out.tb, s, q, e);
            }
        }
    }
    if constexpr (TCK != kTcNone) {
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            e2 += __shfl_xor_sync(0xffffffffu, e2, d);
            ff t;
            t.hi = __shfl_xor_sync(0xffffffffu, q2.hi, d);
            t.lo = __shfl_xor_sync(0xffffffffu, q2.lo, d);
            q2 = ff_add(q2, t);
        }
        const float half = 0.5f * q2.hi;
        const float hi = TCK == kTcBf16 ? __bfloat162float(__float2bfloat16_rn(half)) : to_tf32(half);
        const float rest = __fsub_rn(half, hi);
        const float lo = TCK == kTcBf16 ? __bfloat162float(__float2bfloat16_rn(rest)) : to_tf32(rest);
        if (lane < 2) {  // columns 136 .. 139 and 140 .. 143
            const float ea[4] = {lane ? 0.f : 1.f, lane ? 0.f : 1.f, 0.f, 0.f};
            const float eb[4] = {lane ? 0.f : -hi, lane ? 0.f : -lo, 0.f, 0.f};
            store4<TCK>(out.xa, out.ta, s, kCols4 + lane, ea);
            store4<TCK>(out.xb, out.tb, s, kCols4 + lane, eb);
        }
        if (lane == 0) {
            out.nsq[s] = q2.hi;
            out.err[s] = __fsqrt_ru(__fmul_ru(e2, 1.001f));
            out.nrm[s] = __fsqrt_ru(__fadd_ru(q2.hi, q2.lo));
        }
    }
}

// Metadata of every 128-row block, a warp per block (a thread per block walked
// its rows one dependent load after another: 24 us at 1,500 contigs and 39 us
// at 250,000, 4.3 and 6.7 us so).
__global__ void k_meta(PrepSet v, uint64_t nblk, const double* __restrict__ ls_s, const float* __restrict__ err,
                       const float* __restrict__ nrm, const float* __restrict__ proj,
                       const uint32_t* __restrict__ perm, BlockMeta* __restrict__ meta, BlockMeta* __restrict__ meta32,
                       float2* __restrict__ prange) {
    const uint64_t b = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint32_t lane = threadIdx.x & 31;
    if (b >= nblk) return;
    PrepSeg seg;
    seg_of(v, b * MDET_BLK, seg);
    const uint64_t s0 = b * MDET_BLK, end = (uint64_t)seg.base + seg.n;
    BlockMeta m;
    m.emax = m.nmax = 0.f;
    // the block's range of GC projections (one set only); empty for padding
    float plo = __int_as_float(0x7f800000), phi = -plo;
    if (s0 >= end) {
        m.lo = m.hi = (float)ls_s[end - 1];
    } else {
        // true range (the rows need not be in size order); NaN is the identity of fmin/fmax
        const uint64_t s1 = min(end, s0 + MDET_BLK);
        double lo = __longlong_as_double(0x7ff8000000000000ll), hi = lo;
        float e = 0.f, nm = 0.f;
        for (uint64_t s = s0 + lane; s < s1; s += 32) {
            lo = fmin(lo, ls_s[s]);
            hi = fmax(hi, ls_s[s]);
            if (err) {
                e = fmaxf(e, err[s]);
                nm = fmaxf(nm, nrm[s]);
            }
            if (prange) {
                const float p = proj[perm[s]], inf = __int_as_float(0x7f800000);
                plo = fminf(plo, p == p ? p : -inf);
                phi = fmaxf(phi, p == p ? p : inf);
            }
        }
#pragma unroll
        for (int d = 16; d; d >>= 1) {
            plo = fminf(plo, __shfl_xor_sync(0xffffffffu, plo, d));
            phi = fmaxf(phi, __shfl_xor_sync(0xffffffffu, phi, d));
            lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, d));
            hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, d));
            e = fmaxf(e, __shfl_xor_sync(0xffffffffu, e, d));
            nm = fmaxf(nm, __shfl_xor_sync(0xffffffffu, nm, d));
        }
        m.lo = __double2float_rd(lo);
        m.hi = __double2float_ru(hi);
        m.emax = e;
        m.nmax = nm;
    }
    if (lane) return;
    if (prange) prange[b] = make_float2(plo, phi);
    if (meta) meta[b] = m;
    m.emax = 0.f;
    m.nmax = 0.f;
    meta32[b] = m;
}

// ---- d* table ----

constexpr int kPts = 4 * MDET_TBL + 1;

// F_m and G_m at the table's 1,025 grid points: axis[m][p], axis[4 + m][p].
// The grid comes from device memory when `grid` is given.
__global__ void k_dstar_axis(const TableGrid* __restrict__ grid, double lmin, double h, ModelSplit ms,
                             double* __restrict__ axis) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= kPts) return;
    if (grid) {
        lmin = grid->lmin;
        h = grid->h;
    }
    const double x = lmin + p * (h / 4);
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        axis[m * kPts + p] = poly(ms.F[m], 7, x);
        const double g[7] = {0, ms.G[m][1], ms.G[m][2], ms.G[m][3], ms.G[m][4], ms.G[m][5], ms.G[m][6]};
        axis[(4 + m) * kPts + p] = poly(g, 6, x);
    }
}

// d* at log sizes x <= y with F(x) and G(y) given (+inf where the model is
// not decreasing in d).
__device__ __forceinline__ double dstar_at(double x, double y, const double (&F)[4], const double (&G)[4], double L,
                                           const ModelSplit& ms) {
    const double ln9 = 2.1972245773362196, t = x * y;
    const double inf = __longlong_as_double(0x7ff0000000000000ll);
    auto coef = [&](int m) {
        const double h[6] = {0, ms.H[m][1], ms.H[m][2], ms.H[m][3], ms.H[m][4], ms.H[m][5]};
        return F[m] + G[m] + poly(h, 5, t);
    };
    const double c1 = coef(1);
    if (!(c1 > 0)) return inf;
    const double c0 = coef(0);
    if (L >= ln9) return (-L - c0) / c1;
    const double c3 = coef(3);
    if (!(c3 > 0)) return inf;
    const double d1 = (-ln9 - c0) / c1;
    const double d2 = (-L - coef(2)) / c3;
    return d1 > d2 ? d1 : d2;
}

// Block per cell row a: the 5 x 5 points of every cell (a, b), b >= a (the
// points are symmetric, so cell (b, a) is the same), then the cell's bound
// with its slack.  The one-variable polynomials come from k_dstar_axis, so a
// point costs the x * y terms and the divisions.
__global__ void __launch_bounds__(MDET_TBL) k_dstar_cells(const TableGrid* __restrict__ grid, double lmin, double h,
                                                          double L, ModelSplit ms, const double* __restrict__ axis,
                                                          float* __restrict__ st0) {
    __shared__ float pts[5][kPts + 3];
    const int a = blockIdx.x, b = threadIdx.x;
    if (grid) {
        lmin = grid->lmin;
        h = grid->h;
    }
    // point (4a + i, q), q from 4a + i up
    for (int i = 0; i < 5; ++i) {
        const int pa = 4 * a + i;
        double F[4], G[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) F[m] = axis[m * kPts + pa];
        for (int q = pa + b; q < kPts; q += MDET_TBL) {
#pragma unroll
            for (int m = 0; m < 4; ++m) G[m] = axis[(4 + m) * kPts + q];
            pts[i][q] = __double2float_ru(dstar_at(lmin + pa * (h / 4), lmin + q * (h / 4), F, G, L, ms));
        }
    }
    __syncthreads();
    if (b < a) return;
    float mx = -__int_as_float(0x7f800000), mn = __int_as_float(0x7f800000);
    for (int i = 0; i <= 4; ++i)
        for (int j = 0; j <= 4; ++j) {
            const int pa = 4 * a + i, pb = 4 * b + j;
            const float v = pa <= pb ? pts[i][pb] : pts[pb - 4 * a][pa];
            mx = fmaxf(mx, v);
            mn = fminf(mn, v);
        }
    float T = mx + 0.5f * (mx - mn) + 1e-6f + 1e-5f * fabsf(mx);
    if (isinf(mx) || isnan(mx)) T = __int_as_float(0x7f800000);
    st0[a * MDET_TBL + b] = T;
    st0[b * MDET_TBL + a] = T;
}

// Suffix maximum along x (the min-size axis): cell (a, b) then bounds every
// cell (a', b) with a' >= a, so a box [x0, x1] x [y0, y1] is bounded by row
// x0 alone.  d* falls as the smaller contig grows, so this costs little.
// A warp per column (eight cells a lane, then a scan over the lanes), eight
// columns per block.
__global__ void __launch_bounds__(256) k_suffix_x(float* __restrict__ st0) {
    __shared__ float t[MDET_TBL][9];
    const int c0 = blockIdx.x * 8;
    for (int i = threadIdx.x; i < MDET_TBL * 8; i += 256) t[i >> 3][i & 7] = st0[(i >> 3) * MDET_TBL + c0 + (i & 7)];
    __syncthreads();
    const int col = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float v[8], m = -__int_as_float(0x7f800000);
#pragma unroll
    for (int i = 7; i >= 0; --i) {
        m = fmaxf(m, t[8 * lane + i][col]);
        v[i] = m;
    }
    float after = m;  // inclusive suffix maximum over the lanes
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float u = __shfl_down_sync(0xffffffffu, after, o);
        if (lane + o < 32) after = fmaxf(after, u);
    }
    const float next = __shfl_down_sync(0xffffffffu, after, 1);
#pragma unroll
    for (int i = 0; i < 8; ++i) t[8 * lane + i][col] = lane < 31 ? fmaxf(v[i], next) : v[i];
    __syncthreads();
    for (int i = threadIdx.x; i < MDET_TBL * 8; i += 256) st0[(i >> 3) * MDET_TBL + c0 + (i & 7)] = t[i >> 3][i & 7];
}

// The sparse table's upper levels, block per row.
__global__ void __launch_bounds__(MDET_TBL) k_sparse(float* __restrict__ st) {
    __shared__ float lev[2][MDET_TBL];
    const int a = blockIdx.x, b = threadIdx.x;
    lev[0][b] = st[a * MDET_TBL + b];
    __syncthreads();
    for (int k = 1; k < MDET_TBL_LEVELS; ++k) {
        const float* prev = lev[(k - 1) & 1];
        const float m = fmaxf(prev[b], prev[min(b + (1 << (k - 1)), MDET_TBL - 1)]);
        lev[k & 1][b] = m;
        st[(size_t)k * MDET_TBL * MDET_TBL + a * MDET_TBL + b] = m;
        __syncthreads();
    }
}

// Builds a table into st: the grid is (lmin, h), or *grid on the device.
// Four launches, 78 us (eleven, 300 us, in the first form: 204 us for the
// points, each with all eight polynomials, and 58 us for the suffix maxima of
// one thread per column).
int launch_table(mdet_ctx* ctx, const TableGrid* grid, double lmin, double h, double logit_cut, float* st) {
    cudaStream_t s = ctx->stream;
    double* axis = (double*)ctx_scratch(ctx, "tbl.axis", (size_t)8 * kPts * 8);
    if (!axis) return MDET_ERR_NOMEM;
    k_dstar_axis<<<(kPts + 63) / 64, 64, 0, s>>>(grid, lmin, h, model_split(), axis);
    MDET_LAUNCHED(ctx, "k_dstar_axis");
    k_dstar_cells<<<MDET_TBL, MDET_TBL, 0, s>>>(grid, lmin, h, logit_cut, model_split(), axis, st);
    MDET_LAUNCHED(ctx, "k_dstar_cells");
    k_suffix_x<<<MDET_TBL / 8, 256, 0, s>>>(st);
    MDET_LAUNCHED(ctx, "k_suffix_x");
    k_sparse<<<MDET_TBL, MDET_TBL, 0, s>>>(st);
    MDET_LAUNCHED(ctx, "k_sparse");
    return MDET_OK;
}

// union of (lo, hi) ranges -> table grid (one warp)
__global__ void k_grid_from_ranges(const double* __restrict__ r, uint32_t count, TableGrid* __restrict__ g) {
    double lo = INFINITY, hi = -INFINITY;
    for (uint32_t k = threadIdx.x; k < count; k += 32)
        if (r[2 * k] <= r[2 * k + 1]) {
            lo = fmin(lo, r[2 * k]);
            hi = fmax(hi, r[2 * k + 1]);
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (threadIdx.x) return;
    if (!(lo <= hi)) lo = hi = 0;
    double h = (hi - lo) / MDET_TBL;
    if (!(h > 1e-7)) h = 1e-7;
    lo -= 1e-9;
    g->lmin = lo;
    g->h = h;
    g->lminf = (float)lo;
    g->inv_hf = (float)(1.0 / h);
}

// Range of the log sizes: a one-block scan.
__global__ void k_minmax(const double* __restrict__ ls_s, uint64_t n, double* __restrict__ out) {
    __shared__ double smin[32], smax[32];
    double lo = INFINITY, hi = -INFINITY;
    for (uint64_t i = threadIdx.x; i < n; i += blockDim.x) {
        lo = fmin(lo, ls_s[i]);
        hi = fmax(hi, ls_s[i]);
    }
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if ((threadIdx.x & 31) == 0) {
        smin[threadIdx.x >> 5] = lo;
        smax[threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
            lo = fmin(lo, smin[w]);
            hi = fmax(hi, smax[w]);
        }
        out[0] = lo;
        out[1] = hi;
    }
}

}  // namespace

ModelHFF model_h_ff() {
    const ModelH h = model_h();
    ModelHFF r;
    for (int m = 0; m < 4; ++m)
        for (int k = 0; k < 6; ++k) {
            const float hi = (float)h.h[m][k];
            r.h[m][k].hi = hi;
            r.h[m][k].lo = (float)(h.h[m][k] - (double)hi);
        }
    return r;
}

ModelH model_h() {
    ModelH h;
    const ModelSplit& s = model_split();
    for (int m = 0; m < 4; ++m)
        for (int k = 0; k < 6; ++k) h.h[m][k] = s.H[m][k];
    return h;
}

// The double whose order-preserving key is k.
static double size_of_key(unsigned long long k) {
    const unsigned long long b = (k & 0x8000000000000000ull) ? (k & 0x7fffffffffffffffull) : ~k;
    double v;
    memcpy(&v, &b, 8);
    return v;
}

int prep_alloc(mdet_ctx* ctx, const char* tag, uint64_t rows, int tck, uint32_t sets, GraphPrep* g) {
    const std::string t(tag);
    const uint64_t nblk = rows / MDET_BLK;
    g->perm = (uint32_t*)ctx_scratch(ctx, (t + ".perm").c_str(), rows * 4);
    g->inv = (uint32_t*)ctx_scratch(ctx, (t + ".inv").c_str(), rows * 4);
    g->x32 = (float*)ctx_scratch(ctx, (t + ".x32").c_str(), rows * MDET_NTNF * 4);
    g->ls = (double*)ctx_scratch(ctx, (t + ".ls").c_str(), rows * 8);
    g->parts = (PartsFF*)ctx_scratch(ctx, (t + ".parts").c_str(), rows * sizeof(PartsFF));
    g->meta32 = (BlockMeta*)ctx_scratch(ctx, (t + ".meta32").c_str(), nblk * sizeof(BlockMeta));
    g->prange = nullptr;
    g->mu = (float*)ctx_scratch(ctx, (t + ".mu").c_str(), (uint64_t)sets * MDET_NTNF * 4);
    g->xa = g->xb = nullptr;
    g->ta = g->tb = nullptr;
    g->tck = tck;
    g->nsq = nullptr;
    g->meta = nullptr;
    if (tck == kTcBf16) {
        g->xa = (uint16_t*)ctx_scratch(ctx, (t + ".xa").c_str(), rows * MDET_KPAD * 2);
        g->xb = (uint16_t*)ctx_scratch(ctx, (t + ".xb").c_str(), rows * MDET_KPAD * 2);
        if (!g->xa || !g->xb) return MDET_ERR_NOMEM;
    } else if (tck == kTcTf32) {
        g->ta = (float*)ctx_scratch(ctx, (t + ".ta").c_str(), rows * MDET_KPAD * 4);
        g->tb = (float*)ctx_scratch(ctx, (t + ".tb").c_str(), rows * MDET_KPAD * 4);
        if (!g->ta || !g->tb) return MDET_ERR_NOMEM;
    }
    if (tck != kTcNone) {
        g->nsq = (float*)ctx_scratch(ctx, (t + ".nsq").c_str(), rows * 4);
        g->meta = (BlockMeta*)ctx_scratch(ctx, (t + ".meta").c_str(), nblk * sizeof(BlockMeta));
        if (!g->nsq || !g->meta) return MDET_ERR_NOMEM;
    }
    if (!g->perm || !g->inv || !g->x32 || !g->ls || !g->parts || !g->meta32 || !g->mu) return MDET_ERR_NOMEM;
    return MDET_OK;
}

// Zeroed accumulators of k_scan in one buffer: the statistics, the column
// sums and finished-block counts per segment.
struct ScanBuf {
    ScanStat* stat;
    double* sums;
    uint32_t* done;
};

static int scan_rows(mdet_ctx* ctx, const PrepSet& set, uint64_t rows, int tck, bool stat, float* mu, float* proj,
                     ScanBuf* out) {
    static const GcVector gc = gc_vector();
    const uint64_t nsum = (uint64_t)set.count * MDET_NTNF;
    const size_t bytes = sizeof(ScanStat) + nsum * 8 + set.count * 4ull;
    unsigned char* p = (unsigned char*)ctx_scratch(ctx, "pre.scan", bytes);
    if (!p) return MDET_ERR_NOMEM;
    out->stat = (ScanStat*)p;
    out->sums = (double*)(p + sizeof(ScanStat));
    out->done = (uint32_t*)(out->sums + nsum);
    MDET_CUDA(ctx, cudaMemsetAsync(p, 0, bytes, ctx->stream));
    const uint32_t rpb = rows <= 65536 ? 64 : 256;
    k_scan<<<(unsigned)(rows / rpb), kScanWarps * 32, 0, ctx->stream>>>(
        set, rpb, tck != kTcNone ? out->sums : nullptr, out->done, mu, stat ? out->stat : nullptr, proj, gc);
    MDET_LAUNCHED(ctx, "k_scan");
    return MDET_OK;
}

// Bands of log size per unit in a whole graph's order.  Within a band the blocks
// are narrow in the GC projection, so wider bands (more blocks in each) leave more
// tiles empty but loosen the tiles' distance bound (more candidates to score).
// The graph's time in us at 5, 10, 20 and 40 bands: 9,000 contigs 420, 408, 404, 400;
// 30,000 876, 859, 870, 905; 100,000 2,966, 2,759, 2,790, 2,863; 250,000 8,971, 8,891,
// 9,066, 9,362; 600,000 31.9, 31.0, 31.1, 32.2 ms; 1,000,000 74.1, 71.6, 70.9, 72.6.
static float band_inv_width(uint64_t n) { return n > 700000 ? 20.f : 10.f; }

// Everything after the scan: the order, the rows, the metadata.  With proj (one
// set) the order is by size bands and GC projection, else by size or the
// caller's.
static int prep_rows(mdet_ctx* ctx, const PrepSet& set, uint64_t rows, int tck, const GraphPrep& g,
                     const uint32_t* order, const float* proj) {
    cudaStream_t s = ctx->stream;
    const uint64_t nblk = rows / MDET_BLK;
    // one set: its n contigs are sorted; several: every row, padding included
    const uint64_t ns = set.segs ? rows : set.one.n;
    if (order) {
        // caller's order (original index per position)
        MDET_CUDA(ctx, cudaMemcpyAsync(g.perm, order, ns * 4, cudaMemcpyDeviceToDevice, s));
    } else {
        unsigned long long* keys = (unsigned long long*)ctx_scratch(ctx, "pre.keys", ns * 8);
        unsigned long long* keys2 = (unsigned long long*)ctx_scratch(ctx, "pre.keys2", ns * 8);
        uint32_t* vals = (uint32_t*)ctx_scratch(ctx, "pre.vals", ns * 4);
        if (!keys || !keys2 || !vals) return MDET_ERR_NOMEM;
        const unsigned blocks = (unsigned)((ns + 255) / 256);
        if (proj) {
            uint32_t *k32 = (uint32_t*)keys, *k32b = (uint32_t*)keys2;
            k_band_keys<<<blocks, 256, 0, s>>>(set.one.ls, proj, ns, band_inv_width(ns), k32, vals);
            MDET_LAUNCHED(ctx, "k_band_keys");
            size_t tb = 0;
            cub::DeviceRadixSort::SortPairs(nullptr, tb, k32, k32b, vals, g.perm, (int)ns, 0, 32, s);
            void* tmp = ctx_scratch(ctx, "pre.cubtmp", tb);
            if (!tmp) return MDET_ERR_NOMEM;
            MDET_CUDA(ctx, cub::DeviceRadixSort::SortPairs(tmp, tb, k32, k32b, vals, g.perm, (int)ns, 0, 32, s));
        } else {
            k_keys<<<blocks, 256, 0, s>>>(set, ns, keys, vals);
            MDET_LAUNCHED(ctx, "k_keys");
            // several sets: by size, then (stable) by set -- two sorts over all
            // rows cost less than one per set
            uint32_t* vals2 = set.segs ? (uint32_t*)ctx_scratch(ctx, "pre.vals2", ns * 4) : g.perm;
            if (!vals2) return MDET_ERR_NOMEM;
            size_t t1 = 0, t2 = 0;
            cub::DeviceRadixSort::SortPairs(nullptr, t1, keys, keys2, vals, vals2, (int)ns, 0, 64, s);
            int bits = 1;
            uint32_t *k32 = (uint32_t*)keys, *k32b = (uint32_t*)keys2;
            if (set.segs) {
                while (bits < 32 && (set.count - 1) >> bits) ++bits;
                cub::DeviceRadixSort::SortPairs(nullptr, t2, k32, k32b, vals2, g.perm, (int)ns, 0, bits, s);
            }
            size_t tb = t1 > t2 ? t1 : t2;
            void* tmp = ctx_scratch(ctx, "pre.cubtmp", tb);
            if (!tmp) return MDET_ERR_NOMEM;
            MDET_CUDA(ctx, cub::DeviceRadixSort::SortPairs(tmp, t1, keys, keys2, vals, vals2, (int)ns, 0, 64, s));
            if (set.segs) {
                k_seg_keys<<<blocks, 256, 0, s>>>(set, ns, vals2, k32);
                MDET_LAUNCHED(ctx, "k_seg_keys");
                MDET_CUDA(ctx, cub::DeviceRadixSort::SortPairs(tmp, t2, k32, k32b, vals2, g.perm, (int)ns, 0, bits, s));
            }
        }
    }
    RowsOut out{g.perm, g.inv, g.x32, g.ls, g.parts, g.xa, g.xb, g.ta, g.tb, g.nsq, nullptr, nullptr, g.mu};
    if (tck != kTcNone) {
        out.err = (float*)ctx_scratch(ctx, "pre.err", rows * 4);
        out.nrm = (float*)ctx_scratch(ctx, "pre.nrm", rows * 4);
        if (!out.err || !out.nrm) return MDET_ERR_NOMEM;
    }
    const unsigned pblocks = (unsigned)(rows / 256), grid = pblocks + (unsigned)(rows / 8);
    if (tck == kTcBf16)
        k_rows<kTcBf16><<<grid, 256, 0, s>>>(set, rows, pblocks, out, model_split());
    else if (tck == kTcTf32)
        k_rows<kTcTf32><<<grid, 256, 0, s>>>(set, rows, pblocks, out, model_split());
    else
        k_rows<kTcNone><<<grid, 256, 0, s>>>(set, rows, pblocks, out, model_split());
    MDET_LAUNCHED(ctx, "k_rows");
    k_meta<<<(unsigned)((nblk * 32 + 255) / 256), 256, 0, s>>>(set, nblk, g.ls, out.err, out.nrm, proj, g.perm,
                                                             tck != kTcNone ? g.meta : nullptr, g.meta32, g.prange);
    MDET_LAUNCHED(ctx, "k_meta");
    return MDET_OK;
}

int prep_set(mdet_ctx* ctx, const PrepSet& set, uint64_t rows, int tck, const GraphPrep& g) {
    ScanBuf sb;
    MDET_TRY(scan_rows(ctx, set, rows, tck, false, g.mu, nullptr, &sb));
    return prep_rows(ctx, set, rows, tck, g, nullptr, nullptr);
}

// Rows in bands of size, strictly by size, or in the caller's order.  A preparation
// of the very same inputs that is still in place (same pointers and contents, no
// count since) is used as it is: the search and the graph of one assembly share it,
// and a call that takes any order (PrepOrder::any) leaves it there.
int prep_sorted(mdet_ctx* ctx, const float* d_tnf, const double* d_ls, uint64_t n, int tck, GraphPrep* g,
                const uint32_t* order, PrepOrder how) {
    g->n = (uint32_t)n;
    g->npad = (uint32_t)((n + 255) / 256 * 256);
    MDET_TRY(prep_alloc(ctx, "pre", g->npad, tck, 1, g));
    const PrepSet set{1, PrepSeg{d_tnf, d_ls, (uint32_t)n, 0}, nullptr, nullptr};
    auto& c = ctx->prep_cache;
    ScanBuf sb;
    if (order) {
        c.valid = false;
        MDET_TRY(scan_rows(ctx, set, g->npad, tck, false, g->mu, nullptr, &sb));
        return prep_rows(ctx, set, g->npad, tck, *g, order, nullptr);
    }
    const bool by_size =
        how == PrepOrder::any ? !(c.valid && c.tnf == d_tnf && c.ls == d_ls && c.n == n) || c.by_size : how == PrepOrder::size;
    float* proj = nullptr;
    if (!by_size) {
        proj = (float*)ctx_scratch(ctx, "pre.proj", n * 4);
        g->prange = (float2*)ctx_scratch(ctx, "pre.prange", (uint64_t)g->npad / MDET_BLK * sizeof(float2));
        if (!proj || !g->prange) return MDET_ERR_NOMEM;
    }
    // the scan writes the means, so a preparation it confirms keeps equal ones
    MDET_TRY(scan_rows(ctx, set, g->npad, tck, true, g->mu, proj, &sb));
    ScanStat st;
    MDET_CUDA(ctx, cudaMemcpyAsync(&st, sb.stat, sizeof(st), cudaMemcpyDeviceToHost, ctx->stream));
    MDET_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    g->lrange[0] = size_of_key(~st.min_inv);
    g->lrange[1] = size_of_key(st.max);
    // a preparation with other reduced-precision rows (or none) is remade:
    // nsq and the block metadata describe the rows last made
    if (c.valid && c.tnf == d_tnf && c.ls == d_ls && c.n == n && (c.tck == tck || tck == kTcNone) &&
        c.by_size == by_size && c.hash == st.hash && c.x32 == g->x32 && (tck == kTcNone || (c.xa == g->xa && c.ta == g->ta)) &&
        c.gen == ctx->scratch_gen)
        return MDET_OK;
    c.valid = false;
    MDET_TRY(prep_rows(ctx, set, g->npad, tck, *g, nullptr, proj));
    c.valid = true;
    c.by_size = by_size;
    c.tnf = d_tnf;
    c.ls = d_ls;
    c.n = n;
    c.tck = tck;
    c.hash = st.hash;
    c.x32 = g->x32;
    c.xa = g->xa;
    c.ta = g->ta;
    c.gen = ctx->scratch_gen;
    return MDET_OK;
}

int grid_from_ranges(mdet_ctx* ctx, const double* ranges, uint32_t count, TableGrid* grid) {
    k_grid_from_ranges<<<1, 32, 0, ctx->stream>>>(ranges, count, grid);
    MDET_LAUNCHED(ctx, "k_grid_from_ranges");
    return MDET_OK;
}

int build_dstar_table_dev(mdet_ctx* ctx, const TableGrid* grid, double logit_cut, float* st, DstarTable* out) {
    MDET_TRY(launch_table(ctx, grid, 0, 0, logit_cut, st));
    out->st = st;
    out->lmin = 0.f;
    out->inv_h = 0.f;
    out->dyn = &grid->lminf;
    return MDET_OK;
}

int build_dstar_table(mdet_ctx* ctx, const double* d_ls, uint64_t n, double logit_cut, DstarTable* out,
                      const double* range) {
    out->dyn = nullptr;
    cudaStream_t s = ctx->stream;
    double lmin, lmax;
    if (range) {
        lmin = range[0];
        lmax = range[1];
    } else {
        // the range is needed on the host to place the grid
        double* mm = (double*)ctx_scratch(ctx, "tbl.mm", 16);
        if (!mm) return MDET_ERR_NOMEM;
        double r[2];
        k_minmax<<<1, 1024, 0, s>>>(d_ls, n, mm);
        MDET_LAUNCHED(ctx, "k_minmax");
        MDET_CUDA(ctx, cudaMemcpyAsync(r, mm, 16, cudaMemcpyDeviceToHost, s));
        MDET_CUDA(ctx, cudaStreamSynchronize(s));
        lmin = r[0];
        lmax = r[1];
    }
    double h = (lmax - lmin) / MDET_TBL;
    if (!(h > 1e-7)) h = 1e-7;
    // a table already built for this cutoff and size range?
    int slot = -1, lru = 0;
    for (int k = 0; k < 4; ++k) {
        const auto& t = ctx->tbl[k];
        if (t.valid && t.L == logit_cut && t.lmin == lmin && t.lmax == lmax) slot = k;
        if (ctx->tbl[k].used < ctx->tbl[lru].used) lru = k;
    }
    const bool hit = slot >= 0;
    if (!hit) slot = lru;
    const std::string name = "tbl.st" + std::to_string(slot);
    float* st = (float*)ctx_scratch(ctx, name.c_str(), (size_t)MDET_TBL_LEVELS * MDET_TBL * MDET_TBL * 4);
    if (!st) return MDET_ERR_NOMEM;
    auto& t = ctx->tbl[slot];
    t.used = ++ctx->tbl_clock;
    out->st = st;
    out->lmin = (float)(lmin - 1e-9);
    out->inv_h = (float)(1.0 / h);
    if (hit) return MDET_OK;
    t.valid = false;
    MDET_TRY(launch_table(ctx, nullptr, lmin - 1e-9, h, logit_cut, st));
    t.valid = true;
    t.L = logit_cut;
    t.lmin = lmin;
    t.lmax = lmax;
    return MDET_OK;
}

// ---- tiles that can hold a pair ----
// A pair of rows a, b has |v . (a - b)| <= ||a - b|| for the unit vector v, so a
// tile whose blocks' ranges of v . x lie further apart than its distance bound
// holds no pair within the bound.  (1M contigs in bands: two thirds of the
// tiles, which the filter then never loads.)
namespace {

template <int W>  // 128-row blocks per column tile
__device__ __forceinline__ bool tile_kept(const BlockMeta* __restrict__ meta, const float2* __restrict__ pr,
                                          const DstarTable& tbl, uint32_t I, uint32_t J, uint32_t nblk) {
    const uint32_t b0 = W * J, b1 = min(W * J + W - 1, nblk - 1);
    const BlockMeta ma = meta[I], m0 = meta[b0], m1 = meta[b1];
    const float2 pa = pr[I], p0 = pr[b0], p1 = pr[b1];
    const float gap = fmaxf(fminf(p0.x, p1.x) - pa.y, pa.x - fmaxf(p0.y, p1.y));
    // a projection is ten roundings of partial sums below 9.3 (entries up to
    // 1.0625, the direction's add up to 8.7): 6e-6 off at most, a difference twice that
    const float R = tile_dstar(tbl, ma.lo, ma.hi, fminf(m0.lo, m1.lo), fmaxf(m0.hi, m1.hi)) * (1.f + 2e-5f) + 2e-5f;
    return !(gap > R);
}

// Warp per row tile I: how many of its column tiles are kept, or (list) which,
// in order.
template <int W>
__global__ void __launch_bounds__(256) k_tile_keep(const BlockMeta* __restrict__ meta, const float2* __restrict__ pr,
                                                   DstarTable tbl, uint32_t ta, uint32_t tb, uint32_t nblk,
                                                   unsigned long long* __restrict__ cnt,
                                                   const unsigned long long* __restrict__ off,
                                                   uint32_t* __restrict__ list, uint32_t* __restrict__ mid) {
    const uint32_t I = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (I >= ta) {
        if (I == ta && lane == 0 && !list) cnt[ta] = 0;  // the scan's last entry is then the total
        return;
    }
    unsigned long long at = list ? off[I] : 0ull;
    uint32_t c = 0;
    for (uint32_t j = I / W; j < tb; j += 32) {
        const uint32_t J = j + lane;
        const bool keep = J < tb && tile_kept<W>(meta, pr, tbl, I, J, nblk);
        const uint32_t bal = __ballot_sync(0xffffffffu, keep);
        if (list && keep) list[at + __popc(bal & ((1u << lane) - 1u))] = I * tb + J;
        at += __popc(bal);
        c += __popc(bal);
    }
    if (!list && lane == 0) {
        cnt[I] = c;
        if (mid) {  // sorts like the middle of the tile's projections
            const uint32_t f = __float_as_uint(pr[I].x + pr[I].y);
            mid[I] = (f & 0x80000000u) ? ~f : (f | 0x80000000u);
            mid[ta + I] = I;
        }
    }
}

// The list in one launch: warp per row tile, lane k keeps the ballot of the k-th 32
// column tiles, and the row's entries go where the counter says, in no order of the
// rows.  Up to 65,536 contigs (the graph in us with two passes and a scan, and so: 20,011
// contigs 646 and 631, 50,000 1,322 and 1,311); larger sets want neighbouring row tiles in
// turn (100,000: 2,759 and 2,850).
constexpr uint32_t kListRows = 65536;
template <int W>
__global__ void __launch_bounds__(256) k_tile_list(const BlockMeta* __restrict__ meta, const float2* __restrict__ pr,
                                                   DstarTable tbl, uint32_t ta, uint32_t tb, uint32_t nblk,
                                                   unsigned long long* __restrict__ total,
                                                   uint32_t* __restrict__ list) {
    const uint32_t I = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31, j0 = I / W;
    if (I >= ta) return;
    uint32_t mine = 0;
    for (uint32_t j = j0, k = 0; j < tb; j += 32, ++k) {
        const uint32_t J = j + lane;
        const bool keep = J < tb && tile_kept<W>(meta, pr, tbl, I, J, nblk);
        const uint32_t bal = __ballot_sync(0xffffffffu, keep);
        if (lane == k) mine = bal;
    }
    const uint32_t own = __popc(mine);
    uint32_t upto = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= (uint32_t)o) upto += u;
    }
    unsigned long long at = 0;
    if (lane == 31 && upto) at = atomicAdd(total, (unsigned long long)upto);
    at = __shfl_sync(0xffffffffu, at, 31) + (upto - own);
    for (; mine; mine &= mine - 1) list[at++] = I * tb + j0 + 32 * lane + __ffs(mine) - 1;
}

// Key of the row tile at every position of the order by projection: its group
// of `group` tiles, within the group the longest list first.
__global__ void k_wave_keys(const uint32_t* __restrict__ by_mid, const unsigned long long* __restrict__ cnt,
                            uint32_t ta, uint32_t group, uint32_t* __restrict__ keys) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= ta) return;
    const unsigned long long c = cnt[by_mid[r]];
    keys[r] = (r / group) << 18 | (0x3ffffu - (uint32_t)(c < 0x3ffffull ? c : 0x3ffffull));
}

}  // namespace

int kept_tiles(mdet_ctx* ctx, const GraphPrep& g, const DstarTable& tbl, int bn, uint32_t wave, TileList* out) {
    cudaStream_t s = ctx->stream;
    const uint32_t nblk = g.npad / MDET_BLK, ta = (g.n + 127) / 128, tb = (g.n + bn - 1) / bn;
    const uint64_t most = (uint64_t)ta * tb / 2 + 2ull * ta + tb;  // the triangle, diagonal tiles included
    unsigned long long* cnt = (unsigned long long*)ctx_scratch(ctx, "tl.cnt", ((uint64_t)ta + 1) * 8);
    unsigned long long* off = (unsigned long long*)ctx_scratch(ctx, "tl.off", ((uint64_t)ta + 1) * 8);
    uint32_t* list = (uint32_t*)ctx_scratch(ctx, "tl.list", most * 4);
    size_t tmpb = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tmpb, cnt, off, (int)ta + 1, s);
    void* tmp = ctx_scratch(ctx, "tl.cubtmp", tmpb);
    if (!cnt || !off || !list || !tmp) return MDET_ERR_NOMEM;
    uint32_t* mid = nullptr;  // five arrays of ta: keys, tiles, their sorted copies, the order
    if (wave && !(mid = (uint32_t*)ctx_scratch(ctx, "tl.mid", 5ull * ta * 4))) return MDET_ERR_NOMEM;
    const BlockMeta* meta = g.meta ? g.meta : g.meta32;
    const unsigned blocks = (unsigned)(((uint64_t)(ta + 1) * 32 + 255) / 256);
    if (!wave && g.n <= kListRows) {  // at most 512 column tiles, 32 a lane
        MDET_CUDA(ctx, cudaMemsetAsync(off + ta, 0, 8, s));
        if (bn == 256)
            k_tile_list<2><<<blocks, 256, 0, s>>>(meta, g.prange, tbl, ta, tb, nblk, off + ta, list);
        else
            k_tile_list<1><<<blocks, 256, 0, s>>>(meta, g.prange, tbl, ta, tb, nblk, off + ta, list);
        MDET_LAUNCHED(ctx, "k_tile_list");
        *out = TileList{list, nullptr, off + ta, nullptr};
        return MDET_OK;
    }
    for (int fill = 0; fill < 2; ++fill) {
        if (bn == 256)
            k_tile_keep<2><<<blocks, 256, 0, s>>>(meta, g.prange, tbl, ta, tb, nblk, cnt, off, fill ? list : nullptr,
                                                  mid);
        else
            k_tile_keep<1><<<blocks, 256, 0, s>>>(meta, g.prange, tbl, ta, tb, nblk, cnt, off, fill ? list : nullptr,
                                                  mid);
        MDET_LAUNCHED(ctx, "k_tile_keep");
        if (!fill) MDET_CUDA(ctx, cub::DeviceScan::ExclusiveSum(tmp, tmpb, cnt, off, (int)ta + 1, s));
    }
    out->list = list;
    out->rowoff = off;
    out->total = off + ta;
    out->row_order = nullptr;
    if (wave) {
        uint32_t *keys = mid, *vals = mid + ta, *keys2 = mid + 2ull * ta, *vals2 = mid + 3ull * ta;
        uint32_t* order = mid + 4ull * ta;
        size_t sb = 0;
        cub::DeviceRadixSort::SortPairs(nullptr, sb, keys, keys2, vals, vals2, (int)ta, 0, 32, s);
        void* stmp = ctx_scratch(ctx, "tl.sorttmp", sb);
        if (!stmp) return MDET_ERR_NOMEM;
        MDET_CUDA(ctx, cub::DeviceRadixSort::SortPairs(stmp, sb, keys, keys2, vals, vals2, (int)ta, 0, 32, s));
        k_wave_keys<<<(ta + 255) / 256, 256, 0, s>>>(vals2, cnt, ta, kWaveGroup * wave, keys);
        MDET_LAUNCHED(ctx, "k_wave_keys");
        MDET_CUDA(ctx, cub::DeviceRadixSort::SortPairs(stmp, sb, keys, keys2, vals2, order, (int)ta, 0, 32, s));
        out->row_order = order;
    }
    return MDET_OK;
}
