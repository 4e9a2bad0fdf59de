// graph_exact.cu -- exact scoring of filtered pairs and per-contig top-k.
//
// Every pair that passed a distance filter is scored again from the FP32
// TNF rows: the reference's terms float((a_k - b_k)^2) (cuda/Cuda2.cu:194-196)
// summed with compensated FP32 arithmetic, the square root and the MetaBAT2
// logistic model (cuda/Cuda2.cu:199-240) in float-float arithmetic (ff.cuh,
// about 48 significant bits) from per-contig parts F(x), G(y) and the pair
// term H(x*y).  A pair is an edge when its
// pre-probability beats logit(cutoff) (cuda/Cuda2.cu:257-260); its score is
// sigmoid(pre).  Edges are then grouped per contig (both directions), each
// contig keeps its best max_edges by (score desc, original column asc), and
// (i, j) is emitted for i < j in original indices (cuda/Cuda2.cu:921-946).
#include <cub/cub.cuh>

#include "exact.cuh"

using namespace mdet_exact;

namespace {

struct ExactArgs {
    const uint2* cand;
    unsigned long long ncand;
    const uint32_t* row_map;  // maxprob: sample slot -> sorted position; graph: null
    bool swapped;             // maxprob: pairs are (sorted position, sample slot)
    const float* x32;
    const PartsFF* parts;
    ModelHFF H;
    double L;
    ff Lff;
    const BlkCut* blk_L;  // optional per-256-row-block cutoff
    const unsigned long long* ncand_dev;  // optional device candidate count (ncand is then its cap)
    const uint8_t* low;   // optional abundance gate per sorted position (graph only)
    // graph outputs
    Edge* edges;
    unsigned long long* nedges;
    uint32_t* deg;
    // maxprob output
    unsigned long long* maxkey;
};

// Squared distances of 32 candidates per warp: candidate base + L belongs to
// lane L.  Eight lanes share one candidate at a time, so each row is read in
// coalesced 128-byte runs (lane k of the group takes float4 columns k, k+8,
// k+16 and k+24 and column 128+k); partial sums keep their rounding errors
// (TwoSum) through the group reduction.  Returns the owner lane's (sum, error)
// pair and its rows.
__device__ __forceinline__ ff warp_dist2(const uint2* __restrict__ cand, unsigned long long ncand,
                                         unsigned long long base, const uint32_t* __restrict__ row_map,
                                         const float* __restrict__ x32, uint32_t lane, uint32_t& si, uint32_t& sj,
                                         bool swapped = false) {
    const uint32_t grp = lane >> 3, sub = lane & 7;
    // every lane loads its own candidate once (one coalesced read for the
    // warp); the rounds below take the row indices by shuffle, so the row
    // reads of a round depend on no further load
    const bool own = base + lane < ncand;
    si = sj = 0;
    if (own) {
        uint2 cd = cand[base + lane];
        if (swapped) cd = make_uint2(cd.y, cd.x);
        si = row_map ? row_map[cd.x] : cd.x;
        sj = cd.y;
    }
    float ms = 0.f, mc = 0.f;
#pragma unroll 1
    for (uint32_t it = 0; it < 8; ++it) {
        const uint32_t from = it * 4 + grp;  // lane owning the candidate of this group and round
        const unsigned long long k = base + from;
        const uint32_t a = __shfl_sync(0xffffffffu, si, from);
        const uint32_t b = __shfl_sync(0xffffffffu, sj, from);
        float s = 0.f, c = 0.f;
        if (k < ncand) {
            const float* ra = x32 + (uint64_t)a * MDET_NTNF;
            const float* rb = x32 + (uint64_t)b * MDET_NTNF;
            f32x2 s2 = 0, c2 = 0;  // two chains, {0, 0}
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) {
                const ulonglong2 x = __ldg(reinterpret_cast<const ulonglong2*>(ra) + sub + 8 * q);
                const ulonglong2 y = __ldg(reinterpret_cast<const ulonglong2*>(rb) + sub + 8 * q);
                const f32x2 d0 = sub2(x.x, y.x), d1 = sub2(x.y, y.y);
                two_sum_acc2(s2, c2, square2(d0));
                two_sum_acc2(s2, c2, square2(d1));
            }
            const float d = __fsub_rn(__ldg(ra + 128 + sub), __ldg(rb + 128 + sub));
            const float2 sv = unpack2(s2), cv = unpack2(c2);
            const ff t = two_sum(sv.x, sv.y);
            s = t.hi;
            c = __fadd_rn(__fadd_rn(cv.x, cv.y), t.lo);
            two_sum_acc(s, c, __fmul_rn(d, d));
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const float s2 = __shfl_xor_sync(0xffffffffu, s, o);
            const float c2 = __shfl_xor_sync(0xffffffffu, c, o);
            const ff t = two_sum(s, s2);
            s = t.hi;
            c = __fadd_rn(__fadd_rn(c, c2), t.lo);
        }
        // candidate base + L was handled in round L / 4 by group L % 4
        const uint32_t src = 8 * (lane & 3);
        const float vs = __shfl_sync(0xffffffffu, s, src);
        const float vc = __shfl_sync(0xffffffffu, c, src);
        if ((lane >> 2) == it) {
            ms = vs;
            mc = vc;
        }
    }
    return quick_two_sum(ms, mc);
}

constexpr uint32_t kEdgeQueue = 96;

// Bound by the row reads: from DRAM at a million contigs, by instruction issue
// where the rows fit L2.  The kernel may take 80 registers (three blocks an
// SM), so that a round's ten row loads are in flight at once (1,000,000 contigs:
// 21.4 ms in 40 registers, 17.3 in 68); a warp collects its edges in shared
// memory and reserves list slots 65 to 96 at a time, without a barrier.  20,000
// contigs (2.85 M candidates): 281 us with 40 registers, six blocks and a
// block-wide reservation, 243 us with packed arithmetic, 209 us here;
// 1,000,000: 19.6 -> 17.3 ms.
__global__ void __launch_bounds__(256, 3) k_exact_graph(ExactArgs p) {
    __shared__ Edge queue[8][kEdgeQueue];
    if (p.ncand_dev) p.ncand = min(*p.ncand_dev, p.ncand);
    const bool model2 = p.L < kLn9;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    Edge* q = queue[w];
    uint32_t held = 0;  // edges in the warp's queue
    const unsigned long long step = gridDim.x * 256ull;
    for (unsigned long long base = blockIdx.x * 256ull + 32ull * w; base < p.ncand; base += step) {
        uint32_t si, sj;
        const ff d2 = warp_dist2(p.cand, p.ncand, base, nullptr, p.x32, lane, si, sj);
        bool edge = false;
        double sim = 0;
        // a pair of two contigs without a depth above 1 is never an edge (is_nz)
        if (base + lane < p.ncand && !(p.low && p.low[si] && p.low[sj])) {
            ff Lc = p.Lff;
            bool m2 = model2;
            if (p.blk_L) {
                const BlkCut bc = p.blk_L[si >> 8];
                Lc = bc.L;
                m2 = bc.model2 != 0;
            }
            const ff pre = pre_prob(p.parts[si], p.parts[sj], ff_sqrt(d2), p.H, m2);
            if (ff_gt(pre, Lc)) {
                edge = true;
                sim = sim_of(pre);
            }
        }
        const uint32_t bal = __ballot_sync(0xffffffffu, edge);
        if (edge) {
            Edge e;
            e.i = si;
            e.j = sj;
            e.sim = sim;
            q[held + __popc(bal & ((1u << lane) - 1u))] = e;
            atomicAdd(&p.deg[si], 1u);
            atomicAdd(&p.deg[sj], 1u);
        }
        held += __popc(bal);
        // flush when another 32 may not fit, and after the warp's last candidates
        if (held > kEdgeQueue - 32 || (base + step >= p.ncand && held)) {
            __syncwarp();
            unsigned long long at = 0;
            if (lane == 0) at = atomicAdd(p.nedges, (unsigned long long)held);
            at = __shfl_sync(0xffffffffu, at, 0);
            for (uint32_t k = lane; k < held; k += 32) p.edges[at + k] = q[k];
            held = 0;
            __syncwarp();
        }
    }
}

__global__ void __launch_bounds__(256, 3) k_exact_maxprob(ExactArgs p) {
    const uint32_t lane = threadIdx.x & 31;
    const unsigned long long warps = (unsigned long long)gridDim.x * (blockDim.x / 32);
    for (unsigned long long base = ((unsigned long long)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5)) * 32;
         base < p.ncand; base += warps * 32) {
        uint32_t si, sj;
        const ff d2 = warp_dist2(p.cand, p.ncand, base, p.row_map, p.x32, lane, si, sj, p.swapped);
        const unsigned long long idx = base + lane;
        if (idx < p.ncand && si != sj) {  // skip the sampled contig itself
            const ff pre = pre_prob(p.parts[si], p.parts[sj], ff_sqrt(d2), p.H, true);
            const uint2 cd = p.cand[idx];
            atomicMax(&p.maxkey[p.swapped ? cd.y : cd.x], dkey(ff_to_double(pre)));
        }
    }
}

// Distance and probability of given pairs (original indices, mapped through inv).
__global__ void k_pair_scores(const uint64_t* __restrict__ pairs, uint64_t m, const uint32_t* __restrict__ inv,
                              const float* __restrict__ x32, const PartsFF* __restrict__ parts, ModelHFF H,
                              double* __restrict__ dist, double* __restrict__ prob) {
    for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < m; q += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t i = inv[pairs[2 * q]], j = inv[pairs[2 * q + 1]];
        const ff d = exact_dist(x32 + (uint64_t)i * MDET_NTNF, x32 + (uint64_t)j * MDET_NTNF);
        const ff pre = pre_prob(parts[i], parts[j], d, H, true);
        if (dist) dist[q] = ff_to_double(d);
        if (prob) prob[q] = sim_of(pre);
    }
}

__global__ void k_scatter(const Edge* __restrict__ edges, unsigned long long ne_cap,
                          const unsigned long long* __restrict__ ne_dev, const uint32_t* __restrict__ perm,
                          const unsigned long long* __restrict__ rowptr, uint32_t* __restrict__ cursor,
                          Ent* __restrict__ list) {
    const unsigned long long ne = ne_dev ? min(*ne_dev, ne_cap) : ne_cap;
    for (unsigned long long e = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; e < ne;
         e += (unsigned long long)gridDim.x * blockDim.x) {
        Edge ed = edges[e];
        uint32_t a = atomicAdd(&cursor[ed.i], 1u);
        uint32_t b = atomicAdd(&cursor[ed.j], 1u);
        Ent x;
        x.sim = ed.sim;
        x.pad = 0;
        x.ocol = perm[ed.j];
        list[rowptr[ed.i] + a] = x;
        x.ocol = perm[ed.i];
        list[rowptr[ed.j] + b] = x;
    }
}

__device__ __forceinline__ bool before(const Ent& a, const Ent& b) {
    return a.sim > b.sim || (a.sim == b.sim && a.ocol < b.ocol);
}

constexpr int kWarpCap = 1024;
constexpr int kTopkWarps = 4;

// Warp per contig (sorted position s) with at most 1024 edges: bitonic sort
// in shared memory, keep the best max_edges in place.
__global__ void __launch_bounds__(kTopkWarps * 32) k_topk_warp(
    const unsigned long long* __restrict__ rowptr, const uint32_t* __restrict__ deg, const uint32_t* __restrict__ perm,
    uint32_t n, uint32_t max_edges, Ent* __restrict__ list, uint32_t* __restrict__ out_cnt,
    uint32_t* __restrict__ big, unsigned int* __restrict__ nbig) {
    extern __shared__ __align__(16) unsigned char sm[];
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Ent* e = reinterpret_cast<Ent*>(sm) + (size_t)w * kWarpCap;
    for (uint32_t s = blockIdx.x * kTopkWarps + w; s < n; s += gridDim.x * kTopkWarps) {
        const uint32_t cnt = deg[s];
        const uint32_t orow = perm[s];
        if (cnt > kWarpCap) {
            if (lane == 0) big[atomicAdd(nbig, 1u)] = s;
            continue;
        }
        Ent* row = list + rowptr[s];
        uint32_t P = 1;
        while (P < cnt) P <<= 1;
        if (cnt > max_edges || cnt > 1) {
            for (uint32_t i = lane; i < P; i += 32) {
                if (i < cnt)
                    e[i] = row[i];
                else {
                    e[i].sim = -1.0;
                    e[i].ocol = 0xFFFFFFFFu;
                }
            }
            __syncwarp();
            for (uint32_t k = 2; k <= P; k <<= 1)
                for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                    for (uint32_t i = lane; i < P; i += 32) {
                        uint32_t ixj = i ^ j;
                        if (ixj > i) {
                            Ent a = e[i], b = e[ixj];
                            bool up = (i & k) == 0;
                            if (up ? before(b, a) : before(a, b)) {
                                e[i] = b;
                                e[ixj] = a;
                            }
                        }
                    }
                    __syncwarp();
                }
        } else {
            for (uint32_t i = lane; i < cnt; i += 32) e[i] = row[i];
            __syncwarp();
        }
        const uint32_t keep = cnt < max_edges ? cnt : max_edges;
        uint32_t c = 0;
        for (uint32_t i = lane; i < keep; i += 32) {
            row[i] = e[i];
            c += e[i].ocol > orow;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        if (lane == 0) out_cnt[orow] = c;
        __syncwarp();
    }
}

constexpr int kBigCap = 8192;

// Block per contig with more than 1024 edges: repeated sort of the running
// best plus the next chunk in a 8192-entry shared buffer.
__global__ void __launch_bounds__(1024) k_topk_big(const uint32_t* __restrict__ big, const unsigned int* __restrict__ nbig,
                                                   const unsigned long long* __restrict__ rowptr,
                                                   const uint32_t* __restrict__ deg, const uint32_t* __restrict__ perm,
                                                   uint32_t max_edges, Ent* __restrict__ list,
                                                   uint32_t* __restrict__ out_cnt) {
    extern __shared__ __align__(16) unsigned char sm[];
    Ent* e = reinterpret_cast<Ent*>(sm);
    __shared__ uint32_t red;
    const uint32_t nb = *nbig;
    for (uint32_t bi = blockIdx.x; bi < nb; bi += gridDim.x) {
        const uint32_t s = big[bi];
        const uint32_t cnt = deg[s], orow = perm[s];
        Ent* row = list + rowptr[s];
        uint32_t kept = 0, base = 0;
        while (base < cnt) {
            uint32_t take = min((uint32_t)kBigCap - kept, cnt - base);
            for (uint32_t i = threadIdx.x; i < (uint32_t)kBigCap - kept; i += blockDim.x) {
                if (i < take)
                    e[kept + i] = row[base + i];
                else {
                    e[kept + i].sim = -1.0;
                    e[kept + i].ocol = 0xFFFFFFFFu;
                }
            }
            __syncthreads();
            for (uint32_t k = 2; k <= (uint32_t)kBigCap; k <<= 1)
                for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                    for (uint32_t i = threadIdx.x; i < (uint32_t)kBigCap; i += blockDim.x) {
                        uint32_t ixj = i ^ j;
                        if (ixj > i) {
                            Ent a = e[i], b = e[ixj];
                            bool up = (i & k) == 0;
                            if (up ? before(b, a) : before(a, b)) {
                                e[i] = b;
                                e[ixj] = a;
                            }
                        }
                    }
                    __syncthreads();
                }
            base += take;
            kept = min(max_edges, kept + take);
            __syncthreads();
        }
        if (threadIdx.x == 0) red = 0;
        __syncthreads();
        uint32_t c = 0;
        for (uint32_t i = threadIdx.x; i < kept; i += blockDim.x) {
            row[i] = e[i];
            c += e[i].ocol > orow;
        }
        atomicAdd(&red, c);
        __syncthreads();
        if (threadIdx.x == 0) out_cnt[orow] = red;
        __syncthreads();
    }
}

// ---- selection top-k: warp per contig --------------------------------------
// A row's kept set is its max_edges best entries under (sim descending, ocol
// ascending).  Ordered as the 96-bit key (bits of sim, ~ocol) -- sim is a
// positive double, so its bits order like its value -- the kept set is every
// entry whose key is >= the max_edges-th largest key, found by a radix
// select (8-bit digits, most significant first).  Only kept entries with ocol
// above the row's own index are emitted, so only those are sorted (bitonic
// network in registers) and written to the front of the row.  topk_row does
// this on 64-bit values; topk_any, on the full keys, takes any row.

// Keys are the bit patterns of positive doubles, which order like the
// values, so every comparison is an integer one (FP64 is slow on this part).
__device__ __forceinline__ bool kv_less(unsigned long long s1, uint32_t c1, unsigned long long s2, uint32_t c2) {
    return s1 > s2 || (s1 == s2 && c1 < c2);
}

// In-lane compare-exchange of slots e and e | JE (stride >= 32 entries).
template <int E, int JE>
__device__ __forceinline__ void stage_in_lane(unsigned long long (&s)[E], uint32_t (&c)[E], uint32_t lane,
                                              uint32_t k) {
#pragma unroll
    for (int e = 0; e < E; ++e) {
        if ((e & JE) == 0) {
            const int e2 = e | JE;
            const bool up = ((((uint32_t)e * 32u + lane) & k) == 0);
            const bool sw = up ? kv_less(s[e2], c[e2], s[e], c[e]) : kv_less(s[e], c[e], s[e2], c[e2]);
            const unsigned long long s1 = sw ? s[e2] : s[e], s2 = sw ? s[e] : s[e2];
            const uint32_t c1 = sw ? c[e2] : c[e], c2 = sw ? c[e] : c[e2];
            s[e] = s1;
            s[e2] = s2;
            c[e] = c1;
            c[e2] = c2;
        }
    }
}

template <int E>
__device__ __forceinline__ void bitonic_stage(unsigned long long (&s)[E], uint32_t (&c)[E], uint32_t lane, uint32_t k,
                                              uint32_t j) {
    if (j >= 32) {
        const uint32_t je = j >> 5;
        if (E >= 2 && je == 1) stage_in_lane<E, 1>(s, c, lane, k);
        if (E >= 4 && je == 2) stage_in_lane<E, (E >= 4 ? 2 : 1)>(s, c, lane, k);
        if (E >= 8 && je == 4) stage_in_lane<E, (E >= 8 ? 4 : 1)>(s, c, lane, k);
        if (E >= 16 && je == 8) stage_in_lane<E, (E >= 16 ? 8 : 1)>(s, c, lane, k);
    } else {
        const bool lower = (lane & j) == 0;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const bool up = ((((uint32_t)e * 32u + lane) & k) == 0);
            const unsigned long long os = __shfl_xor_sync(0xffffffffu, s[e], (int)j);
            const uint32_t oc = __shfl_xor_sync(0xffffffffu, c[e], (int)j);
            const bool take = (lower == up) ? kv_less(os, oc, s[e], c[e]) : kv_less(s[e], c[e], os, oc);
            s[e] = take ? os : s[e];
            c[e] = take ? oc : c[e];
        }
    }
}

// Sorts entries [0, m) of the warp's staging buffer best-first into row[0, m).
template <int E>
__device__ __forceinline__ void sort_out(const unsigned long long* __restrict__ key, const uint32_t* __restrict__ col,
                                         uint32_t m, uint32_t lane, Ent* __restrict__ row) {
    unsigned long long s[E];
    uint32_t c[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const uint32_t i = (uint32_t)e * 32u + lane;
        s[e] = i < m ? key[i] : 0ull;  // padding sorts last (every real key is a positive double)
        c[e] = i < m ? col[i] : 0xFFFFFFFFu;
    }
    uint32_t P = 32u * E;
    while (P / 2 >= m && P > 64) P >>= 1;  // the network only needs the next power of two
#pragma unroll 1
    for (uint32_t k = 2; k <= P; k <<= 1)
#pragma unroll 1
        for (uint32_t j = k >> 1; j > 0; j >>= 1) bitonic_stage<E>(s, c, lane, k, j);
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const uint32_t i = (uint32_t)e * 32u + lane;
        if (i < m) {
            Ent x;
            x.sim = __longlong_as_double((long long)s[e]);
            x.ocol = c[e];
            x.pad = 0;
            row[i] = x;
        }
    }
}

constexpr int kSelWarps = 4;

__device__ __forceinline__ uint32_t sel_digit(unsigned long long hi, uint32_t lo, int p) {
    return p < 8 ? (uint32_t)(hi >> (56 - 8 * p)) & 255u : (lo >> (24 - 8 * (p - 8))) & 255u;
}

// key (hi, lo) agrees with the prefix (P_hi, P_lo) on its first p digits
__device__ __forceinline__ bool sel_match(unsigned long long hi, uint32_t lo, unsigned long long P_hi, uint32_t P_lo,
                                          int p) {
    if (p == 0) return true;
    if (p < 8) return (hi >> (64 - 8 * p)) == (P_hi >> (64 - 8 * p));
    if (hi != P_hi) return false;
    return p == 8 || (lo >> (32 - 8 * (p - 8))) == (P_lo >> (32 - 8 * (p - 8)));
}

// The highest bin of a 256-bin histogram at which the count from the top
// reaches `need` (>= 1, at most the total), the count above it and its own.
__device__ __forceinline__ void sel_bin(const uint32_t* __restrict__ hist, uint32_t lane, uint32_t need, uint32_t& bin,
                                        uint32_t& above, uint32_t& count) {
    // lane L owns bins [8L, 8L + 8); count the bins above each lane's
    const uint4 b0 = *reinterpret_cast<const uint4*>(hist + 8 * lane);
    const uint4 b1 = *reinterpret_cast<const uint4*>(hist + 8 * lane + 4);
    const uint32_t b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
    uint32_t own = 0;
#pragma unroll
    for (int t = 0; t < 8; ++t) own += b[t];
    uint32_t suf = own;  // inclusive sum over lanes >= lane
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_down_sync(0xffffffffu, suf, o);
        if (lane + o < 32) suf += v;
    }
    uint32_t at = suf - own;
    int found = -1;
    uint32_t cnt = 0;
    if (at < need && need <= suf) {
#pragma unroll
        for (int t = 7; t >= 0; --t) {
            if (found < 0 && at + b[t] >= need) {
                found = (int)(lane * 8 + t);
                cnt = b[t];
            }
            if (found < 0) at += b[t];
        }
    }
    const uint32_t who = __ffs(__ballot_sync(0xffffffffu, found >= 0)) - 1;
    bin = (uint32_t)__shfl_sync(0xffffffffu, found, who);
    above = __shfl_sync(0xffffffffu, at, who);
    count = __shfl_sync(0xffffffffu, cnt, who);
}

__device__ __forceinline__ void sel_clear(uint32_t* __restrict__ hist, uint32_t lane) {
    *reinterpret_cast<uint4*>(hist + 8 * lane) = make_uint4(0, 0, 0, 0);
    *reinterpret_cast<uint4*>(hist + 8 * lane + 4) = make_uint4(0, 0, 0, 0);
    __syncwarp();
}

// A row of any length and with any scores: the entries are read from memory in
// every pass, keys are the full 96 bits.
template <int EMAX>
__device__ __noinline__ uint32_t topk_any(uint32_t cnt, uint32_t orow, uint32_t max_edges, Ent* __restrict__ row,
                                          unsigned long long* __restrict__ key, uint32_t* __restrict__ col,
                                          uint32_t* __restrict__ hist, uint32_t lane) {
    // threshold key (P_hi, P_lo): kept iff key >= it
    unsigned long long P_hi = 0;
    uint32_t P_lo = 0;
    if (cnt > max_edges) {
        uint32_t need = max_edges;
        for (int p = 0; p < 12; ++p) {
            sel_clear(hist, lane);
            for (uint32_t i = lane; i < cnt; i += 32) {
                const Ent x = row[i];
                const unsigned long long hi = (unsigned long long)__double_as_longlong(x.sim);
                const uint32_t lo = ~x.ocol;
                if (sel_match(hi, lo, P_hi, P_lo, p)) atomicAdd(&hist[sel_digit(hi, lo, p)], 1u);
            }
            __syncwarp();
            uint32_t bin, above, count;
            sel_bin(hist, lane, need, bin, above, count);
            __syncwarp();
            need -= above;
            if (p < 8)
                P_hi |= (unsigned long long)bin << (56 - 8 * p);
            else
                P_lo |= bin << (24 - 8 * (p - 8));
            if (count == need) break;
        }
    }
    // compact the kept entries with ocol > orow
    uint32_t m = 0;
    for (uint32_t base = 0; base < cnt; base += 32) {
        const uint32_t i = base + lane;
        unsigned long long hi = 0;
        uint32_t c = 0;
        bool take = false;
        if (i < cnt) {
            const Ent x = row[i];
            hi = (unsigned long long)__double_as_longlong(x.sim);
            c = x.ocol;
            const uint32_t lo = ~c;
            take = c > orow && (hi > P_hi || (hi == P_hi && lo >= P_lo));
        }
        const uint32_t bal = __ballot_sync(0xffffffffu, take);
        const uint32_t q = m + __popc(bal & ((1u << lane) - 1u));
        if (take && q < max_edges) {
            key[q] = hi;
            col[q] = c;
        }
        m += __popc(bal);
    }
    __syncwarp();
    m = min(m, max_edges);
    if (m <= 64)
        sort_out<2>(key, col, m, lane, row);
    else if (m <= 128)
        sort_out<4>(key, col, m, lane, row);
    else
        sort_out<EMAX>(key, col, m, lane, row);
    return m;
}

// Exchange of two values, the larger first when `up`.
__device__ __forceinline__ void order2(unsigned long long& a, unsigned long long& b, bool up) {
    const bool sw = (b > a) == up;
    const unsigned long long t = sw ? b : a;
    b = sw ? a : b;
    a = t;
}

// Sorts 32 * E distinct values (zeros may repeat) in shared memory, largest
// first: value i in lane i / E, slot i % E, so that strides below E stay in
// the lane.
template <int E>
__device__ __forceinline__ void sort_desc(unsigned long long* __restrict__ v, uint32_t m, uint32_t lane) {
    unsigned long long x[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const uint32_t i = (uint32_t)e * 32u + lane;
        x[e] = i < m ? v[i] : 0ull;
    }
    __syncwarp();
    // every lane's slots, alternate lanes in opposite order
#pragma unroll
    for (int k = 2; k <= E; k <<= 1)
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1)
#pragma unroll
            for (int e = 0; e < E; ++e)
                if (!(e & j)) order2(x[e], x[e | j], k == E ? (lane & 1) == 0 : (e & k) == 0);
    // merges of 2, 4, .. 32 lanes
#pragma unroll 1
    for (uint32_t k = 2; k <= 32; k <<= 1) {
        const bool up = (lane & k) == 0;
#pragma unroll 1
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            const bool large = ((lane & j) == 0) == up;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const unsigned long long o = __shfl_xor_sync(0xffffffffu, x[e], (int)j);
                x[e] = (o > x[e]) == large ? o : x[e];
            }
        }
#pragma unroll
        for (int j = E >> 1; j > 0; j >>= 1)
#pragma unroll
            for (int e = 0; e < E; ++e)
                if (!(e & j)) order2(x[e], x[e | j], up);
    }
#pragma unroll
    for (int e = 0; e < E; ++e) v[lane * E + e] = x[e];
    __syncwarp();
}

// The first m of the row's values, largest first (shared memory).
template <int EMAX>
__device__ __forceinline__ void sort_row(unsigned long long* __restrict__ x, uint32_t m, uint32_t lane) {
    if (m <= 64)
        sort_desc<2>(x, m, lane);
    else if (m <= 128)
        sort_desc<4>(x, m, lane);
    else if (EMAX == 8 || m <= 256)
        sort_desc<8>(x, m, lane);
    else
        sort_desc<EMAX>(x, m, lane);
}

// The same out of line: one copy for both sorts of a row where registers are short
// (limits to 256: rows of 99 and 499 entries 74 and 174 us inline, 63 and 166 so; larger
// limits 301 inline and 328 out of line at 499), and for the second sort.
template <int EMAX>
__device__ __noinline__ void sort_again(unsigned long long* __restrict__ x, uint32_t m, uint32_t lane) {
    sort_row<EMAX>(x, m, lane);
}

// A row of at most 1,024 entries.  A value is the score's bits above the
// row's smallest, plus one (53 bits), then the entry's slot (10) and whether the
// row emits it (1): distinct, and ordered like the scores.  Equal scores go by
// column: at the border of the kept set by a selection among them, and in the
// emitted list by a second sort.  (40,000 contigs in genomes of 500, limit 200: 166 us,
// and 233 to 424 with equal contigs in pairs or in groups of 5, 20, 40 or 500; 784 to
// 1,270 where such rows went to topk_any.  Genomes of 800: 229 us, 625 by topk_any.)
// Returns the number of edges, or ~0 where
// this form does not do: scores that span 53 bits.
// col: the entries' columns in shared memory, or (kStaged false) none; they are then
// read from the row, which is written last.
template <int EMAX, bool kStaged>
__device__ __forceinline__ uint32_t topk_row(uint32_t cnt, uint32_t orow, uint32_t max_edges, Ent* __restrict__ row,
                                             unsigned long long* __restrict__ x, uint32_t* __restrict__ col,
                                             uint32_t* __restrict__ hist, uint32_t lane) {
    auto column = [&](unsigned long long v) {
        const uint32_t slot = (uint32_t)(v >> 1) & 1023u;
        return kStaged ? col[slot] : row[slot].ocol;
    };
    unsigned long long lo = ~0ull, hi = 0;
#pragma unroll 4
    for (uint32_t i = lane; i < cnt; i += 32) {
        const Ent t = row[i];
        const unsigned long long v = (unsigned long long)__double_as_longlong(t.sim);
        x[i] = v;
        if (kStaged) col[i] = t.ocol;
        lo = v < lo ? v : lo;
        hi = v > hi ? v : hi;
    }
#pragma unroll 1
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long l2 = __shfl_xor_sync(0xffffffffu, lo, o), h2 = __shfl_xor_sync(0xffffffffu, hi, o);
        lo = l2 < lo ? l2 : lo;
        hi = h2 > hi ? h2 : hi;
    }
    if (hi - lo >= (1ull << 53) - 2) return ~0u;
    // the max_edges-th largest value: histograms of 8 bits from the top of the
    // row's range down, until the bin has at most 32 values
    const bool select = cnt > max_edges;
    int shift = max(11, 64 - __clzll((long long)((hi - lo + 2) << 11)) - 8);  // score bits only
    if (select) sel_clear(hist, lane);
#pragma unroll 2
    for (uint32_t i = lane; i < cnt; i += 32) {
        const uint32_t c = kStaged ? col[i] : row[i].ocol;
        const unsigned long long v = (x[i] - lo + 1) << 11 | i << 1 | (c > orow ? 1u : 0u);
        x[i] = v;
        if (select) atomicAdd(&hist[(uint32_t)(v >> shift)], 1u);
    }
    unsigned long long T = 1;
    if (select) {
        uint32_t need = max_edges, bin, above, count;
        unsigned long long pre = 0;
        int width = 8;
#pragma unroll 1
        while (true) {
            __syncwarp();
            sel_bin(hist, lane, need, bin, above, count);
            __syncwarp();
            need -= above;
            pre = pre << width | bin;
            if (count <= 32 || shift == 11) break;
            width = shift - 11 < 8 ? shift - 11 : 8;
            shift -= width;
            sel_clear(hist, lane);
            for (uint32_t i = lane; i < cnt; i += 32) {
                const unsigned long long v = x[i] >> shift;
                if (v >> width == pre) atomicAdd(&hist[(uint32_t)v & ((1u << width) - 1u)], 1u);
            }
        }
        if (count > 32) {
            // that many have the border's score: the `need` smallest columns of them, by
            // histograms of the columns' complements; the others drop out
            uint32_t kpre = 0;
            int ks = 24;
#pragma unroll 1
            for (;; ks -= 8) {
                sel_clear(hist, lane);
                for (uint32_t i = lane; i < cnt; i += 32) {
                    const unsigned long long v = x[i];
                    const uint32_t key = v >> 11 == pre ? ~column(v) : 0u;
                    if (v >> 11 == pre && (ks == 24 || key >> (ks + 8) == kpre)) atomicAdd(&hist[key >> ks & 255u], 1u);
                }
                __syncwarp();
                sel_bin(hist, lane, need, bin, above, count);
                __syncwarp();
                need -= above;
                kpre = kpre << 8 | bin;
                if (count == need || ks == 0) break;
            }
            for (uint32_t i = lane; i < cnt; i += 32)
                if (x[i] >> 11 == pre && ~column(x[i]) >> ks < kpre) x[i] = 0ull;
            T = pre << 11;
        } else {
            // the bin's values, one a lane (in the histogram's place); the need-th largest
            unsigned long long* few = reinterpret_cast<unsigned long long*>(hist);
            uint32_t c = 0;
            for (uint32_t base = 0; base < cnt; base += 32) {
                const unsigned long long v = base + lane < cnt ? x[base + lane] : 0ull;
                const bool in = v && v >> shift == pre;
                const uint32_t bal = __ballot_sync(0xffffffffu, in);
                if (in) few[c + __popc(bal & ((1u << lane) - 1u))] = v;
                c += __popc(bal);
            }
            __syncwarp();
            const unsigned long long mine = lane < c ? few[lane] : 0ull;
            uint32_t rank = 0;
#pragma unroll 1
            for (uint32_t k = 0; k < c; ++k) rank += few[k] > mine;
            T = __shfl_sync(0xffffffffu, mine, __ffs(__ballot_sync(0xffffffffu, lane < c && rank + 1 == need)) - 1);
            // all values of T's score are in the bin; one left out makes the border a
            // tie: of them as many as are kept go by the smallest columns
            const bool eq = lane < c && mine >> 11 == T >> 11;
            if (__any_sync(0xffffffffu, eq && mine < T)) {
                const uint32_t all = __ballot_sync(0xffffffffu, eq);
                const uint32_t keep = __popc(__ballot_sync(0xffffffffu, eq && mine >= T));
                const uint32_t my = eq ? column(mine) : 0u;
                uint32_t before = 0;
#pragma unroll 1
                for (uint32_t m = all; m; m &= m - 1) before += __shfl_sync(0xffffffffu, my, __ffs(m) - 1) < my;
                if (eq && before >= keep) x[(uint32_t)(mine >> 1) & 1023u] = 0ull;
                T = T >> 11 << 11;
            }
        }
    }
    // the values to emit to the front
    uint32_t m = 0;
    __syncwarp();
    for (uint32_t base = 0; base < cnt; base += 32) {
        const unsigned long long v = base + lane < cnt ? x[base + lane] : 0ull;
        const bool take = v >= T && (v & 1);
        const uint32_t bal = __ballot_sync(0xffffffffu, take);  // every lane has read its value
        if (take) x[m + __popc(bal & ((1u << lane) - 1u))] = v;
        m += __popc(bal);
    }
    __syncwarp();
    if (EMAX == 8)
        sort_again<EMAX>(x, m, lane);
    else
        sort_row<EMAX>(x, m, lane);
    bool tie = false;
    for (uint32_t i = lane; i + 1 < m; i += 32) tie |= x[i] >> 11 == x[i + 1] >> 11;
    if (__any_sync(0xffffffffu, tie)) {
        // equal scores by column: the columns sorted behind their run's first place,
        // in the values' upper half (a place keeps its score, so only columns move)
        unsigned long long* y = x + 32 * EMAX;
        uint32_t run = 0;  // where the run of the last value before this lane's starts
        for (uint32_t base = 0; base < m; base += 32) {
            const uint32_t i = base + lane;
            const bool first = i < m && (i == 0 || x[i - 1] >> 11 != x[i] >> 11);
            const uint32_t heads = __ballot_sync(0xffffffffu, first) & (0xffffffffu >> (31 - lane));
            const uint32_t at = heads ? base + 31 - __clz(heads) : run;
            if (i < m) y[i] = ~((unsigned long long)at << 32 | column(x[i]));
            run = __shfl_sync(0xffffffffu, at, 31);
        }
        __syncwarp();
        sort_again<EMAX>(y, m, lane);
        for (uint32_t i = lane; i < m; i += 32) {
            Ent e;
            e.sim = __longlong_as_double((long long)((x[i] >> 11) - 1 + lo));
            e.ocol = ~(uint32_t)y[i];
            e.pad = 0;
            row[i] = e;
        }
        return m;
    }
    if (kStaged) {
        for (uint32_t i = lane; i < m; i += 32) {
            const unsigned long long v = x[i];
            Ent e;
            e.sim = __longlong_as_double((long long)((v >> 11) - 1 + lo));
            e.ocol = column(v);
            e.pad = 0;
            row[i] = e;
        }
    } else {
        // the columns of all edges, kept beside the sorted values, before the row is written
        uint32_t c[EMAX];
#pragma unroll
        for (int e = 0; e < EMAX; ++e) c[e] = e * 32 + lane < m ? column(x[e * 32 + lane]) : 0u;
        __syncwarp();
#pragma unroll
        for (int e = 0; e < EMAX; ++e) {
            const uint32_t i = e * 32 + lane;
            if (i >= m) break;
            Ent t;
            t.sim = __longlong_as_double((long long)((x[i] >> 11) - 1 + lo));
            t.ocol = c[e];
            t.pad = 0;
            row[i] = t;
        }
    }
    return m;
}

// Entries staged in shared memory per row, the columns beside them or (kLong) the
// values alone: limits to 256 fit seven blocks an SM with 7 KB a warp, the larger ones
// run four blocks, with room for every slot.
template <int EMAX>
struct RowCaps {
    static constexpr uint32_t kShort = EMAX == 8 ? 512 : 1024, kLong = EMAX == 8 ? 880 : 1024;
    static_assert(kShort >= 64 * EMAX, "the emitted values and the columns of equal ones");
    static constexpr uint32_t kBytes = kShort * 12 > kLong * 8 ? kShort * 12 : kLong * 8;
};

// Bound by issue (the entries are read once, about 2,000 instructions a row): one
// 64-bit value per entry, staged in shared memory so that the passes are short
// loops.  Held in registers, the unrolled passes outgrew the instruction cache:
// 48 assemblies of 400 to 6,000 contigs 613 us, 1,000,000 contigs 10.0 ms, with
// this form 324 us and 5.9 ms (96-bit keys and twelve digit passes: 1,098 us and
// 9.9 ms).  Seven blocks fit an SM's shared memory; 72 registers for them beat
// 113 at four blocks (382 us, 6.8 ms).
template <int EMAX>
__global__ void __launch_bounds__(kSelWarps * 32, EMAX == 8 ? 7 : 4)
    k_topk_sel(const unsigned long long* __restrict__ rowptr, const uint32_t* __restrict__ deg,
               const uint32_t* __restrict__ perm, uint32_t n, uint32_t max_edges_all,
               const uint32_t* __restrict__ blk_K, Ent* __restrict__ list, uint32_t* __restrict__ out_cnt) {
    using C = RowCaps<EMAX>;
    extern __shared__ __align__(16) unsigned char sel_smem[];
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char* base = sel_smem + w * (C::kBytes + 1024);
    uint32_t* hist = reinterpret_cast<uint32_t*>(base);
    unsigned long long* x = reinterpret_cast<unsigned long long*>(base + 1024);
    uint32_t* col = reinterpret_cast<uint32_t*>(base + 1024 + C::kShort * 8);
    for (uint32_t sp = blockIdx.x * kSelWarps + w; sp < n; sp += gridDim.x * kSelWarps) {
        const uint32_t cnt = deg[sp], orow = perm[sp];
        const uint32_t max_edges = blk_K ? blk_K[sp >> 8] : max_edges_all;
        Ent* row = list + rowptr[sp];
        uint32_t m = cnt ? ~0u : 0u;
        if (cnt && cnt <= C::kShort)
            m = topk_row<EMAX, true>(cnt, orow, max_edges, row, x, col, hist, lane);
        else if (EMAX == 8 && cnt && cnt <= C::kLong)
            m = topk_row<EMAX, false>(cnt, orow, max_edges, row, x, col, hist, lane);
        __syncwarp();
        if (m == ~0u) m = topk_any<EMAX>(cnt, orow, max_edges, row, x, col, hist, lane);
        if (lane == 0) out_cnt[orow] = m;
        __syncwarp();
    }
}

// Warp per original row: write its kept edges with ocol > row, in order.
// compacted: the row starts with exactly those edges (selection top-k).
// Rows (original index o) outside the sorted-position range [k0, k1) emit nothing.
__global__ void k_keep_rows(const uint32_t* __restrict__ inv, uint32_t n, uint32_t k0, uint32_t k1,
                            uint32_t* __restrict__ out_cnt) {
    const uint32_t o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= n) return;
    const uint32_t s = inv[o];
    if (s < k0 || s >= k1) out_cnt[o] = 0;
}

__global__ void k_emit(const uint32_t* __restrict__ inv, const unsigned long long* __restrict__ rowptr,
                       const uint32_t* __restrict__ deg, const Ent* __restrict__ list,
                       const unsigned long long* __restrict__ outptr, uint32_t n, uint32_t max_edges, int compacted,
                       uint64_t* __restrict__ from, uint64_t* __restrict__ to, double* __restrict__ stnf) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t o = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); o < n; o += gridDim.x * (blockDim.x / 32)) {
        const uint32_t s = inv[o];
        const uint32_t keep = compacted ? (uint32_t)(outptr[o + 1] - outptr[o]) : min(deg[s], max_edges);
        const Ent* row = list + rowptr[s];
        unsigned long long pos = outptr[o];
        for (uint32_t b = 0; b < keep; b += 32) {
            uint32_t i = b + lane;
            Ent x;
            bool ok = false;
            if (i < keep) {
                x = row[i];
                ok = x.ocol > o;
            }
            uint32_t bal = __ballot_sync(0xffffffffu, ok);
            if (ok) {
                unsigned long long q = pos + __popc(bal & ((1u << lane) - 1u));
                from[q] = o;
                to[q] = x.ocol;
                stnf[q] = x.sim;
            }
            pos += __popc(bal);
        }
    }
}

__global__ void k_maxprob_finish(const unsigned long long* __restrict__ maxkey, const uint32_t* __restrict__ slot_of,
                                 uint64_t m, double* __restrict__ out) {
    uint64_t b = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (b >= m) return;
    double pre = dkey_inv(maxkey[slot_of[b]]);
    // the reference seeds its running max with DBL_MIN (cuda/Cuda2.cu:287)
    const double dbl_min = 2.2250738585072014e-308;
    if (!(pre > dbl_min)) pre = dbl_min;
    out[b] = 1. - (1. / (1. + exp(pre)));
}

__global__ void k_widen(const uint32_t* __restrict__ src, uint64_t n, unsigned long long* __restrict__ dst) {
    uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i < n) dst[i] = src[i];
    if (i == n) dst[i] = 0;
}

__global__ void k_fill_u64(unsigned long long* p, uint64_t n, unsigned long long v) {
    uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i < n) p[i] = v;
}

}  // namespace

// ------------------------------------------------------------ host side --

int exact_graph(mdet_ctx* ctx, const GraphPrep& g, const uint2* cand, unsigned long long ncand, double L,
                Edge** edges_out, unsigned long long* nedges_out, uint32_t** deg_out, const BlkCut* blk_L,
                const unsigned long long* ncand_dev, unsigned long long** nedges_dev) {
    cudaStream_t s = ctx->stream;
    Edge* edges = (Edge*)ctx_scratch(ctx, "ex.edges", (ncand ? ncand : 1) * sizeof(Edge));
    unsigned long long* cnt = (unsigned long long*)ctx_scratch(ctx, "ex.cnt", 8);
    uint32_t* deg = (uint32_t*)ctx_scratch(ctx, "ex.deg", (uint64_t)g.n * 4);
    if (!edges || !cnt || !deg) return MDET_ERR_NOMEM;
    MDET_CUDA(ctx, cudaMemsetAsync(cnt, 0, 8, s));
    MDET_CUDA(ctx, cudaMemsetAsync(deg, 0, (uint64_t)g.n * 4, s));
    if (ncand) {
        ExactArgs p;
        memset(&p, 0, sizeof(p));
        p.cand = cand;
        p.ncand = ncand;
        p.x32 = g.x32;
        p.parts = g.parts;
        p.H = model_h_ff();
        p.L = L;
        p.Lff.hi = (float)L;
        p.Lff.lo = (float)(L - (double)p.Lff.hi);
        p.blk_L = blk_L;
        p.ncand_dev = ncand_dev;
        p.low = g.low;
        p.edges = edges;
        p.nedges = cnt;
        p.deg = deg;
        // three blocks fit an SM.  Rows that stay in L2 (half of it: each die
        // keeps its own copies): eight waves, for a short tail (20,000 contigs:
        // 222 us with one wave, 209 with eight).  Larger sets: one wave, so that
        // the list is swept once and near candidates find their rows in L2
        // (1,000,000 contigs: 16.3 -> 15.8 ms, 28 GB from DRAM instead of 78).
        const bool in_l2 = (uint64_t)g.n * MDET_NTNF * 4 <= (64ull << 20);
        const unsigned long long blocks = (ncand + 255) / 256;
        const unsigned long long cap = (unsigned long long)ctx->num_sms * (in_l2 ? 24 : 3);
        ctx_timer_begin(ctx, "k_exact_graph");
        k_exact_graph<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, s>>>(p);
        ctx_timer_end(ctx, "k_exact_graph");
        MDET_LAUNCHED(ctx, "k_exact_graph");
    }
    *edges_out = edges;
    *deg_out = deg;
    if (nedges_dev) {  // counts stay on the device (capturable); ncand bounds the edges
        *nedges_dev = cnt;
        *nedges_out = ncand;
        return MDET_OK;
    }
    MDET_CUDA(ctx, cudaMemcpyAsync(nedges_out, cnt, 8, cudaMemcpyDeviceToHost, s));
    MDET_CUDA(ctx, cudaStreamSynchronize(s));
    return MDET_OK;
}

int exact_maxprob(mdet_ctx* ctx, const GraphPrep& g, const uint2* cand, unsigned long long ncand,
                  const uint32_t* row_map, uint64_t m, const uint32_t* slot_of, double* d_out, bool swapped) {
    cudaStream_t s = ctx->stream;
    unsigned long long* maxkey = (unsigned long long*)ctx_scratch(ctx, "mp.maxkey", (m ? m : 1) * 8);
    if (!maxkey) return MDET_ERR_NOMEM;
    k_fill_u64<<<(unsigned)((m + 255) / 256), 256, 0, s>>>(maxkey, m, 0ull);
    MDET_LAUNCHED(ctx, "k_fill_u64");
    if (ncand) {
        ExactArgs p;
        memset(&p, 0, sizeof(p));
        p.cand = cand;
        p.ncand = ncand;
        p.row_map = row_map;
        p.swapped = swapped;
        p.x32 = g.x32;
        p.parts = g.parts;
        p.H = model_h_ff();
        p.maxkey = maxkey;
        unsigned long long blocks = (ncand + 255) / 256;
        int fit = 0;
        MDET_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k_exact_maxprob, 256, 0));
        unsigned long long cap = (unsigned long long)ctx->num_sms * (fit < 1 ? 1 : fit);
        ctx_timer_begin(ctx, "k_exact_maxprob");
    k_exact_maxprob<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, s>>>(p);
        ctx_timer_end(ctx, "k_exact_maxprob");
    MDET_LAUNCHED(ctx, "k_exact_maxprob");
    }
    k_maxprob_finish<<<(unsigned)((m + 255) / 256), 256, 0, s>>>(maxkey, slot_of, m, d_out);
    MDET_LAUNCHED(ctx, "k_maxprob_finish");
    return MDET_OK;
}

int pair_scores(mdet_ctx* ctx, const GraphPrep& g, const uint64_t* pairs, uint64_t m, double* dist, double* prob) {
    if (m == 0) return MDET_OK;
    const uint64_t blocks = std::min<uint64_t>((m + 255) / 256, (uint64_t)ctx->num_sms * 16);
    k_pair_scores<<<(unsigned)blocks, 256, 0, ctx->stream>>>(pairs, m, g.inv, g.x32, g.parts, model_h_ff(), dist, prob);
    MDET_LAUNCHED(ctx, "k_pair_scores");
    return MDET_OK;
}

int select_topk(mdet_ctx* ctx, const GraphPrep& g, const Edge* edges, unsigned long long ne, uint32_t* deg,
                uint32_t max_edges, uint64_t* n_out, const uint32_t* blk_K, const unsigned long long* ne_dev,
                uint32_t keep0, uint32_t keep1) {
    cudaStream_t s = ctx->stream;
    const uint32_t n = g.n;
    unsigned long long* rowptr = (unsigned long long*)ctx_scratch(ctx, "tk.rowptr", ((uint64_t)n + 1) * 8);
    uint32_t* cursor = (uint32_t*)ctx_scratch(ctx, "tk.cursor", (uint64_t)n * 4);
    Ent* list = (Ent*)ctx_scratch(ctx, "tk.list", (ne ? 2 * ne : 1) * sizeof(Ent));
    uint32_t* out_cnt = (uint32_t*)ctx_scratch(ctx, "tk.outcnt", (uint64_t)n * 4);
    unsigned long long* outptr = (unsigned long long*)ctx_scratch(ctx, "tk.outptr", ((uint64_t)n + 1) * 8);
    uint32_t* big = (uint32_t*)ctx_scratch(ctx, "tk.big", (uint64_t)n * 4);
    unsigned int* nbig = (unsigned int*)ctx_scratch(ctx, "tk.nbig", 8);
    if (!rowptr || !cursor || !list || !out_cnt || !outptr || !big || !nbig) return MDET_ERR_NOMEM;
    // 64-bit scans: widen the per-row counts (plus a trailing zero) first
    unsigned long long* w64 = (unsigned long long*)ctx_scratch(ctx, "tk.w64", ((uint64_t)n + 1) * 8);
    if (!w64) return MDET_ERR_NOMEM;
    size_t tb = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tb, w64, rowptr, (int)n + 1, s);
    void* tmp = ctx_scratch(ctx, "tk.cubtmp", tb);
    if (!tmp) return MDET_ERR_NOMEM;
    const unsigned wblocks = (unsigned)(((uint64_t)n + 1 + 255) / 256);
    k_widen<<<wblocks, 256, 0, s>>>(deg, n, w64);
    MDET_LAUNCHED(ctx, "k_widen");
    MDET_CUDA(ctx, cub::DeviceScan::ExclusiveSum(tmp, tb, w64, rowptr, (int)n + 1, s));
    MDET_CUDA(ctx, cudaMemsetAsync(cursor, 0, (uint64_t)n * 4, s));
    if (ne) {
        unsigned long long blocks = (ne + 255) / 256, cap = (unsigned long long)ctx->num_sms * 16;
        ctx_timer_begin(ctx, "k_scatter");
        k_scatter<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, s>>>(edges, ne, ne_dev, g.perm, rowptr, cursor,
                                                                           list);
        ctx_timer_end(ctx, "k_scatter");
        MDET_LAUNCHED(ctx, "k_scatter");
    }
    MDET_CUDA(ctx, cudaMemsetAsync(nbig, 0, 4, s));
    MDET_CUDA(ctx, cudaMemsetAsync(out_cnt, 0, (uint64_t)n * 4, s));
    if (max_edges <= 512) {
        // selection top-k, warp per row
        const unsigned blocks =
            (unsigned)std::min<uint64_t>(((uint64_t)n + kSelWarps - 1) / kSelWarps, (uint64_t)ctx->num_sms * 32);
        ctx_timer_begin(ctx, "k_topk_sel");
        if (max_edges <= 256) {
            constexpr size_t dyn = kSelWarps * (RowCaps<8>::kBytes + 1024);
            k_topk_sel<8><<<blocks, kSelWarps * 32, dyn, s>>>(rowptr, deg, g.perm, n, max_edges, blk_K, list, out_cnt);
        } else {
            constexpr size_t dyn = kSelWarps * (RowCaps<16>::kBytes + 1024);
            MDET_CUDA(ctx, cudaFuncSetAttribute(k_topk_sel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
            k_topk_sel<16><<<blocks, kSelWarps * 32, dyn, s>>>(rowptr, deg, g.perm, n, max_edges, blk_K, list, out_cnt);
        }
        ctx_timer_end(ctx, "k_topk_sel");
        MDET_LAUNCHED(ctx, "k_topk_sel");
    } else {
        if (blk_K) return ctx_fail(ctx, MDET_ERR_INVALID, "per-row max_edges needs max_edges <= 512");
        size_t dyn = (size_t)kTopkWarps * kWarpCap * sizeof(Ent);
        static bool set[64] = {false};
        if (!set[ctx->device & 63]) {
            MDET_CUDA(ctx, cudaFuncSetAttribute(k_topk_warp, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
            MDET_CUDA(ctx, cudaFuncSetAttribute(k_topk_big, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                (int)(kBigCap * sizeof(Ent))));
            set[ctx->device & 63] = true;
        }
        unsigned blocks = (unsigned)std::min<uint64_t>(((uint64_t)n + kTopkWarps - 1) / kTopkWarps,
                                                       (uint64_t)ctx->num_sms * 32);
        k_topk_warp<<<blocks, kTopkWarps * 32, dyn, s>>>(rowptr, deg, g.perm, n, max_edges, list, out_cnt, big, nbig);
        MDET_LAUNCHED(ctx, "k_topk_warp");
        k_topk_big<<<ctx->num_sms, 1024, kBigCap * sizeof(Ent), s>>>(big, nbig, rowptr, deg, g.perm, max_edges, list,
                                                                    out_cnt);
        MDET_LAUNCHED(ctx, "k_topk_big");
    }
    if (keep0 > 0 || keep1 < n) {
        if (max_edges > 512) return ctx_fail(ctx, MDET_ERR_INVALID, "row shards need max_edges <= 512");
        k_keep_rows<<<wblocks, 256, 0, s>>>(g.inv, n, keep0, keep1, out_cnt);
        MDET_LAUNCHED(ctx, "k_keep_rows");
    }
    k_widen<<<wblocks, 256, 0, s>>>(out_cnt, n, w64);
    MDET_LAUNCHED(ctx, "k_widen");
    MDET_CUDA(ctx, cub::DeviceScan::ExclusiveSum(tmp, tb, w64, outptr, (int)n + 1, s));
    if (ne_dev) {  // capturable: the total stays on the device (outptr[n])
        *n_out = 0;
        return MDET_OK;
    }
    unsigned long long total = 0;
    MDET_CUDA(ctx, cudaMemcpyAsync(&total, outptr + n, 8, cudaMemcpyDeviceToHost, s));
    MDET_CUDA(ctx, cudaStreamSynchronize(s));
    *n_out = total;
    return MDET_OK;
}

int emit_topk(mdet_ctx* ctx, const GraphPrep& g, uint32_t max_edges, uint64_t* d_from, uint64_t* d_to,
              double* d_stnf, uint64_t total) {
    cudaStream_t s = ctx->stream;
    const uint32_t n = g.n;
    const unsigned long long* rowptr = (const unsigned long long*)ctx->bufs["tk.rowptr"].p;
    const unsigned long long* outptr = (const unsigned long long*)ctx->bufs["tk.outptr"].p;
    const Ent* list = (const Ent*)ctx->bufs["tk.list"].p;
    const uint32_t* deg = (const uint32_t*)ctx->bufs["ex.deg"].p;
    if (total) {
        unsigned blocks = (unsigned)std::min<uint64_t>(((uint64_t)n + 7) / 8, (uint64_t)ctx->num_sms * 32);
        k_emit<<<blocks, 256, 0, s>>>(g.inv, rowptr, deg, list, outptr, n, max_edges, max_edges <= 512 ? 1 : 0,
                                      d_from, d_to, d_stnf);
        MDET_LAUNCHED(ctx, "k_emit");
    }
    return MDET_OK;
}
