// abundance.cu -- the coverage side of the graph: the pair gate of the
// abundance form (is_nz, cuda/Cuda2.cu:845-856, applied at 925) and the
// sTNF -> sSCR conversion of the edges (cuda/Cuda2.cu:1921-1971 with
// cal_abd_dist2 / cal_abd_dist 667-719, cal_abd_corr 1219-1245 and the ranks
// of cuda/ranker.h:56-80).
//
// Layout: the context keeps the reference's ABD (mean depth) and ABD_VAR
// (variance) as n x nabd row-major FP64 matrices in the original contig order,
// plus one byte per contig that says whether none of its depths exceeds 1,
// and, formed once when the depths are set, each contig's per-sample variance,
// clamped mean and CDF scale and its correlation deviations (k_abd_prep).
// sSCR runs one thread per edge over its nabd samples -- the crossing points
// of the two normal densities in float-float (abd_dist2_ff; in FP64 as the
// reference forms them where the variances are close), the four normal CDFs
// per sample in float-float from this project's erfc table, the
// correlation's cross sum --
// then three radix sorts (the abundance
// similarities, sTNF and the depth correlations) turn values into ranks and
// the ranks into quantiles of the similarity distribution.
//
// This unit is compiled without FMA contraction: sums and products round
// separately, as in the reference, so the depth correlations -- whose ranks
// pick quantiles -- come out bit-identical to a host evaluation.
#include <cub/cub.cuh>

#include "erfc_table.cuh"
#include "graph.cuh"

namespace {

// erfc(z), z >= 0, in float-float from this project's own table
// (erfc_table.cuh, generated by gen_erfc_table.py): degree-13 interpolants on
// 26 pieces of [0, 6.5], absolute error ~5e-16 before the float-float
// evaluation; 0 beyond 6.5 (erfc < 4e-20 there).  The FP32 pipes run this far
// faster than the FP64 pipe runs the double erfc.  The terms from degree 8 up
// run in FP32: they sum to less than 7e-10, so rounding them costs 4e-17, a
// tenth of the table's own error; degrees 7 to 2 (below 8e-3) take the shorter
// float-float sum, whose error is 2^-47 of its operands.  Kept out of line:
// the score kernel calls it from several places, and inlined copies stall the
// kernel on instruction fetch.  tab: the table in shared memory
// (load_erfc_table) -- the lanes sit on different pieces, and rows kErfcRow
// words apart put 16 of the 26 pieces on banks of their own, where reads of
// the table in global memory filled 60 % of the L1's wavefronts.
constexpr int kErfcRow = 2 * (MDET_ERFC_DEG + 2);
constexpr int kErfcWords = MDET_ERFC_PIECES * kErfcRow;
__device__ __forceinline__ void load_erfc_table(float* tab) {
    for (int i = threadIdx.x; i < MDET_ERFC_PIECES * (MDET_ERFC_DEG + 1); i += blockDim.x) {
        const int p = i / (MDET_ERFC_DEG + 1), j = i % (MDET_ERFC_DEG + 1);
        tab[p * kErfcRow + 2 * j] = kErfcTable[p][j][0];
        tab[p * kErfcRow + 2 * j + 1] = kErfcTable[p][j][1];
    }
    __syncthreads();
}
__device__ __noinline__ ff erfc_pos(ff z, const float* tab) {
    if (!(z.hi < 6.5f)) return z.hi != z.hi ? z : ff_make(0.f, 0.f);  // NaN stays
    const int p = min((int)(z.hi * 4.f), MDET_ERFC_PIECES - 1);
    // u = (z - centre) * 8, exact scaling of an exact difference
    ff u = ff_add_f(z, -((float)p + 0.5f) * 0.25f);
    u.hi *= 8.f;
    u.lo *= 8.f;
    const float2* c = reinterpret_cast<const float2*>(tab + p * kErfcRow);
    float h = c[MDET_ERFC_DEG].x;
#pragma unroll
    for (int j = MDET_ERFC_DEG - 1; j >= 8; --j) h = __fmaf_rn(h, u.hi, c[j].x);
    ff r = ff_make(h, 0.f);
#pragma unroll
    for (int j = 7; j >= 2; --j) {
        const ff m = ff_mul(r, u);
        const float2 k = c[j];
        const ff t = two_sum(m.hi, k.x);
        r = quick_two_sum(t.hi, __fadd_rn(t.lo, __fadd_rn(m.lo, k.y)));
    }
#pragma unroll
    for (int j = 1; j >= 0; --j) {
        const float2 k = c[j];
        r = ff_add(ff_mul(r, u), ff_make(k.x, k.y));
    }
    return r;
}

// erfc(-z) = 2 - erfc(z)
__device__ __forceinline__ ff erfc_ff(ff z, const float* tab) {
    const bool neg = z.hi < 0.f;
    const ff r = erfc_pos(neg ? ff_neg(z) : z, tab);
    return neg ? ff_add_f(ff_neg(r), 2.f) : r;
}

// 1 / (sd * sqrt(2)) in float-float: the per-(contig, sample) factor of the
// normal CDF below.
__device__ __forceinline__ ff cdf_scale(double sd) {
    return ff_recip(ff_mul(ff_from_double(sd), ff_make(0x1.6a09e6p+0f, 0x1.9fcef4p-26f)));  // sqrt(2)
}

// Boost's normal CDF, erfc(-(x - mean) / (sd * sqrt(2))) / 2 (the function
// the reference calls), with x - mean formed in FP64 as the reference forms
// it and the rest in float-float (isd = cdf_scale(sd)); returned in double.
__device__ __forceinline__ double normal_cdf_ff(double mean, ff isd, double x, const float* tab) {
    const ff diff = ff_from_double(x - mean);
    const ff z = ff_mul(diff, isd);
    return ff_to_double(erfc_ff(ff_neg(z), tab)) * 0.5;
}

// What the scoring needs of one contig's depths, formed once when the depths
// are set (everything here depends on one contig alone, so per edge it would
// be formed again for every edge the contig is in):
//   vv[i]   = s * s, s = sqrt(max(var[i], 1)) (the variance the FP64 crossing
//             points use);
//   ratio[i] = (i + 1) / (i + 2.0), as the reference forms it;
//   rec[i]  = everything the float-float path reads of sample i, side by
//             side (AbdRec): the clamped mean max(abd[i], 1e-6) as three
//             floats whose sum is exactly that double, cdf_scale(s), vv[i] and
//             its logarithm in float-float, and the deviation of depth i from
//             the running mean of depths 0 .. i - 1 (FP64);
//   sx      = sqrt of the running sum of squared deviations times i / (i + 1):
//             with the deviations, the one-row steps of cal_abd_corr, in its
//             order.  The edge's correlation is then (sum (dev1[i] * dev2[i]) *
//             ratio[i]) / (sx1 * sx2): the reference's operations on the
//             reference's values.
struct __align__(16) AbdRec {
    float m[3], isd_hi;
    float isd_lo, v_hi, v_lo, lv_hi;
    float lv_lo, pad;
    double dev;
};

__global__ void k_abd_prep(const double* __restrict__ abd, const double* __restrict__ var, uint64_t n, uint32_t nabd,
                           double* __restrict__ vv, double* __restrict__ ratio, AbdRec* __restrict__ rec,
                           double* __restrict__ sx) {
    const uint64_t t0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (t0 + 1 < nabd) ratio[t0] = (t0 + 1) / (t0 + 2.0);
    for (uint64_t r = t0; r < n; r += (uint64_t)gridDim.x * blockDim.x) {
        const double* a = abd + r * nabd;
        const double* w = var + r * nabd;
        double sxx = 0., mx = 0.;
        for (uint32_t i = 0; i < nabd; ++i) {
            const double u = w[i];
            const double sd = sqrt(u < 1 ? 1. : u);
            AbdRec q;
            vv[r * nabd + i] = sd * sd;
            const ff f = cdf_scale(sd), fv = ff_from_double(sd * sd), fl = ff_from_double(log(sd * sd));
            q.isd_hi = f.hi;
            q.isd_lo = f.lo;
            q.v_hi = fv.hi;
            q.v_lo = fv.lo;
            q.lv_hi = fl.hi;
            q.lv_lo = fl.lo;
            const double x = a[i];
            // the clamped mean as three floats that sum to it exactly
            const double mc = x < 1e-6 ? 1e-6 : x;
            q.m[0] = __double2float_rn(mc);
            const double r1 = mc - (double)q.m[0];
            q.m[1] = __double2float_rn(r1);
            q.m[2] = __double2float_rn(r1 - (double)q.m[1]);
            q.pad = 0.f;
            q.dev = 0.;
            if (i == 0) {
                mx = x;
            } else {
                const double t = i / (i + 1.0);
                const double dx = x - mx;
                sxx += dx * dx * t;
                mx += dx / (i + 1.0);
                q.dev = dx;
            }
            rec[r * nabd + i] = q;
        }
        sx[r] = sqrt(sxx);
    }
}

__global__ void k_abd_low(const double* __restrict__ abd, uint64_t n, uint32_t nabd, uint8_t* __restrict__ low) {
    for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < n; r += (uint64_t)gridDim.x * blockDim.x) {
        bool any = false;
        for (uint32_t i = 0; i < nabd; ++i) any = any || abd[r * nabd + i] > 1.;
        low[r] = any ? 0 : 1;
    }
}

__global__ void k_low_sorted(const uint32_t* __restrict__ perm, const uint8_t* __restrict__ low, uint64_t n,
                             uint8_t* __restrict__ out) {
    for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < n; s += (uint64_t)gridDim.x * blockDim.x)
        out[s] = low[perm[s]];
}


// Overlap of two normal densities from their crossing points k1 <= k2, the
// narrower distribution evaluated first (cal_abd_dist2), the FP64 form: the
// crossing points, whose numerator cancels when the variances are close, in
// FP64 in the reference's order; the four CDF values in float-float.  Used
// where abd_dist2_ff declines.
__device__ __noinline__ double abd_dist2(double m1, double v1, ff f1, double m2, double v2, ff f2, const float* tab) {
    double k1, k2;
    if (fabs(v2 - v1) < 1e-4) {
        k1 = k2 = (m1 + m2) / 2;
    } else {
        const double t = sqrt(v1 * v2 * ((m1 - m2) * (m1 - m2) - 2 * (v1 - v2) * log(sqrt(v2 / v1))));
        k1 = (t - m1 * v2 + m2 * v1) / (v1 - v2);
        k2 = (t + m1 * v2 - m2 * v1) / (v2 - v1);
    }
    if (k1 > k2) {
        const double x = k1;
        k1 = k2;
        k2 = x;
    }
    double ma = m1, mb = m2;
    ff fa = f1, fb = f2;
    if (v1 > v2) {
        ma = m2;
        fa = f2;
        mb = m1;
        fb = f1;
    }
    if (k1 == k2) return fabs(normal_cdf_ff(ma, fa, k1, tab) - normal_cdf_ff(mb, fb, k1, tab));
    return fabs(normal_cdf_ff(ma, fa, k2, tab) - normal_cdf_ff(ma, fa, k1, tab) + normal_cdf_ff(mb, fb, k1, tab) -
                normal_cdf_ff(mb, fb, k2, tab));
}

// One contig's sample as the float-float path reads it.
struct Rec {
    float m0, m1, m2;  // the clamped mean, exactly
    ff isd, v, lv;
    double dev;
};
__device__ __forceinline__ Rec load_rec(const AbdRec* __restrict__ p) {
    const float4* q = reinterpret_cast<const float4*>(p);
    const float4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
    Rec r;
    r.m0 = a.x, r.m1 = a.y, r.m2 = a.z;
    r.isd = ff_make(a.w, b.x);
    r.v = ff_make(b.y, b.z);
    r.lv = ff_make(b.w, c.x);
    r.dev = __hiloint2double(__float_as_int(c.w), __float_as_int(c.z));
    return r;
}

// The mean of r (three floats, each the rounding of what the ones before leave)
// against another double in that form: the first floats that differ decide.
__device__ __forceinline__ bool mean_gt(const Rec& r, float3 c) {
    return r.m0 > c.x || (r.m0 == c.x && (r.m1 > c.y || (r.m1 == c.y && r.m2 > c.z)));
}
__device__ __forceinline__ bool same_mean(const Rec& a, const Rec& b) {
    return a.m0 == b.m0 && a.m1 == b.m1 && a.m2 == b.m2;
}

// k - mean in float-float: error ~2^-48 of the result.
__device__ __forceinline__ ff ff_sub_mean(ff k, const Rec& r) {
    ff s = two_sum(k.hi, -r.m0);
    s = ff_add_f(s, k.lo);
    s = ff_add_f(s, -r.m1);
    return ff_add_f(s, -r.m2);
}

// Twice the normal CDF at k is n + t, n = 0 or 2 and t the tail the table
// gives: t keeps its relative accuracy where the CDF is near 1.
__device__ __forceinline__ ff cdf2_tail(ff k, const Rec& r, float& n, const float* tab) {
    const ff z = ff_mul(ff_sub_mean(k, r), r.isd);
    const bool up = z.hi >= 0.f;
    const ff e = erfc_pos(up ? z : ff_neg(z), tab);
    n = up ? 2.f : 0.f;
    return up ? ff_neg(e) : e;
}

// 1 - |n + tl| / 2, n = 0 or +-2
__device__ __forceinline__ ff sim_of_parts(float n, ff tl) {
    if (n != 0.f) {  // |n + tl| = 2 + (n > 0 ? tl : -tl)
        const float h = n > 0.f ? -0.5f : 0.5f;
        return ff_make(tl.hi * h, tl.lo * h);
    }
    if (tl.hi < 0.f) tl = ff_neg(tl);
    return ff_add_f(ff_make(-0.5f * tl.hi, -0.5f * tl.lo), 1.f);
}

// 1 - cal_abd_dist2 with the crossing points in float-float.  At the crossing
// points the two densities are equal, so the overlap is stationary in k1
// and k2: an error e in either moves it by O((e / sd)^2).  Where the
// variances differ by at least 1e-3 of the larger one, the crossing points'
// cancellation is bounded by that ratio, and float-float places them within
// ~1e-9 sd of the true points (the reference's FP64 points are nearer
// still), so the overlap agrees with the reference's to ~1e-18 -- far inside
// the CDFs' own error.  The CDF arguments are formed from the three-float
// means to float-float accuracy.  Each doubled CDF value is its integer part
// and a tail; the integers cancel exactly, to d = |n + t| / 2 with n = 0 or
// +-2, so 1 - d is |t| / 2 where d is near 1 and keeps the tails' relative
// accuracy without FP64 (three FP64 sums of the four converted values cost
// half of the kernel on this part's narrow FP64 unit).  Returns hi = -1 where
// the FP64 path decides instead: closer variances, values out of the
// float-float range, crossing points that do not separate.
__device__ __forceinline__ ff abd_sim_ff(const Rec& a, const Rec& b, const float* tab) {
    const ff none = ff_make(-1.f, 0.f);
    if (!(a.v.hi < 1e15f && b.v.hi < 1e15f && a.m0 < 1e15f && b.m0 < 1e15f)) return none;
    const ff m1 = ff_make(a.m0, a.m1), m2 = ff_make(b.m0, b.m1);
    // Equal variances (a depth's variance below 1 counts as 1): one crossing
    // point, half way, where the overlap is stationary too.
    if (a.v.hi == b.v.hi && a.v.lo == b.v.lo) {
        ff k = ff_add(m1, m2);
        k.hi *= 0.5f;
        k.lo *= 0.5f;
        float na, nb;
        const ff ta = cdf2_tail(k, a, na, tab), tb = cdf2_tail(k, b, nb, tab);
        return sim_of_parts(na - nb, ff_add(ta, ff_neg(tb)));
    }
    // in FP32: variances (>= 1) this far apart also pass the reference's own
    // |v2 - v1| >= 1e-4 test, and their order is that of the FP64 values
    if (!(fabsf(a.v.hi - b.v.hi) >= 1e-3f * fmaxf(a.v.hi, b.v.hi))) return none;
    const ff L = ff_add(b.lv, ff_neg(a.lv));  // 2 log(sqrt(v2 / v1))
    const ff dm = ff_add(m1, ff_neg(m2));
    const ff dv = ff_add(a.v, ff_neg(b.v));
    // t = sqrt(v1 v2 ((m1 - m2)^2 - 2 (v1 - v2) log(sqrt(v2 / v1))))
    const ff A = ff_add(ff_mul(dm, dm), ff_neg(ff_mul(dv, L)));
    const ff t = ff_sqrt(ff_mul(ff_mul(a.v, b.v), A));
    const ff c = ff_add(ff_mul(m1, b.v), ff_neg(ff_mul(m2, a.v)));  // m1 v2 - m2 v1
    const ff idv = ff_recip(dv);
    ff k1 = ff_mul(ff_add(t, ff_neg(c)), idv);  // (t - m1 v2 + m2 v1) / (v1 - v2)
    ff k2 = ff_mul(ff_add(t, c), ff_neg(idv));  // (t + m1 v2 - m2 v1) / (v2 - v1)
    if (!(fabsf(k1.hi) < 1e30f && fabsf(k2.hi) < 1e30f &&
          fabsf(k1.hi - k2.hi) > 0x1p-30f * (fabsf(k1.hi) + fabsf(k2.hi))))
        return none;
    if (ff_gt(k1, k2)) {
        const ff x = k1;
        k1 = k2;
        k2 = x;
    }
    // the doubled overlap of the narrower distribution minus that of the wider
    // one is n + tl, up to its sign, which the absolute value drops
    float n2a, n1a, n1b, n2b;
    const ff t2a = cdf2_tail(k2, a, n2a, tab), t1a = cdf2_tail(k1, a, n1a, tab);
    const ff t1b = cdf2_tail(k1, b, n1b, tab), t2b = cdf2_tail(k2, b, n2b, tab);
    return sim_of_parts((n2a - n1a) + (n1b - n2b), ff_add(ff_add(t2a, ff_neg(t1a)), ff_add(t1b, ff_neg(t2b))));
}

struct ScoreArgs {
    const uint64_t* from;
    const uint64_t* to;
    uint64_t ne, n;
    const double* abd;
    const double* vv;     // per contig and sample (k_abd_prep)
    const AbdRec* rec;
    const double* sx;     // per contig
    const double* ratio;
    uint32_t nabd;
    double min_cv;
    float3 cv3;      // min_cv as three floats
    bool cv_clamped; // min_cv >= 1e-6: the clamped means compare with it as the depths do
    bool corr;
    double* raw;     // mean abundance similarity per edge
    uint32_t* nnz;   // samples where either depth exceeds min_cv
    double* cor;     // depth correlation per edge (corr only)
    uint32_t* idx;   // 0 .. ne-1, the values of the rank sorts
    unsigned long long* bad;  // edges with an index out of range or no covered sample
};

// The ends of a sample's similarity, 1 - min(max(d, 1e-6), 1 - 1e-6) as FP64
// forms them, and in float-float (the upper one needs all 53 bits, so the
// values that reach an end take the FP64 one).
constexpr double kSimMin = 1. - (1. - 1e-6), kSimMax = 1. - 1e-6;
constexpr float kSimMinHi = (float)kSimMin, kSimMinLo = (float)(kSimMin - (double)kSimMinHi);
constexpr float kSimMaxHi = (float)kSimMax, kSimMaxLo = (float)(kSimMax - (double)kSimMaxHi);

// cal_abd_dist of one sample by the FP64 path: its similarity 1 - d.
__device__ __noinline__ double abd_sim64(const ScoreArgs& p, uint64_t i1, uint64_t i2, ff f1, ff f2,
                                         const float* tab) {
    const double x = p.abd[i1], y = p.abd[i2];
    const double m1 = x < 1e-6 ? 1e-6 : x, m2 = y < 1e-6 ? 1e-6 : y;
    double d = 0.;
    if (m1 != m2) d = abd_dist2(m1, p.vv[i1], f1, m2, p.vv[i2], f2, tab);
    d = d < 1e-6 ? 1e-6 : d;  // std::min(std::max(d, 1e-6), 1 - 1e-6), NaN kept
    d = (1. - 1e-6) < d ? 1. - 1e-6 : d;
    return 1. - d;
}

// One thread per edge: r1 = to[e], r2 = from[e] (the reference's order).  The
// FP64 left is the correlation's cross sum and the sum of the similarities.
// (3.8M edges, 10 samples: 3,358 us with the similarities combined and compared
// in FP64, a logarithm per pair and all 14 table terms in float-float; 1,931 us
// so, issue slots 79 % used.)
__global__ void k_abd_score(ScoreArgs p) {
    __shared__ __align__(16) float tab[kErfcWords];
    load_erfc_table(tab);
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < p.ne;
         e += (uint64_t)gridDim.x * blockDim.x) {
        p.idx[e] = (uint32_t)e;
        const uint64_t r1 = p.to[e], r2 = p.from[e];
        if (r1 >= p.n || r2 >= p.n) {
            atomicAdd(p.bad, 1ull);
            p.raw[e] = 0.;
            p.nnz[e] = 0;
            if (p.corr) p.cor[e] = 0.;
            continue;
        }
        const AbdRec* q1 = p.rec + r1 * p.nabd;
        const AbdRec* q2 = p.rec + r2 * p.nabd;
        double sum = 0.;
        uint32_t k = 0;
        // the cross sum of the Pearson correlation (cal_abd_corr), from the
        // rows' own deviations
        double sxy = 0.;
        const ff lo = ff_make(kSimMinHi, kSimMinLo), hi = ff_make(kSimMaxHi, kSimMaxLo);
        for (uint32_t i = 0; i < p.nabd; ++i) {
            const Rec a = load_rec(q1 + i), b = load_rec(q2 + i);
            // cal_abd_dist for sample i
            bool covered;
            if (p.cv_clamped)
                covered = mean_gt(a, p.cv3) || mean_gt(b, p.cv3);
            else
                covered = p.abd[r1 * p.nabd + i] > p.min_cv || p.abd[r2 * p.nabd + i] > p.min_cv;
            if (covered) {
                ff s = hi;
                if (!same_mean(a, b)) s = abd_sim_ff(a, b, tab);
                if (s.hi >= 0.f) {
                    sum += !ff_gt(s, lo) ? kSimMin : !ff_gt(hi, s) ? kSimMax : ff_to_double(s);
                } else {
                    sum += abd_sim64(p, r1 * p.nabd + i, r2 * p.nabd + i, a.isd, b.isd, tab);
                }
                ++k;
            }
            if (i > 0) sxy += a.dev * b.dev * __ldg(p.ratio + i - 1);
        }
        if (k == 0) atomicAdd(p.bad, 1ull);
        const double mean = sum / (double)k;
        p.raw[e] = mean != mean ? __longlong_as_double(0x7ff8000000000000ll) : mean;  // a NaN sorts last, whatever its sign was on the way
        p.nnz[e] = k;
        if (p.corr) p.cor[e] = sxy / (__ldg(p.sx + r1) * __ldg(p.sx + r2));
    }
}

// ---- ranks by 32-bit sorts -------------------------------------------------
// A radix sort of FP64 keys with indices takes eight passes over 12 bytes an
// edge; the sorts here run on a 32-bit key that is monotone in the value (four
// passes over 8 bytes), and runs of equal 32-bit keys that are out of order by
// their full keys are put in order afterwards (k_mark_runs, k_fix_runs).
//
// The similarities and sTNF are positive and span a few octaves: their key is
// the top 32 bits of the bit pattern's offset from the smallest (k_key_range;
// NaN is set aside, so that it does not stretch the range).  Correlations change
// sign and crowd at both ends -- two contigs of a genome, few samples -- so
// their key is the bit pattern of 1 - |c| to either side of the middle, with 25
// bits of every octave of the distance from +-1 (corr_key).  (A restatement of
// 60,000 contigs' 3.8M edges: 19 % of the correlations in runs, the longest 6 to 7
// long at 3 to 10 samples; by the pattern's offset from the smallest, 63 bits wide over
// both signs, 78 % and 71 to 16,877.)  Runs out of order and longer than kFixRun
// raise a flag, and those values are sorted by their full keys instead, before any
// score is written.  Two samples' correlations are +-1 but for the last
// bits, two runs of half the edges: they go by their full keys at once.
//
// The ranks by either route, 10 samples: 3.8M edges 1,186 us by the full keys and
// 969 by these, 7.2M 1,920 and 1,612, 16M 3,693 and 3,505, 32M 7,667 and 8,375 (more
// edges crowd the runs), 80M 20.7 and 26.5 ms; so up to 2^24 edges.
constexpr uint64_t kTopBitsMost = 1ull << 24;
constexpr uint32_t kFixRun = 48;

struct KeyRange {
    unsigned long long min_inv, max;  // of the order keys; min complemented, so that zeros start both
};

// The order of the radix sort: negative values reversed, -0 as 0; NaN lies
// beyond the infinities, on its sign's side.
__device__ __forceinline__ unsigned long long order_key(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v == 0. ? 0. : v);
    return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}

// Correlation to 32 bits, monotone: 1 - |c| is in [2^-53, 1] or not positive.
__device__ __forceinline__ uint32_t corr_key(double c) {
    if (c != c) return __double2hiint(c) < 0 ? 0u : ~0u;
    const long long base = (1023ll - 54) << 52, one = 1023ll << 52;
    const long long t = __double_as_longlong(1. - fabs(c));  // negative when |c| rounds above 1
    const uint32_t k = (uint32_t)((one - (t > base ? t : base)) >> 27);  // below 2^31: 54 octaves of 25 bits
    return c >= 0. ? 0x80000000u + k : 0x7fffffffu - k;
}

struct RankArrays {  // blockIdx.y: which; the last one holds the correlations
    const double* v[3];
    uint32_t* key[3];
};

__global__ void __launch_bounds__(256) k_key_range(RankArrays A, uint64_t ne, KeyRange* __restrict__ r) {
    const double* v = A.v[blockIdx.y];
    unsigned long long lo = 0, hi = 0;
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < ne; e += (uint64_t)gridDim.x * blockDim.x) {
        const double x = v[e];
        if (x != x) continue;
        const unsigned long long k = order_key(x);
        lo = lo > ~k ? lo : ~k;
        hi = hi > k ? hi : k;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long l2 = __shfl_xor_sync(0xffffffffu, lo, o), h2 = __shfl_xor_sync(0xffffffffu, hi, o);
        lo = lo > l2 ? lo : l2;
        hi = hi > h2 ? hi : h2;
    }
    __shared__ unsigned long long part[2][8];
    if ((threadIdx.x & 31) == 0) {
        part[0][threadIdx.x >> 5] = lo;
        part[1][threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) {
            lo = lo > part[0][w] ? lo : part[0][w];
            hi = hi > part[1][w] ? hi : part[1][w];
        }
        if (lo | hi) {
            atomicMax(&r[blockIdx.y].min_inv, lo);
            atomicMax(&r[blockIdx.y].max, hi);
        }
    }
}

__global__ void k_key32(RankArrays A, uint64_t ne, const KeyRange* __restrict__ r) {
    const double* v = A.v[blockIdx.y];
    uint32_t* key = A.key[blockIdx.y];
    const uint64_t e0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, step = (uint64_t)gridDim.x * blockDim.x;
    if (blockIdx.y == 2) {
        for (uint64_t e = e0; e < ne; e += step) key[e] = corr_key(v[e]);
        return;
    }
    const unsigned long long lo = ~r[blockIdx.y].min_inv, span = r[blockIdx.y].max - lo;
    const int sh = max(0, 32 - __clzll((long long)span));
    for (uint64_t e = e0; e < ne; e += step) {
        const double x = v[e];
        // 0 and ~0 are the NaNs'
        const unsigned long long k = (order_key(x) - lo) >> sh;
        key[e] = x != x ? (__double2hiint(x) < 0 ? 0u : ~0u) : 1u + (uint32_t)(k < 0xfffffffdull ? k : 0xfffffffdull);
    }
}

// Runs of equal 32-bit keys that are not in order by their full keys: the thread
// at a position whose full key belongs before its predecessor's marks the run's
// start.  Every position is looked at by a thread of its own, so a long run that
// is in order (equal values: pairs at a similarity's end, say) costs no more
// than others; a walk is at most kFixRun long.
__global__ void k_mark_runs(const uint32_t* __restrict__ ks, const double* __restrict__ v,
                            const uint32_t* __restrict__ os, uint64_t ne, bool descending, uint8_t* __restrict__ mark,
                            unsigned long long* __restrict__ overflow) {
    for (uint64_t q = 1 + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < ne;
         q += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t k = ks[q];
        if (ks[q - 1] != k) continue;
        const unsigned long long a = order_key(v[os[q - 1]]), b = order_key(v[os[q]]);
        if (descending ? b <= a : b >= a) continue;
        uint64_t first = q - 1;
        while (first > 0 && q - first < kFixRun && ks[first - 1] == k) --first;
        if (first > 0 && ks[first - 1] == k)
            atomicAdd(overflow, 1ull);
        else
            mark[first] = 1;
    }
}

// The thread at the start of a marked run sorts the run's indices by the full
// keys (insertion, stable).
__global__ void k_fix_runs(const uint32_t* __restrict__ ks, const double* __restrict__ v,
                           const uint8_t* __restrict__ mark, uint64_t ne, bool descending, uint32_t* __restrict__ os,
                           unsigned long long* __restrict__ overflow) {
    for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < ne; q += (uint64_t)gridDim.x * blockDim.x) {
        if (!mark[q]) continue;
        const uint32_t k = ks[q];
        uint64_t end = q + 1;
        while (end < ne && end - q <= kFixRun && ks[end] == k) ++end;
        if (end - q > kFixRun) {
            atomicAdd(overflow, 1ull);
            continue;
        }
        for (uint64_t i = q + 1; i < end; ++i) {
            const uint32_t x = os[i];
            const unsigned long long f = order_key(v[x]);
            uint64_t j = i;
            for (; j > q; --j) {
                const unsigned long long g = order_key(v[os[j - 1]]);
                if (descending ? g >= f : g <= f) break;
                os[j] = os[j - 1];
            }
            os[j] = x;
        }
    }
}

__global__ void k_gather_sorted(const double* __restrict__ v, const uint32_t* __restrict__ os, uint64_t ne,
                                double* __restrict__ out) {
    for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < ne; q += (uint64_t)gridDim.x * blockDim.x)
        out[q] = v[os[q]];
}

// Sorted position p starts its run of equal values: p, else 0 (a max-scan then
// gives every position the start of its run).  os: the values' places when
// they are not sorted themselves.
__global__ void k_run_heads(const double* __restrict__ keys, const uint32_t* __restrict__ os, uint64_t ne,
                            uint32_t* __restrict__ head) {
    for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < ne; q += (uint64_t)gridDim.x * blockDim.x) {
        bool first = q == 0;
        if (q) first = os ? keys[os[q]] != keys[os[q - 1]] : keys[q] != keys[q - 1];
        head[q] = first ? (uint32_t)q : 0u;
    }
}

// Ranks from the run starts: ascending sort -> the run's first rank ("min");
// descending sort -> the run's last rank in ascending order ("max").
__global__ void k_run_ranks(const uint32_t* __restrict__ order, const uint32_t* __restrict__ start, uint64_t ne,
                            bool descending, uint32_t* __restrict__ rank) {
    for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < ne; q += (uint64_t)gridDim.x * blockDim.x)
        rank[order[q]] = descending ? (uint32_t)(ne - start[q]) : start[q] + 1u;
}

// The weighted geometric mean pow(raw, 1 - w) * pow(t, w), w = 1 / (1 + nnz)
// (times the correlation's quantile, square-rooted, with enough samples),
// as exp((1 - w) log raw + w log t) in float-float: ff_log and ff_exp are
// good to ~1e-14, so sSCR is within ~1e-13 relative of the reference's FP64
// pows (the values lie in [1e-6, 1]: every similarity term is at least
// 1e-6).  The three FP64 pows cost ~250 FP64 operations an edge.
// overflow: with any of the three counts set the ranks do not stand, and
// nothing is written: out may be the sTNF values, which are then ranked again.
__global__ void k_sscr(const double* __restrict__ raw, const uint32_t* __restrict__ nnz,
                       const uint32_t* __restrict__ rt, const uint32_t* __restrict__ rc,
                       const double* __restrict__ distr, uint64_t ne, bool corr,
                       const unsigned long long* __restrict__ overflow, double* __restrict__ out) {
    if (overflow && (overflow[0] | overflow[1] | overflow[2])) return;
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < ne; e += (uint64_t)gridDim.x * blockDim.x) {
        const ff t = ff_from_double(distr[rt[e] - 1]);
        const ff w = ff_recip(ff_make((float)(1 + nnz[e]), 0.f));
        const ff l = ff_add(ff_mul(ff_add_f(ff_neg(w), 1.f), ff_log(ff_from_double(raw[e]))), ff_mul(w, ff_log(t)));
        const ff sc = ff_exp(l);
        out[e] = ff_to_double(corr ? ff_sqrt(ff_mul(sc, ff_from_double(distr[rc[e] - 1]))) : sc);
    }
}

struct MaxOp {
    __device__ __forceinline__ uint32_t operator()(uint32_t a, uint32_t b) const { return a > b ? a : b; }
};

unsigned grid_for(mdet_ctx* ctx, uint64_t items, unsigned block) {
    const uint64_t want = (items + block - 1) / block, cap = (uint64_t)ctx->num_sms * 16;
    return (unsigned)(want < 1 ? 1 : (want < cap ? want : cap));
}

// ranks from sorted values (ks, or keys at os) into rank (ascending "min" or,
// descending, "max")
int ranks_of(mdet_ctx* ctx, const double* keys, const uint32_t* by, const uint32_t* os, uint64_t ne, bool descending,
             uint32_t* head, uint32_t* start, uint32_t* rank, void* tmp, size_t tmpb) {
    cudaStream_t s = ctx->stream;
    k_run_heads<<<grid_for(ctx, ne, 256), 256, 0, s>>>(keys, by, ne, head);
    MDET_LAUNCHED(ctx, "k_run_heads");
    size_t tb = tmpb;
    MDET_CUDA(ctx, cub::DeviceScan::InclusiveScan(tmp, tb, head, start, MaxOp(), (int)ne, s));
    k_run_ranks<<<grid_for(ctx, ne, 256), 256, 0, s>>>(os, start, ne, descending, rank);
    MDET_LAUNCHED(ctx, "k_run_ranks");
    return MDET_OK;
}

// the same from a sort of the full keys
int rank_runs(mdet_ctx* ctx, const double* keys, const uint32_t* idx, uint64_t ne, bool descending, double* ks,
              uint32_t* os, uint32_t* head, uint32_t* start, uint32_t* rank, void* tmp, size_t tmpb) {
    cudaStream_t s = ctx->stream;
    size_t tb = tmpb;
    if (descending)
        MDET_CUDA(ctx, cub::DeviceRadixSort::SortPairsDescending(tmp, tb, keys, ks, idx, os, (int)ne, 0, 64, s));
    else
        MDET_CUDA(ctx, cub::DeviceRadixSort::SortPairs(tmp, tb, keys, ks, idx, os, (int)ne, 0, 64, s));
    return ranks_of(ctx, ks, nullptr, os, ne, descending, head, start, rank, tmp, tmpb);
}

int sscr_core(mdet_ctx* ctx, const uint64_t* from, const uint64_t* to, const double* stnf, uint64_t ne,
              double min_cv, uint32_t min_sample, double* out) {
    cudaStream_t s = ctx->stream;
    if (ne == 0) return MDET_OK;
    if (ctx->abd_nabd == 0) {  // no abundance: sSCR = sTNF
        MDET_CUDA(ctx, cudaMemcpyAsync(out, stnf, ne * 8, cudaMemcpyDeviceToDevice, s));
        return MDET_OK;
    }
    if (ne >= (1ull << 31)) return ctx_fail(ctx, MDET_ERR_INVALID, "too many edges (%llu)", (unsigned long long)ne);
    const bool corr = ctx->abd_nabd >= min_sample;
    double* raw = (double*)ctx_scratch(ctx, "abd.raw", ne * 8);
    uint32_t* nnz = (uint32_t*)ctx_scratch(ctx, "abd.nnz", ne * 4);
    double* cor = (double*)ctx_scratch(ctx, "abd.cor", ne * 8);
    uint32_t* idx = (uint32_t*)ctx_scratch(ctx, "abd.idx", ne * 4);
    double* ks = (double*)ctx_scratch(ctx, "abd.ks", ne * 8);
    uint32_t* os = (uint32_t*)ctx_scratch(ctx, "abd.os", ne * 4);
    uint32_t* head = (uint32_t*)ctx_scratch(ctx, "abd.head", ne * 4);
    uint32_t* start = (uint32_t*)ctx_scratch(ctx, "abd.start", ne * 4);
    uint32_t* rt = (uint32_t*)ctx_scratch(ctx, "abd.rt", ne * 4);
    uint32_t* rc = (uint32_t*)ctx_scratch(ctx, "abd.rc", ne * 4);
    double* distr = (double*)ctx_scratch(ctx, "abd.distr", ne * 8);
    // [0] bad edges, [1 ..] runs too long to fix in each array of values, [4 ..] the key ranges
    const size_t bad_bytes = 32 + 3 * sizeof(KeyRange);
    unsigned long long* bad = (unsigned long long*)ctx_scratch(ctx, "abd.bad", bad_bytes);
    uint32_t* k32 = (uint32_t*)ctx_scratch(ctx, "abd.k32", ne * 12);
    uint32_t* k32s = (uint32_t*)ctx_scratch(ctx, "abd.k32s", ne * 4);
    uint8_t* mark = (uint8_t*)ctx_scratch(ctx, "abd.mark", ne);
    if (!k32 || !k32s || !mark) return MDET_ERR_NOMEM;
    if (!raw || !nnz || !cor || !idx || !ks || !os || !head || !start || !rt || !rc || !distr || !bad)
        return MDET_ERR_NOMEM;
    size_t t1 = 0, t2 = 0, t3 = 0, t4 = 0;
    MDET_CUDA(ctx, cub::DeviceRadixSort::SortKeys(nullptr, t1, raw, distr, (int)ne, 0, 64, s));
    MDET_CUDA(ctx, cub::DeviceRadixSort::SortPairs(nullptr, t2, stnf, ks, idx, os, (int)ne, 0, 64, s));
    MDET_CUDA(ctx, cub::DeviceRadixSort::SortPairsDescending(nullptr, t3, cor, ks, idx, os, (int)ne, 0, 64, s));
    MDET_CUDA(ctx, cub::DeviceScan::InclusiveScan(nullptr, t4, head, start, MaxOp(), (int)ne, s));
    size_t t5 = 0, t6 = 0;
    MDET_CUDA(ctx, cub::DeviceRadixSort::SortPairs(nullptr, t5, k32, k32s, idx, os, (int)ne, 0, 32, s));
    MDET_CUDA(ctx, cub::DeviceRadixSort::SortPairsDescending(nullptr, t6, k32, k32s, idx, os, (int)ne, 0, 32, s));
    const size_t tmpb = std::max(std::max(std::max(t1, t2), std::max(t3, t4)), std::max(t5, t6));
    void* tmp = ctx_scratch(ctx, "abd.cubtmp", tmpb);
    if (!tmp) return MDET_ERR_NOMEM;
    MDET_CUDA(ctx, cudaMemsetAsync(bad, 0, bad_bytes, s));

    ScoreArgs p;
    p.from = from;
    p.to = to;
    p.ne = ne;
    p.n = ctx->abd_n;
    p.abd = (const double*)ctx->bufs["abd.m"].p;
    p.vv = (const double*)ctx->bufs["abd.vv"].p;
    p.rec = (const AbdRec*)ctx->bufs["abd.rec"].p;
    p.sx = (const double*)ctx->bufs["abd.sx"].p;
    p.ratio = (const double*)ctx->bufs["abd.ratio"].p;
    p.nabd = ctx->abd_nabd;
    p.min_cv = min_cv;
    p.cv_clamped = min_cv >= 1e-6 && min_cv < 1e30;
    p.cv3.x = (float)min_cv;
    p.cv3.y = (float)(min_cv - (double)p.cv3.x);
    p.cv3.z = (float)(min_cv - (double)p.cv3.x - (double)p.cv3.y);
    p.corr = corr;
    p.raw = raw;
    p.nnz = nnz;
    p.cor = cor;
    p.idx = idx;
    p.bad = bad;
    ctx_timer_begin(ctx, "k_abd_score");
    k_abd_score<<<grid_for(ctx, ne, 128), 128, 0, s>>>(p);
    ctx_timer_end(ctx, "k_abd_score");
    MDET_LAUNCHED(ctx, "k_abd_score");

    // the abundance similarities in ascending order (partial_sort_copy), the
    // ranks of sTNF and of the correlations, then the scores
    const unsigned g = grid_for(ctx, ne, 256);
    const int arrays = corr ? 3 : 2;
    // array k of the values by its full keys
    auto by_full_keys = [&](int k) -> int {
        size_t tb = tmpb;
        if (k == 0)
            MDET_CUDA(ctx, cub::DeviceRadixSort::SortKeys(tmp, tb, raw, distr, (int)ne, 0, 64, s));
        else if (k == 1)
            MDET_TRY(rank_runs(ctx, stnf, idx, ne, false, ks, os, head, start, rt, tmp, tmpb));
        else
            MDET_TRY(rank_runs(ctx, cor, idx, ne, true, ks, os, head, start, rc, tmp, tmpb));
        return MDET_OK;
    };
    auto by_top_bits = [&]() -> int {
        const RankArrays A{{raw, stnf, cor}, {k32, k32 + ne, k32 + 2 * ne}};
        KeyRange* range = (KeyRange*)(bad + 4);
        const dim3 g3(g, arrays), gr(std::min<unsigned>(g, ctx->num_sms * 4), 2);
        k_key_range<<<gr, 256, 0, s>>>(A, ne, range);
        MDET_LAUNCHED(ctx, "k_key_range");
        k_key32<<<g3, 256, 0, s>>>(A, ne, range);
        MDET_LAUNCHED(ctx, "k_key32");
        for (int k = 0; k < arrays; ++k) {
            if (k == 2 && p.nabd == 2) {
                MDET_TRY(by_full_keys(k));
                continue;
            }
            size_t tb = tmpb;
            if (k == 2)
                MDET_CUDA(ctx, cub::DeviceRadixSort::SortPairsDescending(tmp, tb, A.key[k], k32s, idx, os, (int)ne, 0,
                                                                         32, s));
            else
                MDET_CUDA(ctx, cub::DeviceRadixSort::SortPairs(tmp, tb, A.key[k], k32s, idx, os, (int)ne, 0, 32, s));
            MDET_CUDA(ctx, cudaMemsetAsync(mark, 0, ne, s));
            k_mark_runs<<<g, 256, 0, s>>>(k32s, A.v[k], os, ne, k == 2, mark, bad + 1 + k);
            MDET_LAUNCHED(ctx, "k_mark_runs");
            k_fix_runs<<<g, 256, 0, s>>>(k32s, A.v[k], mark, ne, k == 2, os, bad + 1 + k);
            MDET_LAUNCHED(ctx, "k_fix_runs");
            if (k == 0) {
                k_gather_sorted<<<g, 256, 0, s>>>(raw, os, ne, distr);
                MDET_LAUNCHED(ctx, "k_gather_sorted");
            } else {
                MDET_TRY(ranks_of(ctx, A.v[k], os, os, ne, k == 2, head, start, k == 1 ? rt : rc, tmp, tmpb));
            }
        }
        return MDET_OK;
    };
    const bool top_bits = ne <= kTopBitsMost;
    unsigned long long h_bad[4] = {0, 0, 0, 0};
    ctx_timer_begin(ctx, "abd_ranks");
    if (top_bits)
        MDET_TRY(by_top_bits());
    else
        for (int k = 0; k < arrays; ++k) MDET_TRY(by_full_keys(k));
    ctx_timer_end(ctx, "abd_ranks");
    for (bool again = false;; again = true) {
        ctx_timer_begin(ctx, "k_sscr");
        k_sscr<<<g, 256, 0, s>>>(raw, nnz, rt, rc, distr, ne, corr, top_bits && !again ? bad + 1 : nullptr, out);
        ctx_timer_end(ctx, "k_sscr");
        MDET_LAUNCHED(ctx, "k_sscr");
        MDET_CUDA(ctx, cudaMemcpyAsync(h_bad, bad, 32, cudaMemcpyDeviceToHost, s));
        MDET_CUDA(ctx, cudaStreamSynchronize(s));
        if (again || h_bad[0] || !(h_bad[1] | h_bad[2] | h_bad[3])) break;
        ctx_timer_begin(ctx, "abd_ranks_full");
        for (int k = 0; k < arrays; ++k)
            if (h_bad[1 + k]) MDET_TRY(by_full_keys(k));
        ctx_timer_end(ctx, "abd_ranks_full");
    }
    if (h_bad[0])
        return ctx_fail(ctx, MDET_ERR_INVALID,
                        "%llu edges have a contig index out of range or no sample with depth above min_cv", h_bad[0]);
    return MDET_OK;
}

}  // namespace

int abd_gate(mdet_ctx* ctx, GraphPrep& g) {
    g.low = nullptr;
    if (ctx->abd_nabd == 0) return MDET_OK;
    if (ctx->abd_n != g.n)
        return ctx_fail(ctx, MDET_ERR_INVALID, "the abundance set on the context covers %llu contigs, the graph %llu",
                        (unsigned long long)ctx->abd_n, (unsigned long long)g.n);
    uint8_t* low_s = (uint8_t*)ctx_scratch(ctx, "abd.lows", g.n);
    if (!low_s) return MDET_ERR_NOMEM;
    k_low_sorted<<<grid_for(ctx, g.n, 256), 256, 0, ctx->stream>>>(g.perm, (const uint8_t*)ctx->bufs["abd.low"].p,
                                                                    g.n, low_s);
    MDET_LAUNCHED(ctx, "k_low_sorted");
    g.low = low_s;
    return MDET_OK;
}

extern "C" {

int mdet_ctx_set_abundance(mdet_ctx* ctx, const double* abd, const double* abd_var, uint64_t n, uint32_t nabd) {
    if (!ctx) return MDET_ERR_INVALID;
    MDET_CUDA(ctx, cudaSetDevice(ctx->device));
    if (nabd == 0 || n == 0 || !abd) {
        ctx->abd_n = 0;
        ctx->abd_nabd = 0;
        return MDET_OK;
    }
    if (!abd_var) return ctx_fail(ctx, MDET_ERR_INVALID, "null variance matrix");
    if (n >= (1ull << 31)) return ctx_fail(ctx, MDET_ERR_INVALID, "too many contigs");
    cudaStream_t s = ctx->stream;
    double* dm = (double*)ctx_scratch(ctx, "abd.m", n * nabd * 8);
    double* dv = (double*)ctx_scratch(ctx, "abd.v", n * nabd * 8);
    uint8_t* low = (uint8_t*)ctx_scratch(ctx, "abd.low", n);
    double* vv = (double*)ctx_scratch(ctx, "abd.vv", n * nabd * 8);
    AbdRec* rec = (AbdRec*)ctx_scratch(ctx, "abd.rec", n * nabd * sizeof(AbdRec));
    double* sx = (double*)ctx_scratch(ctx, "abd.sx", n * 8);
    double* ratio = (double*)ctx_scratch(ctx, "abd.ratio", nabd * 8);
    if (!dm || !dv || !low || !vv || !rec || !sx || !ratio) return MDET_ERR_NOMEM;
    MDET_CUDA(ctx, cudaMemcpyAsync(dm, abd, n * nabd * 8, cudaMemcpyHostToDevice, s));
    MDET_CUDA(ctx, cudaMemcpyAsync(dv, abd_var, n * nabd * 8, cudaMemcpyHostToDevice, s));
    k_abd_low<<<grid_for(ctx, n, 256), 256, 0, s>>>(dm, n, nabd, low);
    MDET_LAUNCHED(ctx, "k_abd_low");
    k_abd_prep<<<std::max<unsigned>(grid_for(ctx, n, 256), (nabd + 255) / 256), 256, 0, s>>>(dm, dv, n, nabd, vv,
                                                                                            ratio, rec, sx);
    MDET_LAUNCHED(ctx, "k_abd_prep");
    MDET_CUDA(ctx, cudaStreamSynchronize(s));
    ctx->abd_n = n;
    ctx->abd_nabd = nabd;
    return MDET_OK;
}

int mdet_edges_sscr_dev(mdet_ctx* ctx, const uint64_t* d_from, const uint64_t* d_to, const double* d_stnf,
                        uint64_t n_edges, double min_cv, uint32_t min_sample, double* d_sscr) {
    if (!ctx) return MDET_ERR_INVALID;
    MDET_CUDA(ctx, cudaSetDevice(ctx->device));
    ctx->launches = 0;
    if (n_edges && (!d_from || !d_to || !d_stnf || !d_sscr)) return ctx_fail(ctx, MDET_ERR_INVALID, "null pointer");
    return sscr_core(ctx, d_from, d_to, d_stnf, n_edges, min_cv, min_sample, d_sscr);
}

int mdet_edges_sscr(mdet_ctx* ctx, const uint64_t* from, const uint64_t* to, const double* stnf, uint64_t n_edges,
                    double min_cv, uint32_t min_sample, double* sscr) {
    if (!ctx) return MDET_ERR_INVALID;
    MDET_CUDA(ctx, cudaSetDevice(ctx->device));
    ctx->launches = 0;
    if (n_edges == 0) return MDET_OK;
    if (!from || !to || !stnf || !sscr) return ctx_fail(ctx, MDET_ERR_INVALID, "null pointer");
    cudaStream_t s = ctx->stream;
    uint64_t* df = (uint64_t*)ctx_scratch(ctx, "io.efrom", n_edges * 8);
    uint64_t* dt = (uint64_t*)ctx_scratch(ctx, "io.eto", n_edges * 8);
    double* ds = (double*)ctx_scratch(ctx, "io.estnf", n_edges * 8);
    double* dout = (double*)ctx_scratch(ctx, "io.esscr", n_edges * 8);
    if (!df || !dt || !ds || !dout) return MDET_ERR_NOMEM;
    MDET_CUDA(ctx, cudaMemcpyAsync(df, from, n_edges * 8, cudaMemcpyHostToDevice, s));
    MDET_CUDA(ctx, cudaMemcpyAsync(dt, to, n_edges * 8, cudaMemcpyHostToDevice, s));
    MDET_CUDA(ctx, cudaMemcpyAsync(ds, stnf, n_edges * 8, cudaMemcpyHostToDevice, s));
    MDET_TRY(sscr_core(ctx, df, dt, ds, n_edges, min_cv, min_sample, dout));
    MDET_CUDA(ctx, cudaMemcpyAsync(sscr, dout, n_edges * 8, cudaMemcpyDeviceToHost, s));
    MDET_CUDA(ctx, cudaStreamSynchronize(s));
    return MDET_OK;
}

}  // extern "C"
