// fasta_index.cu -- FASTA ingest on the device: the reference reader's record
// split (cuda/Cuda2.cu:1486-1553) over the file's bytes in HBM, so that a
// caller can go from the raw file to TNF rows without a host pass over it.
//
// Record rules (the reference's loop read sequentially): a '>' starts a record
// wherever it stands, except inside the name line of the record before it;
// so the record starts are exactly the first '>' of each line.  The name is
// the rest of that line cut at its first space; the sequence view runs from
// after the name line's newline to the next record's '>' (or the end), inner
// newlines kept, one trailing newline dropped; the size is the view's bytes
// before that drop minus its newlines.  A name line that reaches the end of
// the buffer without a newline is not a record.
//
// Pass 1 (k_fa_scan) reads every byte once in 16-byte loads, a warp per 2 KB,
// and leaves the number of newlines of every 64 bytes in a byte array (1/64 of
// the file).  A thread that sees a '>' settles whether it is the
// first of its line from its own 16 bytes or, when the line began in an
// earlier chunk, by walking back to the line's previous '\n' or '>'.  A block
// takes a contiguous range of at most 384 KB and leaves its starts in order, so one
// small launch (k_fa_compact) joins them; a file with more records in a range
// than a block's queue holds (records of less than 170 bytes) is scanned again
// with the starts appended as they come, and sorted.  Pass 2 (k_fa_records) gives each record a warp: it finds the name line's newline and
// first space with ballots over 32-byte windows, and the view's newlines are
// the byte array's sum over its whole 64-byte blocks and a count over the bytes
// at its two ends, so the sequence is not read again.  A scan of the
// size-class flags places the records with size >= min_contig in file order.
#include <algorithm>
#include <cstring>

#include <cub/cub.cuh>

#include "common.cuh"

namespace {

constexpr uint64_t kNone = ~0ull;

__device__ __forceinline__ unsigned char byte_of(const uint4& q, int j) {
    const uint32_t w = j < 4 ? q.x : j < 8 ? q.y : j < 12 ? q.z : q.w;
    return (unsigned char)(w >> (8 * (j & 3)));
}

// Is the '>' whose line reaches back before position p (exclusive) the first
// of its line?  Walks back to the previous '\n' (yes) or '>' (no); the
// buffer's start is a line start.
__device__ bool line_has_no_gt_before(const unsigned char* __restrict__ b, uint64_t p) {
    while (p > 0) {
        const unsigned char c = b[--p];
        if (c == '\n') return true;
        if (c == '>') return false;
    }
    return true;
}

constexpr uint32_t kBlk = 64;  // bytes per newline count

// 0x80 in every byte of w that equals '\n'
__device__ __forceinline__ uint32_t newline_bits(uint32_t w) {
    const uint32_t z = w ^ 0x0A0A0A0Au;
    return ~(((z & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | z | 0x7F7F7F7Fu);
}

// 0x80 in every byte of w that equals '>'
__device__ __forceinline__ uint32_t gt_bits(uint32_t w) {
    const uint32_t z = w ^ 0x3E3E3E3Eu;
    return ~(((z & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | z | 0x7F7F7F7Fu);
}

// not 0 when a byte of w is '>'
__device__ __forceinline__ uint32_t has_gt(uint32_t w) {
    const uint32_t z = w ^ 0x3E3E3E3Eu;
    return (z - 0x01010101u) & ~z & 0x80808080u;
}

// the byte flags (0x80) of four words as 16 bits
__device__ __forceinline__ uint32_t flags16(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    auto four = [](uint32_t m) { return ((m >> 7) * 0x01020408u) >> 24; };  // byte k -> bit k
    return four(a) | four(b) << 4 | four(c) << 8 | four(d) << 12;
}

// Record starts found by a block, in shared memory until the block ends: an
// atomic on the file's one counter per record start was what the scan waited
// for at 4 KB a record.
// A range is at most kRange bytes (and the file's last 2 KB), so that records of 170
// bytes and more, a raw assembly's shortest, never fill a queue: with a grid that did not
// grow with the file, 4.3M records of 280 bytes took 5.8 ms for the second scan and
// the sort, 3.2 so.
constexpr uint32_t kQueue = 2304;
constexpr uint64_t kRange = 384 * 1024;
struct StartQueue {
    uint32_t pos[kQueue];  // from the range's first byte
    uint32_t n;
    uint64_t base;
};

// The '>' bytes of one 16-byte chunk at base: queues the record starts, or
// (sq null) appends them.
__device__ __noinline__ void chunk_starts(const unsigned char* __restrict__ b, uint64_t base, uint4 q,
                                          StartQueue* sq, uint64_t* __restrict__ starts, uint64_t cap,
                                          unsigned long long* __restrict__ count) {
    uint32_t gt = flags16(gt_bits(q.x), gt_bits(q.y), gt_bits(q.z), gt_bits(q.w));
    const uint32_t nl = flags16(newline_bits(q.x), newline_bits(q.y), newline_bits(q.z), newline_bits(q.w));
    const uint32_t all = gt | nl;
    while (gt) {
        const uint32_t j = __ffs(gt) - 1;
        gt &= gt - 1;
        const uint32_t before = all & ((1u << j) - 1u);  // the last of these decides
        const bool first = before ? (nl >> (31 - __clz(before))) & 1u : line_has_no_gt_before(b, base);
        if (!first) continue;
        if (sq) {
            const uint32_t slot = atomicAdd(&sq->n, 1u);
            if (slot < kQueue) sq->pos[slot] = (uint32_t)(base + j - sq->base);
        } else {
            const unsigned long long pos = atomicAdd(count, 1ull);
            if (pos < cap) starts[pos] = base + j;
        }
    }
}

// The newlines of one 16-byte chunk (0 .. 16) and whether it has a '>'.
__device__ __forceinline__ uint32_t chunk_newlines(const uint4& q, uint32_t& gt) {
    gt = has_gt(q.x) | has_gt(q.y) | has_gt(q.z) | has_gt(q.w);
    const uint32_t acc = (newline_bits(q.x) >> 7) + (newline_bits(q.y) >> 7) + (newline_bits(q.z) >> 7) +
                         (newline_bits(q.w) >> 7);
    return __dp4a(acc, 0x01010101u, 0u);
}

// First 2-KB tile of block k of a grid of g (k = g: past the last).
__device__ __forceinline__ uint64_t range_tile(uint64_t ntile, uint32_t k, uint32_t g) { return ntile * k / g; }

// A warp per 2 KB: lane l takes the 16-byte chunks l, l + 32, l + 64 and
// l + 96, all four loads in flight.  The four chunk counts ride in one word's
// bytes, so two shuffle-adds make the sums of all 32 64-byte blocks, a byte per
// lane to write.
//
// kAppend false: the block's starts go to found[blockIdx.x * kQueue ..] in order,
// from the first byte of its range on, and their number (which may exceed the queue) to nfound[blockIdx.x].
// (0.93 GB, 220,000 records: 465 us with a global atomic per start, 179 us so.)
template <bool kAppend>
__global__ void __launch_bounds__(256) k_fa_scan(const unsigned char* __restrict__ b, uint64_t nbytes,
                                                 uint8_t* __restrict__ nlc, uint32_t* __restrict__ found,
                                                 uint32_t* __restrict__ nfound, uint64_t* __restrict__ starts,
                                                 uint64_t cap, unsigned long long* __restrict__ count) {
    __shared__ StartQueue queue;
    StartQueue* sq = kAppend ? nullptr : &queue;
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t ntile = nbytes / 2048;
    const uint64_t t0 = range_tile(ntile, blockIdx.x, gridDim.x), t1 = range_tile(ntile, blockIdx.x + 1, gridDim.x);
    if (threadIdx.x == 0) {
        queue.n = 0;
        queue.base = t0 * 2048;
    }
    __syncthreads();
    for (uint64_t tile = t0 + (threadIdx.x >> 5); tile < t1; tile += blockDim.x >> 5) {
        const uint4* p = reinterpret_cast<const uint4*>(b + tile * 2048) + lane;
        uint4 q[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) q[u] = __ldg(p + 32 * u);
        uint32_t sum = 0, gt[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) sum |= chunk_newlines(q[u], gt[u]) << (8 * u);
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        nlc[tile * 32 + 8 * (lane & 3) + (lane >> 2)] = (uint8_t)(sum >> (8 * (lane & 3)));
        if (gt[0] | gt[1] | gt[2] | gt[3]) {
#pragma unroll 1
            for (int u = 0; u < 4; ++u) {
                const uint4 c = u == 0 ? q[0] : u == 1 ? q[1] : u == 2 ? q[2] : q[3];
                if (u == 0 ? gt[0] : u == 1 ? gt[1] : u == 2 ? gt[2] : gt[3])
                    chunk_starts(b, tile * 2048 + 16 * lane + 512 * u, c, sq, starts, cap, count);
            }
        }
    }
    // the rest of the file, less than 2 KB: a lane per 64-byte block (the
    // newlines of a ragged last block are counted by its record)
    const uint64_t g = ntile * 32 + lane;
    if (blockIdx.x + 1 == gridDim.x && threadIdx.x < 32 && g * kBlk < nbytes) {
        uint32_t nl = 0;
        for (uint64_t base = g * kBlk; base < g * kBlk + kBlk && base < nbytes; base += 16) {
            uint32_t w[4] = {0, 0, 0, 0};
            for (uint64_t j = 0; j < 16 && base + j < nbytes; ++j) w[j >> 2] |= (uint32_t)b[base + j] << (8 * (j & 3));
            const uint4 c = make_uint4(w[0], w[1], w[2], w[3]);
            uint32_t gt;
            nl += chunk_newlines(c, gt);
            if (gt) chunk_starts(b, base, c, sq, starts, cap, count);
        }
        if ((g + 1) * kBlk <= nbytes) nlc[g] = (uint8_t)nl;
    }
    if (kAppend) return;
    __syncthreads();
    const uint32_t n = queue.n;
    if (threadIdx.x == 0) {
        nfound[blockIdx.x] = n;
        if (n) atomicAdd(count, (unsigned long long)n);
        if (n > kQueue) atomicMax(count + 1, (unsigned long long)n);
    }
    if (n > kQueue) return;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {  // its place is how many lie before it
        const uint32_t v = queue.pos[i];
        uint32_t at = 0;
        for (uint32_t k = 0; k < n; ++k) at += queue.pos[k] < v;
        found[(uint64_t)blockIdx.x * kQueue + at] = v;
    }
}

// Joins the blocks' starts: block k's go after those of blocks 0 .. k - 1, which
// it counts unless `before` says how many they are.
__global__ void __launch_bounds__(256) k_fa_compact(const uint32_t* __restrict__ found,
                                                    const uint32_t* __restrict__ nfound,
                                                    const uint32_t* __restrict__ before, uint64_t nbytes,
                                                    uint64_t* __restrict__ starts) {
    __shared__ uint32_t part[8];
    uint64_t at = 0;
    if (before) {
        at = before[blockIdx.x];
    } else {
        uint32_t sum = 0;
        for (uint32_t k = threadIdx.x; k < blockIdx.x; k += blockDim.x) sum += nfound[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sum;
        __syncthreads();
        for (int w = 0; w < 8; ++w) at += part[w];
    }
    const uint32_t n = nfound[blockIdx.x];
    const uint64_t base = range_tile(nbytes / 2048, blockIdx.x, gridDim.x) * 2048;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x)
        starts[at + i] = base + found[(uint64_t)blockIdx.x * kQueue + i];
}

// (0.93 GB, 220,000 records: k_fa_records 661 us while it read the whole views
// and counted its records with one global atomic each, 96 us so; the sort of
// the starts took 48 us, k_fa_compact takes 6.)
struct RecArgs {
    const unsigned char* b;
    uint64_t nbytes;
    const uint8_t* nlc;  // newlines of every whole 64-byte block
    const uint64_t* starts;
    uint64_t nr;
    uint64_t min_contig;
    uint64_t* off;       // per record: sequence view offset
    uint64_t* len;       // view length
    uint64_t* size;      // bases
    uint64_t* name_off;
    uint32_t* name_len;
    uint32_t* large;     // 1: a record with size >= min_contig
    unsigned long long* n_valid;
    unsigned long long* n_small;
};

// A warp per record.
__global__ void k_fa_records(RecArgs p) {
    __shared__ unsigned int tally[2];  // the block's valid and small records
    if (threadIdx.x < 2) tally[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t nw = (uint64_t)gridDim.x * (blockDim.x >> 5);
    for (uint64_t r = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; r < p.nr; r += nw) {
        const uint64_t g = p.starts[r];
        const uint64_t nx = r + 1 < p.nr ? p.starts[r + 1] : p.nbytes;
        const unsigned char last = p.b[nx - 1];  // nx > g: in flight beside the name line
        // name line: its newline h and the first space before it
        uint64_t h = kNone, sp = kNone;
        for (uint64_t q0 = g + 1; q0 < nx; q0 += 32) {
            const uint64_t q = q0 + lane;
            const unsigned char ch = q < nx ? p.b[q] : 0;
            const uint32_t nlm = __ballot_sync(0xffffffffu, ch == '\n');
            const uint32_t spm = __ballot_sync(0xffffffffu, ch == ' ');
            const uint32_t lim = nlm ? (nlm & (0u - nlm)) - 1u : 0xffffffffu;  // lanes before the newline
            if (sp == kNone && (spm & lim)) sp = q0 + __ffs(spm & lim) - 1;
            if (nlm) {
                h = q0 + __ffs(nlm) - 1;
                break;
            }
        }
        if (h == kNone) {  // the name line runs into the end of the buffer: no record
            if (lane == 0) p.large[r] = 0;
            continue;
        }
        const uint64_t s0 = h + 1, s1 = nx;
        // newlines of the view [s0, s1): the bytes before its first whole
        // block and after its last, and the blocks' counts, four per load
        const uint64_t B0 = (s0 + kBlk - 1) / kBlk, B1 = s1 / kBlk;
        const uint64_t h1 = B0 < B1 ? B0 * kBlk : s1, t0 = B0 < B1 ? B1 * kBlk : s1;
        uint32_t nl = 0;
        for (uint64_t q = s0 + lane; q < h1; q += 32) nl += p.b[q] == '\n';
        for (uint64_t q = t0 + lane; q < s1; q += 32) nl += p.b[q] == '\n';
        const uint32_t* words = reinterpret_cast<const uint32_t*>(p.nlc);
        for (uint64_t w = B0 / 4 + lane; B0 < B1 && w < (B1 + 3) / 4; w += 32) {
            uint32_t v = words[w];
            if (4 * w < B0) v &= ~0u << (8 * (uint32_t)(B0 - 4 * w));
            if (4 * w + 4 > B1) v &= ~0u >> (8 * (uint32_t)(4 * w + 4 - B1));
            nl = __dp4a(v, 0x01010101u, nl);
        }
#pragma unroll
        for (int d = 16; d; d >>= 1) nl += __shfl_xor_sync(0xffffffffu, nl, d);
        if (lane == 0) {
            uint64_t view = s1 - s0;
            const uint64_t sz = view - nl;
            if (view > 0 && last == '\n') --view;
            p.off[r] = s0;
            p.len[r] = view;
            p.size[r] = sz;
            p.name_off[r] = g + 1;
            p.name_len[r] = (uint32_t)((sp != kNone ? sp : h) - (g + 1));
            p.large[r] = sz >= p.min_contig ? 1u : 0u;
            atomicAdd(&tally[0], 1u);
            if (sz < p.min_contig && sz >= 1000) atomicAdd(&tally[1], 1u);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && tally[0]) {
        atomicAdd(p.n_valid, (unsigned long long)tally[0]);
        if (tally[1]) atomicAdd(p.n_small, (unsigned long long)tally[1]);
    }
}

struct EmitArgs {
    uint64_t nr, cap;
    const uint32_t* large;
    const uint32_t* dst;
    const uint64_t *off, *len, *size, *name_off;
    const uint32_t* name_len;
    uint64_t *o_off, *o_len, *o_size, *o_name_off;
    double* o_log_size;
    uint32_t* o_name_len;
};

__global__ void k_fa_emit(EmitArgs p) {
    for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < p.nr;
         r += (uint64_t)gridDim.x * blockDim.x) {
        if (!p.large[r]) continue;
        const uint64_t k = p.dst[r];
        if (k >= p.cap) continue;
        p.o_off[k] = p.off[r];
        p.o_len[k] = p.len[r];
        const uint64_t sz = p.size[r];
        if (p.o_size) p.o_size[k] = sz;
        // log10(min(size, 500000)) (cuda/Cuda2.cu:1535)
        if (p.o_log_size) p.o_log_size[k] = log10((double)(sz < 500000 ? sz : 500000));
        if (p.o_name_off) p.o_name_off[k] = p.name_off[r];
        if (p.o_name_len) p.o_name_len[k] = p.name_len[r];
    }
}

unsigned grid_for(mdet_ctx* ctx, uint64_t items, unsigned block) {
    const uint64_t want = (items + block - 1) / block, cap = (uint64_t)ctx->num_sms * 16;
    return (unsigned)(want < 1 ? 1 : (want < cap ? want : cap));
}

struct FastaOut {
    uint64_t *off, *len, *size, *name_off;
    double* log_size;
    uint32_t* name_len;
};

int index_core(mdet_ctx* ctx, const char* d_bytes, uint64_t nbytes, uint64_t min_contig, uint64_t capacity,
               const FastaOut& o, mdet_fasta_stats* st) {
    cudaStream_t s = ctx->stream;
    const unsigned char* b = (const unsigned char*)d_bytes;
    unsigned long long* cnt = (unsigned long long*)ctx_scratch(ctx, "fa.cnt", 3 * 8);
    if (!cnt) return MDET_ERR_NOMEM;
    uint8_t* nlc = (uint8_t*)ctx_scratch(ctx, "fa.nlc", nbytes / kBlk + 4);
    // sixteen blocks an SM, or as many as keep a range within kRange, in whole waves of
    // eight an SM
    unsigned sgrid = grid_for(ctx, nbytes / kBlk, 256);
    if (nbytes / kRange + 1 > sgrid) {
        const uint64_t wave = (uint64_t)ctx->num_sms * 8;
        sgrid = (unsigned)((nbytes / kRange + wave) / wave * wave);
    }
    uint32_t* found = (uint32_t*)ctx_scratch(ctx, "fa.found", (uint64_t)sgrid * kQueue * 4);
    uint32_t* nfound = (uint32_t*)ctx_scratch(ctx, "fa.nfound", sgrid * 4ull);
    if (!nlc || !found || !nfound) return MDET_ERR_NOMEM;
    // pass 1: record starts, queued per block
    unsigned long long h_cnt[3] = {0, 0, 0};
    MDET_CUDA(ctx, cudaMemsetAsync(cnt, 0, 3 * 8, s));
    ctx_timer_begin(ctx, "k_fa_scan");
    k_fa_scan<false><<<sgrid, 256, 0, s>>>(b, nbytes, nlc, found, nfound, nullptr, 0, cnt);
    ctx_timer_end(ctx, "k_fa_scan");
    MDET_LAUNCHED(ctx, "k_fa_scan");
    MDET_CUDA(ctx, cudaMemcpyAsync(h_cnt, cnt, 16, cudaMemcpyDeviceToHost, s));
    MDET_CUDA(ctx, cudaStreamSynchronize(s));
    const bool queued = h_cnt[1] == 0;
    const uint64_t nr = h_cnt[0];
    if (nr >= (1ull << 31)) return ctx_fail(ctx, MDET_ERR_INVALID, "too many FASTA records (%llu)", (unsigned long long)nr);
    st->n_records = st->n_large = st->n_small = 0;
    if (nr == 0) return MDET_OK;
    uint64_t* sorted = (uint64_t*)ctx_scratch(ctx, "fa.sorted", nr * 8);
    uint64_t* starts = queued ? nullptr : (uint64_t*)ctx_scratch(ctx, "fa.starts", nr * 8);
    if (!queued && !starts) return MDET_ERR_NOMEM;
    uint64_t* r_off = (uint64_t*)ctx_scratch(ctx, "fa.off", nr * 8);
    uint64_t* r_len = (uint64_t*)ctx_scratch(ctx, "fa.len", nr * 8);
    uint64_t* r_size = (uint64_t*)ctx_scratch(ctx, "fa.size", nr * 8);
    uint64_t* r_noff = (uint64_t*)ctx_scratch(ctx, "fa.noff", nr * 8);
    uint32_t* r_nlen = (uint32_t*)ctx_scratch(ctx, "fa.nlen", nr * 4);
    uint32_t* large = (uint32_t*)ctx_scratch(ctx, "fa.large", (nr + 1) * 4);
    uint32_t* dst = (uint32_t*)ctx_scratch(ctx, "fa.dst", (nr + 1) * 4);
    if (!sorted || !r_off || !r_len || !r_size || !r_noff || !r_nlen || !large || !dst) return MDET_ERR_NOMEM;
    size_t t1 = 0, t2 = 0;
    int bits = 1;
    while (bits < 64 && (nbytes >> bits)) ++bits;
    if (!queued) MDET_CUDA(ctx, cub::DeviceRadixSort::SortKeys(nullptr, t1, starts, sorted, (int)nr, 0, bits, s));
    MDET_CUDA(ctx, cub::DeviceScan::ExclusiveSum(nullptr, t2, large, dst, (int)nr + 1, s));
    // each block's sum over the blocks before it, up to 3 GB; beyond, one scan
    size_t t3 = 0;
    uint32_t* before = nullptr;
    if (queued && sgrid > 8192) {
        before = (uint32_t*)ctx_scratch(ctx, "fa.before", sgrid * 4ull);
        if (!before) return MDET_ERR_NOMEM;
        MDET_CUDA(ctx, cub::DeviceScan::ExclusiveSum(nullptr, t3, nfound, before, (int)sgrid, s));
    }
    void* tmp = ctx_scratch(ctx, "fa.cubtmp", std::max(std::max(t1, t2), t3));
    if (!tmp) return MDET_ERR_NOMEM;
    MDET_CUDA(ctx, cudaMemsetAsync(cnt, 0, 3 * 8, s));
    if (queued) {
        if (before) MDET_CUDA(ctx, cub::DeviceScan::ExclusiveSum(tmp, t3, nfound, before, (int)sgrid, s));
        k_fa_compact<<<sgrid, 256, 0, s>>>(found, nfound, before, nbytes, sorted);
        MDET_LAUNCHED(ctx, "k_fa_compact");
    } else {
        ctx_timer_begin(ctx, "k_fa_scan_append");
        k_fa_scan<true><<<sgrid, 256, 0, s>>>(b, nbytes, nlc, nullptr, nullptr, starts, nr, cnt);
        ctx_timer_end(ctx, "k_fa_scan_append");
        MDET_LAUNCHED(ctx, "k_fa_scan");
        MDET_CUDA(ctx, cub::DeviceRadixSort::SortKeys(tmp, t1, starts, sorted, (int)nr, 0, bits, s));
    }

    RecArgs ra{b, nbytes, nlc, sorted, nr, min_contig, r_off, r_len, r_size, r_noff, r_nlen, large, cnt + 1, cnt + 2};
    ctx_timer_begin(ctx, "k_fa_records");
    k_fa_records<<<grid_for(ctx, nr * 32, 256), 256, 0, s>>>(ra);
    ctx_timer_end(ctx, "k_fa_records");
    MDET_LAUNCHED(ctx, "k_fa_records");
    // the scan runs over nr + 1 flags so that dst[nr] is the count
    MDET_CUDA(ctx, cudaMemsetAsync(large + nr, 0, 4, s));
    MDET_CUDA(ctx, cub::DeviceScan::ExclusiveSum(tmp, t2, large, dst, (int)nr + 1, s));
    EmitArgs ea{nr, capacity, large, dst, r_off, r_len, r_size, r_noff, r_nlen,
                o.off, o.len, o.size, o.name_off, o.log_size, o.name_len};
    k_fa_emit<<<grid_for(ctx, nr, 256), 256, 0, s>>>(ea);
    MDET_LAUNCHED(ctx, "k_fa_emit");
    uint32_t nlarge = 0;
    MDET_CUDA(ctx, cudaMemcpyAsync(&nlarge, dst + nr, 4, cudaMemcpyDeviceToHost, s));
    MDET_CUDA(ctx, cudaMemcpyAsync(h_cnt + 1, cnt + 1, 16, cudaMemcpyDeviceToHost, s));
    MDET_CUDA(ctx, cudaStreamSynchronize(s));
    st->n_records = h_cnt[1];
    st->n_large = nlarge;
    st->n_small = h_cnt[2];
    if (nlarge > capacity)
        return ctx_fail(ctx, MDET_ERR_CAPACITY, "%llu contigs of at least %llu bases, capacity %llu",
                        (unsigned long long)nlarge, (unsigned long long)min_contig, (unsigned long long)capacity);
    return MDET_OK;
}

}  // namespace

extern "C" {

int mdet_fasta_index_dev(mdet_ctx* ctx, const char* d_bytes, uint64_t nbytes, uint64_t min_contig,
                         uint64_t capacity, uint64_t* d_seq_off, uint64_t* d_seq_len, uint64_t* d_size,
                         double* d_log_size, uint64_t* d_name_off, uint32_t* d_name_len, mdet_fasta_stats* stats) {
    if (!ctx || !stats) return MDET_ERR_INVALID;
    MDET_CUDA(ctx, cudaSetDevice(ctx->device));
    ctx->launches = 0;
    memset(stats, 0, sizeof(*stats));
    if (nbytes == 0) return MDET_OK;
    if (!d_bytes) return ctx_fail(ctx, MDET_ERR_INVALID, "null pointer");
    if (((uintptr_t)d_bytes & 15) != 0) return ctx_fail(ctx, MDET_ERR_INVALID, "FASTA buffer must be 16-byte aligned");
    if (capacity && (!d_seq_off || !d_seq_len)) return ctx_fail(ctx, MDET_ERR_INVALID, "null output pointer");
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, ctx->stream);
    const FastaOut o{d_seq_off, d_seq_len, d_size, d_name_off, d_log_size, d_name_len};
    int rc = index_core(ctx, d_bytes, nbytes, min_contig, capacity, o, stats);
    cudaEventRecord(e1, ctx->stream);
    float ms = 0;
    cudaEventSynchronize(e1);
    cudaEventElapsedTime(&ms, e0, e1);
    stats->ms_total = ms;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return rc;
}

int mdet_fasta_index(mdet_ctx* ctx, const char* bytes, uint64_t nbytes, uint64_t min_contig, uint64_t capacity,
                     uint64_t* seq_off, uint64_t* seq_len, uint64_t* size, double* log_size, uint64_t* name_off,
                     uint32_t* name_len, mdet_fasta_stats* stats) {
    if (!ctx || !stats) return MDET_ERR_INVALID;
    MDET_CUDA(ctx, cudaSetDevice(ctx->device));
    memset(stats, 0, sizeof(*stats));
    if (nbytes == 0) return MDET_OK;
    if (!bytes) return ctx_fail(ctx, MDET_ERR_INVALID, "null pointer");
    cudaStream_t s = ctx->stream;
    char* d_bytes = (char*)ctx_scratch(ctx, "io.bytes", nbytes + 64);
    const uint64_t c = capacity ? capacity : 1;
    uint64_t* d_off = (uint64_t*)ctx_scratch(ctx, "io.fa_off", c * 8);
    uint64_t* d_len = (uint64_t*)ctx_scratch(ctx, "io.fa_len", c * 8);
    uint64_t* d_size = (uint64_t*)ctx_scratch(ctx, "io.fa_size", c * 8);
    double* d_ls = (double*)ctx_scratch(ctx, "io.fa_ls", c * 8);
    uint64_t* d_noff = (uint64_t*)ctx_scratch(ctx, "io.fa_noff", c * 8);
    uint32_t* d_nlen = (uint32_t*)ctx_scratch(ctx, "io.fa_nlen", c * 4);
    if (!d_bytes || !d_off || !d_len || !d_size || !d_ls || !d_noff || !d_nlen) return MDET_ERR_NOMEM;
    MDET_CUDA(ctx, cudaMemcpyAsync(d_bytes, bytes, nbytes, cudaMemcpyHostToDevice, s));
    int rc = mdet_fasta_index_dev(ctx, d_bytes, nbytes, min_contig, capacity, d_off, d_len, d_size, d_ls, d_noff,
                                  d_nlen, stats);
    if (rc != MDET_OK) return rc;
    const uint64_t k = stats->n_large;
    if (k) {
        if (seq_off) MDET_CUDA(ctx, cudaMemcpyAsync(seq_off, d_off, k * 8, cudaMemcpyDeviceToHost, s));
        if (seq_len) MDET_CUDA(ctx, cudaMemcpyAsync(seq_len, d_len, k * 8, cudaMemcpyDeviceToHost, s));
        if (size) MDET_CUDA(ctx, cudaMemcpyAsync(size, d_size, k * 8, cudaMemcpyDeviceToHost, s));
        if (log_size) MDET_CUDA(ctx, cudaMemcpyAsync(log_size, d_ls, k * 8, cudaMemcpyDeviceToHost, s));
        if (name_off) MDET_CUDA(ctx, cudaMemcpyAsync(name_off, d_noff, k * 8, cudaMemcpyDeviceToHost, s));
        if (name_len) MDET_CUDA(ctx, cudaMemcpyAsync(name_len, d_nlen, k * 4, cudaMemcpyDeviceToHost, s));
    }
    MDET_CUDA(ctx, cudaStreamSynchronize(s));
    return MDET_OK;
}

}  // extern "C"
