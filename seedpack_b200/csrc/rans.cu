// Segment-parallel rANS over a plain symbol stream with per-block context tables (the residual-codec
// microbenchmark, and the engine the QR and BF16 coders share): histogram, table preparation, encode,
// prefix-sum + gather of the per-segment slots, decode.
//
// Stream model: `nsym` byte symbols cut into blocks of `block_len` symbols (a quantised block's codes);
// block b is coded with context table block_tab[b]; segments of `seg_len` symbols (a multiple of block_len
// and of 16) are independent rANS streams, one lane each.  Arithmetic and byte order follow the
// reference's coder (seedpack/qr.py:651-663, seedpack/rans.py:54-105 with PROB_BITS = PB).
#include "api_util.h"
#include "rans.cuh"

namespace sg {

// ---- tables: frequencies -> encoder entries (+ decoder LUT) ---------------------------------------------
// Replaces cum_of (seedpack/gpu2.py:483-486) and build_lut (seedpack/qr.py:889-895).  One CTA per table.
__global__ void __launch_bounds__(256) k_rans_tables(const uint16_t* __restrict__ freq, int pb, RansSym* __restrict__ enc,
                                                     uint8_t* __restrict__ lut, int* __restrict__ status) {
    __shared__ unsigned cum[257];
    const int t = blockIdx.x, s = threadIdx.x;
    const unsigned f = freq[t * 256 + s];
    // inclusive scan of 256 frequencies
    __shared__ unsigned warp_tot[8];
    unsigned v = f;
    for (int o = 1; o < 32; o <<= 1) { const unsigned n = __shfl_up_sync(0xffffffffu, v, o); if ((s & 31) >= o) v += n; }
    if ((s & 31) == 31) warp_tot[s >> 5] = v;
    __syncthreads();
    unsigned base = 0;
    for (int w = 0; w < (s >> 5); ++w) base += warp_tot[w];
    const unsigned incl = v + base;
    cum[s + 1] = incl;
    if (s == 0) cum[0] = 0;
    __syncthreads();
    const bool whole = cum[256] == (1u << pb);                                             // a used table must sum to 2^PB
    if (s == 255 && incl != 0 && !whole) atomicOr(status, SG_ST_CORRUPT);
    const unsigned c = incl - f;
    RansSym e;
    e.fc = f | (c << 16);
    if (f >= 2) {
        const unsigned sh = rans_shift(f);
        e.rcp = (unsigned)((((unsigned long long)1 << (sh + 31)) + f - 1) / f);
    } else e.rcp = 0xffffffffu;
    enc[t * 256 + s] = e;
    if (lut && pb == 15) {            // compact: one entry per 128 slots (the decoder scans on from it), then the symbols' words
        uint8_t* l = lut + (size_t)t * RANS_COMPACT;
        if (whole) for (unsigned b = (c + 127) >> 7; (b << 7) < incl; ++b) l[b] = (uint8_t)s;
        else l[s] = 0;                // (k_r2_dec stages unused tables like the others: zeros)
        reinterpret_cast<unsigned*>(l + 256)[s] = whole ? e.fc : 0u;
    } else if (lut && whole) {        // any other row would write outside its 2^PB slots: its LUT is left alone
        uint8_t* l = lut + ((size_t)t << pb);
        for (unsigned i = c; i < incl; ++i) l[i] = (uint8_t)s;
    }
}

// ---- histogram -------------------------------------------------------------------------------------------
// One lane per block.  Zero symbols (the bulk of a residual stream) are counted in registers and added once
// per warp and table; the others go out individually.
__global__ void __launch_bounds__(256) k_rans_hist(const uint8_t* __restrict__ sym, const uint16_t* __restrict__ block_tab,
                                                   int block_len, long long nblocks, unsigned* __restrict__ counts) {
    const long long b = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = b < nblocks;
    unsigned tab = 0xffffffffu, zeros = 0;
    if (live) {
        tab = block_tab[b];
        const uint4* p = reinterpret_cast<const uint4*>(sym + b * block_len);
        for (int i = 0; i < block_len / 16; ++i) {
            const uint4 v = __ldg(p + i);
            const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const unsigned s = (w[k] >> (8 * j)) & 0xff;
                    if (s == 0) ++zeros; else atomicAdd(counts + tab * 256 + s, 1u);
                }
            }
        }
    }
    const unsigned peers = __match_any_sync(0xffffffffu, tab);
    const unsigned total = __reduce_add_sync(peers, zeros);
    if (live && (threadIdx.x & 31) == (unsigned)(__ffs(peers) - 1) && total) atomicAdd(counts + tab * 256, total);
}

// ---- encode ----------------------------------------------------------------------------------------------
// Bound by the chain of a lane (one per segment) - x, comparisons, reciprocal, multiply-add - as long as nothing else is on
// it: symbols and table ids are loaded three batches of 16 symbols ahead, the table's entry for 0 two, the other entries
// one.  Most residual symbols are 0: only lanes with another symbol load (the lanes of a warp use different tables: a load
// by all of them touches 32 lines).  `spw` segments per warp: few segments are spread over all SMs' schedulers.
template <int PB>
__global__ void __launch_bounds__(32) k_rans_encode(const uint8_t* __restrict__ sym, const uint16_t* __restrict__ block_tab,
                                                    int block_len, long long nsym, int seg_len, const RansSym* __restrict__ enc,
                                                    uint8_t* __restrict__ out, size_t cap, unsigned* __restrict__ out_len, int nseg, int spw) {
    const long long sl = (long long)blockIdx.x * spw + threadIdx.x;
    if ((int)threadIdx.x >= spw || sl >= nseg) return;
    const int s = (int)sl;
    const long long s0 = (long long)s * seg_len;
    const int n = (int)min((long long)seg_len, nsym - s0), nb = n / 16;            // n: a multiple of 16
    const int sub = block_len / 16;                                                // 16 | block_len: one table per batch of 16
    const uint4* __restrict__ src = reinterpret_cast<const uint4*>(sym + s0);
    const uint16_t* __restrict__ bt = block_tab + s0 / block_len;
    uint8_t* slot = out + (size_t)s * cap;
    ByteWriterDown w;
    w.init(slot + cap);
    unsigned x = RANS_L;
    int li = nb - 1, lblk = li / sub, lrem = li - lblk * sub;                      // next batch to load
    uint4 v0, v1;                                                                  // symbols: just asked for / with their table known
    unsigned t0 = 0;
    const RansSym* tab1 = enc;
    RansSym e01;
    auto load = [&]() {
        if (li >= 0) { v0 = __ldg(src + li); t0 = __ldg(bt + lblk); }
        --li;
        if (--lrem < 0) { lrem = sub - 1; --lblk; }
    };
    auto table = [&]() { v1 = v0; tab1 = enc + (size_t)t0 * 256; e01 = tab1[0]; };
    auto look = [&](RansSym (&e)[16]) {
        const unsigned wv[4] = {v1.x, v1.y, v1.z, v1.w};
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const unsigned sy = (wv[k >> 2] >> (8 * (k & 3))) & 0xff;
            e[k] = e01;
            if (sy) e[k] = tab1[sy];
        }
    };
    RansSym cur[16], nxt[16];
    load(); table(); load();
    look(cur);
    table(); load();
    for (int i = nb - 1; i >= 0; --i) {
        if (i > 0) look(nxt);
        table(); load();
#pragma unroll
        for (int k = 15; k >= 0; k -= 2) rans_put2<PB>(x, w, cur[k], cur[k - 1]);
        if (w.ptr() < slot + 64) { out_len[s] = 0xffffffffu; return; }             // 16 symbols write at most 32 bytes
#pragma unroll
        for (int k = 0; k < 16; ++k) cur[k] = nxt[k];
    }
    rans_flush(x, w);
    w.flush();
    out_len[s] = w.bad() ? LEN_NOFREQ : (unsigned)(slot + cap - w.ptr());
}

// ---- scan + gather ---------------------------------------------------------------------------------------
// Replaces cumsum + gather (seedpack/qr.py:1054-1056, 880-887).  k_scan: exclusive prefix sum of the
// segment lengths by one CTA (segments number in the thousands to hundreds of thousands);
// k_gather: one warp per segment copies its bytes to its place.
__global__ void __launch_bounds__(1024) k_scan_lens(const unsigned* __restrict__ len, int nseg, unsigned long long* __restrict__ off,
                                                    int* __restrict__ status) {
    __shared__ unsigned long long wsum[32];
    __shared__ unsigned long long carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < nseg; base += 1024) {
        const int i = base + threadIdx.x;
        unsigned l = i < nseg ? len[i] : 0;
        if (l == LEN_OVERFLOW) { atomicOr(status, SG_ST_OVERFLOW); l = 0; }
        else if (l == LEN_NOFREQ) { atomicOr(status, SG_ST_CORRUPT); l = 0; }
        unsigned long long v = l;
        for (int o = 1; o < 32; o <<= 1) { const unsigned long long n = __shfl_up_sync(0xffffffffu, v, o); if ((threadIdx.x & 31) >= o) v += n; }
        if ((threadIdx.x & 31) == 31) wsum[threadIdx.x >> 5] = v;
        __syncthreads();
        unsigned long long pre = carry;
        for (int w = 0; w < (threadIdx.x >> 5); ++w) pre += wsum[w];
        if (i < nseg) off[i] = pre + v - l;
        __syncthreads();
        if (threadIdx.x == 1023) carry = pre + v;
        __syncthreads();
    }
    if (threadIdx.x == 0) off[nseg] = carry;
}

__global__ void __launch_bounds__(256) k_gather(const uint8_t* __restrict__ src, size_t cap, const unsigned* __restrict__ len,
                                                const unsigned long long* __restrict__ off, int nseg, uint8_t* __restrict__ dst,
                                                unsigned long long dst_cap) {
    const int s = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (s >= nseg) return;
    const unsigned l = len[s];
    if (l >= LEN_NOFREQ || off[s] + l > dst_cap) return;
    const uint8_t* a = src + (size_t)(s + 1) * cap - l;
    uint8_t* d = dst + off[s];
    for (unsigned i = lane; i < l; i += 32) d[i] = a[i];
}

// ---- decode ----------------------------------------------------------------------------------------------
template <int PB>
__global__ void __launch_bounds__(64) k_rans_decode(const uint8_t* __restrict__ in, const unsigned long long* __restrict__ off,
                                                    const uint16_t* __restrict__ block_tab, int block_len, long long nsym, int seg_len,
                                                    const RansSym* __restrict__ enc, const uint8_t* __restrict__ lut,
                                                    uint8_t* __restrict__ sym, int nseg, int* __restrict__ status) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nseg) return;
    const long long s0 = (long long)s * seg_len;
    const long long n = min((long long)seg_len, nsym - s0);
    ByteReaderUp r;
    r.init(in + off[s], in + off[s + 1]);
    unsigned x = rans_init(r);
    const RansSym* tab = nullptr;
    const uint8_t* l = nullptr;
    long long cur_block = -1;
    for (long long i = 0; i < n; i += 16) {
        const long long blk = (s0 + i) / block_len;
        if (blk != cur_block) { cur_block = blk; const unsigned t = block_tab[blk]; tab = enc + (size_t)t * 256; l = lut + ((size_t)t << PB); }
        unsigned wv[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            unsigned word = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) word |= rans_get<PB>(x, r, l, tab) << (8 * j);
            wv[k] = word;
        }
        *reinterpret_cast<uint4*>(sym + s0 + i) = make_uint4(wv[0], wv[1], wv[2], wv[3]);
        if (r.over) { atomicOr(status, SG_ST_CORRUPT); return; }
    }
    if (x != RANS_L || r.p != r.end) atomicOr(status, SG_ST_CORRUPT);     // a well-formed segment ends in the initial state
}

// The same decoder with the tables it needs in shared memory.  A residual stream is mostly the symbol 0, whose slots are
// [0, freq(0)) of every table: for those the step is x = freq(0) (x >> PB) + slot with freq(0) from a small array in
// shared memory.  The other slots of a table - [freq(0), 2^PB), few when zeros dominate - get one 4-byte entry each,
// symbol | (slot - cum) << 8 | (freq - 1) << 20, also in shared memory as far as they fit (tables in id order; the rest
// keep the two dependent global loads lut[slot] -> enc[symbol]).  Every CTA builds the entries from enc / lut itself
// (a few per cent of its decoding time; all 512 threads): the caller passes no further buffer.  One CTA per SM, whose first
// `per` threads then decode a segment each: the segments are spread over all SMs before a CTA takes more of them.
constexpr unsigned NOFIT = 0xffffffffu;
template <int PB>
__global__ void __launch_bounds__(512, 1) k_rans_decode_sm(const uint8_t* __restrict__ in, const unsigned long long* __restrict__ off,
                                                           const uint16_t* __restrict__ block_tab, int block_len, long long nsym, int seg_len,
                                                           const RansSym* __restrict__ enc, const uint8_t* __restrict__ lut,
                                                           uint8_t* __restrict__ sym, int nseg, int ntab, unsigned cap, int per,
                                                           int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned smem[];
    constexpr unsigned SLOTS = 1u << PB;
    unsigned* base = smem;                                   // [ntab] first entry of the table, NOFIT if not staged
    unsigned* ring = smem + ntab;                            // [per / 32][RING_ROWS][32]
    unsigned* ent = smem + max((int)SLOTS, ntab + RING_ROWS * per);        // [cap]; SLOTS words before it can be read
    unsigned short* f0 = reinterpret_cast<unsigned short*>(ent + cap);     // [ntab] freq(0)
    for (int t = threadIdx.x; t < ntab; t += blockDim.x) {
        const unsigned first = enc[(size_t)t * 256].fc & 0xffffu, last = enc[(size_t)t * 256 + 255].fc;
        const bool used = (last >> 16) + (last & 0xffffu) == SLOTS;
        f0[t] = (unsigned short)(used ? first : 0);
        base[t] = used ? SLOTS - first : 0;                  // for now: the number of entries the table needs
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned run = 0;
        for (int t = 0; t < ntab; ++t) {
            const unsigned n = base[t];
            if (n == 0 && f0[t] == 0) { base[t] = NOFIT; continue; }           // an unused table
            if (run + n <= cap) { base[t] = run; run += n; } else base[t] = NOFIT;
        }
    }
    __syncthreads();
    for (int t = threadIdx.x >> 5; t < ntab; t += blockDim.x >> 5) {
        const unsigned b = base[t];
        if (b == NOFIT) continue;
        const unsigned f = f0[t];
        for (unsigned slot = f + (threadIdx.x & 31); slot < SLOTS; slot += 32) {
            const unsigned s = lut[((size_t)t << PB) + slot];
            const unsigned fc = enc[(size_t)t * 256 + s].fc;
            ent[b + slot - f] = s | ((slot - (fc >> 16)) << 8) | (((fc & 0xffffu) - 1u) << 20);
        }
    }
    __syncthreads();
    const long long sl = (long long)blockIdx.x * per + threadIdx.x;
    if ((int)threadIdx.x >= per || sl >= nseg) return;
    const int s = (int)sl;
    const long long s0 = (long long)s * seg_len;
    const int n = (int)min((long long)seg_len, nsym - s0);
    RingReader<32> r;
    r.init(in + off[s], in + off[s + 1], ring + (threadIdx.x >> 5) * (RING_ROWS * 32) + (threadIdx.x & 31));
    unsigned x = r.state();
    const uint16_t* __restrict__ bt = block_tab + s0 / block_len;
    const int nblk = n / block_len;
    unsigned tid_next = bt[0];
    for (int b = 0; b < nblk; ++b) {
        const unsigned tid = tid_next, tf0 = f0[tid], tb = base[tid];
        if (b + 1 < nblk) tid_next = __ldg(bt + b + 1);
        // both kinds of slot without a branch: with 32 segments in a warp some lane meets a symbol other than 0 at most
        // steps.  ent[] is read whatever the slot: for a slot of the symbol 0 that is some word before the table's entries
        const unsigned* te = ent + (int)(tb == NOFIT ? 0u : tb) - (int)tf0;
        const unsigned e0 = (tf0 - 1u) << 20;
        for (int i = 0; i < block_len; i += 16) {
            r.top_up();
            unsigned wv[4];
            if (tb != NOFIT) {
#pragma unroll
                for (int k = 0; k < 16; ++k) {
                    const unsigned slot = x & (SLOTS - 1), xs = x >> PB, en = te[slot];
                    const unsigned e = slot >= tf0 ? en : e0 + (slot << 8);
                    x = (e >> 20) * xs + (xs + ((e >> 8) & (SLOTS - 1)));
                    r.renorm(x);
                    wv[k >> 2] = (k & 3) == 0 ? e & 0xffu : wv[k >> 2] | (e & 0xffu) << (8 * (k & 3));
                }
            } else {
#pragma unroll 1
                for (int k = 0; k < 4; ++k) {
                    unsigned word = 0;
#pragma unroll 1
                    for (int j = 0; j < 4; ++j) {
                        const unsigned slot = x & (SLOTS - 1), sy = lut[((size_t)tid << PB) + slot], fc = enc[(size_t)tid * 256 + sy].fc;
                        x = (fc & 0xffffu) * (x >> PB) + slot - (fc >> 16);
                        r.renorm(x);
                        word |= sy << (8 * j);
                    }
                    wv[0] = k == 0 ? word : wv[0]; wv[1] = k == 1 ? word : wv[1]; wv[2] = k == 2 ? word : wv[2]; wv[3] = k == 3 ? word : wv[3];
                }
            }
            *reinterpret_cast<uint4*>(sym + s0 + (long long)b * block_len + i) = make_uint4(wv[0], wv[1], wv[2], wv[3]);
            if (r.over()) { atomicOr(status, SG_ST_CORRUPT); return; }
        }
    }
    if (x != RANS_L || !r.at_end()) atomicOr(status, SG_ST_CORRUPT);      // a well-formed segment ends in the initial state
}

}  // namespace sg

using namespace sg;

static int stream_args_ok(const void* sym, const void* block_tab, int block_len, long long nsym, int seg_len) {
    if (!sym || !block_tab || nsym < 0) return SG_ERR_ARG;
    if (block_len <= 0 || block_len % 16 || seg_len <= 0 || seg_len % block_len || nsym % block_len) return SG_ERR_SHAPE;
    if ((uintptr_t)sym % 16 || (uintptr_t)block_tab % 2) return SG_ERR_ALIGN;
    return SG_OK;
}

extern "C" int sg_rans_hist(int device, void* stream, const unsigned char* sym, const unsigned short* block_tab, int block_len,
                            long long nsym, unsigned* counts) {
    if (!counts) return SG_ERR_ARG;
    int rc = stream_args_ok(sym, block_tab, block_len, nsym, block_len);
    if (rc != SG_OK) return rc;
    if (nsym == 0) return SG_OK;
    rc = use_device(device);
    if (rc != SG_OK) return rc;
    const long long nblocks = nsym / block_len, grid = (nblocks + 255) / 256;
    if (grid > 0x7fffffffLL) return SG_ERR_LIMIT;
    k_rans_hist<<<(unsigned)grid, 256, 0, (cudaStream_t)stream>>>(sym, block_tab, block_len, nblocks, counts);
    return cuda_ok(cudaGetLastError());
}

extern "C" int sg_rans_tables(int device, void* stream, const unsigned short* freq, int ntab, int pb, void* enc_tab, unsigned char* lut) {
    if (!freq || !enc_tab || ntab < 0 || (pb != 12 && pb != 14 && pb != 15)) return SG_ERR_ARG;
    if ((uintptr_t)enc_tab % 8) return SG_ERR_ALIGN;
    if (ntab == 0) return SG_OK;
    int rc = use_device(device);
    if (rc != SG_OK) return rc;
    k_rans_tables<<<ntab, 256, 0, (cudaStream_t)stream>>>(freq, pb, (RansSym*)enc_tab, lut, status_word(device));
    return cuda_ok(cudaGetLastError());
}

extern "C" int sg_rans_encode(int device, void* stream, const unsigned char* sym, const unsigned short* block_tab, int block_len,
                              long long nsym, int seg_len, int pb, const void* enc_tab, unsigned char* slots, size_t cap,
                              unsigned* out_len) {
    if (!enc_tab || !slots || !out_len || pb != 12) return SG_ERR_ARG;
    int rc = stream_args_ok(sym, block_tab, block_len, nsym, seg_len);
    if (rc != SG_OK) return rc;
    if (cap < 128 || cap % 16 || (uintptr_t)slots % 16) return SG_ERR_ALIGN;
    if (nsym == 0) return SG_OK;
    rc = use_device(device);
    if (rc != SG_OK) return rc;
    const long long nseg = (nsym + seg_len - 1) / seg_len;
    if (nseg > 0x7fffffffLL) return SG_ERR_LIMIT;
    const int spw = segs_per_warp(nseg);
    k_rans_encode<12><<<(unsigned)((nseg + spw - 1) / spw), 32, 0, (cudaStream_t)stream>>>(
        sym, block_tab, block_len, nsym, seg_len, (const RansSym*)enc_tab, slots, cap, out_len, (int)nseg, spw);
    return cuda_ok(cudaGetLastError());
}

extern "C" int sg_scan_gather(int device, void* stream, const unsigned char* slots, size_t cap, const unsigned* out_len, int nseg,
                              unsigned char* dst, unsigned long long dst_cap, unsigned long long* off) {
    if (!slots || !out_len || !off || nseg < 0 || (!dst && dst_cap)) return SG_ERR_ARG;
    int rc = use_device(device);
    if (rc != SG_OK) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    k_scan_lens<<<1, 1024, 0, st>>>(out_len, nseg, off, status_word(device));
    rc = cuda_ok(cudaGetLastError());
    if (rc != SG_OK || nseg == 0 || !dst) return rc;
    k_gather<<<(nseg + 7) / 8, 256, 0, st>>>(slots, cap, out_len, off, nseg, dst, dst_cap);
    return cuda_ok(cudaGetLastError());
}

extern "C" int sg_rans_decode(int device, void* stream, const unsigned char* in, const unsigned long long* off,
                              const unsigned short* block_tab, int block_len, long long nsym, int seg_len, int pb,
                              const void* enc_tab, const unsigned char* lut, int ntab, unsigned char* sym_out) {
    if (!in || !off || !enc_tab || !lut || pb != 12 || ntab < 0) return SG_ERR_ARG;
    int rc = stream_args_ok(sym_out, block_tab, block_len, nsym, seg_len);
    if (rc != SG_OK) return rc;
    if ((uintptr_t)in % 16) return SG_ERR_ALIGN;
    if (nsym == 0) return SG_OK;
    rc = use_device(device);
    if (rc != SG_OK) return rc;
    const long long nseg = (nsym + seg_len - 1) / seg_len;
    if (nseg > 0x7fffffffLL) return SG_ERR_LIMIT;
    cudaStream_t st = (cudaStream_t)stream;
    // tables staged in shared memory when their number is given and small enough to leave room for entries
    const size_t smem_max = 220 * 1024;
    if (ntab > 0 && (size_t)ntab * 6 + 16384 + 256 * RING_ROWS * 4 <= smem_max) {
        // segments per CTA: as few as fill the SMs (a warp's worth at least), 256 at most (their rings take 128 bytes each)
        long long per = (nseg + 147) / 148;
        per = per <= 32 ? 32 : per >= 256 ? 256 : (per + 31) / 32 * 32;
        const size_t head = (size_t)ntab * 4 + (size_t)per * RING_ROWS * 4, front = head > (4 << 12) ? head : 4 << 12;
        const unsigned cap = (unsigned)((smem_max - front - (size_t)ntab * 2 - 16) / 4);
        const size_t smem = front + (size_t)cap * 4 + (size_t)ntab * 2 + 16;
        static bool configured[64] = {false};
        if (device < 64 && !configured[device]) {
            rc = cuda_ok(cudaFuncSetAttribute(k_rans_decode_sm<12>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max + 1024));
            if (rc != SG_OK) return rc;
            configured[device] = true;
        }
        k_rans_decode_sm<12><<<(unsigned)((nseg + per - 1) / per), 512, smem, st>>>(in, off, block_tab, block_len, nsym, seg_len,
                                                                                (const RansSym*)enc_tab, lut, sym_out, (int)nseg, ntab, cap,
                                                                                (int)per, status_word(device));
        return cuda_ok(cudaGetLastError());
    }
    k_rans_decode<12><<<(unsigned)((nseg + 63) / 64), 64, 0, st>>>(in, off, block_tab, block_len, nsym, seg_len,
                                                                  (const RansSym*)enc_tab, lut, sym_out, (int)nseg, status_word(device));
    return cuda_ok(cudaGetLastError());
}
