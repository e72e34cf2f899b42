// Byte-renormalising rANS coder core, one 32-bit state per segment, one segment per lane.
//
// The bitstream is fixed by the reference (seedpack/qr.py:651-663 PUT / GET, seedpack/bf16v2.py:84-137,
// seedpack/rans.py:54-105): state in [2^23, 2^31), static per-context tables with frequencies summing to
// 2^PB, the encoder walks its symbols backwards writing bytes downwards from the end of a private slot and
// finishes with the 4 state bytes, so that a segment's stream reads forwards as state (big endian)
// followed by the renormalisation bytes in decode order.
//
// What differs from the reference is only how a lane gets there:
//   * x / f and x % f use a per-(table, symbol) 32-bit reciprocal (exact for x < 2^31, which the
//     renormalisation guarantees) instead of integer division;
//   * a coder step has no branch: the number of bytes it moves (0, 1 or 2) is two comparisons, the bytes enter or
//     leave a shift register.  The lanes of a warp sit in different segments and renormalise at different symbols, so
//     that a branch per byte ran on nearly every symbol of the warp: 280 - 360 cycles a symbol before, see the kernels.
#pragma once
#include "common.cuh"

namespace sg {

constexpr unsigned RANS_L = 1u << 23;
constexpr unsigned LEN_OVERFLOW = 0xffffffffu;     // out_len of a segment whose slot was too small (retry with more)
constexpr unsigned LEN_NOFREQ   = 0xfffffffeu;     // out_len of a segment that met a symbol its table gives no frequency

// encoder entry for one (table, symbol): rcp = ceil(2^(31+s) / freq) with s = ceil(log2 freq); fc = freq | cum << 16
struct __align__(8) RansSym { unsigned rcp, fc; };

SG_DEVINL unsigned rans_shift(unsigned freq) { return freq < 2 ? 0u : 32u - __clz(freq - 1); }

// ---- downward byte writer ----------------------------------------------------------------------------
// Writes bytes at decreasing addresses ending at `end` (4-byte aligned).  Pending bytes sit in `acc`, the last one lowest;
// whenever four are there the oldest four leave as one aligned word.
struct ByteWriterDown {
    uint8_t* p;                    // lowest address stored so far
    unsigned long long acc;        // pending bytes (what is above them has left already)
    int cnt;                       // how many: 0 .. 3 between calls
    unsigned bad;                  // set when a symbol with frequency 0 was coded (tables not made from these symbols)
    SG_DEVINL void init(uint8_t* end) { p = end; acc = 0; cnt = 0; bad = 0; }
    SG_DEVINL bool push(unsigned x, int n) {                   // the n <= 2 low bytes of x, the lowest first
        const unsigned v = n == 2 ? __byte_perm(x, 0, 0x4401) : n ? x & 0xffu : 0u;
        acc = (acc << (8 * n)) | v;
        cnt += n;
        return cnt >= 4;
    }
    SG_DEVINL void emit(unsigned x, int n) {
        if (push(x, n)) { cnt -= 4; p -= 4; *reinterpret_cast<unsigned*>(p) = (unsigned)(acc >> (8 * cnt)); }
    }
    // bytes written so far end at this address (the lowest written byte)
    SG_DEVINL uint8_t* ptr() const { return p - cnt; }
    // store the pending bytes
    SG_DEVINL void flush() { for (; cnt > 0; --cnt) *--p = (uint8_t)(acc >> (8 * (cnt - 1))); }
};

// ---- forward byte reader -----------------------------------------------------------------------------
// Reads bytes at increasing addresses from [p, end) through aligned 16-byte loads; reads past `end` return 0
// and set `over`.
struct ByteReaderUp {
    const uint8_t* win;            // aligned address of the loaded window
    unsigned long long lo, hi;     // the window
    unsigned long long nlo, nhi;   // the window after it, fetched when this one was entered (its latency is off the chain)
    const uint8_t* p;
    const uint8_t* end;
    bool over;
    SG_DEVINL void fetch_next() {
        if (win + 16 < end) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(win + 16);
            nlo = v.x; nhi = v.y;
        }
    }
    SG_DEVINL void init(const uint8_t* begin, const uint8_t* e) {
        p = begin; end = e; over = false;
        win = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(begin) & ~(uintptr_t)15);
        lo = hi = nlo = nhi = 0;
        if (begin < e) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(win);
            lo = v.x; hi = v.y;
            fetch_next();
        }
    }
    SG_DEVINL unsigned get() {
        if (p >= end) { over = true; return 0; }
        const int k = (int)(p - win);
        const unsigned b = (unsigned)((k >= 8 ? hi >> (8 * (k - 8)) : lo >> (8 * k)) & 0xff);
        ++p;
        if (k == 15) { win += 16; lo = nlo; hi = nhi; fetch_next(); }
        return b;
    }
};

// ---- forward reader through a ring in shared memory --------------------------------------------------------
// For kernels whose lanes decode side by side.  A register that is refilled by a load when a lane has used it up makes
// the whole warp wait for that load, and with 8 - 32 segments per warp some lane refills at almost every symbol.  Here all
// lanes top their rings up together, every few symbols, with the 32 bytes that were asked for at the last top-up; a
// symbol takes its next four bytes from two shared-memory words, off the state's own chain.
// A lane's ring: 32 words at a stride of `pitch` words.  Between two top-ups a lane may take 32 bytes (16 symbols).
constexpr int RING_WORDS = 32;
struct RingReader {
    const uint8_t* src;            // next 32 bytes to ask for (16-byte aligned)
    const uint8_t* end;
    uint4 c0, c1;                  // the 32 bytes asked for last
    unsigned* ring; int pitch;
    int pos, have, len;            // bytes from the aligned start: taken, put into the ring, in the stream
    unsigned top;                  // the next four bytes, the first one highest
    SG_DEVINL void fetch() {
        c0 = c1 = make_uint4(0, 0, 0, 0);
        if (src < end) c0 = *reinterpret_cast<const uint4*>(src);
        if (src + 16 < end) c1 = *reinterpret_cast<const uint4*>(src + 16);
        src += 32;
    }
    SG_DEVINL void put(const uint4 v, int w) {
        const unsigned a[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) ring[((w + i) & (RING_WORDS - 1)) * pitch] = __byte_perm(a[i], 0, 0x0123);
    }
    SG_DEVINL void top_up() {
        if (have - pos <= 4 * RING_WORDS - 32) {
            put(c0, have >> 2); put(c1, (have >> 2) + 4);
            have += 32;
            fetch();
        }
    }
    SG_DEVINL void look() {
        const unsigned hi = ring[((pos >> 2) & (RING_WORDS - 1)) * pitch], lo = ring[((pos >> 2) + 1 & (RING_WORDS - 1)) * pitch];
        top = __funnelshift_l(lo, hi, 8 * (pos & 3));
    }
    SG_DEVINL void init(const uint8_t* begin, const uint8_t* e, unsigned* r, int stride) {
        ring = r; pitch = stride;
        src = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(begin) & ~(uintptr_t)15);
        pos = (int)(begin - src); have = 0;
        end = e > begin ? e : begin;
        len = (int)min((long long)(end - src), 0x7fffff00LL);
        if (end == begin) end = src;                           // nothing to read
        fetch();
        top_up(); top_up(); top_up();
        look();
    }
    SG_DEVINL bool over() const { return pos > len; }
    SG_DEVINL bool at_end() const { return pos == len; }
    // x after a step: take bytes until x >= 2^23 (a stream that was coded needs at most two)
    SG_DEVINL void renorm(unsigned& x) {
        int n = x < (1u << 15) ? 2 : x < RANS_L ? 1 : 0;
        x = __funnelshift_l(top, x, 8 * n);
        pos += n;
        look();
        if (x < RANS_L && n) {                                 // damaged streams only
#pragma unroll 1
            for (int guard = 0; guard < 2 && x < RANS_L; ++guard) { x = __funnelshift_l(top, x, 8); ++pos; look(); }
        }
    }
    SG_DEVINL unsigned state() { const unsigned x = top; pos += 4; look(); return x; }
};

// ---- coder steps -------------------------------------------------------------------------------------
// The chain from state to state: two comparisons, a shift, the reciprocal's high product, a shift, one multiply-add.  What
// depends on the entry alone (xm, the shift, the bias) is off it.  f = 1: the reciprocal 2^32 - 1 gives x - 1, made up
// for in the bias.
// Segments per warp of a kernel with one lane per segment: its time is that of one lane's chain, so a warp takes more than 8
// only once every scheduler of the 148 SMs has one.
inline int segs_per_warp(long long nseg) {
    const long long n = (nseg + 148 * 4 - 1) / (148 * 4);
    return n <= 8 ? 8 : n >= 32 ? 32 : (int)n;
}
constexpr unsigned RANS_NOP_RCP = 1u << 31;        // with freq = 2^12, cum = 0 (12 bits): an entry that leaves the state as it is
template <int PB, class W>
SG_DEVINL void rans_put(unsigned& x, W& w, const RansSym e) {
    const unsigned f = e.fc & 0xffffu, c = e.fc >> 16;
    const unsigned xm = f << (31 - PB);
    // x < 2^31 and xm >= 2^(31 - PB) for f >= 1: at most two bytes leave per symbol (PB <= 15); a zero frequency marks the segment
    w.bad |= (unsigned)(f == 0);
    const int n = x >= xm ? ((x >> 8) >= xm ? 2 : 1) : 0;
    w.emit(x, n);
    x >>= 8 * n;
    const unsigned sh = f < 2 ? 0u : 31u - __clz(f - 1), bias = f < 2 ? c + (1u << PB) - 1u : c;
    const unsigned q = __umulhi(x, e.rcp) >> sh;
    x = q * ((1u << PB) - f) + (x + bias);
}
template <class W> SG_DEVINL void rans_flush(unsigned x, W& w) {
#pragma unroll
    for (int i = 0; i < 4; ++i) { w.emit(x, 1); x >>= 8; }
}
template <class R> SG_DEVINL unsigned rans_init(R& r) {
    unsigned x = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) x = (x << 8) | r.get();
    return x;
}
// decode one symbol of table `t`: lut = symbol per slot, tab = encoder entries of the same table (freq, cum)
template <int PB, class R>
SG_DEVINL unsigned rans_get(unsigned& x, R& r, const uint8_t* __restrict__ lut, const RansSym* __restrict__ tab) {
    const unsigned slot = x & ((1u << PB) - 1);
    const unsigned s = lut[slot];
    const unsigned fc = tab[s].fc;
    x = (fc & 0xffffu) * (x >> PB) + slot - (fc >> 16);
#pragma unroll 1
    for (int guard = 0; guard < 4 && x < RANS_L; ++guard) x = (x << 8) | r.get();
    return s;
}

// The same through a compact table (RANS_COMPACT bytes per context: 256 coarse entries, one per 2^(PB - 8) slots = the
// symbol whose range holds the bucket's first slot, then the 256 symbols' freq | cum << 16 words) and a walk over the
// words from the coarse entry: 1.25 KiB per context instead of 2^PB + 2 KiB.
constexpr int RANS_COMPACT = 256 + 256 * 4;
template <int PB, class R>
SG_DEVINL unsigned rans_get_compact(unsigned& x, R& r, const uint8_t* __restrict__ ct) {
    const unsigned* __restrict__ words = reinterpret_cast<const unsigned*>(ct + 256);
    const unsigned slot = x & ((1u << PB) - 1);
    unsigned s = ct[slot >> (PB - 8)];
    unsigned fc = words[s];
#pragma unroll 1
    while (slot >= (fc >> 16) + (fc & 0xffffu) && s < 255u) fc = words[++s];
    x = (fc & 0xffffu) * (x >> PB) + slot - (fc >> 16);
#pragma unroll 1
    for (int guard = 0; guard < 4 && x < RANS_L; ++guard) x = (x << 8) | r.get();
    return s;
}

}  // namespace sg
