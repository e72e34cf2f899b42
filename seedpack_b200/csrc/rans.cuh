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
// Writes bytes at decreasing addresses ending at `end` (4-byte aligned).  Pending bytes sit at the top of a 64-bit register,
// the last one highest: a step shifts the low bytes of its state in (two funnel shifts).  Whenever four are pending the
// oldest four leave as one aligned word; two steps between flushes are the most that fits.
struct ByteWriterDown {
    uint8_t* p;                    // lowest address stored so far
    unsigned hi, lo;               // pending bytes
    int bits;                      // 8 x how many
    unsigned minf;                 // smallest frequency coded: 0 = tables not made from these symbols
    SG_DEVINL void init(uint8_t* end) { p = end; hi = lo = 0; bits = 0; minf = 1; }
    SG_DEVINL void push(unsigned x, int n8) {                  // the n8 / 8 <= 2 low bytes of x, the lowest first
        lo = __funnelshift_r(lo, hi, n8);
        hi = __funnelshift_r(hi, x, n8);
        bits += n8;
    }
    SG_DEVINL unsigned oldest() const { return __byte_perm(__funnelshift_rc(lo, hi, 64 - bits), 0, 0x0123); }       // bits >= 32
    SG_DEVINL void drain() {                                   // (a predicated store: a branch would end the block of independent steps)
        const bool four = bits >= 32;
        uint8_t* q = p - 4;
        asm volatile("{\n\t.reg .pred t;\n\tsetp.ne.u32 t, %0, 0;\n\t@t st.global.u32 [%1], %2;\n\t}" ::"r"((unsigned)four), "l"(q), "r"(oldest()) : "memory");
        p = four ? q : p;
        bits -= four ? 32 : 0;
    }
    SG_DEVINL bool bad() const { return minf == 0; }
    // bytes written so far end at this address (the lowest written byte)
    SG_DEVINL uint8_t* ptr() const { return p - (bits >> 3); }
    // store the pending bytes
    SG_DEVINL void flush() {
        drain();
        const int n = bits >> 3;
        for (int k = 0; k < n; ++k) p[-1 - k] = (uint8_t)(hi >> (32 - bits + 8 * k));
        p -= n; bits = 0;
    }
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
// A lane's ring: 32 words and a copy of the first (a read takes two neighbours) at a pitch of P words.  Between two
// top-ups a lane may take 32 bytes (16 symbols).
constexpr int RING_WORDS = 32, RING_ROWS = RING_WORDS + 1;
template <int P>
struct RingReader {
    const uint8_t* src;            // next 32 bytes to ask for (16-byte aligned)
    const uint8_t* end;
    uint4 c0, c1;                  // the 32 bytes asked for last
    unsigned* ring;
    unsigned pos, have;            // bits from the aligned start, modulo 2^32: taken, put into the ring (`have` is never far ahead)
    long long left;                // bits of the stream that are not in the ring yet; negative: it holds some past the end
    unsigned top;                  // the next four bytes, the first one highest
    SG_DEVINL void fetch() {
        c0 = c1 = make_uint4(0, 0, 0, 0);
        if (src < end) c0 = *reinterpret_cast<const uint4*>(src);
        if (src + 16 < end) c1 = *reinterpret_cast<const uint4*>(src + 16);
        src += 32;
    }
    SG_DEVINL void top_up() {
        if ((int)(have - pos) <= 8 * (4 * RING_WORDS - 32)) {
            const unsigned w = (have >> 5) & (RING_WORDS - 1); // a multiple of 8
            unsigned* r = ring + w * P;
            const unsigned a[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) r[i * P] = __byte_perm(a[i], 0, 0x0123);
            if (w == 0) ring[RING_WORDS * P] = __byte_perm(a[0], 0, 0x0123);
            have += 256;
            left -= 256;
            fetch();
        }
    }
    SG_DEVINL void look() {
        const unsigned off = (P >= 8 ? pos * (P / 8) : pos / (8 / P)) & ((RING_WORDS - 1) * P * 4);
        const unsigned* r = reinterpret_cast<const unsigned*>(reinterpret_cast<const char*>(ring) + off);
        top = __funnelshift_l(r[P], r[0], pos);                // (the shift counts modulo 32)
    }
    SG_DEVINL void init(const uint8_t* begin, const uint8_t* e, unsigned* r) {
        ring = r;
        src = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(begin) & ~(uintptr_t)15);
        pos = 8 * (unsigned)(begin - src); have = 0;
        end = e > begin ? e : begin;
        left = 8LL * (end - src);
        if (end == begin) end = src;                           // nothing to read
        fetch();
        top_up(); top_up(); top_up();
        look();
    }
    // (a stream may be longer than 2^32 bits: only distances are compared)
    SG_DEVINL bool over() const { return (int)(pos - have) > left; }
    SG_DEVINL bool at_end() const { return (int)(pos - have) == left; }
    // x after a step: the bytes that bring it to 2^23 or more.  A coder's state is 2^23 or more before a step, hence 2^8 or
    // more after it: two bytes at most.  (A damaged stream may leave it smaller; it is found out at the segment's end.)
    SG_DEVINL void renorm(unsigned& x) {
        const int n8 = x < (1u << 15) ? 16 : x < RANS_L ? 8 : 0;
        x = __funnelshift_l(top, x, n8);
        pos += n8;
        look();
    }
    SG_DEVINL unsigned state() { const unsigned x = top; pos += 32; look(); return x; }
};

// ---- coder steps -------------------------------------------------------------------------------------
// The chain from state to state: a shift, the reciprocal's high product, a shift, one multiply-add, two selects.  What
// depends on the entry alone (xm, the shift, the bias) is off it.  f = 1: the reciprocal 2^32 - 1 gives x - 1, made up
// for in the bias.
// Segments per warp of a kernel with one lane per segment: its time is that of one lane's chain, so a warp takes more than 8
// only once every scheduler of the 148 SMs has one.
inline int segs_per_warp(long long nseg) {
    const long long n = (nseg + 148 * 4 - 1) / (148 * 4);
    return n <= 8 ? 8 : n >= 32 ? 32 : (int)n;
}
constexpr unsigned RANS_NOP_RCP = 1u << 31;        // with freq = 2^12, cum = 0 (12 bits): an entry that leaves the state as it is
// what a step needs of an entry
struct RansStep { unsigned xm, rcp, sh_comp, bias; };                              // sh_comp = shift | (2^PB - freq) << 5
template <int PB> SG_DEVINL RansStep rans_step_of(const RansSym e) {
    const unsigned f = e.fc & 0xffffu, c = e.fc >> 16;
    const unsigned sh = f < 2 ? 0u : 31u - __clz(f - 1);
    return {e.fc << (31 - PB), e.rcp, sh | ((1u << PB) - f) << 5, f < 2 ? c + (1u << PB) - 1u : c};
}
template <class W>
SG_DEVINL void rans_put(unsigned& x, W& w, const RansStep t) {
    // x < 2^31 and xm >= 2^(31 - PB) for f >= 1: at most two bytes leave per symbol (PB <= 15).  The step is worked out for no,
    // one and two bytes side by side and chosen at the end, so that the comparisons are not on the chain
    const unsigned y1 = x >> 8, y2 = x >> 16, sh = t.sh_comp & 31u, comp = t.sh_comp >> 5;
    const bool one = x >= t.xm, two = y1 >= t.xm;
    const unsigned r0 = (__umulhi(x, t.rcp) >> sh) * comp + (x + t.bias);
    const unsigned r1 = (__umulhi(y1, t.rcp) >> sh) * comp + (y1 + t.bias);
    const unsigned r2 = (__umulhi(y2, t.rcp) >> sh) * comp + (y2 + t.bias);
    w.push(x, two ? 16 : one ? 8 : 0);
    x = two ? r2 : one ? r1 : r0;
}
// one symbol, or two with one look at the pending bytes
template <int PB, class W>
SG_DEVINL void rans_put(unsigned& x, W& w, const RansSym e) {
    w.minf = min(w.minf, e.fc & 0xffffu);
    rans_put(x, w, rans_step_of<PB>(e));
    w.drain();
}
template <int PB, class W>
SG_DEVINL void rans_put2(unsigned& x, W& w, const RansSym e, const RansSym f) {
    w.minf = min(w.minf, min(e.fc & 0xffffu, f.fc & 0xffffu));
    rans_put(x, w, rans_step_of<PB>(e));
    rans_put(x, w, rans_step_of<PB>(f));
    w.drain();
}
template <class W> SG_DEVINL void rans_flush(unsigned x, W& w) {
#pragma unroll
    for (int i = 0; i < 4; ++i) { w.push(x, 8); w.drain(); x >>= 8; }
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
