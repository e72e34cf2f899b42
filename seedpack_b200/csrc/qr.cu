// QR residual coder kernels: histogram, encode, decode of a batch of stored blocks against their predictions.
//
// Replaces qr_hist / qr_enc / qr_dec (seedpack/qr.py:674-807).  Format and symbol order are the reference's:
// per segment (seg_blocks(T) blocks, one rANS state) and per block, in decode order: the "equals its prediction"
// flag (context: previous block's flag), then for a differing block its scale fields and its codes.  The encoder
// walks the same symbols backwards.
//
// What is done differently: block equality comes from a separate memory-bound pass (sg_residual_blocks: one
// coalesced sweep over F and P, one flag byte per block) instead of a byte loop inside the serial walk, so the
// per-segment lanes only touch the few blocks that differ; the coder uses the reciprocal / register-window
// engine of rans.cuh; histogram counts of the flag symbols are accumulated per lane and added once.
#include "api_util.h"
#include "qr_model.cuh"
#include "rans.cuh"

namespace sg {
namespace qr {

struct Setup {
    SG g; TM m; int qk, bs, nf, sublen, hboff;
    const uchar* sbase;
};
SG_DEVINL Setup setup(int T, const uchar* seed, const TM* tm, const SG* sg, int s) {
    Setup u;
    u.g = sg[s]; u.m = tm[u.g.t];
    u.qk = qk_of(T); u.bs = bs_of(T); u.nf = nfield(T); u.sublen = sublen_of(T);
    u.sbase = seed + u.m.seed_off;
    u.hboff = u.m.seed_type == 98 ? HBOFF_COL : 8;
    return u;
}

// symbols of one field delta, in decode order, through `emit(tab, sym)`
template <class E> SG_DEVINL void field_symbols(int kd, int any, int tv, int dl, E&& emit) {
    if (kd < 2 && (dl < -127 || dl > 127)) { emit(fctx(kd, any), 128); emit(FESC_LO, tv & 255); emit(FESC_HI, tv >> 8); }
    else emit(fctx(kd, any), dl & 255);
}

// ---- one coder for the three passes ---------------------------------------------------------------------------
struct Coder {
    int mode;                       // 0 histogram (symbols in decode order), 1 encode (symbols in reverse decode order),
                                    // 3 stage: like encode, but the (table, symbol) pairs are only written down
    unsigned* counts;
    unsigned* stage; int nstaged;
    const RansSym* enc;
    unsigned x; ByteWriterDown wr; uchar* slot; bool ovf;
    SG_DEVINL void put(int tab, int s) {
        if (mode == 0) { atomicAdd(counts + tab * 256 + s, 1u); return; }
        if (mode == 3) { stage[nstaged++] = (unsigned)(tab * 256 + s); return; }
        if (ovf) return;
        rans_put<12>(x, wr, enc[tab * 256 + s]);
        if (wr.ptr() < slot + 64) ovf = true;
    }
};

// ---- grid types: rank of the true lattice point among all points, by weighted distance to the seed -------------
// Per pair of weights a table in shared memory holds the weighted squared error of every pair of levels, so the
// distance of a lattice point is N/2 lookups (qr.py:496-515).  Laid out [entry][thread]: conflict-free.
constexpr int TOPK = 16;
constexpr int QR_TPB = 64;

template <int N, bool SGN>
SG_DEVINL void pair_tables(float* tab, const float* uu, const float* ww, float dl) {
    constexpr int B = N == 8 ? 2 : 3, L = 1 << B, E = L * L;
    for (int p = 0; p < N / 2; ++p)
        for (int e = 0; e < E; ++e) {
            const int la = e & (L - 1), lb = e >> B;
            const float qa = SGN ? (float)(2 * la + 1) : (float)(la - 1) + dl;
            const float qb = SGN ? (float)(2 * lb + 1) : (float)(lb - 1) + dl;
            const float ea = qa - uu[2 * p], eb = qb - uu[2 * p + 1];
            tab[(p * E + e) * QR_TPB + threadIdx.x] = ww[2 * p] * (ea * ea) + ww[2 * p + 1] * (eb * eb);
        }
}
template <int N> SG_DEVINL float point_dist(const float* tab, unsigned key) {
    constexpr int B = N == 8 ? 2 : 3, E = 1 << (2 * B);
    float d = 0.f;
#pragma unroll
    for (int p = 0; p < N / 2; ++p) d = d + tab[(p * E + ((key >> (2 * B * p)) & (E - 1))) * QR_TPB + threadIdx.x];
    return isnan(d) ? __int_as_float(0x7f800000) : d;
}
// the two smallest distances and the rank of point t in the order (distance, index)        (encode / histogram)
// Keys are read two at a time (gs is even, gk 4-byte aligned); points before t count when they are at most as far as
// t, points from t on when they are strictly closer (t itself is not).
template <int N> SG_DEVINL void scan_rank(const float* tab, const uint16_t* __restrict__ gk, int gs, int t, float& d1, float& d2, int& rank) {
    const float inf = __int_as_float(0x7f800000);
    const float dt = point_dist<N>(tab, gk[t]);
    const unsigned* gk2 = reinterpret_cast<const unsigned*>(gk);
    d1 = inf; d2 = inf; rank = 0;
    auto two_smallest = [&](float d) { d2 = fminf(d2, fmaxf(d1, d)); d1 = fminf(d1, d); };
    for (int k = 0; k < gs / 2; ++k) {              // every lane runs the same trip count
        const unsigned kk = __ldg(gk2 + k);
        const float da = point_dist<N>(tab, kk & 0xffffu), db = point_dist<N>(tab, kk >> 16);
        two_smallest(da); two_smallest(db);
        rank += (2 * k < t ? da <= dt : da < dt) + (2 * k + 1 < t ? db <= dt : db < dt);
    }
}
// all symbols of one differing block of a grid type after its scale fields (qr.py:553-637), in the encoder's order.
// fb: stored block, tv: its unpacked fields.
template <int N, bool SGN>
SG_DEVINL void grid_block(Coder& c, int T, int mv, uchar* fb, const uchar* pb, const int* tv, const uint16_t* __restrict__ gk,
                          long long gw0, int st, const uchar* sbase, int cols, const float* im, float* tab) {
    constexpr int B = N == 8 ? 2 : 3, ng = 8 / N;
    const int gs = grid_size(T);
    const bool par = parity_type(T);
    float sx2 = 0.f;
    for (int i = 0; i < 256; ++i) { float xv, hv; seed_val(st, sbase, gw0 + i, xv, hv, cols); sx2 += xv * xv; }
    const float sigma2 = (T == 16 || T == 17) ? sx2 * (1.0f / 256.f) : 2.f * sx2 * (1.0f / 256.f);
    const long long col0 = cols > 0 ? gw0 % cols : 0;
    for (int ui = 0; ui < 32; ++ui) {
        const int u = 31 - ui;
        const int p4 = pos4(col0 + 8 * u, cols);
        const int rank0 = mv >= 2 ? GRANK2 + 4 * p4 : GRID_RANK;
        const int sign0 = mv >= 2 ? GSIGN2 + 16 * p4 : GRID_SIGN;
        float gu[8], gw[8], gs_, gdl;
        int pn[8];
        gscale(T, fb, tv, u, gs_, gdl);
        {
            float x[8], v[8];
            for (int i = 0; i < 8; ++i) {
                const long long gwi = gw0 + 8 * u + i;
                float hv; seed_val(st, sbase, gwi, x[i], hv, cols);
                float wi = sqrtf(sigma2 + x[i] * x[i]);
                if (im) wi = wi * im[gwi % cols];
                gw[i] = wi;
                pn[i] = x[i] < 0.f;
                v[i] = SGN ? fabsf(x[i]) : x[i];
            }
            if (SGN && par) {                  // an odd number of negatives: the least weighty one flips back
                int cnt = 0;
                for (int i = 0; i < 8; ++i) cnt += pn[i];
                if (cnt & 1) {
                    int imin = 0; float mn = gw[0] * x[0] * x[0];
                    for (int i = 1; i < 8; ++i) { const float a = gw[i] * x[i] * x[i]; if (a < mn) { mn = a; imin = i; } }
                    pn[imin] ^= 1; v[imin] = -v[imin];
                }
            }
            for (int i = 0; i < 8; ++i) gu[i] = v[i] / gs_;
        }
        int tg[2] = {0, 0};
        auto sign_ctx = [&](int j) {
            const int lev = (gk[tg[j / N]] >> (B * (j % N))) & ((1 << B) - 1);
            const float m4 = fabsf(gu[j]) * 4.f;
            return sign0 + (lev == 0) * 8 + (m4 < 7.f ? (int)m4 : 7);
        };
        for (int gg = 0; gg < ng; ++gg) tg[gg] = get_gidx(T, fb, u * ng + gg);
        if (SGN) for (int j = 7; j >= 0; --j) {
            if (par && j == 7) continue;
            c.put(sign_ctx(j), get_neg(T, fb, 8 * u + j) ^ pn[j]);
        }
        for (int gg = ng - 1; gg >= 0; --gg) {
            pair_tables<N, SGN>(tab, gu + gg * N, gw + gg * N, gdl);
            int rank; float d1, d2;
            scan_rank<N>(tab, gk, gs, tg[gg], d1, d2, rank);
            const int ctx = rank0 + gapctx(d1, d2);
            if (rank >= TOPK) { c.put(FESC_HI, tg[gg] >> 8); c.put(FESC_LO, tg[gg] & 255); c.put(ctx, TOPK); }
            else c.put(ctx, rank);
        }
        if (T == 29) c.put(GRID_SHIFT, get_shift(fb, u) ^ get_shift(pb, u));
        if (c.ovf) return;
    }
}
SG_DEVINL void grid_code(Coder& c, int T, int mv, uchar* fb, const uchar* pb, const int* tv, const uint16_t* gk, long long gw0, int st,
                         const uchar* sbase, int cols, const float* im, float* tab) {
    switch (T) {
        case 18: case 21: grid_block<4, true>(c, T, mv, fb, pb, tv, gk, gw0, st, sbase, cols, im, tab); return;
        case 19: case 29: grid_block<8, false>(c, T, mv, fb, pb, tv, gk, gw0, st, sbase, cols, im, tab); return;
        default: grid_block<8, true>(c, T, mv, fb, pb, tv, gk, gw0, st, sbase, cols, im, tab);
    }
}

// ---- the three passes -------------------------------------------------------------------------------------------
extern __shared__ float gtab[];          // grid types only: 64 (IQ3: 128) floats per thread

struct Args {
    int T, mv, nseg;
    const uchar *F, *P, *ne, *seed;
    const TM* tm; const SG* sg;
    const uint16_t* gk; const float* imx;
};

// scalar-code types: the codes of one differing block, forwards (histogram) or backwards (encode, stage)
SG_DEVINL void scalar_codes(Coder& c, int T, int mv, uchar* fb, const uchar* pb, const int* tv, const Setup& u, long long gw0) {
    const long long col0 = u.m.cols > 0 ? gw0 % u.m.cols : 0;
    const bool fwd = c.mode == 0;
    int tsub = -1; float ta = 0.f, tc = 0.f;
    for (int i = 0; i < u.qk; ++i) {
        const int w = fwd ? i : u.qk - 1 - i;
        if (w / u.sublen != tsub) { tsub = w / u.sublen; wscale(T, tv, tsub, ta, tc); }
        float xv, hv; seed_val(u.m.seed_type, u.sbase, gw0 + w, xv, hv, u.m.cols);
        int r, sgn, ctx; predict_code(T, ta, tc, pb, w, xv, hv, u.hboff, r, sgn, ctx, mv, pos8(col0 + w, u.m.cols));
        c.put(ctx, (sgn * (get_code(T, fb, w) - r)) & 255);
    }
}

__global__ void __launch_bounds__(QR_TPB) k_qr_hist(const Args a, unsigned* __restrict__ counts) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= a.nseg) return;
    const int T = a.T, mv = a.mv;
    const Setup u = setup(T, a.seed, a.tm, a.sg, s);
    const float* im = u.m.imx_off >= 0 ? a.imx + u.m.imx_off : nullptr;
    Coder c; c.mode = 0; c.counts = counts; c.ovf = false;
    unsigned flagc[4] = {0, 0, 0, 0};                 // [prev * 2 + eq], added once per lane
    int prev = 1;
    for (long long b = u.g.b0; b < u.g.b0 + u.g.nb; ++b) {
        const int eq = !a.ne[b];
        ++flagc[prev * 2 + eq];
        prev = eq;
        if (eq) continue;
        const uchar* fb = a.F + b * u.bs; const uchar* pb = a.P + b * u.bs;
        int tv[MAXF], pv[MAXF];
        unpack_fields(T, fb, tv); unpack_fields(T, pb, pv);
        int any = 0;
        for (int k = 0; k < u.nf; ++k) {
            const int kd = fkind(T, k), dl = tv[k] - fpred(T, mv, pv, k, tv[0], u.nf > 1 ? tv[1] : 0);
            if (kd < 2 && (dl < -127 || dl > 127)) { c.put(fctx(kd, any), 128); c.put(FESC_LO, tv[k] & 255); c.put(FESC_HI, tv[k] >> 8); }
            else c.put(fctx(kd, any), dl & 255);
            any |= dl != 0;
        }
        const long long gw0 = (b - u.m.blk0) * u.qk;
        if (is_grid(T)) grid_code(c, T, mv, const_cast<uchar*>(fb), pb, tv, a.gk, gw0, u.m.seed_type, u.sbase, u.m.cols, im, gtab);
        else scalar_codes(c, T, mv, const_cast<uchar*>(fb), pb, tv, u, gw0);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) if (flagc[i]) atomicAdd(counts + (FLAG + (i >> 1)) * 256 + (i & 1), flagc[i]);
}

__global__ void __launch_bounds__(QR_TPB) k_qr_enc(const Args a, const RansSym* __restrict__ enc, uchar* __restrict__ out, size_t cap,
                                                   unsigned* __restrict__ out_len) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= a.nseg) return;
    const int T = a.T, mv = a.mv;
    const Setup u = setup(T, a.seed, a.tm, a.sg, s);
    const float* im = u.m.imx_off >= 0 ? a.imx + u.m.imx_off : nullptr;
    Coder c; c.mode = 1; c.enc = enc; c.slot = out + (size_t)s * cap; c.wr.init(c.slot + cap); c.x = RANS_L; c.ovf = false;
    for (long long b = u.g.b0 + u.g.nb - 1; b >= u.g.b0 && !c.ovf; --b) {
        const int eq = !a.ne[b];
        const int prev = b > u.g.b0 ? !a.ne[b - 1] : 1;
        if (eq) { c.put(FLAG + prev, 1); continue; }
        const uchar* fb = a.F + b * u.bs; const uchar* pb = a.P + b * u.bs;
        int tv[MAXF], pv[MAXF];
        unpack_fields(T, fb, tv); unpack_fields(T, pb, pv);
        const long long gw0 = (b - u.m.blk0) * u.qk;
        if (is_grid(T)) grid_code(c, T, mv, const_cast<uchar*>(fb), pb, tv, a.gk, gw0, u.m.seed_type, u.sbase, u.m.cols, im, gtab);
        else scalar_codes(c, T, mv, const_cast<uchar*>(fb), pb, tv, u, gw0);
        {   // fields, last to first; anyk = what the decoder will have seen before field k
            int dl[MAXF], anyk[MAXF], any = 0;
            for (int k = 0; k < u.nf; ++k) {
                dl[k] = tv[k] - fpred(T, mv, pv, k, tv[0], u.nf > 1 ? tv[1] : 0);
                anyk[k] = any; any |= dl[k] != 0;
            }
            for (int k = u.nf - 1; k >= 0; --k) {
                const int kd = fkind(T, k);
                if (kd < 2 && (dl[k] < -127 || dl[k] > 127)) { c.put(FESC_HI, tv[k] >> 8); c.put(FESC_LO, tv[k] & 255); c.put(fctx(kd, anyk[k]), 128); }
                else c.put(fctx(kd, anyk[k]), dl[k] & 255);
            }
        }
        c.put(FLAG + prev, 0);
    }
    if (c.ovf) { out_len[s] = 0xffffffffu; return; }
    rans_flush(c.x, c.wr);
    c.wr.flush();
    out_len[s] = c.wr.bad() ? LEN_NOFREQ : (unsigned)(c.slot + cap - c.wr.ptr());
}

// ---- decoder of the scalar-code types: a warp per segment ------------------------------------------------------------
// A segment is one rANS chain, so its symbols come out one after the other; but what a block's code symbols are coded
// WITH (context, predicted code, sign) depends only on the seed, the prediction and the block's scale fields, which
// are decoded first.  So the warp decodes flag and fields in lockstep (every lane runs the same chain on the same
// bytes, which costs what one lane would), then its lanes work out contexts and predictions of the block's weights
// side by side into shared memory, the chain runs over the staged contexts, and the lanes put the codes together.
// Table lookups for the symbols 0 and 1 (by far the most frequent) stay off global memory.
constexpr int DW_WARPS = 4;
struct __align__(8) DecWarpSmem {
    unsigned ring[RING_ROWS + 1];           // (a word more: the arrays below are read eight bytes at a time)
    unsigned fblk[56], pblk[56];            // the block being rebuilt / its prediction (block sizes <= 210 bytes)
    unsigned short ctx[256];
    short pred[256];
    signed char sgn[256];
    uchar sym[256];
};
// a segment's decoder, run by several lanes in lockstep over one ring
struct QrDec {
    unsigned x; RingReader<1> r; const RansSym* enc; const uchar* lut; const unsigned* f01;
    // w = f01[tab].  Symbols 0 and 1 without a load
    SG_DEVINL int step(int tab, unsigned w) {
        const unsigned slot = x & 4095u, f0 = w & 0xffffu, f1 = w >> 16;
        const bool one = slot >= f0;
        int s = one;
        unsigned f = one ? f1 : f0, d = one ? slot - f0 : slot;
        if (slot >= f0 + f1) {
            s = lut[((size_t)tab << 12) + slot];
            const unsigned fc = enc[tab * 256 + s].fc;
            f = fc & 0xffffu; d = slot - (fc >> 16);
        }
        x = f * (x >> 12) + d;
        r.renorm(x);
        return s;
    }
    SG_DEVINL int get(int tab) { return step(tab, f01[tab]); }
};
SG_DEVINL void or_byte(unsigned* blk, int i, unsigned v) { atomicOr(blk + (i >> 2), (v & 255u) << (8 * (i & 3))); }
// a code's bits OR-ed into a zeroed block in shared memory, safe for lanes that share a byte (4-bit single-part codes go in
// unmasked, qr.py:156-175)
SG_DEVINL void put_code_shared(int T, unsigned* blk, int w, int q) {
    const CodeLoc L = code_loc(T, w);
    if (T == 8) { or_byte(blk, L.lo_byte, (unsigned)q); return; }
    if (L.hi_bits) {
        or_byte(blk, L.lo_byte, (unsigned)((q & ((1 << L.lo_bits) - 1)) << L.lo_shift));
        or_byte(blk, L.hi_byte, (unsigned)(((q >> L.lo_bits) & ((1 << L.hi_bits) - 1)) << L.hi_shift));
    } else if (L.lo_bits == 2) or_byte(blk, L.lo_byte, (unsigned)((q & 3) << L.lo_shift));
    else or_byte(blk, L.lo_byte, (unsigned)(q << L.lo_shift));
}

// W lanes per segment, 32 / W segments per warp.  A chain instruction issued by a warp advances 32 / W chains, so a
// small W wastes fewer issue slots on the lockstep parts, a large W spreads the per-weight work wider.  The warp's
// control flow is kept uniform (every segment of the warp is at its j-th block; segments whose block equals its
// prediction, or that have ended, sit the phases out), so the lane groups stay converged.
// B CTAs per SM at least.  6 (80 registers) once the segments fill five per SM: with its 93 - 96 registers a kernel of Q2_K, Q4_K,
// Q5_K or Q2_0 gets five, and a last wave of a few CTAs took as long as all others (Q4_K, 12288 segments: 8.0 ms against 5.7).
// 1 below, where the registers are worth 4 % (2048 segments: 3.47 against 3.60 ms).
template <int T, int W, int B>
__global__ void __launch_bounds__(DW_WARPS * 32, B) k_qr_dec_warp(const Args a, const uchar* __restrict__ in, const unsigned long long* __restrict__ off,
                                                               const RansSym* __restrict__ enc, const uchar* __restrict__ lut,
                                                               uchar* __restrict__ F, int* __restrict__ status) {
    constexpr int SPW = 32 / W;
    constexpr int qk = qk_of(T), bs = bs_of(T), nf = nfield(T), sublen = sublen_of(T);
    __shared__ unsigned f01[NTAB2];
    __shared__ DecWarpSmem wsm[DW_WARPS * SPW];
    for (int t = threadIdx.x; t < NTAB2; t += blockDim.x) f01[t] = (enc[t * 256].fc & 0xffffu) | (enc[t * 256 + 1].fc << 16);
    __syncthreads();
    const int lane = threadIdx.x & 31, sub = lane % W, grp = (threadIdx.x >> 5) * SPW + lane / W;
    const int s = blockIdx.x * (DW_WARPS * SPW) + grp;
    const bool have = s < a.nseg;
    DecWarpSmem& m = wsm[grp];
    const int mv = a.mv;
    const unsigned group = (W == 32 ? 0xffffffffu : (1u << (W & 31)) - 1u) << (lane / W * W);
    const Setup u = setup(T, a.seed, a.tm, a.sg, have ? s : a.nseg - 1);
    QrDec c; c.enc = enc; c.lut = lut; c.f01 = f01;
    if (have) { c.r.init(in + off[s], in + off[s + 1], m.ring); c.x = c.r.state(); }
    else { c.r.init(in, in, m.ring); c.x = RANS_L; }
    // (the ring is one for the segment's lanes: none runs ahead into a top-up)
    auto top_up = [&]() { __syncwarp(group); c.r.top_up(); };
    uchar* fb = reinterpret_cast<uchar*>(m.fblk);
    const uchar* pbs = reinterpret_cast<const uchar*>(m.pblk);
    const int nb = have ? u.g.nb : 0;
    const int nbmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)nb);
    int prev = 1;
    for (int j = 0; j < nbmax; ++j) {
        const bool live = j < nb && !c.r.over();
        const long long b = u.g.b0 + j;
        const uchar* pg = a.P + b * bs;
        uchar* fg = F + b * bs;
        int eq = 1;
        if (live) { top_up(); eq = c.get(FLAG + prev); prev = eq; }
        if (live && eq) for (int i = sub; i < bs; i += W) fg[i] = pg[i];
        const bool code = live && !eq;
        if (!__any_sync(0xffffffffu, code)) continue;
        __syncwarp();
        if (code) {
            for (int i = sub; i < 56; i += W) m.fblk[i] = 0;
            for (int i = sub; i < bs; i += W) reinterpret_cast<uchar*>(m.pblk)[i] = pg[i];
        }
        __syncwarp();
        int tv[MAXF];
        if (code) {
            int pv[MAXF];
            unpack_fields(T, pbs, pv);
            int any = 0;
#pragma unroll
            for (int k = 0; k < nf; ++k) {
                if ((k & 3) == 0) top_up();
                const int kd = fkind(T, k);
                const int pr = fpred(T, mv, pv, k, k > 0 ? tv[0] : 0, k > 1 ? tv[1] : 0);
                const int sym = c.get(fctx(kd, any));
                int t;
                if (kd < 2 && sym == 128) { const int lo = c.get(FESC_LO), hi = c.get(FESC_HI); t = lo | (hi << 8); }
                else {
                    t = pr + (int)(signed char)sym;
                    if (kd < 2) t &= 0xffff;
                    else if (T == 14) t = (int)(signed char)(t & 255);
                }
                tv[k] = t; any |= t != pr;
            }
            if (sub == 0) pack_fields(T, fb, tv);
            // contexts and predictions of the block's weights, side by side
            const long long gw0 = (b - u.m.blk0) * qk;
            const long long col0 = u.m.cols > 0 ? gw0 % u.m.cols : 0;
            int tsub = -1; float ta = 0.f, tc = 0.f;
            for (int w = sub; w < qk; w += W) {
                if (w / sublen != tsub) { tsub = w / sublen; wscale(T, tv, tsub, ta, tc); }
                float xv, hv; seed_val(u.m.seed_type, u.sbase, gw0 + w, xv, hv, u.m.cols);
                int r, sgn, ctx; predict_code(T, ta, tc, pbs, w, xv, hv, u.hboff, r, sgn, ctx, mv, pos8(col0 + w, u.m.cols));
                m.ctx[w] = (unsigned short)ctx; m.pred[w] = (short)r; m.sgn[w] = (signed char)sgn;
            }
        }
        __syncwarp();
        if (code) {
#pragma unroll 1
            for (int w = 0; w < qk; w += 4) {          // four contexts per load, four symbols per store
                if ((w & 15) == 0) top_up();
                const uint2 cx = *reinterpret_cast<const uint2*>(m.ctx + w);
                unsigned sy = (unsigned)c.get((int)(cx.x & 0xffffu));
                sy |= (unsigned)c.get((int)(cx.x >> 16)) << 8;
                sy |= (unsigned)c.get((int)(cx.y & 0xffffu)) << 16;
                sy |= (unsigned)c.get((int)(cx.y >> 16)) << 24;
                if (sub == 0) *reinterpret_cast<unsigned*>(m.sym + w) = sy;
            }
        }
        __syncwarp();
        if (code) {
            for (int w = sub; w < qk; w += W) {
                int q = m.pred[w] + m.sgn[w] * (int)(signed char)m.sym[w];
                if (T == 8) q = (int)(signed char)(q & 255);
                put_code_shared(T, m.fblk, w, q);
            }
        }
        __syncwarp();
        if (code) for (int i = sub; i < bs; i += W) fg[i] = fb[i];
    }
    if (have && sub == 0 && (c.r.over() || c.x != RANS_L || !c.r.at_end())) atomicOr(status, SG_ST_CORRUPT);
}

// ---- decoder of the lattice types: a CTA per segment -------------------------------------------------------------------
// What makes these blocks expensive is the ordering of all 256 - 2048 lattice points by their weighted distance to the
// seed, once per group of 4 / 8 weights.  It depends on the seed and on the block's scale fields only, so that once the
// fields are decoded the CTA's warps rank all groups of the block side by side, four units of 8 weights at a time: the closest
// points and the gap context of every group go to shared memory.  The first warp then runs the chain - ranks and signs - over
// them, all lanes in lockstep, while the others fetch the next block and sum its squares.  A rank that is not among the
// closest four is looked up when it occurs; so is the group's order where IQ1_M's shift bit is not the prediction's, on which the
// level offset hangs.  (One warp per segment that ranked a group when the chain came to it: 13.2 ms for the 1024 x 3072
// weights of an IQ3_S tensor against 4.9, 60 ms for 2 x 4096 x 12288 against 39.)
// Bound by the chain with few segments, by the issue of the ranking with many: B CTAs per SM, that is 64 registers a thread.
constexpr int GTOP = 4;                            // ranked points kept per group
template <int T, int GW> struct GridSmem {           // GW: warps per CTA
    unsigned f01[NTAB2];                           // per table: frequency of symbol 0 | of symbol 1 << 16
    unsigned ring[RING_ROWS];
    unsigned fblk[28], pblk[2][28];                // block sizes <= 110 bytes
    float xs[2][256];                              // the block's seed values; this block and the next
    float sx2[2];
    float tab[GW][128];                            // pair tables of the group a warp ranks: [pair][levels]
    float dist[grid_size(T)];                      // distance of every lattice point (ranks beyond GTOP)
    float gu[256], gw[256];                        // per weight: seed value over the unit's scale (sign-folded), search weight
    unsigned short gk[grid_size(T)];               // the lattice's points
    unsigned short top[64][GTOP];                  // per group: closest points in order, NOPOINT, NOTKNOWN
    unsigned char gap[64];
    unsigned char pn[32], neg[32], shift[32];      // per unit: negative seed values; decoded sign symbols, shift bit
    unsigned short tg[64];
    int tv[MAXF];
    int eq;
};
template <int N> SG_DEVINL float point_dist_w(const float* tab, unsigned key) {
    constexpr int B = N == 8 ? 2 : 3, E = 1 << (2 * B);
    float d = 0.f;
#pragma unroll
    for (int p = 0; p < N / 2; ++p) d = d + tab[p * E + ((key >> (2 * B * p)) & (E - 1))];
    return fminf(d, __int_as_float(0x7f800000));   // (NaN: infinity)
}
// pair tables of the group of weights w0 .. w0 + N - 1, entries spread over the lanes
template <int N, bool SGN, class S> SG_DEVINL void group_tables(float* tab, const S& m, int w0, float gdl, int lane) {
    constexpr int B = N == 8 ? 2 : 3, L = 1 << B, E = L * L;
#pragma unroll
    for (int e = lane; e < (N / 2) * E; e += 32) {
        const int p = e / E, ee = e % E, la = ee & (L - 1), lb = ee >> B;
        const float qa = SGN ? (float)(2 * la + 1) : (float)(la - 1) + gdl;
        const float qb = SGN ? (float)(2 * lb + 1) : (float)(lb - 1) + gdl;
        const float ea = qa - m.gu[w0 + 2 * p], eb = qb - m.gu[w0 + 2 * p + 1];
        tab[e] = m.gw[w0 + 2 * p] * (ea * ea) + m.gw[w0 + 2 * p + 1] * (eb * eb);
    }
}
// a float's bits in an unsigned order (no NaN comes here)
SG_DEVINL unsigned ordered_bits(float d) { const unsigned u = __float_as_uint(d); return u ^ ((unsigned)((int)u >> 31) | 0x80000000u); }

// The lattice's points in shared memory: a word holds the points k and k + 32 of every 64
SG_DEVINL int gk_at(int k) { return (k & ~63) + 2 * (k & 31) + ((k >> 5) & 1); }

// Closest GTOP points of one group in the order (distance, index), and its gap context.  Every lane keeps the closest two of
// its own points (lane, lane + 32, ...; met in index order): a point goes in before the first one that is further away, so
// after its equals, and what stands there moves down one place, whatever the distances.  The warp's next one is then an
// arg-min over the lanes' lists.  Points at infinite distance never come up.  A lane that has given both of its points leaves
// the ranks after them unknown: looked up where one is coded.  (Lists of four cost as much as the distances themselves: IQ1_S
// 24576 segments 187 ms, with lists of two 142.)
constexpr int NOPOINT = 0xffff, NOTKNOWN = 0xfffe, LLEN = 2;
template <int N, bool SGN, int gs, class S> SG_DEVINL void rank_group(S& m, float* tab, int w0, float gdl, int lane, unsigned short* top, unsigned char* gap) {
    const float inf = __int_as_float(0x7f800000);
    __syncwarp();
    group_tables<N, SGN>(tab, m, w0, gdl, lane);
    __syncwarp();
    float D[LLEN]; int K[LLEN];
#pragma unroll
    for (int l = 0; l < LLEN; ++l) { D[l] = inf; K[l] = NOPOINT; }
    auto insert = [&](float d, int k) {
        bool lt[LLEN];
#pragma unroll
        for (int l = 0; l < LLEN; ++l) lt[l] = d < D[l];
#pragma unroll
        for (int l = LLEN - 1; l > 0; --l) { D[l] = fminf(fmaxf(d, D[l - 1]), D[l]); K[l] = lt[l - 1] ? K[l - 1] : lt[l] ? k : K[l]; }
        D[0] = fminf(d, D[0]); K[0] = lt[0] ? k : K[0];
    };
    const unsigned* gk2 = reinterpret_cast<const unsigned*>(m.gk) + lane;
#pragma unroll 4
    for (int k = 0; k < gs; k += 64) {
        const unsigned kk = gk2[k / 2];
        insert(point_dist_w<N>(tab, kk & 0xffffu), k + lane);
        insert(point_dist_w<N>(tab, kk >> 16), k + 32 + lane);
    }
    float d1 = inf, d2 = inf;
    int given = 0;
    bool known = true;
#pragma unroll
    for (int j = 0; j < GTOP; ++j) {
        const unsigned key = ordered_bits(D[0]), best = __reduce_min_sync(0xffffffffu, key);
        const unsigned bk = __reduce_min_sync(0xffffffffu, key == best ? (unsigned)K[0] : (unsigned)NOPOINT);
        if (lane == 0) top[j] = (unsigned short)(known ? bk : NOTKNOWN);
        if (j < 2) {
            const float d = __uint_as_float(best ^ ((best >> 31) ? 0x80000000u : 0xffffffffu));
            if (j == 0) d1 = d; else d2 = d;
        }
        if (key == best && (unsigned)K[0] == bk && bk != NOPOINT) {
#pragma unroll
            for (int l = 0; l + 1 < LLEN; ++l) { D[l] = D[l + 1]; K[l] = K[l + 1]; }
            D[LLEN - 1] = inf; K[LLEN - 1] = NOPOINT;
            ++given;
        }
        if (j + 1 >= LLEN && j + 1 < GTOP) known = known && !__any_sync(0xffffffffu, given == LLEN);
    }
    if (lane == 0) *gap = (unsigned char)gapctx(d1, d2);
}
// the point of rank r, by the first warp: distances to shared memory, then r + 1 rounds of an arg-min
template <int N, bool SGN, int gs, class S> SG_DEVINL int deep_rank(S& m, int w0, float gdl, int r, int lane) {
    const float inf = __int_as_float(0x7f800000);
    __syncwarp();
    group_tables<N, SGN>(m.tab[0], m, w0, gdl, lane);
    __syncwarp();
    float md = inf; int mk = 0x7fffffff;
    for (int k = lane; k < gs; k += 32) {
        const float d = point_dist_w<N>(m.tab[0], m.gk[gk_at(k)]);
        m.dist[k] = d;
        if (d < md) { md = d; mk = k; }
    }
    int bk = 0x7fffffff;
    for (int j = 0; j <= r; ++j) {
        float bd = md; bk = mk;
#pragma unroll
        for (int sft = 16; sft > 0; sft >>= 1) {
            const float od = __shfl_xor_sync(0xffffffffu, bd, sft);
            const int ok = __shfl_xor_sync(0xffffffffu, bk, sft);
            if (od < bd || (od == bd && ok < bk)) { bd = od; bk = ok; }
        }
        if (bk == mk && bk != 0x7fffffff) {
            m.dist[mk] = inf;
            md = inf; mk = 0x7fffffff;
            for (int k = lane; k < gs; k += 32) { const float d = m.dist[k]; if (d < md) { md = d; mk = k; } }
        }
        __syncwarp();
    }
    return bk == 0x7fffffff ? r : bk;              // slots beyond the points at finite distance keep their own number
}

template <int T, int GW, int B>
__global__ void __launch_bounds__(GW * 32, B) k_qr_dec_grid(const Args a, const uchar* __restrict__ in, const unsigned long long* __restrict__ off,
                                                         const RansSym* __restrict__ enc, const uchar* __restrict__ lut,
                                                         uchar* __restrict__ F, int* __restrict__ status) {
    constexpr int N = T == 18 || T == 21 ? 4 : 8, ng = 8 / N, LB = N == 8 ? 2 : 3, gs = grid_size(T), bs = bs_of(T), nf = nfield(T);
    constexpr bool SGN = T != 19 && T != 29, par = parity_type(T);
    __shared__ __align__(16) GridSmem<T, GW> m;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, s = blockIdx.x, mv = a.mv;
    const Setup u = setup(T, a.seed, a.tm, a.sg, s);
    const float* im = u.m.imx_off >= 0 ? a.imx + u.m.imx_off : nullptr;
    for (int t = threadIdx.x; t < NTAB2; t += GW * 32) m.f01[t] = (enc[t * 256].fc & 0xffffu) | (enc[t * 256 + 1].fc << 16);
    for (int k = threadIdx.x; k < gs; k += GW * 32) m.gk[gk_at(k)] = a.gk[k];
    // prediction / seed values of block j of the segment into buffer j & 1, by the warps w0 .. GW - 1
    auto fetch = [&](int j, int w0) {
        const long long b = u.g.b0 + j;
        if (j < u.g.nb) for (int i = (int)threadIdx.x - 32 * w0; i < bs; i += 32 * (GW - w0)) reinterpret_cast<uchar*>(m.pblk[j & 1])[i] = a.P[b * bs + i];
    };
    auto fetch_seed = [&](int j, int w0) {
        const long long gw0 = (u.g.b0 + j - u.m.blk0) * 256;
        for (int i = (int)threadIdx.x - 32 * w0; i < 256; i += 32 * (GW - w0)) {
            float xv, hv; seed_val(u.m.seed_type, u.sbase, gw0 + i, xv, hv, u.m.cols); m.xs[j & 1][i] = xv;
        }
    };
    auto sum_squares = [&](int j) {                // in order; one warp, every lane the same
        float sx2 = 0.f;
#pragma unroll 16
        for (int i = 0; i < 256; ++i) { const float xv = m.xs[j & 1][i]; sx2 += xv * xv; }
        if (lane == 0) m.sx2[j & 1] = sx2;
    };
    fetch(0, 0);
    __syncthreads();
    bool ahead = false;                            // block j's seed values are there
    QrDec c; c.enc = enc; c.lut = lut; c.f01 = m.f01;
    int prev = 1;
    if (warp == 0) { c.r.init(in + off[s], in + off[s + 1], m.ring); c.x = c.r.state(); }
    uchar* fb = reinterpret_cast<uchar*>(m.fblk);
    for (int j = 0; j < u.g.nb; ++j) {
        const long long b = u.g.b0 + j, gw0 = (b - u.m.blk0) * 256;
        const uchar* pbs = reinterpret_cast<const uchar*>(m.pblk[j & 1]);
        if (warp == 0) {
            __syncwarp();                          // (the ring is one for all lanes: no lane runs ahead into a top-up)
            c.r.top_up();
            int eq = c.get(FLAG + prev);
            prev = eq;
            if (c.r.over()) eq = 2;                // a damaged stream: no more blocks
            if (eq == 0) {
                int pv[MAXF], tv[MAXF];
                unpack_fields(T, pbs, pv);
                int any = 0;
#pragma unroll
                for (int k = 0; k < nf; ++k) {
                    if ((k & 3) == 0) { __syncwarp(); c.r.top_up(); }
                    const int kd = fkind(T, k);
                    const int pr = fpred(T, mv, pv, k, k > 0 ? tv[0] : 0, k > 1 ? tv[1] : 0);
                    const int sym = c.get(fctx(kd, any));
                    int t;
                    if (kd < 2 && sym == 128) { const int lo = c.get(FESC_LO), hi = c.get(FESC_HI); t = lo | (hi << 8); }
                    else {
                        t = pr + (int)(signed char)sym;
                        if (kd < 2) t &= 0xffff;
                    }
                    tv[k] = t; any |= t != pr;
                }
                if (lane < 28) m.fblk[lane] = 0;
                __syncwarp();
                if (lane == 0) {
                    pack_fields(T, fb, tv);
#pragma unroll
                    for (int k = 0; k < nf; ++k) m.tv[k] = tv[k];
                }
            }
            if (lane == 0) m.eq = eq;
        }
        __syncthreads();
        const int eq = m.eq;
        if (eq == 2) break;
        const long long col0 = u.m.cols > 0 ? gw0 % u.m.cols : 0;
        if (eq == 0 && !ahead) {
            fetch_seed(j, 0);
            __syncthreads();
            if (warp == 1) sum_squares(j);
            __syncthreads();
        }
        if (eq == 0) {
            // four units at a time, a weight per lane: search weight, sign folding with the parity repair, value over scale
#pragma unroll 1
            for (int part = warp; part < 8; part += GW) {
                const int un = 4 * part + (lane >> 3), i = lane & 7, w = 32 * part + lane;
                const float sx2 = m.sx2[j & 1], sigma2 = (T == 16 || T == 17) ? sx2 * (1.0f / 256.f) : 2.f * sx2 * (1.0f / 256.f);
                float gs_, gdl;
                gscale(T, fb, m.tv, un, gs_, gdl); // (the scale does not depend on IQ1_M's shift bit)
                const float x = m.xs[j & 1][w];
                float wi = sqrtf(sigma2 + x * x);
                if (im) wi = wi * im[(gw0 + w) % u.m.cols];
                float v = SGN ? fabsf(x) : x;
                unsigned pnb = (__ballot_sync(0xffffffffu, x < 0.f) >> (8 * (lane >> 3))) & 255u;
                if (SGN && par) {                  // an odd number of negatives: the least weighty one flips back
                    const float e = wi * x * x;
                    int imin = 0; float mn = __shfl_sync(0xffffffffu, e, 0, 8);
#pragma unroll
                    for (int q = 1; q < 8; ++q) { const float o = __shfl_sync(0xffffffffu, e, q, 8); if (o < mn) { mn = o; imin = q; } }
                    if (__popc(pnb) & 1) { pnb ^= 1u << imin; if (i == imin) v = -v; }
                }
                m.gu[w] = v / gs_; m.gw[w] = wi;
                if (i == 0) m.pn[un] = (unsigned char)pnb;
                __syncwarp();
#pragma unroll 1
                for (int q = 0; q < 4 * ng; ++q) {
                    const int g = 4 * ng * part + q;
                    float sc, dl;
                    gscale(T, fb, m.tv, g / ng, sc, dl);
                    if (T == 29) dl = get_shift(pbs, g) ? -0.125f : 0.125f;      // (the chain decodes whether the shift bit is the prediction's)
                    rank_group<N, SGN, gs>(m, m.tab[warp], N * g, dl, lane, m.top[g], &m.gap[g]);
                }
            }
        }
        __syncthreads();
        if (warp > 0) {
            fetch(j + 1, 1);
            if (eq == 0 && j + 1 < u.g.nb) {       // after a block that differs the next one is expected to differ as well
                fetch_seed(j + 1, 1);
                asm volatile("bar.sync 1, %0;" ::"n"((GW - 1) * 32) : "memory");
                if (warp == 1) sum_squares(j + 1);
            }
        } else if (eq) {
            for (int i = lane; i < bs; i += 32) F[b * bs + i] = pbs[i];
        } else {
#pragma unroll 1
            for (int un = 0; un < 32; ++un) {
                __syncwarp();
                c.r.top_up();                      // a unit takes 14 symbols at most
                const int p4 = pos4(col0 + 8 * un, u.m.cols);
                const int rank0 = mv >= 2 ? GRANK2 + 4 * p4 : GRID_RANK;
                const int sign0 = mv >= 2 ? GSIGN2 + 16 * p4 : GRID_SIGN;
                int h = 0;
                float gs_, gdl;
                gscale(T, fb, m.tv, un, gs_, gdl);
                if (T == 29) {
                    const int sp = get_shift(pbs, un);
                    h = (c.get(GRID_SHIFT) ^ sp) != 0; gdl = h ? -0.125f : 0.125f;
                    if (h != sp) { rank_group<N, SGN, gs>(m, m.tab[0], N * un, gdl, lane, m.top[un], &m.gap[un]); __syncwarp(); }
                }
                int tg[2] = {0, 0};
#pragma unroll
                for (int gg = 0; gg < ng; ++gg) {
                    const int g = un * ng + gg;
                    const int r = c.get(rank0 + m.gap[g]);
                    int t = r < GTOP ? m.top[g][r] : NOTKNOWN;
                    if (r >= TOPK) { const int lo = c.get(FESC_LO), hi = c.get(FESC_HI); t = (lo | (hi << 8)) % gs; }
                    else if (t == NOTKNOWN) t = deep_rank<N, SGN, gs>(m, N * g, gdl, r, lane);
                    else if (t == NOPOINT) t = r;
                    tg[gg] = t;
                }
                unsigned neg = 0;
                if (SGN) {
                    // lane j works out the context of sign j; the chain then takes the contexts' tables from the lanes
                    const int j8 = lane & 7, lev = (m.gk[gk_at(ng == 2 && j8 >= 4 ? tg[1] : tg[0])] >> (LB * (j8 % N))) & ((1 << LB) - 1);
                    const float m4 = fabsf(m.gu[8 * un + j8]) * 4.f;
                    const int sctx = sign0 + (lev == 0) * 8 + (m4 < 7.f ? (int)m4 : 7);
                    const unsigned sw = m.f01[sctx], pn = m.pn[un];
#pragma unroll
                    for (int q = 0; q < (par ? 7 : 8); ++q) {
                        const int tq = __shfl_sync(0xffffffffu, sctx, q);
                        const unsigned wq = __shfl_sync(0xffffffffu, sw, q);
                        if (c.step(tq, wq) ^ (int)((pn >> q) & 1u)) neg |= 1u << q;
                    }
                }
                if (lane < ng) m.tg[un * ng + lane] = (unsigned short)(lane ? tg[1] : tg[0]);
                if (lane == 0) { m.neg[un] = (unsigned char)neg; m.shift[un] = (unsigned char)h; }
                if (c.r.over()) break;
            }
            __syncwarp();
            // the block's bytes, a unit per lane (lanes share bytes)
            auto orb = [&](int i, unsigned v) { or_byte(m.fblk, i, v); };
            if (!c.r.over()) {
#pragma unroll
                for (int gg = 0; gg < ng; ++gg) put_gidx(T, orb, lane * ng + gg, m.tg[lane * ng + gg]);
                if (SGN) for (int q = 0; q < 8; ++q) if ((m.neg[lane] >> q) & 1) put_neg(T, orb, 8 * lane + q);
                if (T == 29 && m.shift[lane]) put_shift(orb, lane);
            }
            __syncwarp();
            for (int i = lane; i < bs; i += 32) F[b * bs + i] = fb[i];
        }
        ahead = eq == 0;
        __syncthreads();
    }
    if (threadIdx.x == 0 && (c.r.over() || c.x != RANS_L || !c.r.at_end())) atomicOr(status, SG_ST_CORRUPT);
}

// ---- encoding in two steps ---------------------------------------------------------------------------------------
// The model (fields, predictions, contexts, lattice ranks) of a block does not depend on the coder's state, only the
// rANS walk does.  So one lane per BLOCK first writes the block's (table, symbol) pairs down in the order the encoder
// consumes them; the histogram is a count over those pairs, and the coder proper is one lane per segment walking
// staged pairs.  The model runs once instead of twice, on seg_blocks(T) times as many lanes.
// Staging: cnt[b] pairs of block b at stage[b * capb ...], a pair is table * 256 + symbol.
__global__ void __launch_bounds__(QR_TPB) k_qr_stage(const Args a, int segb, unsigned* __restrict__ stage, unsigned short* __restrict__ cnt,
                                                     int capb) {
    const long long lane = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int s = (int)(lane / segb), j = (int)(lane % segb);
    if (s >= a.nseg) return;
    const int T = a.T, mv = a.mv;
    const Setup u = setup(T, a.seed, a.tm, a.sg, s);
    if (j >= u.g.nb) return;
    const long long b = u.g.b0 + j;
    const float* im = u.m.imx_off >= 0 ? a.imx + u.m.imx_off : nullptr;
    Coder c; c.mode = 3; c.stage = stage + (size_t)b * capb; c.nstaged = 0; c.ovf = false;
    const int eq = !a.ne[b];
    const int prev = j > 0 ? !a.ne[b - 1] : 1;
    if (eq) c.put(FLAG + prev, 1);
    else {
        const uchar* fb = a.F + b * u.bs; const uchar* pb = a.P + b * u.bs;
        int tv[MAXF], pv[MAXF];
        unpack_fields(T, fb, tv); unpack_fields(T, pb, pv);
        const long long gw0 = (b - u.m.blk0) * u.qk;
        if (is_grid(T)) grid_code(c, T, mv, const_cast<uchar*>(fb), pb, tv, a.gk, gw0, u.m.seed_type, u.sbase, u.m.cols, im, gtab);
        else scalar_codes(c, T, mv, const_cast<uchar*>(fb), pb, tv, u, gw0);
        int dl[MAXF], anyk[MAXF], any = 0;
        for (int k = 0; k < u.nf; ++k) {
            dl[k] = tv[k] - fpred(T, mv, pv, k, tv[0], u.nf > 1 ? tv[1] : 0);
            anyk[k] = any; any |= dl[k] != 0;
        }
        for (int k = u.nf - 1; k >= 0; --k) {
            const int kd = fkind(T, k);
            if (kd < 2 && (dl[k] < -127 || dl[k] > 127)) { c.put(FESC_HI, tv[k] >> 8); c.put(FESC_LO, tv[k] & 255); c.put(fctx(kd, anyk[k]), 128); }
            else c.put(fctx(kd, anyk[k]), dl[k] & 255);
        }
        c.put(FLAG + prev, 0);
    }
    cnt[b] = (unsigned short)c.nstaged;
}

// counts over the staged pairs, equal pairs of a warp added once.  A warp takes 32 blocks at a time: blocks with a
// single pair (equal to their prediction: just the flag) are counted one per lane, the others one after the other
// by the whole warp.
__global__ void __launch_bounds__(256) k_qr_stage_hist(long long nblocks, const unsigned* __restrict__ stage, const unsigned short* __restrict__ cnt,
                                                        int capb, unsigned* __restrict__ counts) {
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    auto add = [&](unsigned e, bool live) {
        const unsigned peers = __match_any_sync(0xffffffffu, live ? e : 0xffffffffu);
        if (live && lane == __ffs(peers) - 1) atomicAdd(counts + e, (unsigned)__popc(peers));
    };
    for (long long b0 = warp * 32; b0 < nblocks; b0 += nwarps * 32) {
        const long long b = b0 + lane;
        const int n = b < nblocks ? cnt[b] : 0;
        add(n == 1 ? stage[(size_t)b * capb] : 0u, n == 1);
        unsigned many = __ballot_sync(0xffffffffu, n > 1);
        while (many) {
            const int src = __ffs(many) - 1;
            many &= many - 1;
            const int nn = __shfl_sync(0xffffffffu, n, src);
            const unsigned* p = stage + (size_t)(b0 + src) * capb;
            for (int i0 = 0; i0 < nn; i0 += 32) add(i0 + lane < nn ? p[i0 + lane] : 0u, i0 + lane < nn);
        }
    }
}

// The coder proper: one lane per segment, blocks last to first, each block's staged pairs in order.  Bound by the lane's
// chain: pairs are taken eight at a time, asked for two groups ahead, their table entries one group ahead; a block's last
// group is filled with entries that leave the state as it is, so that the step has no branch.
__global__ void __launch_bounds__(32) k_qr_stage_code(const SG* __restrict__ sg, int nseg, const unsigned* __restrict__ stage,
                                                      const unsigned short* __restrict__ cnt, int capb, const RansSym* __restrict__ enc,
                                                      uchar* __restrict__ out, size_t cap, unsigned* __restrict__ out_len, int spw) {
    const int s = blockIdx.x * spw + threadIdx.x;
    if ((int)threadIdx.x >= spw || s >= nseg) return;
    const SG g = sg[s];
    uchar* slot = out + (size_t)s * cap;
    ByteWriterDown wr; wr.init(slot + cap);
    unsigned x = RANS_L;
    long long b = g.b0 + g.nb;                          // block of the group asked for last
    int i = 0, n = 0, nn = g.nb > 0 ? cnt[b - 1] : 0;   // next pair of it, its pairs, the pairs of the block before it
    uint4 pa = make_uint4(0, 0, 0, 0), pc = pa;
    int m0 = 0;
    auto load = [&]() {                                 // m0 = 0: no group left (a block has one pair at least)
        if (i >= n) {
            --b; i = 0;
            n = b >= g.b0 ? nn : 0;
            if (b - 1 >= g.b0) nn = cnt[b - 1];
        }
        m0 = min(8, n - i);
        if (m0 > 0) {
            const unsigned* p = stage + (size_t)b * capb + i;
            pa = *reinterpret_cast<const uint4*>(p);
            if (m0 > 4) pc = *reinterpret_cast<const uint4*>(p + 4);
        } else { m0 = 0; n = i = 0; b = g.b0; }
        i += 8;
    };
    const RansSym nop = {RANS_NOP_RCP, 4096u};
    auto look = [&](RansSym (&e)[8]) {
        const unsigned w[8] = {pa.x, pa.y, pa.z, pa.w, pc.x, pc.y, pc.z, pc.w};
#pragma unroll
        for (int k = 0; k < 8; ++k) { e[k] = nop; if (k < m0) e[k] = enc[w[k]]; }
    };
    RansSym cur[8], nxt[8];
    load();
    look(cur);
    int m = m0;
    load();
    while (m > 0) {
        look(nxt);
        m = m0;
        load();
#pragma unroll
        for (int k = 0; k < 8; k += 2) rans_put2<12>(x, wr, cur[k], cur[k + 1]);
        if (wr.ptr() < slot + 64) { out_len[s] = LEN_OVERFLOW; return; }       // 8 symbols write at most 16 bytes
#pragma unroll
        for (int k = 0; k < 8; ++k) cur[k] = nxt[k];
    }
    rans_flush(x, wr);
    wr.flush();
    out_len[s] = wr.bad() ? LEN_NOFREQ : (unsigned)(slot + cap - wr.ptr());
}

}  // namespace qr
}  // namespace sg

using namespace sg;
using namespace sg::qr;

static size_t grid_smem(int T) {
    switch (T) { case 18: case 21: return (size_t)QR_TPB * 4 * 128; case 16: case 17: case 19: case 22: case 29: return (size_t)QR_TPB * 4 * 64; }
    return 0;
}
static int grid_table_index(int T) {
    switch (T) { case 16: return 0; case 17: return 1; case 19: case 29: return 2; case 22: return 3; case 18: return 4; case 21: return 5; }
    return -1;
}
namespace sg { const uint16_t* device_grid_keys(int device, int which); }      // tables.cu

static int qr_args(int device, Args& a, int T, const void* F, const void* P, const void* ne, const void* seed, const void* tm,
                   const void* sgp, int nseg, const float* imx, int mv) {
    if (!P || !seed || !tm || !sgp || nseg < 0 || (mv != 1 && mv != 2)) return SG_ERR_ARG;
    int qk, bs;
    if (sg_type_info(T, &qk, &bs) != SG_OK) return SG_ERR_TYPE;
    a.T = T; a.mv = mv; a.nseg = nseg;
    a.F = (const uchar*)F; a.P = (const uchar*)P; a.ne = (const uchar*)ne; a.seed = (const uchar*)seed;
    a.tm = (const TM*)tm; a.sg = (const SG*)sgp; a.imx = imx; a.gk = nullptr;
    const int gi = grid_table_index(T);
    if (gi >= 0) {
        a.gk = device_grid_keys(device, gi);
        if (!a.gk) return SG_ERR_TABLES;
    }
    return SG_OK;
}

extern "C" int sg_qr_hist(int device, void* stream, int T, const unsigned char* F, const unsigned char* P, const unsigned char* ne,
                          const unsigned char* seed, const void* tm, const void* sgp, int nseg, const float* imx, unsigned* counts, int mv) {
    Args a;
    int rc = qr_args(device, a, T, F, P, ne, seed, tm, sgp, nseg, imx, mv);
    if (rc != SG_OK) return rc;
    if (!F || !ne || !counts) return SG_ERR_ARG;
    if (nseg == 0) return SG_OK;
    rc = use_device(device);
    if (rc != SG_OK) return rc;
    k_qr_hist<<<(nseg + QR_TPB - 1) / QR_TPB, QR_TPB, grid_smem(T), (cudaStream_t)stream>>>(a, counts);
    return cuda_ok(cudaGetLastError());
}

extern "C" int sg_qr_encode(int device, void* stream, int T, const unsigned char* F, const unsigned char* P, const unsigned char* ne,
                            const unsigned char* seed, const void* tm, const void* sgp, int nseg, const float* imx, const void* enc_tab,
                            unsigned char* slots, size_t cap, unsigned* out_len, int mv) {
    Args a;
    int rc = qr_args(device, a, T, F, P, ne, seed, tm, sgp, nseg, imx, mv);
    if (rc != SG_OK) return rc;
    if (!F || !ne || !enc_tab || !slots || !out_len) return SG_ERR_ARG;
    if (cap < 128 || cap % 16 || (uintptr_t)slots % 16) return SG_ERR_ALIGN;
    if (nseg == 0) return SG_OK;
    rc = use_device(device);
    if (rc != SG_OK) return rc;
    k_qr_enc<<<(nseg + QR_TPB - 1) / QR_TPB, QR_TPB, grid_smem(T), (cudaStream_t)stream>>>(a, (const RansSym*)enc_tab, slots, cap, out_len);
    return cuda_ok(cudaGetLastError());
}

extern "C" int sg_qr_decode(int device, void* stream, int T, const unsigned char* in, const unsigned long long* off,
                            const unsigned char* P, const unsigned char* seed, const void* tm, const void* sgp, int nseg, const float* imx,
                            const void* enc_tab, const unsigned char* lut, unsigned char* F, int mv) {
    Args a;
    int rc = qr_args(device, a, T, nullptr, P, nullptr, seed, tm, sgp, nseg, imx, mv);
    if (rc != SG_OK) return rc;
    if (!in || !off || !enc_tab || !lut || !F) return SG_ERR_ARG;
    if ((uintptr_t)in % 16) return SG_ERR_ALIGN;
    if (nseg == 0) return SG_OK;
    rc = use_device(device);
    if (rc != SG_OK) return rc;
    if (qr::is_grid(T)) {
        // up to four CTAs per SM: eight warps rank a block the faster; beyond, twice the segments side by side count for more (IQ1_S:
        // 384 segments 3.97 ms with eight warps and 4.09 with four, 768 segments 6.96 and 6.40, 6144 segments 42.7 and 36.9)
        auto run = [&](auto kernel, int warps) {
            kernel<<<nseg, warps * 32, 0, (cudaStream_t)stream>>>(a, in, off, (const RansSym*)enc_tab, lut, F, status_word(device));
        };
        switch (T) {
#define SG_DEC(t) case t: if (nseg <= 148 * 4) run(k_qr_dec_grid<t, 8, 4>, 8); else run(k_qr_dec_grid<t, 4, 8>, 4); break;
            SG_DEC(16) SG_DEC(17) SG_DEC(18) SG_DEC(19) SG_DEC(21) SG_DEC(22) SG_DEC(29)
#undef SG_DEC
        }
    }
    else
    {
        constexpr int W = 8, per_cta = DW_WARPS * (32 / W);
        auto run = [&](auto kernel) {
            kernel<<<(nseg + per_cta - 1) / per_cta, DW_WARPS * 32, 0, (cudaStream_t)stream>>>(a, in, off, (const RansSym*)enc_tab, lut, F, status_word(device));
        };
        const bool crowded = nseg > 148 * 5 * per_cta;
        switch (T) {
#define SG_DEC(t) case t: if (crowded) run(k_qr_dec_warp<t, W, 6>); else run(k_qr_dec_warp<t, W, 1>); break;
            SG_DEC(2) SG_DEC(3) SG_DEC(6) SG_DEC(7) SG_DEC(8) SG_DEC(10) SG_DEC(11)
            SG_DEC(12) SG_DEC(13) SG_DEC(14) SG_DEC(20) SG_DEC(23) SG_DEC(42)
#undef SG_DEC
            default: return SG_ERR_TYPE;
        }
    }
    return cuda_ok(cudaGetLastError());
}

// pairs one block can produce: flag + fields (an escaped field takes three) + codes, or for a lattice type per unit of
// 8 weights the ranks (an escaped rank takes three), 8 signs and a shift bit; rounded up to a multiple of 4
static int stage_capb(int T) {
    int qk, bs;
    if (sg_type_info(T, &qk, &bs) != SG_OK) return 0;
    const int nf = qr::nfield(T);
    const int n = 1 + 3 * nf + (qr::is_grid(T) ? 32 * (2 * 3 + 8 + 1) : qk);
    return (n + 3) / 4 * 4;
}
static size_t stage_cnt_bytes(long long nblocks) { return ((size_t)nblocks * 2 + 255) / 256 * 256; }

extern "C" size_t sg_qr_stage_bytes(int T, long long nblocks) {
    const int capb = stage_capb(T);
    if (!capb || nblocks < 0) return 0;
    return stage_cnt_bytes(nblocks) + (size_t)nblocks * capb * 4;
}

extern "C" int sg_qr_stage(int device, void* stream, int T, const unsigned char* F, const unsigned char* P, const unsigned char* ne,
                           const unsigned char* seed, const void* tm, const void* sgp, int nseg, const float* imx, int mv,
                           long long nblocks, void* stage, size_t stage_bytes) {
    Args a;
    int rc = qr_args(device, a, T, F, P, ne, seed, tm, sgp, nseg, imx, mv);
    if (rc != SG_OK) return rc;
    if (!F || !ne || !stage || nblocks < 0) return SG_ERR_ARG;
    if ((uintptr_t)stage % 16) return SG_ERR_ALIGN;
    if (stage_bytes < sg_qr_stage_bytes(T, nblocks)) return SG_ERR_SCRATCH;
    if (nseg == 0) return SG_OK;
    rc = use_device(device);
    if (rc != SG_OK) return rc;
    const int segb = 16384 / qr::qk_of(T) > 16 ? 16384 / qr::qk_of(T) : 16, capb = stage_capb(T);      // seg_blocks, qr.py:952-954
    const long long lanes = (long long)nseg * segb;
    k_qr_stage<<<(unsigned)((lanes + QR_TPB - 1) / QR_TPB), QR_TPB, grid_smem(T), (cudaStream_t)stream>>>(
        a, segb, (unsigned*)((uchar*)stage + stage_cnt_bytes(nblocks)), (unsigned short*)stage, capb);
    return cuda_ok(cudaGetLastError());
}

extern "C" int sg_qr_stage_hist(int device, void* stream, int T, long long nblocks, const void* stage, unsigned* counts) {
    const int capb = stage_capb(T);
    if (!capb) return SG_ERR_TYPE;
    if (!stage || !counts || nblocks < 0) return SG_ERR_ARG;
    if (nblocks == 0) return SG_OK;
    int rc = use_device(device);
    if (rc != SG_OK) return rc;
    const long long want = (nblocks + 255) / 256;
    k_qr_stage_hist<<<(unsigned)(want < 148 * 8 ? want : 148 * 8), 256, 0, (cudaStream_t)stream>>>(
        nblocks, (const unsigned*)((const uchar*)stage + stage_cnt_bytes(nblocks)), (const unsigned short*)stage, capb, counts);
    return cuda_ok(cudaGetLastError());
}

extern "C" int sg_qr_stage_encode(int device, void* stream, int T, long long nblocks, const void* stage, const void* sgp, int nseg,
                                  const void* enc_tab, unsigned char* slots, size_t cap, unsigned* out_len) {
    const int capb = stage_capb(T);
    if (!capb) return SG_ERR_TYPE;
    if (!stage || !sgp || !enc_tab || !slots || !out_len || nseg < 0 || nblocks < 0) return SG_ERR_ARG;
    if (cap < 128 || cap % 16 || (uintptr_t)slots % 16 || (uintptr_t)stage % 16) return SG_ERR_ALIGN;
    if (nseg == 0) return SG_OK;
    int rc = use_device(device);
    if (rc != SG_OK) return rc;
    const int spw = segs_per_warp(nseg);
    k_qr_stage_code<<<(nseg + spw - 1) / spw, 32, 0, (cudaStream_t)stream>>>(
        (const SG*)sgp, nseg, (const unsigned*)((const uchar*)stage + stage_cnt_bytes(nblocks)), (const unsigned short*)stage, capb,
        (const RansSym*)enc_tab, slots, cap, out_len, spw);
    return cuda_ok(cudaGetLastError());
}
