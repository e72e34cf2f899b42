// R2: the BF16 base-model codec (context-modelled rANS over exponent, mantissa and sign of every weight) and the
// order-fixed float64 statistics that define its contexts.
//
// Replaces v2_hist / v2_enc / v2_dec / row_hash (seedpack/bf16v2.py:63-155) and the statistics pass `_stats`
// (seedpack/bf16v2.py:225-244) with its detmath kernels (seedpack/detmath.py:67-106).  Format: 15 probability bits,
// segments of 16384 weights, three symbols per weight in decode order exponent, mantissa, sign; contexts
//   exponent: clamp(rfi[row] + cfi[col] + 256, 0, 511)          (predicted log2 sigma in 1/8 octave)
//   mantissa: 512 + clamp(8 * exponent - pred - 952, 0, 127)
//   sign:     640 + scl[col]                                       (column bias class)
// plus the tensor's role offset (656 tables per role).
#include "api_util.h"
#include "detmath.cuh"
#include "rans.cuh"

namespace sg {
namespace r2 {

constexpr int PB = 15;

struct TB { long long doff; int rowlen, rowbase, colbase, tab, rmap, pad; };       // bf16v2.py:158
struct SG { int t, n; long long i0; };                                             // bf16v2.py:159

SG_DEVINL int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

struct Ctx {
    const short* rfi; const short* cfi; const signed char* scl; const int* rowmap;
};

// position of a lane inside its tensor: compact row rc (after duplicate-row removal), column j, original row
struct Cursor {
    TB T; int rc, j, orow; const unsigned short* w;
    SG_DEVINL void seek(const unsigned char* dev, const TB& t, long long i, const int* rowmap) {
        T = t; rc = (int)(i / T.rowlen); j = (int)(i % T.rowlen);
        orow = T.rmap >= 0 ? rowmap[T.rmap + rc] : rc;
        w = reinterpret_cast<const unsigned short*>(dev + T.doff) + (size_t)orow * T.rowlen;
    }
    SG_DEVINL void row(const unsigned char* dev, const int* rowmap) {
        orow = T.rmap >= 0 ? rowmap[T.rmap + rc] : rc;
        w = reinterpret_cast<const unsigned short*>(dev + T.doff) + (size_t)orow * T.rowlen;
    }
};

SG_DEVINL void contexts(const Ctx& c, const TB& T, int orow, int j, int& pred, int& pe, int& sc) {
    pred = c.rfi[T.rowbase + orow] + c.cfi[T.colbase + j];
    pe = clampi(pred + 256, 0, 511);
    sc = clampi(c.scl[T.colbase + j], 0, 15);         // (0..15 by construction, bf16v2.py:243; a damaged side part must not index past the tables)
}
SG_DEVINL int mctx(int ex, int pred) { return clampi(8 * ex - pred - 1016 + 64, 0, 127); }

// Counts do not depend on the order of the weights.  A CTA takes `per` segments, as few as give two CTAs per SM their share,
// and its 16 warps walk through a segment together (coalesced reads, four weights per lane in flight).  Bound by the shared
// memory's atomics, three per weight.  Mantissa symbols are spread over 128 x 128 counters per role, which a CTA collects in
// shared memory (64 KB) and adds to global memory at its end; so are the exponent symbols inside a window of 128 contexts x
// 64 exponents around the CTA's first weight (weights of one tensor keep to a few octaves; what falls outside the window
// goes to global memory directly).  Of the sign's 32 counters every lane has its own copy: they would collide on every step.
constexpr int R2H_THREADS = 512, R2H_U = 4;
constexpr int R2H_SMEM = (128 * 128 + 128 * 64 + 32 * 32) * 4;
__global__ void __launch_bounds__(R2H_THREADS, 2) k_r2_hist(const unsigned char* __restrict__ dev, const TB* __restrict__ tb,
                                                            const SG* __restrict__ sg, int nseg, int per, Ctx c, unsigned* __restrict__ counts) {
    extern __shared__ unsigned mhist[];            // [128 contexts][128 symbols] of the role of the CTA's first segment
    unsigned* ehist = mhist + 128 * 128;           // [128 contexts from pe0][64 exponents from ex0] of the same role
    unsigned* shist = ehist + 128 * 64;            // [16 classes x sign][lane] of the same role
    __shared__ int win[2];
    for (int i = threadIdx.x; i < R2H_SMEM / 4; i += R2H_THREADS) mhist[i] = 0;
    const int lane = threadIdx.x & 31, first = blockIdx.x * per;
    const int cta_tab = tb[sg[first].t].tab;
    if (threadIdx.x == 0) {
        const SG g = sg[first];
        const TB T = tb[g.t];
        const int rc = (int)(g.i0 / T.rowlen), j = (int)(g.i0 % T.rowlen);
        const int orow = T.rmap >= 0 ? c.rowmap[T.rmap + rc] : rc;
        const unsigned u = reinterpret_cast<const unsigned short*>(dev + T.doff)[(size_t)orow * T.rowlen + j];
        int pred, pe, sc; contexts(c, T, orow, j, pred, pe, sc);
        win[0] = pe - 64; win[1] = (int)((u >> 7) & 255) - 40;      // weights mostly lie below the typical magnitude
    }
    __syncthreads();
    const int pe0 = win[0], ex0 = win[1];
    for (int s = first; s < min(nseg, first + per); ++s) {
        const SG g = sg[s];
        const TB T = tb[g.t];
        const bool local = T.tab == cta_tab;
        unsigned* gt = counts + (size_t)T.tab * 256;
        // this lane's weight: compact row rc, column j; a CTA's width further every time (no division inside the loop)
        const int dr = R2H_THREADS / T.rowlen, dj = R2H_THREADS % T.rowlen;
        int rc = (int)((g.i0 + threadIdx.x) / T.rowlen), j = (int)((g.i0 + threadIdx.x) % T.rowlen);
        const unsigned short* base = reinterpret_cast<const unsigned short*>(dev + T.doff);
        for (int k0 = threadIdx.x; k0 < g.n; k0 += R2H_THREADS * R2H_U) {
            unsigned u[R2H_U];
            int pred[R2H_U], pe[R2H_U], sc[R2H_U];
#pragma unroll
            for (int v = 0; v < R2H_U; ++v) {
                if (k0 + v * R2H_THREADS < g.n) {
                    const int orow = T.rmap >= 0 ? c.rowmap[T.rmap + rc] : rc;
                    u[v] = base[(size_t)orow * T.rowlen + j];
                    contexts(c, T, orow, j, pred[v], pe[v], sc[v]);
                }
                j += dj; rc += dr;
                if (j >= T.rowlen) { j -= T.rowlen; ++rc; }
            }
#pragma unroll
            for (int v = 0; v < R2H_U; ++v) {
                if (k0 + v * R2H_THREADS >= g.n) break;
                const int ex = (u[v] >> 7) & 255, man = u[v] & 127, sgn = u[v] >> 15, mc = mctx(ex, pred[v]);
                if (local && (unsigned)(pe[v] - pe0) < 128u && (unsigned)(ex - ex0) < 64u) atomicAdd(ehist + (pe[v] - pe0) * 64 + (ex - ex0), 1u);
                else atomicAdd(gt + pe[v] * 256 + ex, 1u);
                if (local) {
                    atomicAdd(mhist + mc * 128 + man, 1u);
                    atomicAdd(shist + (sc[v] * 2 + sgn) * 32 + lane, 1u);
                } else {
                    atomicAdd(gt + (512 + mc) * 256 + man, 1u);
                    atomicAdd(gt + (640 + sc[v]) * 256 + sgn, 1u);
                }
            }
        }
    }
    __syncthreads();
    unsigned* gt = counts + (size_t)cta_tab * 256;
    for (int i = threadIdx.x; i < 128 * 128; i += R2H_THREADS) {
        const unsigned v = mhist[i];
        if (v) atomicAdd(gt + (512 + (i >> 7)) * 256 + (i & 127), v);
    }
    for (int i = threadIdx.x; i < 128 * 64; i += R2H_THREADS) {
        const unsigned v = ehist[i];
        if (v) atomicAdd(gt + (pe0 + (i >> 6)) * 256 + ex0 + (i & 63), v);
    }
    for (int i = threadIdx.x >> 5; i < 32; i += R2H_THREADS / 32) {
        const unsigned v = __reduce_add_sync(0xffffffffu, shist[i * 32 + lane]);
        if (v && lane == 0) atomicAdd(gt + (640 + (i >> 1)) * 256 + (i & 1), v);
    }
}

// Encoder.  What a weight's three symbols are coded with depends on the data only, not on the coder state, and a segment's
// state is one chain.  So the CTA's first warp runs the chains of its 32 segments, a segment per lane, over table entries
// staged in shared memory, while four more warps stage the next 32 weights of every segment (from the segments' ends
// backwards; four lanes a segment, three dependent loads a weight): the loads' latency is hidden behind the chains.
// Bound by the chain of 96 steps per batch.
constexpr int EB = 32, ESEG = 32, EG = 4, EW = EB / EG;          // weights per batch, segments per CTA, staging lanes per segment
constexpr int E_THREADS = 32 + EG * ESEG, E_PITCH = EB * 3 + 1;  // padded: the chain lanes read the same weight of their rows together
constexpr int E_SMEM = 2 * ESEG * E_PITCH * (int)sizeof(RansStep);
__global__ void __launch_bounds__(E_THREADS) k_r2_enc(const unsigned char* __restrict__ dev, const TB* __restrict__ tb, const SG* __restrict__ sg,
                                                      int nseg, Ctx c, const RansSym* __restrict__ enc, unsigned char* __restrict__ out, size_t cap,
                                                      unsigned* __restrict__ out_len) {
    // per weight of a batch: sign, mantissa, exponent entries (coding order); two batches
    extern __shared__ __align__(16) RansStep s_e[];
    __shared__ int s_nmax;
    __shared__ unsigned s_bad[ESEG];
    const bool chain = threadIdx.x < 32;
    const int grp = chain ? threadIdx.x : (threadIdx.x - 32) / EG, gl = (threadIdx.x - 32) % EG;
    const int s = blockIdx.x * ESEG + grp;
    const bool live = s < nseg;
    SG g; g.t = 0; g.n = 0; g.i0 = 0;
    if (live) g = sg[s];
    const TB T = tb[g.t];
    if (threadIdx.x == 0) s_nmax = 0;
    if (chain) s_bad[grp] = 0;
    __syncthreads();
    if (chain) atomicMax(&s_nmax, g.n);
    __syncthreads();
    const int nb_max = (s_nmax + EB - 1) / EB;
    unsigned char* slot = out + (size_t)(live ? s : 0) * cap;
    ByteWriterDown wr; wr.init(slot + cap);
    unsigned x = RANS_L;
    bool full = false;
    const unsigned short* base = reinterpret_cast<const unsigned short*>(dev + T.doff);
    // batches of 32 weights, the last one first; a staging lane's first weight of the batch: compact row rc, column j
    int rc = 0, j = 0;
    if (!chain && live) {
        const long long i = g.i0 + (long long)(nb_max - 1) * EB + EW * gl;
        rc = (int)(i / T.rowlen); j = (int)(i % T.rowlen);
    }
    for (int it = 0; it <= nb_max; ++it) {
        if (!chain) {
            const int k0 = (nb_max - 1 - it) * EB;
            RansStep* row = s_e + ((it & 1) * ESEG + grp) * E_PITCH + 3 * EW * gl;
            if (live && k0 >= 0 && k0 < g.n) {
                // loads in three waves, each for all of the lane's weights (past the segment's end: its last weight again)
                int r[EW], col[EW], orow[EW];
                unsigned u[EW];
                int pred[EW], pe[EW], sc[EW];
                RansSym e[3 * EW];
#pragma unroll
                for (int v = 0; v < EW; ++v) {
                    r[v] = v ? r[v - 1] : rc; col[v] = v ? col[v - 1] : j;
                    if (v && k0 + EW * gl + v < g.n && ++col[v] == T.rowlen) { col[v] = 0; ++r[v]; }
                }
                if (k0 + EW * gl < g.n) {
#pragma unroll
                    for (int v = 0; v < EW; ++v) orow[v] = T.rmap >= 0 ? c.rowmap[T.rmap + r[v]] : r[v];
#pragma unroll
                    for (int v = 0; v < EW; ++v) {
                        u[v] = base[(size_t)orow[v] * T.rowlen + col[v]];
                        contexts(c, T, orow[v], col[v], pred[v], pe[v], sc[v]);
                    }
                    const RansSym* et = enc + (size_t)T.tab * 256;
#pragma unroll
                    for (int v = 0; v < EW; ++v) {
                        const int ex = (u[v] >> 7) & 255;
                        e[3 * v] = et[(640 + sc[v]) * 256 + (u[v] >> 15)];
                        e[3 * v + 1] = et[(512 + mctx(ex, pred[v])) * 256 + (u[v] & 127)];
                        e[3 * v + 2] = et[pe[v] * 256 + ex];
                    }
                    bool none = false;
#pragma unroll
                    for (int i = 0; i < 3 * EW; ++i) {
                        none |= (e[i].fc & 0xffffu) == 0;
                        row[i] = rans_step_of<PB>(e[i]);
                    }
                    if (none) s_bad[grp] = 1;
                }
            }
            j -= EB;
            if (live) while (j < 0) { j += T.rowlen; --rc; }
        } else if (it > 0 && live && !full) {
            const int n = min(EB, g.n - (nb_max - it) * EB);
            const RansStep* row = s_e + (((it - 1) & 1) * ESEG + grp) * E_PITCH;
            int w = n - 1;
            // four weights, twelve steps, at a time; they take 24 bytes at most
            for (; (w & 3) != 3; --w) {
                if (w < 0) break;
                rans_put(x, wr, row[3 * w]); rans_put(x, wr, row[3 * w + 1]); wr.drain();
                rans_put(x, wr, row[3 * w + 2]); wr.drain();
                if (wr.ptr() < slot + 64) { full = true; break; }
            }
            for (; w >= 3 && !full; w -= 4) {
                const RansStep* q = row + 3 * w;
#pragma unroll
                for (int v = 0; v < 4; v += 2, q -= 6) {
                    rans_put(x, wr, q[0]); rans_put(x, wr, q[1]); wr.drain();
                    rans_put(x, wr, q[2]); rans_put(x, wr, q[-3]); wr.drain();
                    rans_put(x, wr, q[-2]); rans_put(x, wr, q[-1]); wr.drain();
                }
                full = wr.ptr() < slot + 64;
            }
        }
        __syncthreads();
    }
    if (chain && live) {
        if (full) out_len[s] = LEN_OVERFLOW;
        else {
            rans_flush(x, wr);
            wr.flush();
            out_len[s] = s_bad[grp] ? LEN_NOFREQ : (unsigned)(slot + cap - wr.ptr());
        }
    }
}

// Decoder.  A segment is one rANS chain by format, but what a weight's symbols are decoded WITH - the exponent's and the
// sign's tables, the prediction the mantissa's table is picked by - depends on its row and column only.  A CTA (one per SM)
// takes up to 64 segments, as few as fill the SMs: eight warps run the chains, a segment per lane, over contexts that eight
// more warps (four lanes a segment) stage for the next 32 weights while they store the 32 weights before.  A chain warp and
// its staging warp wait for each other only; few lanes to a chain warp, since one lane's walk through a bucket or top-up
// of its ring holds up the others (four chain warps behind one barrier: 10.7 ms for 2 x 4096 x 12288 weights).
// The chain is three table searches per weight, and what they cost is the memory the tables are in: 656 tables do not fit
// the L1.  In shared memory are, of the role of the CTA's first segment, the 128 mantissa tables, 16 sign tables and the
// exponent tables of 128 contexts (16 octaves) around that segment's first weight, each as the cumulated frequencies plus
// the symbol that holds every 128th slot; anything else goes through the tables in global memory.
constexpr int DB = 32, DSEG = 64, DG = 4, DW = DB / DG;          // weights per batch, segments per CTA, staging lanes per segment and their weights
constexpr int D_CHAIN = 256, D_THREADS = D_CHAIN + DG * DSEG;
constexpr int D_ECTX = 128, D_MCTX = 128, D_MP = 256 + 260, D_EP = 256 + 516;       // bytes per table: 256 coarse, 130 / 258 cumulated
struct DecSmem {
    unsigned ring[RING_ROWS * DSEG];
    unsigned ctx[2][DSEG][DB + 1];                               // pe | sc << 9 | pred << 16; rows padded
    unsigned sign[16];                                           // frequency of symbol 0 | of symbol 1 << 16
    unsigned short out[2][DSEG][DB + 2];
    uint8_t mant[D_MCTX * D_MP], expo[D_ECTX * D_EP];
    int nmax, pe0, bad;
};
// stage a compact table; false: it has symbols from `nsym` on, or is not a whole distribution (an unused one)
SG_DEVINL void stage_table(const uint8_t* __restrict__ ct, uint8_t* dst, int nsym, int lane, int& bad) {
    const unsigned* __restrict__ words = reinterpret_cast<const unsigned*>(ct + 256);
    for (int i = lane; i < 64; i += 32) reinterpret_cast<unsigned*>(dst)[i] = reinterpret_cast<const unsigned*>(ct)[i];
    unsigned short* cum = reinterpret_cast<unsigned short*>(dst + 256);
    for (int i = lane; i < nsym; i += 32) cum[i] = (unsigned short)(words[i] >> 16);
    if (lane == 0) {
        const unsigned w = words[nsym - 1];
        const unsigned tot = (w >> 16) + (w & 0xffffu);
        cum[nsym] = (unsigned short)tot;
        cum[nsym + 1] = (unsigned short)tot;
        if (tot != (1u << PB)) bad = 1;
    }
}
typedef RingReader<DSEG> DecRing;
// The staged search stops at the second symbol of a bucket: a third one (rare symbols share a bucket) sets `miss`, and the
// weight is decoded again with a walk.  So the usual steps have no branch.
template <int NSYM> SG_DEVINL unsigned get_staged(unsigned& x, DecRing& r, const uint8_t* t, bool& miss) {
    const unsigned short* cum = reinterpret_cast<const unsigned short*>(t + 256);
    const unsigned slot = x & ((1u << PB) - 1), xs = x >> PB;
    unsigned s = t[slot >> (PB - 8)];
    if (NSYM < 256) s &= NSYM - 1;                               // (an unused table's place holds anything)
    const unsigned c0 = cum[s], c1 = cum[s + 1], c2 = cum[s + 2];
    const bool up = slot >= c1;
    miss |= slot >= c2;
    const unsigned lo = up ? c1 : c0, hi = up ? c2 : c1;
    x = (hi - lo) * xs + (slot - lo);
    r.renorm(x);
    return s + up;
}
template <int NSYM> SG_DEVINL unsigned get_walk(unsigned& x, DecRing& r, const uint8_t* t) {
    const unsigned short* cum = reinterpret_cast<const unsigned short*>(t + 256);
    const unsigned slot = x & ((1u << PB) - 1);
    unsigned s = t[slot >> (PB - 8)];
    if (NSYM < 256) s &= NSYM - 1;
#pragma unroll 1
    while (slot >= cum[s + 1] && s < NSYM - 1) ++s;
    const unsigned lo = cum[s];
    x = (cum[s + 1] - lo) * (x >> PB) + (slot - lo);
    r.renorm(x);
    return s;
}
SG_DEVINL unsigned get_global(unsigned& x, DecRing& r, const uint8_t* __restrict__ ct) {
    const unsigned* __restrict__ words = reinterpret_cast<const unsigned*>(ct + 256);
    const unsigned slot = x & ((1u << PB) - 1);
    unsigned s = ct[slot >> (PB - 8)];
    unsigned fc = words[s];
#pragma unroll 1
    while (slot >= (fc >> 16) + (fc & 0xffffu) && s < 255u) fc = words[++s];
    x = (fc & 0xffffu) * (x >> PB) + slot - (fc >> 16);
    r.renorm(x);
    return s;
}
__global__ void __launch_bounds__(D_THREADS, 1) k_r2_dec(const unsigned char* __restrict__ in, const unsigned long long* __restrict__ in_off,
                                                         const unsigned long long* __restrict__ in_end, unsigned char* __restrict__ dev,
                                                         const TB* __restrict__ tb, const SG* __restrict__ sg, int nseg, int per, Ctx c,
                                                         const unsigned char* __restrict__ lut, int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char dsm[];
    DecSmem& m = *reinterpret_cast<DecSmem*>(dsm);
    const bool chain = threadIdx.x < D_CHAIN;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int first = blockIdx.x * per;
    const int pair = warp & 7, grp = chain ? (lane < DSEG / 8 ? 8 * lane + pair : DSEG) : 8 * (lane / DG) + pair, gl = lane % DG;
    auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(pair + 1) : "memory"); };
    const int s = first + grp;
    const bool live = grp < per && s < nseg;
    SG g; g.t = 0; g.n = 0; g.i0 = 0;
    if (live) g = sg[s];
    const TB T = tb[g.t];
    const int cta_tab = tb[sg[first].t].tab;
    if (threadIdx.x == 0) {
        const SG f = sg[first];
        const TB F = tb[f.t];
        const int rc = (int)(f.i0 / F.rowlen), j = (int)(f.i0 % F.rowlen);
        int pred, pe, sc; contexts(c, F, F.rmap >= 0 ? c.rowmap[F.rmap + rc] : rc, j, pred, pe, sc);
        m.pe0 = min(max(pe - D_ECTX / 2, 0), 512 - D_ECTX);
        m.nmax = 0; m.bad = 0;
    }
    __syncthreads();
    const int pe0 = m.pe0;
    if (chain && live) atomicMax(&m.nmax, g.n);
    for (int t = warp; t < D_MCTX + D_ECTX; t += D_THREADS / 32) {
        if (t < D_MCTX) {
            const uint8_t* ct = lut + (size_t)(cta_tab + 512 + t) * RANS_COMPACT;
            int bad = 0;
            stage_table(ct, m.mant + t * D_MP, 128, lane, bad);
            // a used table whose distribution goes on past symbol 127 (no encoder writes one): this CTA stays with global memory
            const unsigned w = reinterpret_cast<const unsigned*>(ct + 256)[255];
            if (bad && (w >> 16) + (w & 0xffffu) == (1u << PB)) m.bad = 1;
        } else {
            int bad = 0;
            stage_table(lut + (size_t)(cta_tab + pe0 + t - D_MCTX) * RANS_COMPACT, m.expo + (t - D_MCTX) * D_EP, 256, lane, bad);
        }
    }
    if (threadIdx.x < 16) {
        const unsigned* w = reinterpret_cast<const unsigned*>(lut + (size_t)(cta_tab + 640 + threadIdx.x) * RANS_COMPACT + 256);
        m.sign[threadIdx.x] = (w[0] & 0xffffu) | (w[1] << 16);
    }
    __syncthreads();
    const bool staged = T.tab == cta_tab && !m.bad;
    const int nbatch = (m.nmax + DB - 1) / DB;
    DecRing rd; rd.pos = rd.have = 0; rd.left = 0;
    unsigned x = RANS_L;
    bool bad = false;
    if (chain && live) { rd.init(in + in_off[s], in + in_end[s], m.ring + grp); x = rd.state(); }
    unsigned short* base = reinterpret_cast<unsigned short*>(dev + T.doff);
    // a staging lane's first weight of the batch to stage and of the batch to store: compact row, column
    int rc = 0, j = 0, orc = 0, oj = 0;
    if (!chain && live) { const long long i = g.i0 + DW * gl; orc = rc = (int)(i / T.rowlen); oj = j = (int)(i % T.rowlen); }
    for (int it = 0; it < nbatch + 2; ++it) {
        if (!chain) {
            if (live && it >= 2) {                               // store the batch that was decoded in the last turn
                int r = orc, col = oj, have = -1, orow = 0;
#pragma unroll
                for (int v = 0; v < DW; ++v) {
                    if ((it - 2) * DB + DW * gl + v < g.n) {
                        if (r != have) { orow = T.rmap >= 0 ? c.rowmap[T.rmap + r] : r; have = r; }
                        base[(size_t)orow * T.rowlen + col] = m.out[it & 1][grp][DW * gl + v];
                        if (++col == T.rowlen) { col = 0; ++r; }
                    }
                }
                oj += DB;
                while (oj >= T.rowlen) { oj -= T.rowlen; ++orc; }
            }
            if (live && it < nbatch) {
                int r[DW], col[DW];                              // (past the segment's end: its last weight again)
#pragma unroll
                for (int v = 0; v < DW; ++v) {
                    r[v] = v ? r[v - 1] : rc; col[v] = v ? col[v - 1] : j;
                    if (v && it * DB + DW * gl + v < g.n && ++col[v] == T.rowlen) { col[v] = 0; ++r[v]; }
                }
                if (it * DB + DW * gl < g.n) {
                    unsigned e[DW];
#pragma unroll
                    for (int v = 0; v < DW; ++v) {
                        int pred, pe, sc; contexts(c, T, T.rmap >= 0 ? c.rowmap[T.rmap + r[v]] : r[v], col[v], pred, pe, sc);
                        // (mctx() is constant outside of +-4000)
                        e[v] = (unsigned)pe | (unsigned)sc << 9 | (unsigned)clampi(pred, -4000, 4000) << 16;
                    }
#pragma unroll
                    for (int v = 0; v < DW; ++v) m.ctx[it & 1][grp][DW * gl + v] = e[v];
                }
                j += DB;
                while (j >= T.rowlen) { j -= T.rowlen; ++rc; }
            }
        } else if (live && it >= 1 && !bad) {
            const int n = min(DB, g.n - (it - 1) * DB);
            const unsigned* cx = m.ctx[(it - 1) & 1][grp];
            unsigned short* o = m.out[(it - 1) & 1][grp];
#pragma unroll 1
            for (int w = 0; w < n; ++w) {
                if ((w & 3) == 0) rd.top_up();                   // four weights take 24 bytes at most
                const unsigned e = cx[w];
                const int pe = e & 511, sc = (e >> 9) & 15, pred = (int)e >> 16;
                const unsigned x0 = x, top0 = rd.top;
                const unsigned pos0 = rd.pos;
                const bool near = staged && (unsigned)(pe - pe0) < (unsigned)D_ECTX;
                const uint8_t* te = m.expo + (near ? pe - pe0 : 0) * D_EP;
                bool miss = !near;
                unsigned ex = get_staged<256>(x, rd, te, miss);
                unsigned man = get_staged<128>(x, rd, m.mant + mctx((int)ex, pred) * D_MP, miss);
                unsigned f01 = m.sign[sc];
                if (miss) {
                    x = x0; rd.top = top0; rd.pos = pos0;
                    if (near) {
                        ex = get_walk<256>(x, rd, te);
                        man = get_walk<128>(x, rd, m.mant + mctx((int)ex, pred) * D_MP);
                    } else {
                        const uint8_t* tl = lut + (size_t)T.tab * RANS_COMPACT;
                        ex = get_global(x, rd, tl + (size_t)pe * RANS_COMPACT);
                        man = get_global(x, rd, tl + (size_t)(512 + mctx((int)ex, pred)) * RANS_COMPACT);
                        const unsigned* sw = reinterpret_cast<const unsigned*>(tl + (size_t)(640 + sc) * RANS_COMPACT + 256);
                        f01 = (sw[0] & 0xffffu) | (sw[1] << 16);
                    }
                }
                const unsigned slot = x & ((1u << PB) - 1), f0 = f01 & 0xffffu;
                const bool neg = slot >= f0;                     // (two symbols: the second one starts where the first ends)
                x = (neg ? f01 >> 16 : f0) * (x >> PB) + (slot - (neg ? f0 : 0u));
                rd.renorm(x);
                o[w] = (unsigned short)(((unsigned)neg << 15) | (ex << 7) | man);
            }
            bad = rd.over();
        }
        pair_sync();
    }
    if (chain && live && (bad || rd.over() || x != RANS_L || !rd.at_end())) atomicOr(status, SG_ST_CORRUPT);
}

// duplicate rows copied from their source rows after decoding (bf16v2.py:475-480): pairs = (dup row, source row)
__global__ void __launch_bounds__(256) k_copy_rows(unsigned short* __restrict__ w, int rowlen, const long long* __restrict__ pairs, int npairs) {
    const int p = blockIdx.x;
    if (p >= npairs) return;
    unsigned short* d = w + (size_t)pairs[2 * p] * rowlen;
    const unsigned short* s = w + (size_t)pairs[2 * p + 1] * rowlen;
    for (int j = threadIdx.x; j < rowlen; j += blockDim.x) d[j] = s[j];
}

// ---- row recurrences: fingerprints and sums of squares --------------------------------------------------------------
// Both run along a row, one lane per row, and the row's length is the chain.  The rows' data comes in through shared memory
// in tiles of 32 rows x 64 weights, asked for three tiles ahead by three warps; the fourth runs the chains.  32 rows a CTA:
// a projection's 4096 rows reach 128 SMs.
constexpr int RC_ROWS = 32, RC_STAGES = 4, RC_PITCH = 9;          // 16-byte words per row and tile: 8, and one against bank conflicts
// 64-bit row fingerprints for duplicate-row detection (bf16v2.py:148-155)
struct RowHash {
    unsigned long long* h;
    unsigned long long a;
    SG_DEVINL void init() { a = 1469598103934665603ull; }
    SG_DEVINL void step(unsigned v) { a ^= v; a *= 1099511628211ull; a ^= a >> 29; }
    SG_DEVINL void done(int r, int) { h[r] = a; }
};
// rfi[r] = rint(8 log2 rms(row r)), and rfa[r] = (float) 2^(log2 rms) used to normalise the row in the column pass; the
// float64 sum of squares runs in column order
struct RowRms {
    short* rfi; float* rfa;
    double s;
    SG_DEVINL void init() { s = 0.0; }
    SG_DEVINL void step(unsigned u) { const double v = (double)__uint_as_float(u << 16); s = s + v * v; }
    SG_DEVINL void done(int r, int rowlen) {
        const double rf = dm::log2v(sqrt(s / (double)rowlen) + 1e-30);
        rfa[r] = (float)dm::exp2v(rf);
        rfi[r] = (short)fmin(fmax(rint(rf * 8.0), -32768.0), 32767.0);
    }
};
// WHOLE: every row begins on 16 bytes and is a multiple of them long.  Otherwise a row keeps the place within 16 bytes that it has
// in memory, so that all but its two ends are copied 16 bytes at a time too; the ends are loaded weight by weight (what lies
// beside them may not belong to the buffer).  4096 x 12287 weights: 0.23 ms the hashes, 0.74 when every weight of such rows was a
// load of its own that the next tile waited for.
template <bool WHOLE, class Op>
__global__ void __launch_bounds__(128) k_row_chain(const unsigned short* __restrict__ w, int nrows, int rowlen, Op op) {
    __shared__ __align__(16) uint4 tile[RC_STAGES][RC_ROWS][RC_PITCH];
    const int r0 = blockIdx.x * RC_ROWS, lane = threadIdx.x & 31, ntile = (int)(((long long)rowlen + (WHOLE ? 0 : 7) + 63) / 64);
    auto row_of = [&](int r) { return w + (size_t)(r0 + r) * rowlen; };
    auto shift_of = [&](const unsigned short* row) { return WHOLE ? 0 : (int)(reinterpret_cast<uintptr_t>(row) >> 1 & 7); };
    // a row's ends: the second and third warp load the chunk of 8 weights at the beginning / end of row `lane`, if it is not whole
    const int sh = shift_of(row_of(lane)), stop = sh + rowlen, end_chunk = threadIdx.x < 64 ? 0 : stop >> 3;
    const bool end = r0 + lane < nrows && (threadIdx.x < 64 ? threadIdx.x >= 32 && (sh > 0 || stop < 8) : threadIdx.x < 96 && stop >= 8 && (stop & 7));
    const int end_tile = end ? end_chunk >> 3 : -1;
    auto ask = [&](int t) {
        if (threadIdx.x >= 32 && t < ntile)
            for (int i = threadIdx.x - 32; i < RC_ROWS * 8; i += 96) {
                const int r = i >> 3;
                if (r0 + r >= nrows) break;
                const unsigned short* row = row_of(r);
                const int col = t * 64 + (i & 7) * 8 - shift_of(row);
                if (col >= rowlen) continue;
                if (WHOLE || (col >= 0 && col + 8 <= rowlen))
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(&tile[t % RC_STAGES][r][i & 7])),
                                 "l"(row + col) : "memory");
            }
        if (!WHOLE && t == end_tile) {
            unsigned short* to = reinterpret_cast<unsigned short*>(&tile[t % RC_STAGES][lane][end_chunk & 7]);
            const int col = end_chunk * 8 - sh;
#pragma unroll
            for (int k = 0; k < 8; ++k) if (col + k >= 0 && col + k < rowlen) to[k] = row_of(lane)[col + k];
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    op.init();
    for (int t = 0; t < RC_STAGES - 1; ++t) ask(t);
    for (int t = 0; t < ntile; ++t) {
        asm volatile("cp.async.wait_group %0;" ::"n"(RC_STAGES - 2) : "memory");
        __syncthreads();
        ask(t + RC_STAGES - 1);
        if (threadIdx.x < 32 && r0 + lane < nrows) {
            const uint4* p = tile[t % RC_STAGES][lane];
            const int a = t == 0 ? sh : 0, z = min(64, rowlen + sh - t * 64);
            if (a == 0 && z == 64) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint4 q = p[i];
                    const unsigned v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                    for (int k = 0; k < 4; ++k) { op.step(v[k] & 0xffffu); op.step(v[k] >> 16); }
                }
            } else {
#pragma unroll 1
                for (int i = a >> 3; 8 * i < z; ++i) {
                    const uint4 q = p[i];
                    const unsigned v[4] = {q.x, q.y, q.z, q.w};
                    if (8 * i >= a && 8 * i + 8 <= z) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) { op.step(v[k] & 0xffffu); op.step(v[k] >> 16); }
                    } else {
#pragma unroll
                        for (int k = 0; k < 8; ++k) if (8 * i + k >= a && 8 * i + k < z) op.step(k & 1 ? v[k >> 1] >> 16 : v[k >> 1] & 0xffffu);
                    }
                }
            }
        }
    }
    if (threadIdx.x < 32 && r0 + lane < nrows) op.done(r0 + lane, rowlen);
}
template <class Op> static int row_chain(const void* w, int nrows, int rowlen, Op op, cudaStream_t st) {
    const unsigned grid = (unsigned)((nrows + RC_ROWS - 1) / RC_ROWS);
    const unsigned short* p = (const unsigned short*)w;
    if (rowlen % 8 == 0 && (uintptr_t)w % 16 == 0) k_row_chain<true><<<grid, 128, 0, st>>>(p, nrows, rowlen, op);
    else k_row_chain<false><<<grid, 128, 0, st>>>(p, nrows, rowlen, op);
    return cuda_ok(cudaGetLastError());
}

// ---- statistics ----------------------------------------------------------------------------------------------------
// per (row chunk, column): float64 sums of v^2 and v over the chunk's rows in row order, v = weight / rfa[row] in float32.
// The sums are one dependent chain per column by format; what does not depend on the chain (load, the IEEE division,
// the conversion) is done by all 256 threads of a CTA for a tile of 64 rows x 32 columns into shared memory, and the
// first warp then extends its 32 columns' chains over the tile while the other warps fetch the next one.
__global__ void __launch_bounds__(256) k_r2_colpart(const unsigned short* __restrict__ w, int nrows, int rowlen, int step,
                                                    const float* __restrict__ rfa, double* __restrict__ part) {
    constexpr int TR = 64, TC = 32;
    __shared__ float tile[2][TR][TC + 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = blockIdx.x * TC + lane;
    const int q = blockIdx.y;
    const int r0 = q * step, r1 = min(nrows, r0 + step);
    const bool live = c < rowlen;
    double s2 = 0.0, s1 = 0.0;
    int buf = 0;
    for (int t0 = r0; t0 < r1; t0 += TR, buf ^= 1) {
#pragma unroll
        for (int j = 0; j < TR / 8; ++j) {
            const int r = t0 + warp + 8 * j;
            float f = 0.0f;
            if (live && r < r1) f = __fdiv_rn(__uint_as_float((unsigned)w[(size_t)r * rowlen + c] << 16), rfa[r]);
            tile[buf][warp + 8 * j][lane] = f;
        }
        __syncthreads();
        if (warp == 0) {
            const int n = min(TR, r1 - t0);
            for (int i = 0; i < n; ++i) {
                const double v = (double)tile[buf][i][lane];
                s2 = s2 + v * v;
                s1 = s1 + v;
            }
        }
    }
    if (warp == 0 && live) {
        part[((size_t)q * rowlen + c) * 2] = s2;
        part[((size_t)q * rowlen + c) * 2 + 1] = s1;
    }
}
__global__ void __launch_bounds__(256) k_r2_colfinal(const double* __restrict__ part, int nchunks, int nrows, int rowlen,
                                                     short* __restrict__ cfi, signed char* __restrict__ scl) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= rowlen) return;
    double s2 = 0.0, s1 = 0.0;
    for (int q = 0; q < nchunks; ++q) { s2 = s2 + part[((size_t)q * rowlen + c) * 2]; s1 = s1 + part[((size_t)q * rowlen + c) * 2 + 1]; }
    const double cf = dm::log2v(sqrt(s2 / (double)nrows) + 1e-30);
    const double ci = fmin(fmax(rint(cf * 8.0), -32768.0), 32767.0);
    cfi[c] = (short)ci;
    const double bias = (s1 / (double)nrows) / dm::exp2v((double)(short)ci / 8.0);
    scl[c] = (signed char)fmin(fmax(floor(bias * 16.0) + 8.0, 0.0), 15.0);
}

// ---- generic detmath entry points (seedpack/detmath.py:67-106) --------------------------------------------------------
__global__ void k_dm_log2(const double* x, long long n, double* y) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = dm::log2v(x[i]);
}
__global__ void k_dm_exp2(const double* x, long long n, double* y) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = dm::exp2v(x[i]);
}
__global__ void k_dm_rows(const float* x, long long nr, long long nc, int sq, double* out) {
    const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nr) return;
    const float* p = x + r * nc;
    double s = 0.0;
    if (sq) for (long long j = 0; j < nc; ++j) { const double v = p[j]; s = s + v * v; }
    else for (long long j = 0; j < nc; ++j) s = s + (double)p[j];
    out[r] = s;
}
__global__ void k_dm_cols(const float* x, long long nr, long long nc, int sq, const unsigned char* mask, double* out) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nc) return;
    double s = 0.0;
    for (long long r = 0; r < nr; ++r) {
        if (mask && !mask[r]) continue;
        const double v = x[r * nc + c];
        s = s + (sq ? v * v : v);
    }
    out[c] = s;
}

}  // namespace r2
}  // namespace sg

using namespace sg;
using namespace sg::r2;

static int r2_common(const void* dev, const void* tb, const void* sgp, int nseg, const void* rfi, const void* cfi, const void* scl) {
    if (!dev || !tb || !sgp || !rfi || !cfi || !scl || nseg < 0) return SG_ERR_ARG;
    return SG_OK;
}

extern "C" int sg_r2_hist(int device, void* stream, const unsigned char* dev, const void* tb, const void* sgp, int nseg, const short* rfi,
                          const short* cfi, const signed char* scl, const int* rowmap, unsigned* counts) {
    int rc = r2_common(dev, tb, sgp, nseg, rfi, cfi, scl);
    if (rc != SG_OK || !counts) return rc != SG_OK ? rc : SG_ERR_ARG;
    if (nseg == 0) return SG_OK;
    rc = use_device(device);
    if (rc != SG_OK) return rc;
    Ctx c = {rfi, cfi, scl, rowmap};
    rc = cuda_ok(cudaFuncSetAttribute(k_r2_hist, cudaFuncAttributeMaxDynamicSharedMemorySize, R2H_SMEM));
    if (rc != SG_OK) return rc;
    // clearing and adding up a CTA's counters costs about as much as a segment: at most 64 segments share it
    const int want = (nseg + 2 * 148 - 1) / (2 * 148), per = want > 64 ? 64 : want;
    k_r2_hist<<<(nseg + per - 1) / per, R2H_THREADS, R2H_SMEM, (cudaStream_t)stream>>>(dev, (const TB*)tb, (const SG*)sgp, nseg, per, c, counts);
    return cuda_ok(cudaGetLastError());
}

extern "C" int sg_r2_encode(int device, void* stream, const unsigned char* dev, const void* tb, const void* sgp, int nseg, const short* rfi,
                            const short* cfi, const signed char* scl, const int* rowmap, const void* enc_tab, unsigned char* slots,
                            size_t cap, unsigned* out_len) {
    int rc = r2_common(dev, tb, sgp, nseg, rfi, cfi, scl);
    if (rc != SG_OK) return rc;
    if (!enc_tab || !slots || !out_len) return SG_ERR_ARG;
    if (cap < 128 || cap % 16 || (uintptr_t)slots % 16) return SG_ERR_ALIGN;
    if (nseg == 0) return SG_OK;
    rc = use_device(device);
    if (rc != SG_OK) return rc;
    Ctx c = {rfi, cfi, scl, rowmap};
    rc = cuda_ok(cudaFuncSetAttribute(k_r2_enc, cudaFuncAttributeMaxDynamicSharedMemorySize, E_SMEM));
    if (rc != SG_OK) return rc;
    k_r2_enc<<<(nseg + ESEG - 1) / ESEG, E_THREADS, E_SMEM, (cudaStream_t)stream>>>(dev, (const TB*)tb, (const SG*)sgp, nseg, c, (const RansSym*)enc_tab,
                                                                       slots, cap, out_len);
    return cuda_ok(cudaGetLastError());
}

extern "C" int sg_r2_decode(int device, void* stream, const unsigned char* in, const unsigned long long* in_off,
                            const unsigned long long* in_end, unsigned char* dev, const void* tb, const void* sgp, int nseg, const short* rfi,
                            const short* cfi, const signed char* scl, const int* rowmap, const void* enc_tab, const unsigned char* lut) {
    int rc = r2_common(dev, tb, sgp, nseg, rfi, cfi, scl);
    if (rc != SG_OK) return rc;
    if (!in || !in_off || !in_end || !enc_tab || !lut) return SG_ERR_ARG;
    if ((uintptr_t)in % 16 || (uintptr_t)lut % 8) return SG_ERR_ALIGN;           // (the sign tables' two words are one 8-byte load)
    if (nseg == 0) return SG_OK;
    rc = use_device(device);
    if (rc != SG_OK) return rc;
    Ctx c = {rfi, cfi, scl, rowmap};
    rc = cuda_ok(cudaFuncSetAttribute(k_r2_dec, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DecSmem)));
    if (rc != SG_OK) return rc;
    const int want = (nseg + 147) / 148, per = want > DSEG ? DSEG : want;
    k_r2_dec<<<(nseg + per - 1) / per, D_THREADS, sizeof(DecSmem), (cudaStream_t)stream>>>(in, in_off, in_end, dev, (const TB*)tb, (const SG*)sgp,
                                                                                           nseg, per, c, lut, status_word(device));
    return cuda_ok(cudaGetLastError());
}

extern "C" int sg_row_hash(int device, void* stream, const void* w, int nrows, int rowlen, unsigned long long* h) {
    if (!w || !h || nrows < 0 || rowlen <= 0) return SG_ERR_ARG;
    if (nrows == 0) return SG_OK;
    int rc = use_device(device);
    if (rc != SG_OK) return rc;
    return row_chain(w, nrows, rowlen, RowHash{h, 0}, (cudaStream_t)stream);
}

extern "C" int sg_copy_rows(int device, void* stream, void* w, int rowlen, const long long* pairs, int npairs) {
    if (!w || !pairs || npairs < 0 || rowlen <= 0) return SG_ERR_ARG;
    if (npairs == 0) return SG_OK;
    int rc = use_device(device);
    if (rc != SG_OK) return rc;
    k_copy_rows<<<npairs, 256, 0, (cudaStream_t)stream>>>((unsigned short*)w, rowlen, pairs, npairs);
    return cuda_ok(cudaGetLastError());
}

static int r2_step(int rowlen) { const int s = (16 << 20) / rowlen; return s < 1 ? 1 : s; }

extern "C" size_t sg_r2_stats_scratch_bytes(int nrows, int rowlen) {
    if (nrows <= 0 || rowlen <= 0) return 0;
    const int step = r2_step(rowlen), nchunks = (nrows + step - 1) / step;
    return ((size_t)nrows * 4 + 255) / 256 * 256 + (size_t)nchunks * rowlen * 16;
}

extern "C" int sg_r2_stats(int device, void* stream, const void* w, int nrows, int rowlen, short* rfi, short* cfi, signed char* scl,
                           void* scratch, size_t scratch_bytes) {
    if (!w || !rfi || !cfi || !scl || nrows <= 0 || rowlen <= 0) return SG_ERR_ARG;
    if (!scratch || scratch_bytes < sg_r2_stats_scratch_bytes(nrows, rowlen) || (uintptr_t)scratch % 16) return SG_ERR_SCRATCH;
    int rc = use_device(device);
    if (rc != SG_OK) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    const int step = r2_step(rowlen), nchunks = (nrows + step - 1) / step;
    if (nchunks > 65535) return SG_ERR_LIMIT;
    float* rfa = (float*)scratch;
    double* part = (double*)((unsigned char*)scratch + ((size_t)nrows * 4 + 255) / 256 * 256);
    rc = row_chain(w, nrows, rowlen, RowRms{rfi, rfa, 0.0}, st);
    if (rc != SG_OK) return rc;
    k_r2_colpart<<<dim3((rowlen + 31) / 32, nchunks), 256, 0, st>>>((const unsigned short*)w, nrows, rowlen, step, rfa, part);
    k_r2_colfinal<<<(rowlen + 255) / 256, 256, 0, st>>>(part, nchunks, nrows, rowlen, cfi, scl);
    return cuda_ok(cudaGetLastError());
}

extern "C" int sg_dm_log2(int device, void* stream, const double* x, long long n, double* y) {
    if (n < 0 || (n && (!x || !y))) return SG_ERR_ARG;
    if (n == 0) return SG_OK;
    int rc = use_device(device);
    if (rc != SG_OK) return rc;
    k_dm_log2<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(x, n, y);
    return cuda_ok(cudaGetLastError());
}
extern "C" int sg_dm_exp2(int device, void* stream, const double* x, long long n, double* y) {
    if (n < 0 || (n && (!x || !y))) return SG_ERR_ARG;
    if (n == 0) return SG_OK;
    int rc = use_device(device);
    if (rc != SG_OK) return rc;
    k_dm_exp2<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(x, n, y);
    return cuda_ok(cudaGetLastError());
}
extern "C" int sg_dm_rows(int device, void* stream, const float* x, long long nr, long long nc, int square, double* out) {
    if (nr < 0 || nc < 0 || (nr && (!x || !out))) return SG_ERR_ARG;
    if (nr == 0) return SG_OK;
    int rc = use_device(device);
    if (rc != SG_OK) return rc;
    k_dm_rows<<<(unsigned)((nr + 255) / 256), 256, 0, (cudaStream_t)stream>>>(x, nr, nc, square, out);
    return cuda_ok(cudaGetLastError());
}
extern "C" int sg_dm_cols(int device, void* stream, const float* x, long long nr, long long nc, int square, const unsigned char* mask,
                          double* out) {
    if (nr < 0 || nc < 0 || (nc && (!x || !out))) return SG_ERR_ARG;
    if (nc == 0) return SG_OK;
    int rc = use_device(device);
    if (rc != SG_OK) return rc;
    k_dm_cols<<<(unsigned)((nc + 255) / 256), 256, 0, (cudaStream_t)stream>>>(x, nr, nc, square, mask, out);
    return cuda_ok(cudaGetLastError());
}
