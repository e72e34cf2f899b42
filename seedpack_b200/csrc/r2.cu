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

SG_DEVINL void contexts(const Ctx& c, const TB& T, int orow, int j, int& pred, int& pe, int& sc) {
    pred = c.rfi[T.rowbase + orow] + c.cfi[T.colbase + j];
    pe = clampi(pred + 256, 0, 511);
    sc = clampi(c.scl[T.colbase + j], 0, 15);         // (0..15 by construction, bf16v2.py:243; a damaged side part must not index past the tables)
}
SG_DEVINL int mctx(int ex, int pred) { return clampi(8 * ex - pred - 1016 + 64, 0, 127); }

// The exponent context whose neighbourhood of 64 to either side holds the most of the first weights of the segments first .. first
// + n - 1 (those of the role `tab`; n <= WIN_MAX): one of them alone may lie in a row of zeros.  By the whole CTA.
constexpr int WIN_MAX = 96;
struct WinSmem { int pe[WIN_MAX], best; };
SG_DEVINL int window_of(WinSmem& m, const Ctx& c, const TB* __restrict__ tb, const SG* __restrict__ sg, int first, int n, int tab) {
    const int t = threadIdx.x;
    __syncthreads();
    if (t == 0) m.best = 0;
    if (t < n) {
        const SG g = sg[first + t];
        const TB T = tb[g.t];
        int pred, pe = -1024, sc;
        if (T.tab == tab && g.n > 0) {
            const int rc = (int)(g.i0 / T.rowlen), j = (int)(g.i0 % T.rowlen);
            contexts(c, T, T.rmap >= 0 ? c.rowmap[T.rmap + rc] : rc, j, pred, pe, sc);
        }
        m.pe[t] = pe;
    }
    __syncthreads();
    if (t < n && m.pe[t] >= 0) {
        int k = 0;
        for (int j = 0; j < n; ++j) k += (unsigned)(m.pe[j] - m.pe[t] + 64) < 128u;
        atomicMax(&m.best, k << 9 | m.pe[t]);
    }
    __syncthreads();
    return m.best & 511;
}
// the lowest of 64 exponents to keep at hand around such a context: weights mostly lie below the typical magnitude
SG_DEVINL int window_exponent(int pe) { return ((pe - 256 + 1016) >> 3) - 44; }
// add to global memory, once for the lanes that come with the same counter (rows of zeros do)
SG_DEVINL void hadd(unsigned* counts, unsigned key) {
    const unsigned m = __match_any_sync(__activemask(), key);
    if ((threadIdx.x & 31) == (unsigned)(__ffs(m) - 1)) atomicAdd(counts + key, (unsigned)__popc(m));
}

// Counts do not depend on the order of the weights.  A CTA takes `per` segments, as few as give two CTAs per SM their share,
// and its 16 warps walk through a segment together (coalesced reads, four weights per lane in flight).  Bound by the shared
// memory's atomics, three per weight.  Mantissa symbols are spread over 128 x 128 counters per role, which a CTA collects in
// shared memory (64 KB) and adds to global memory when the role changes and at its end (about the time of a segment); so are
// the exponent symbols inside a window of 128 contexts x 64 exponents (weights of one tensor keep to a few octaves; what falls
// outside the window goes to global memory directly).  Of the sign's 32 counters every lane has its own
// copy: they would collide on every step.
constexpr int R2H_THREADS = 512, R2H_U = 4, R2H_OWN = 4096;
constexpr int R2H_SMEM = (128 * 128 + 128 * 64 + 32 * 32) * 4;
__global__ void __launch_bounds__(R2H_THREADS, 2) k_r2_hist(const unsigned char* __restrict__ dev, const TB* __restrict__ tb,
                                                            const SG* __restrict__ sg, int nseg, int per, Ctx c, unsigned* __restrict__ counts) {
    extern __shared__ unsigned mhist[];            // [128 contexts][128 symbols] of the role `tab`
    __shared__ WinSmem win;
    unsigned* ehist = mhist + 128 * 128;           // [128 contexts from pe0][64 exponents from ex0] of the same role
    unsigned* shist = ehist + 128 * 64;            // [16 classes x sign][lane] of the same role
    for (int i = threadIdx.x; i < R2H_SMEM / 4; i += R2H_THREADS) mhist[i] = 0;
    const int lane = threadIdx.x & 31, first = blockIdx.x * per;
    int tab = -1, pe0 = 0, ex0 = 0;
    auto add_up = [&]() {                          // what was collected to global memory, the counters back to zero
        __syncthreads();
        unsigned* gt = counts + (size_t)tab * 256;
        for (int i = threadIdx.x; i < 128 * 128; i += R2H_THREADS) {
            const unsigned v = mhist[i];
            if (v) { atomicAdd(gt + (512 + (i >> 7)) * 256 + (i & 127), v); mhist[i] = 0; }
        }
        for (int i = threadIdx.x; i < 128 * 64; i += R2H_THREADS) {
            const unsigned v = ehist[i];
            if (v) { atomicAdd(gt + (pe0 + (i >> 6)) * 256 + ex0 + (i & 63), v); ehist[i] = 0; }
        }
        for (int i = threadIdx.x >> 5; i < 32; i += R2H_THREADS / 32) {
            const unsigned v = __reduce_add_sync(0xffffffffu, shist[i * 32 + lane]);
            if (v && lane == 0) atomicAdd(gt + (640 + (i >> 1)) * 256 + (i & 1), v);
            shist[i * 32 + lane] = 0;
        }
    };
    for (int s = first; s < min(nseg, first + per); ++s) {
        const SG g = sg[s];
        const TB T = tb[g.t];
        // another role: its own counters, unless the segment is too small to be worth clearing them
        if (T.tab != tab && (tab < 0 || g.n >= R2H_OWN)) {
            if (tab >= 0) add_up();
            tab = T.tab;
            const int pe = window_of(win, c, tb, sg, s, min(WIN_MAX, min(nseg, first + per) - s), tab);
            pe0 = pe - 64; ex0 = window_exponent(pe);
        }
        const bool local = T.tab == tab;
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
                else hadd(gt, pe[v] * 256 + ex);
                if (local) {
                    atomicAdd(mhist + mc * 128 + man, 1u);
                    atomicAdd(shist + (sc[v] * 2 + sgn) * 32 + lane, 1u);
                } else {
                    hadd(gt, (512 + mc) * 256 + man);
                    hadd(gt, (640 + sc[v]) * 256 + sgn);
                }
            }
        }
    }
    add_up();
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
// takes a piece of up to 96 segments of one role: up to twelve warps run the chains, a segment per lane, over contexts that as
// many warps (four lanes a segment) stage for the next 32 weights while they store the 32 weights before.  A chain warp and
// its staging warp wait for each other only; few lanes to a chain warp, since one lane's walk through a bucket or top-up
// of its ring holds up the others (four chain warps behind one barrier: 10.7 ms for 2 x 4096 x 12288 weights).
// The chain is three table searches per weight, and what they cost is the memory the tables are in: 656 tables do not fit
// the L1.  In shared memory are, of the piece's role, the 128 mantissa tables, 16 sign tables and, of the exponent tables of
// 128 contexts (16 octaves) around the piece's first weight, 64 exponents each, as the cumulated frequencies plus the symbol
// that holds every 128th slot; anything else goes through the tables in global memory.
// Pieces: the segments come in runs of one role, cut evenly.  A CTA of two roles, one of them without tables, took three times
// as long (28 layers of seven projections, layer by layer: 36.6 ms; 22.5 with no tables in shared memory at all).  Runs that are
// too short for that are decoded by k_r2_dec_any from global memory, four lanes a segment: see dec_plan().
constexpr int DB = 32, DG = 4, DW = DB / DG;                     // weights per batch, lanes per segment in the staging warps and their weights
constexpr int D_PAIRS = 12, DSEG = 8 * D_PAIRS, D_THREADS = 2 * 32 * D_PAIRS, D_RING = 128;
constexpr int D_ECTX = 128, D_ESYM = 64, D_MCTX = 128, D_MP = 256 + 260, D_EP = 256 + 132;     // bytes per table: 256 coarse, 130 / 66 cumulated
constexpr int GSEG = D_THREADS / DG, G_RING = 256;               // segments of a CTA that decodes from global memory
constexpr int D_RUNS = 1024;
struct PlanSmem {
    int runs[D_RUNS + 1], warp_sum[D_THREADS / 32], pieces[4], first, count;
    int v_pe[D_THREADS], v_tab[D_THREADS], v_best[64];
};
struct DecSmem {
    PlanSmem plan;
    WinSmem win;
    int nmax, bad;
    unsigned ring[RING_ROWS * D_RING];
    unsigned ctx[2][DSEG][DB + 1];                               // pe | sc << 9 | pred << 16; rows padded
    unsigned sign[16];                                           // frequency of symbol 0 | of symbol 1 << 16
    unsigned short out[2][DSEG][DB + 2];
    uint8_t mant[D_MCTX * D_MP], expo[D_ECTX * D_EP];
};
struct AnySmem {
    PlanSmem plan;
    unsigned ring[RING_ROWS * G_RING];
    unsigned ctx[GSEG][DB + 1];
    unsigned short out[GSEG][DB + 2];
};
static_assert(sizeof(DecSmem) <= 227 * 1024, "one CTA per SM");
typedef RingReader<D_RING> DecRing;
// (mctx() is constant outside of +-4000)
SG_DEVINL unsigned pack_ctx(int pred, int pe, int sc) { return (unsigned)pe | (unsigned)sc << 9 | (unsigned)clampi(pred, -4000, 4000) << 16; }

// How the segments are cut, the same in every CTA: the pieces' number and size; a negative size: pieces of any roles.  A wave of
// pieces takes 4.9 ms with 21 segments each and 6.4 ms with 83, so what counts is the number of waves: a larger piece is
// taken where that saves one.  Segments of any roles, from global memory: 14.3 ms for 6000 in runs of ten, 17.7 for 26000, the
// same again for every further 28416 (192 an SM).  They are decoded that way too if the rows' magnitudes are spread over more
// contexts than a piece has room for (rows over 40 octaves: 8.1 ms for 6144 segments, 13.6 in pieces).
SG_DEVINL int dec_plan(PlanSmem& m, const Ctx& c, const TB* __restrict__ tb, const SG* __restrict__ sg, int nseg, int& per) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int chunk = (nseg + D_THREADS - 1) / D_THREADS;
    const int i0 = (int)min((long long)threadIdx.x * chunk, (long long)nseg), i1 = (int)min((long long)i0 + chunk, (long long)nseg);
    auto starts = [&](auto&& f) {
        int prev = i0 > 0 && i0 < i1 ? sg[i0 - 1].t : -1;
#pragma unroll 4
        for (int i = i0; i < i1; ++i) {
            const int t = sg[i].t;
            if (prev < 0 || (t != prev && tb[t].tab != tb[prev].tab)) f(i);
            prev = t;
        }
    };
    int n = 0;
    starts([&](int) { ++n; });
    int incl = n;
    for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
    if (lane == 31) m.warp_sum[warp] = incl;
    if (threadIdx.x < 4) m.pieces[threadIdx.x] = 0;
    __syncthreads();
    int at = incl - n, nruns = 0;
    for (int w = 0; w < D_THREADS / 32; ++w) { if (w < warp) at += m.warp_sum[w]; nruns += m.warp_sum[w]; }
    const int gwaves = (nseg + 148 * GSEG - 1) / (148 * GSEG), gper = min(GSEG, ((nseg + 148 * gwaves - 1) / (148 * gwaves) + 7) / 8 * 8);
    const int gpieces = (nseg + gper - 1) / gper;
    per = -gper;
    if (nruns > D_RUNS) return gpieces;
    starts([&](int i) { m.runs[at++] = i; });
    if (threadIdx.x == 0) m.runs[nruns] = nseg;
    __syncthreads();
    const int waves0 = (nseg + 148 * DSEG - 1) / (148 * DSEG), even = (nseg + 148 * waves0 - 1) / (148 * waves0);
    const int size[4] = {even, min(DSEG, even * 5 / 4), min(DSEG, even * 3 / 2), min(DSEG, even * 2)};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        int p = 0;
        for (int r = threadIdx.x; r < nruns; r += D_THREADS) p += (m.runs[r + 1] - m.runs[r] + size[k] - 1) / size[k];
        if (p) atomicAdd(&m.pieces[k], p);
    }
    __syncthreads();
    int waves = 0x7fffffff, total = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int w = (m.pieces[k] + 147) / 148;
        if (w < waves) { waves = w; per = size[k]; total = m.pieces[k]; }
    }
    __syncthreads();
    // and how many weights' contexts a piece's window would hold: twelve segments of each of 64 stretches as long as a piece
    const int q = threadIdx.x / 12, i = min((int)((long long)q * nseg / 64) + (int)(threadIdx.x % 12) * per / 12, nseg - 1);
    {
        const SG g = sg[i];
        const TB T = tb[g.t];
        int pred, pe = -1024, sc;
        if (g.n > 0) {
            const int rc = (int)(g.i0 / T.rowlen), j = (int)(g.i0 % T.rowlen);
            contexts(c, T, T.rmap >= 0 ? c.rowmap[T.rmap + rc] : rc, j, pred, pe, sc);
        }
        m.v_pe[threadIdx.x] = pe; m.v_tab[threadIdx.x] = T.tab;
        if (threadIdx.x < 64) m.v_best[threadIdx.x] = 0;
        if (threadIdx.x < 2) m.pieces[threadIdx.x] = 0;
    }
    __syncthreads();
    {
        int held = 0, same = 0;
        for (int k = 12 * q; k < 12 * q + 12; ++k) {
            const bool of_role = m.v_tab[k] == m.v_tab[threadIdx.x];
            same += of_role;
            held += of_role && (unsigned)(m.v_pe[k] - m.v_pe[threadIdx.x] + 64) < 128u;
        }
        atomicMax(&m.v_best[q], held << 8 | same);
    }
    __syncthreads();
    if (threadIdx.x < 64) { atomicAdd(&m.pieces[0], m.v_best[threadIdx.x] >> 8); atomicAdd(&m.pieces[1], m.v_best[threadIdx.x] & 255); }
    __syncthreads();
    // (a lane outside the window holds up its warp: with 16 of 17 inside 9.9 ms, from global memory 8.1)
    if (64LL * waves > 133LL * gwaves + nseg / 600 || 20 * m.pieces[0] < 19 * m.pieces[1]) { per = -gper; total = gpieces; }
    __syncthreads();
    return total;
}

// stage the cumulated frequencies and coarse entries of NSYM symbols of a compact table from s0 on; a coarse entry outside of them
// becomes the nearest of them
template <int NSYM> SG_DEVINL void stage_table(const uint8_t* __restrict__ ct, uint8_t* dst, int s0, int lane) {
    const unsigned* __restrict__ words = reinterpret_cast<const unsigned*>(ct + 256);
    for (int i = lane; i < 64; i += 32) {
        const unsigned v = reinterpret_cast<const unsigned*>(ct)[i];
        unsigned o = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) o |= (unsigned)clampi((int)((v >> (8 * k)) & 255u) - s0, 0, NSYM - 1) << (8 * k);
        reinterpret_cast<unsigned*>(dst)[i] = o;
    }
    unsigned short* cum = reinterpret_cast<unsigned short*>(dst + 256);
    for (int i = lane; i < NSYM + 2; i += 32) {
        const unsigned w = words[min(s0 + i, 255)];
        cum[i] = (unsigned short)((w >> 16) + (s0 + i > 255 ? w & 0xffffu : 0u));
    }
}
// The staged search stops at the second symbol of a bucket: a third one (rare symbols share a bucket) sets `miss`, and the
// weight is decoded again with a walk.  So the usual steps have no branch.  BELOW: there may be symbols before the staged ones.
template <bool BELOW> SG_DEVINL unsigned get_staged(unsigned& x, DecRing& r, const uint8_t* t, bool& miss) {
    const unsigned short* cum = reinterpret_cast<const unsigned short*>(t + 256);
    const unsigned slot = x & ((1u << PB) - 1), xs = x >> PB;
    const unsigned s = t[slot >> (PB - 8)];
    const unsigned c0 = cum[s], c1 = cum[s + 1], c2 = cum[s + 2];
    const bool up = slot >= c1;
    miss |= slot >= c2 || (BELOW && slot < c0);
    const unsigned lo = up ? c1 : c0, hi = up ? c2 : c1;
    x = (hi - lo) * xs + (slot - lo);
    r.renorm(x);
    return s + up;
}
// false: the symbol is not among the staged ones
template <int NSYM> SG_DEVINL bool get_walk(unsigned& x, DecRing& r, const uint8_t* t, unsigned& sym) {
    const unsigned short* cum = reinterpret_cast<const unsigned short*>(t + 256);
    const unsigned slot = x & ((1u << PB) - 1);
    unsigned s = t[slot >> (PB - 8)];
#pragma unroll 1
    while (slot >= cum[s + 1] && s < NSYM) ++s;
    const unsigned lo = cum[s], hi = cum[s + 1];
    if (slot < lo || slot >= hi) return false;
    x = (hi - lo) * (x >> PB) + (slot - lo);
    r.renorm(x);
    sym = s;
    return true;
}
template <class R> SG_DEVINL unsigned get_global(unsigned& x, R& r, const uint8_t* __restrict__ ct) {
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
// exponent, mantissa and the sign's frequencies from the role's tables in global memory
template <class R> SG_DEVINL void weight_global(unsigned& x, R& r, const uint8_t* __restrict__ tl, int pe, int sc, int pred, unsigned& ex,
                                                unsigned& man, unsigned& f01) {
    ex = get_global(x, r, tl + (size_t)pe * RANS_COMPACT);
    man = get_global(x, r, tl + (size_t)(512 + mctx((int)ex, pred)) * RANS_COMPACT);
    const unsigned* sw = reinterpret_cast<const unsigned*>(tl + (size_t)(640 + sc) * RANS_COMPACT + 256);
    f01 = (sw[0] & 0xffffu) | (sw[1] << 16);
}
template <class R> SG_DEVINL bool get_sign(unsigned& x, R& r, unsigned f01) {
    const unsigned slot = x & ((1u << PB) - 1), f0 = f01 & 0xffffu;
    const bool neg = slot >= f0;                                 // (two symbols: the second one starts where the first ends)
    x = (neg ? f01 >> 16 : f0) * (x >> PB) + (slot - (neg ? f0 : 0u));
    r.renorm(x);
    return neg;
}

struct DecArgs {
    const unsigned char* in; const unsigned long long* in_off; const unsigned long long* in_end;
    unsigned char* dev; const TB* tb; const SG* sg; Ctx c; const unsigned char* lut; int* status;
};
// a piece of segments of one role
SG_DEVINL void dec_staged(DecSmem& m, const DecArgs& a, int first, int count) {
    const Ctx& c = a.c;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool chain = warp < D_PAIRS;
    // as many pairs as every scheduler of the SM gets alike: 21 segments in four pairs 4.86 ms, in five 5.31, seven 5.10, eleven 5.72;
    // 42 in eight 5.47, in eleven 5.99
    const int npair = count <= 24 ? 4 : count <= 48 ? 8 : D_PAIRS;
    const int pair = chain ? warp : warp - D_PAIRS, sub = chain ? lane : lane / DG, grp = npair * sub + pair, gl = lane % DG;
    auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(pair + 1) : "memory"); };
    const int s = first + grp;
    const bool live = pair < npair && sub < 8 && grp < count;
    SG g; g.t = 0; g.n = 0; g.i0 = 0;
    if (live) g = a.sg[s];
    const TB T = a.tb[g.t];
    const int tab = a.tb[a.sg[first].t].tab;
    const uint8_t* tl = a.lut + (size_t)tab * RANS_COMPACT;
    if (threadIdx.x == 0) { m.nmax = 0; m.bad = 0; }
    const int pe_mid = window_of(m.win, c, a.tb, a.sg, first, count, tab);
    const int pe0 = clampi(pe_mid - D_ECTX / 2, 0, 512 - D_ECTX), ex0 = clampi(window_exponent(pe_mid), 0, 256 - D_ESYM);
    if (chain && live) atomicMax(&m.nmax, g.n);
    for (int t = warp; t < D_MCTX + D_ECTX; t += D_THREADS / 32) {
        if (t < D_MCTX) {
            const uint8_t* ct = tl + (size_t)(512 + t) * RANS_COMPACT;
            stage_table<128>(ct, m.mant + t * D_MP, 0, lane);
            // a distribution that goes on past symbol 127 (no encoder writes one): this CTA stays with global memory
            const unsigned w = reinterpret_cast<const unsigned*>(ct + 256)[127], z = reinterpret_cast<const unsigned*>(ct + 256)[255];
            if ((w >> 16) + (w & 0xffffu) != (z >> 16) + (z & 0xffffu)) m.bad = 1;
        } else stage_table<D_ESYM>(tl + (size_t)(pe0 + t - D_MCTX) * RANS_COMPACT, m.expo + (t - D_MCTX) * D_EP, ex0, lane);
    }
    if (threadIdx.x < 16) {
        const unsigned* w = reinterpret_cast<const unsigned*>(tl + (size_t)(640 + threadIdx.x) * RANS_COMPACT + 256);
        m.sign[threadIdx.x] = (w[0] & 0xffffu) | (w[1] << 16);
    }
    __syncthreads();
    const bool staged = !m.bad;
    const int nbatch = (m.nmax + DB - 1) / DB;
    if (chain) {
        DecRing rd; rd.pos = rd.have = 0; rd.left = 0;
        unsigned x = RANS_L;
        bool bad = false;
        if (live) { rd.init(a.in + a.in_off[s], a.in + a.in_end[s], m.ring + grp); x = rd.state(); }
        pair_sync();
        for (int it = 0; it < nbatch; ++it) {
            if (live && !bad) {
                const int n = min(DB, g.n - it * DB);
                const unsigned* cx = m.ctx[it & 1][grp];
                unsigned short* o = m.out[it & 1][grp];
#pragma unroll 1
                for (int w = 0; w < n; ++w) {
                    if ((w & 3) == 0) rd.top_up();               // four weights take 24 bytes at most
                    const unsigned e = cx[w];
                    const int pe = e & 511, sc = (e >> 9) & 15, pred = (int)e >> 16;
                    const unsigned x0 = x, top0 = rd.top, pos0 = rd.pos;
                    const bool near = staged && (unsigned)(pe - pe0) < (unsigned)D_ECTX;
                    const uint8_t* te = m.expo + (near ? pe - pe0 : 0) * D_EP;
                    bool miss = !near;
                    unsigned ex = ex0 + get_staged<true>(x, rd, te, miss);
                    unsigned man = get_staged<false>(x, rd, m.mant + mctx((int)ex, pred) * D_MP, miss);
                    unsigned f01 = m.sign[sc];
                    if (miss) {
                        x = x0; rd.top = top0; rd.pos = pos0;
                        if (near && get_walk<D_ESYM>(x, rd, te, ex)) {
                            ex += ex0;
                            if (!get_walk<127>(x, rd, m.mant + mctx((int)ex, pred) * D_MP, man)) bad = true;     // (no table there: a damaged stream)
                        } else weight_global(x, rd, tl, pe, sc, pred, ex, man, f01);
                    }
                    const bool neg = get_sign(x, rd, f01);
                    o[w] = (unsigned short)(((unsigned)neg << 15) | (ex << 7) | man);
                }
                bad |= rd.over();
            }
            pair_sync();
        }
        if (live && (bad || rd.over() || x != RANS_L || !rd.at_end())) atomicOr(a.status, SG_ST_CORRUPT);
    } else {
        unsigned short* base = reinterpret_cast<unsigned short*>(a.dev + T.doff);
        // a staging lane's first weight of the batch to stage and of the batch to store: compact row, column
        int rc = 0, j = 0, orc = 0, oj = 0;
        if (live) { const long long i = g.i0 + DW * gl; orc = rc = (int)(i / T.rowlen); oj = j = (int)(i % T.rowlen); }
        for (int it = 0; it < nbatch + 2; ++it) {
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
                        e[v] = pack_ctx(pred, pe, sc);
                    }
#pragma unroll
                    for (int v = 0; v < DW; ++v) m.ctx[it & 1][grp][DW * gl + v] = e[v];
                }
                j += DB;
                while (j >= T.rowlen) { j -= T.rowlen; ++rc; }
            }
            if (it <= nbatch) pair_sync();
        }
    }
}
// segments of any roles: for every 32 weights the four lanes of a segment look the contexts up side by side, the first of them runs
// the chain over them, all four store
SG_DEVINL void dec_any(AnySmem& m, const DecArgs& a, int first, int count) {
    const Ctx& c = a.c;
    const int grp = threadIdx.x / DG, gl = threadIdx.x % DG, s = first + grp;
    const bool live = grp < count;
    SG g; g.t = 0; g.n = 0; g.i0 = 0;
    if (live) g = a.sg[s];
    const TB T = a.tb[g.t];
    const uint8_t* tl = a.lut + (size_t)T.tab * RANS_COMPACT;
    const int nmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)max(g.n, 0));
    RingReader<G_RING> rd; rd.pos = rd.have = 0; rd.left = 0;
    unsigned x = RANS_L;
    if (live && gl == 0) { rd.init(a.in + a.in_off[s], a.in + a.in_end[s], m.ring + grp); x = rd.state(); }
    unsigned short* base = reinterpret_cast<unsigned short*>(a.dev + T.doff);
    int rc = 0, j = 0;                                           // this lane's first weight of the batch: compact row, column
    if (live) { const long long i = g.i0 + DW * gl; rc = (int)(i / T.rowlen); j = (int)(i % T.rowlen); }
    bool bad = false;
    for (int k0 = 0; k0 < nmax; k0 += DB) {
        size_t at[DW];
        {
            int r = rc, col = j, have = -1, orow = 0;
#pragma unroll
            for (int v = 0; v < DW; ++v) {
                at[v] = 0;
                if (k0 + DW * gl + v < g.n) {
                    if (r != have) { orow = T.rmap >= 0 ? c.rowmap[T.rmap + r] : r; have = r; }
                    int pred, pe, sc; contexts(c, T, orow, col, pred, pe, sc);
                    m.ctx[grp][DW * gl + v] = pack_ctx(pred, pe, sc);
                    at[v] = (size_t)orow * T.rowlen + col;
                    if (++col == T.rowlen) { col = 0; ++r; }
                }
            }
        }
        __syncwarp();
        if (live && gl == 0 && !bad) {
            const int n = min(DB, g.n - k0);
#pragma unroll 1
            for (int w = 0; w < n; ++w) {
                if ((w & 3) == 0) rd.top_up();
                const unsigned e = m.ctx[grp][w];
                unsigned ex, man, f01;
                weight_global(x, rd, tl, e & 511, (e >> 9) & 15, (int)e >> 16, ex, man, f01);
                const bool neg = get_sign(x, rd, f01);
                m.out[grp][w] = (unsigned short)(((unsigned)neg << 15) | (ex << 7) | man);
            }
            bad = rd.over();
        }
        __syncwarp();
#pragma unroll
        for (int v = 0; v < DW; ++v)
            if (k0 + DW * gl + v < g.n) base[at[v]] = m.out[grp][DW * gl + v];
        j += DB;
        if (live) while (j >= T.rowlen) { j -= T.rowlen; ++rc; }
    }
    if (live && gl == 0 && (bad || rd.over() || x != RANS_L || !rd.at_end())) atomicOr(a.status, SG_ST_CORRUPT);
}
// Which of the two ways it is depends on the records, which only the device sees: both kernels are launched, work it out and the one
// that has nothing to do ends (some 10 us).  They are two so that the tables of the second find the L1 that the first's shared
// memory takes from it (rows over 40 octaves: 14.9 ms with both in one, 8.1).
__global__ void __launch_bounds__(D_THREADS, 1) k_r2_dec(const DecArgs a, int nseg) {
    extern __shared__ __align__(16) unsigned char dsm[];
    DecSmem& m = *reinterpret_cast<DecSmem*>(dsm);
    PlanSmem& pl = m.plan;
    int per;
    const int pieces = dec_plan(pl, a.c, a.tb, a.sg, nseg, per);
    if (per < 0) return;
    for (int b = blockIdx.x; b < pieces; b += gridDim.x) {
        if (threadIdx.x == 0) {
            int at = 0, r = 0, k;
            for (;; ++r) {
                k = (pl.runs[r + 1] - pl.runs[r] + per - 1) / per;
                if (b < at + k) break;
                at += k;
            }
            const long long len = pl.runs[r + 1] - pl.runs[r];
            pl.first = pl.runs[r] + (int)(len * (b - at) / k);
            pl.count = pl.runs[r] + (int)(len * (b - at + 1) / k) - pl.first;
        }
        __syncthreads();
        const int first = pl.first, count = pl.count;
        dec_staged(m, a, first, count);
        __syncthreads();
    }
}
__global__ void __launch_bounds__(D_THREADS, 1) k_r2_dec_any(const DecArgs a, int nseg) {
    extern __shared__ __align__(16) unsigned char dsm[];
    AnySmem& m = *reinterpret_cast<AnySmem*>(dsm);
    int per;
    const int pieces = dec_plan(m.plan, a.c, a.tb, a.sg, nseg, per);
    if (per > 0) return;
    per = -per;
    for (int b = blockIdx.x; b < pieces; b += gridDim.x) dec_any(m, a, b * per, min(per, nseg - b * per));     // (its warps are on their own)
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
    if ((uintptr_t)in % 16 || (uintptr_t)lut % 8) return SG_ERR_ALIGN;
    if (nseg == 0) return SG_OK;
    rc = use_device(device);
    if (rc != SG_OK) return rc;
    Ctx c = {rfi, cfi, scl, rowmap};
    rc = cuda_ok(cudaFuncSetAttribute(k_r2_dec, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DecSmem)));
    if (rc != SG_OK) return rc;
    rc = cuda_ok(cudaFuncSetAttribute(k_r2_dec_any, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(AnySmem)));
    if (rc != SG_OK) return rc;
    const DecArgs args = {in, in_off, in_end, dev, (const TB*)tb, (const SG*)sgp, c, lut, status_word(device)};
    // the number of pieces is known to the kernel only: twice what segments of one role need, the CTAs without a piece end at once
    const long long grid = 2LL * 148 * ((nseg + 148LL * DSEG - 1) / (148 * DSEG)), any = 148LL * ((nseg + 148LL * GSEG - 1) / (148 * GSEG));
    k_r2_dec<<<(unsigned)(grid < nseg ? grid : nseg), D_THREADS, sizeof(DecSmem), (cudaStream_t)stream>>>(args, nseg);
    rc = cuda_ok(cudaGetLastError());
    if (rc != SG_OK) return rc;
    k_r2_dec_any<<<(unsigned)(any < nseg ? any : nseg), D_THREADS, sizeof(AnySmem), (cudaStream_t)stream>>>(args, nseg);
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
