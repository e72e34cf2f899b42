// Dequantisers: ggml blocks -> float32, the arithmetic of dequantize_row_<type> (ggml-quants.c:419-589, 961-1968,
// 2489-2766).  Replaces k_dq_<type> (seedpack/gpuquant.py:215-219).  Used where a quantised
// tensor stands in for missing weights (seeds) and by the importance-matrix fit; a minor, write-bound path
// (4 bytes out per weight).  Codes, lattice indices and sign positions come from the locators the residual coder uses; scales
// and fp16 values are read at compile-time places below (unpack_fields() works out all of a block's).
#include "api_util.h"
#include "qr_model.cuh"
#include "quant_extra.cuh"
#include "quant_iq.cuh"

namespace sg {

using namespace qr;

// the IQ4 levels (kv(), all of them whole numbers of 8 bits) of four codes, one signed byte each, by byte selection
SG_DEVINL unsigned iq4_levels(const int (&c)[4]) {
    const unsigned sel = c[0] | (c[1] << 4) | (c[2] << 8) | (c[3] << 12);
    const unsigned lo = __byte_perm(0xbfad9881u, 0xf6eaddcfu, sel & 0x7777u);      // -127 -104 -83 -65 | -49 -35 -22 -10
    const unsigned hi = __byte_perm(0x26190d01u, 0x71594535u, sel & 0x7777u);      // 1 13 25 38 | 53 69 89 113
    const unsigned up = ((sel >> 3) & 1u) | ((sel << 1) & 0x100u) | ((sel << 5) & 0x10000u) | ((sel << 9) & 0x1000000u);
    const unsigned mask = up * 255u;
    return (lo & ~mask) | (hi & mask);
}
SG_DEVINL float lattice_value(int T, int level) {          // dequantisation value of a lattice coordinate
    switch (T) {
        case 16: case 17: case 22: return level == 0 ? 8.f : level == 1 ? 25.f : 43.f;
        case 18: return level == 7 ? 62.f : (float)(4 + 8 * level);
        case 21: return (float)(2 * level + 1);
    }
    return (float)(level - 1);                              // IQ1_S / IQ1_M
}

// ---- one kernel per type: a tile of 4096 weights per CTA --------------------------------------------------------------
// Bound by the 4 bytes written per weight.  The tile's blocks come in through shared memory with 16-byte loads; a thread then
// makes four consecutive weights at a time (their codes are two 16-bit words in every layout but Q2_0's single byte, their
// sub-block scale is one) and stores them as one float4, so a warp writes 512 contiguous bytes.  The type is a template
// argument: one thread per weight that unpacked every scale field of its block through run-time switches took 206 us for
// 4096 x 4096 weights of Q4_K (76 MB), this takes 15.4 us.
constexpr int DQ_TILE = 4096, DQ_TPB = 256;

SG_DEVINL unsigned u16a(const uchar* b) { return *reinterpret_cast<const unsigned short*>(b); }      // b is even
// integer scale (and min) of sub-block s: the entries of unpack_fields() that follow the fp16 values
template <int T> SG_DEVINL int dq_sub(const uchar* b, int s) {
    switch (T) {
        case 10: return b[s] & 15;
        case 11: return q3k_scale(b + 96, s) - 32;
        case 14: return (int)(signed char)b[192 + s];
        case 23: return (((b[4 + (s >> 1)] >> (4 * (s & 1))) & 15) | (((u16a(b + 2) >> (2 * s)) & 3) << 4)) - 32;
        case 16: return b[2 + 8 * s + 7] >> 4;
        case 18: return b[66 + 4 * s + 3] >> 4;
        case 17: return (b[66 + (s >> 1)] >> (4 * (s & 1))) & 15;
        case 22: return (b[74 + (s >> 1)] >> (4 * (s & 1))) & 15;
        case 21: return (b[106 + (s >> 1)] >> (4 * (s & 1))) & 15;
        case 19: return b[34 + 2 * s + 1] >> 4;
        case 29: return (u16a(b + 48 + 2 * (s >> 2)) >> (3 * (s & 3))) & 7;
    }
    return 0;
}
template <int T> SG_DEVINL unsigned dq_fp16(const uchar* b) {
    switch (T) {
        case 10: return u16a(b + 80);
        case 11: return u16a(b + 108);
        case 14: return u16a(b + 208);
        case 29: return (u16a(b + 48) >> 12) | ((u16a(b + 50) >> 8) & 0xf0) | ((u16a(b + 52) >> 4) & 0xf00) | (u16a(b + 54) & 0xf000);
    }
    return u16a(b);
}
// codes of the weights w .. w + 3 (w % 4 == 0): consecutive bytes at one shift, w / l32-indexed planes included
template <int T> SG_DEVINL void dq_codes(const uchar* b, int w, int (&c)[4]) {
    const CodeLoc L = code_loc(T, w);
    if (T == 42) {
        const unsigned q = b[L.lo_byte];
#pragma unroll
        for (int i = 0; i < 4; ++i) c[i] = (q >> (2 * i)) & 3;
        return;
    }
    const unsigned lo = u16a(b + L.lo_byte) | (u16a(b + L.lo_byte + 2) << 16);
    if (T == 8) {
#pragma unroll
        for (int i = 0; i < 4; ++i) c[i] = (int)(signed char)(lo >> (8 * i));
        return;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] = (lo >> (8 * i + L.lo_shift)) & ((1 << L.lo_bits) - 1);
    if (T == 6 || T == 7) {                                  // fifth bits: one bit per weight of a 32-bit word
        const unsigned h = b[L.hi_byte] >> L.hi_shift;
#pragma unroll
        for (int i = 0; i < 4; ++i) c[i] |= ((h >> i) & 1) << 4;
    } else if (L.hi_bits) {
        const unsigned h = u16a(b + L.hi_byte) | (u16a(b + L.hi_byte + 2) << 16);
#pragma unroll
        for (int i = 0; i < 4; ++i) c[i] |= ((h >> (8 * i + L.hi_shift)) & ((1 << L.hi_bits) - 1)) << L.lo_bits;
    }
}
// signs of the 8 weights that w lies in, one bit each
template <int T> SG_DEVINL unsigned dq_signs(const uchar* b, int w) {
    if (!parity_type(T)) return b[sign_bit_pos(T, w & ~7) >> 3];
    const int p = sign_bit_pos(T, w & ~7);
    const unsigned s7 = ((b[p >> 3] | ((unsigned)b[(p >> 3) + 1] << 8)) >> (p & 7)) & 127;
    return s7 | ((__popc(s7) & 1) << 7);
}
template <int T> SG_DEVINL float4 dq4(const uchar* b, int w, const uint16_t* __restrict__ gk) {
    const float d = f16_to_f32((uint16_t)dq_fp16<T>(b));
    float o[4];
    if constexpr (!is_grid(T)) {
        int c[4];
        dq_codes<T>(b, w, c);
        float a = d, m = 0.f;
        if (T == 10) { const int s = w >> 4; a = fmul(d, (float)dq_sub<T>(b, s)); m = fmul(f16_to_f32((uint16_t)u16a(b + 82)), (float)(b[s] >> 4)); }
        else if (T == 12 || T == 13) {
            int sc, mn; scale_min_k4(w >> 5, b + 4, sc, mn);
            a = fmul(d, (float)sc); m = fmul(f16_to_f32((uint16_t)u16a(b + 2)), (float)mn);
        } else if (T == 11 || T == 14) a = fmul(d, (float)dq_sub<T>(b, w >> 4));
        else if (T == 23) a = fmul(d, (float)dq_sub<T>(b, w >> 5));
        else if (T == 3 || T == 7) m = f16_to_f32((uint16_t)u16a(b + 2));
        const unsigned lev = T == 20 || T == 23 ? iq4_levels(c) : 0u;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (T == 20 || T == 23) o[i] = fmul(a, (float)(signed char)(lev >> (8 * i)));
            else if (T == 3 || T == 7) o[i] = fadd(fmul((float)c[i], a), m);
            else if (T == 10 || T == 12 || T == 13) o[i] = fsub(fmul(a, (float)c[i]), m);
            else o[i] = fmul(a, (float)(c[i] - (T == 2 ? 8 : T == 6 ? 16 : T == 42 ? 1 : T == 11 ? 4 : T == 14 ? 32 : 0)));
        }
    } else {
        constexpr int B = (T == 18 || T == 21) ? 3 : 2, N = (T == 18 || T == 21) ? 4 : 8;
        const unsigned key = (unsigned)__ldg(gk + get_gidx(T, b, w / N)) >> (B * (w % N));
        float a, sh = 0.f;
        unsigned neg = 0;
        if (T == 19 || T == 29) {
            const int f = dq_sub<T>(b, w >> (T == 19 ? 5 : 4));
            a = fmul(d, (float)(2 * (T == 19 ? f & 7 : f) + 1));
            sh = (T == 19 ? (f & 8) != 0 : get_shift(b, w >> 3) != 0) ? -0.125f : 0.125f;
        } else {
            const float f = (float)dq_sub<T>(b, w >> ((T == 17 || T == 22) ? 4 : 5));
            a = T == 21 ? fmul(d, fadd(1.f, fmul(2.f, f))) : fmul(fmul(d, fadd(0.5f, f)), T == 18 ? 0.5f : 0.25f);
            neg = dq_signs<T>(b, w) >> (w & 7);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float gv = lattice_value(T, (key >> (B * i)) & ((1 << B) - 1));
            if (T == 19 || T == 29) o[i] = fmul(a, fadd(gv, sh));
            else o[i] = fmul(fmul(a, gv), (neg >> i) & 1 ? -1.f : 1.f);
        }
    }
    return make_float4(o[0], o[1], o[2], o[3]);
}
template <int T> __global__ void __launch_bounds__(DQ_TPB) k_dequant(const uchar* __restrict__ y, float* __restrict__ x, long long n,
                                                                     const uint16_t* __restrict__ gk) {
    constexpr int QK = qk_of(T), BS = bs_of(T), BYTES = DQ_TILE / QK * BS;
    __shared__ __align__(16) uchar tile[BYTES];
    const long long w0 = (long long)blockIdx.x * DQ_TILE;
    const int nw = (int)min((long long)DQ_TILE, n - w0), nbytes = nw / QK * BS;
    const uchar* src = y + w0 / QK * BS;
    int head = 0;                                            // a tile's length is a multiple of 16 bytes: y's alignment decides
    if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
        head = nbytes & ~15;
        for (int i = threadIdx.x * 16; i < head; i += DQ_TPB * 16) *reinterpret_cast<uint4*>(tile + i) = __ldg(reinterpret_cast<const uint4*>(src + i));
    }
    for (int i = head + threadIdx.x; i < nbytes; i += DQ_TPB) tile[i] = src[i];
    __syncthreads();
    const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
#pragma unroll
    for (int j = 0; j < DQ_TILE / (4 * DQ_TPB); ++j) {
        const int w = 4 * (j * DQ_TPB + (int)threadIdx.x);
        if (w >= nw) break;
        const float4 v = dq4<T>(tile + w / QK * BS, w % QK, gk);
        float* o = x + w0 + w;
        if (vec) *reinterpret_cast<float4*>(o) = v;
        else { o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w; }
    }
}

// the five types outside the reference's own table: dequantize_row_q1_0 / mxfp4 / nvfp4 (ggml-quants.c:419-437, 569-612)
// and dequantize_row_tq1_0 / tq2_0 (2429-2487)
__global__ void __launch_bounds__(256) k_dequant_extra(int T, const uchar* __restrict__ y, float* __restrict__ x, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float kvf[16] = {0.f, 1.f, 2.f, 3.f, 4.f, 6.f, 8.f, 12.f, 0.f, -1.f, -2.f, -3.f, -4.f, -6.f, -8.f, -12.f};
    const unsigned pow3[5] = {1, 3, 9, 27, 81};
    float out = 0.f;
    if (T == SG_Q1_0) {
        const uchar* b = y + (i / 128) * 18;
        const int w = (int)(i % 128);
        const float d = f16_to_f32((uint16_t)(b[0] | (b[1] << 8)));
        out = ((b[2 + (w >> 3)] >> (w & 7)) & 1) ? d : -d;
    } else if (T == SG_TQ2_0) {
        const uchar* b = y + (i / 256) * 66;
        const int w = (int)(i % 256);
        const float d = f16_to_f32((uint16_t)(b[64] | (b[65] << 8)));
        const int q = (b[32 * (w >> 7) + (w & 31)] >> (2 * ((w >> 5) & 3))) & 3;
        out = fmul((float)(q - 1), d);
    } else if (T == SG_TQ1_0) {
        const uchar* b = y + (i / 256) * 54;
        const int w = (int)(i % 256);
        const float d = f16_to_f32((uint16_t)(b[52] | (b[53] << 8)));
        unsigned byte, n;
        if (w < 160) { byte = b[w & 31]; n = w >> 5; }
        else if (w < 240) { byte = b[32 + ((w - 160) & 15)]; n = (w - 160) >> 4; }
        else { byte = b[48 + ((w - 240) & 3)]; n = (w - 240) >> 2; }
        const unsigned q = (byte * pow3[n]) & 0xffu;
        out = fmul((float)((int)((q * 3) >> 8) - 1), d);
    } else if (T == SG_MXFP4) {
        const uchar* b = y + (i / 32) * 17;
        const int w = (int)(i % 32);
        const float d = e8m0_half(b[0]);
        out = fmul(kvf[w < 16 ? b[1 + w] & 15 : b[1 + w - 16] >> 4], d);
    } else {
        const uchar* b = y + (i / 64) * 36;
        const int w = (int)(i % 64), sb = w >> 4, j = w & 15;
        const float d = ue4m3_to_f32(b[sb]);
        out = fmul(kvf[j < 8 ? b[4 + 8 * sb + j] & 15 : b[4 + 8 * sb + j - 8] >> 4], d);
    }
    x[i] = out;
}

// BF16 / F16 / F32 conversions of unquantised tensors (norms, embeddings kept in float): replaces
// M28RepoGPU._float_dev (seedpack/repo3.py:673-689).  To BF16: round to nearest even by integer add on the bits.
__global__ void __launch_bounds__(256) k_convert_float(const void* __restrict__ src, int st, void* __restrict__ dst, int dt, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float f;
    if (st == SG_DT_BF16) f = bf16_to_f32(static_cast<const uint16_t*>(src)[i]);
    else if (st == SG_DT_F16) f = f16_to_f32(static_cast<const uint16_t*>(src)[i]);
    else f = static_cast<const float*>(src)[i];
    if (dt == SG_DT_F32) static_cast<float*>(dst)[i] = f;
    else if (dt == SG_DT_F16) static_cast<uint16_t*>(dst)[i] = f32_to_f16(f);
    else { const unsigned u = __float_as_uint(f); static_cast<uint16_t*>(dst)[i] = (uint16_t)((u + 0x7FFFu + ((u >> 16) & 1u)) >> 16); }
}

const uint16_t* device_grid_keys(int device, int which);

}  // namespace sg

using namespace sg;

extern "C" int sg_dequantize(int device, void* stream, int T, const unsigned char* y, float* x, long long n_weights) {
    int qk, bs;
    if (sg_type_info(T, &qk, &bs) != SG_OK) return SG_ERR_TYPE;
    if (n_weights < 0 || (n_weights && (!y || !x))) return SG_ERR_ARG;
    if (n_weights % qk) return SG_ERR_SHAPE;
    if (n_weights == 0) return SG_OK;
    int rc = use_device(device);
    if (rc != SG_OK) return rc;
    const uint16_t* gk = nullptr;
    if (T == 16 || T == 17 || T == 18 || T == 19 || T == 21 || T == 22 || T == 29) {
        const int gi = T == 16 ? 0 : T == 17 ? 1 : (T == 19 || T == 29) ? 2 : T == 22 ? 3 : T == 18 ? 4 : 5;
        gk = device_grid_keys(device, gi);
        if (!gk) return SG_ERR_TABLES;
    }
    const long long grid = (n_weights + 255) / 256;
    if (grid > 0x7fffffffLL) return SG_ERR_LIMIT;
    const unsigned tiles = (unsigned)((n_weights + DQ_TILE - 1) / DQ_TILE);
    if (T == SG_Q1_0 || T == SG_TQ1_0 || T == SG_TQ2_0 || T == SG_MXFP4 || T == SG_NVFP4)
        k_dequant_extra<<<(unsigned)grid, 256, 0, (cudaStream_t)stream>>>(T, y, x, n_weights);
    else
        switch (T) {
#define SG_DQ(t) case t: k_dequant<t><<<tiles, DQ_TPB, 0, (cudaStream_t)stream>>>(y, x, n_weights, gk); break;
            SG_DQ(2) SG_DQ(3) SG_DQ(6) SG_DQ(7) SG_DQ(8) SG_DQ(10) SG_DQ(11) SG_DQ(12) SG_DQ(13) SG_DQ(14) SG_DQ(20) SG_DQ(23) SG_DQ(42)
            SG_DQ(16) SG_DQ(17) SG_DQ(18) SG_DQ(19) SG_DQ(21) SG_DQ(22) SG_DQ(29)
#undef SG_DQ
            default: return SG_ERR_TYPE;
        }
    return cuda_ok(cudaGetLastError());
}

extern "C" int sg_convert_float(int device, void* stream, const void* src, int src_dtype, void* dst, int dst_dtype, long long n) {
    if (n < 0 || (n && (!src || !dst))) return SG_ERR_ARG;
    if (src_dtype < 0 || src_dtype > 2 || dst_dtype < 0 || dst_dtype > 2) return SG_ERR_ARG;
    if (n == 0) return SG_OK;
    int rc = use_device(device);
    if (rc != SG_OK) return rc;
    const long long grid = (n + 255) / 256;
    if (grid > 0x7fffffffLL) return SG_ERR_LIMIT;
    k_convert_float<<<(unsigned)grid, 256, 0, (cudaStream_t)stream>>>(src, src_dtype, dst, dst_dtype, n);
    return cuda_ok(cudaGetLastError());
}

// nearest_int of every element: the rounding helper of all quantisers, exposed so that it can be swept on its own
__global__ void __launch_bounds__(256) k_nearest_int(const float* __restrict__ x, int* __restrict__ out, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = sg::nearest_int(x[i]);
}

extern "C" int sg_selftest_nearest_int(int device, void* stream, const float* x, int* out, long long n) {
    if (n < 0 || (n && (!x || !out))) return SG_ERR_ARG;
    if (n == 0) return SG_OK;
    int rc = use_device(device);
    if (rc != SG_OK) return rc;
    const long long grid = (n + 255) / 256;
    if (grid > 0x7fffffffLL) return SG_ERR_LIMIT;
    k_nearest_int<<<(unsigned)grid, 256, 0, (cudaStream_t)stream>>>(x, out, n);
    return cuda_ok(cudaGetLastError());
}
