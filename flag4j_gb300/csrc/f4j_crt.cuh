// f4j_crt.cuh -- the split GEMM's residue form: the same fixed-point operands,
// multiplied modulo small coprime numbers instead of slice by slice.
//
// The operands become the slice form's integers Y = round(x 2^(F - e)),
// F = 4 + 5 (s - 1) bits for the same s.  Their product C' = Y_A Y_B is an
// integer below k 2^(2F), so it is known once it is known modulo pairwise
// coprime p_1 .. p_L with p_1 ... p_L > 2 k 2^(2F) (Chinese remainder theorem;
// the residue-number form of error-free GEMM emulation, Ozaki, Uchino and
// Imamura 2025).  Residues here are E4M3 numbers:
//  - b odd, b <= 49, or b <= 32: each residue mod b has a representative d with
//    |d| <= 16, or even and |d| <= 32, which E4M3 holds exactly.  C' mod b is
//    one FP8 product.
//  - b^2: with x = x0 + b x1 (digits as above), x y = x0 y0 + b (x0 y1 + x1 y0)
//    modulo b^2 (b^2 x1 y1 vanishes): three FP8 products in two accumulators.
// A product of 8192 terms at F = 49 needs 112 bits: eight squares and seven
// single moduli, 31 FP8 products where the slices take 55 (66 -> 34 or 35 at
// F = 54), and no slice product is dropped: C' is exact and C is C' 2^(..)
// rounded once (where that is subnormal, to 53 bits first).
//
//  k_crt_planes   Y of each element, then its residues' digits, one E4M3 plane
//                 per digit (K-major, as the slice planes).
//  k_crt_gemm     for each modulus and 256 x 256 tile of C, the FP8 products on
//                 CTA pairs (tcgen05 cta_group::2), exact in FP32 (|sum| <= 2^24
//                 over at most 8192 terms), reduced mod p and multiplied by the
//                 modulus's weight (M / p)^-1: an int16 plane per modulus.
//  k_crt_combine  sum_l y_l (M / p_l) in 32-bit words, reduced mod M, rounded to
//                 double and scaled.
//
// Included by f4j_split.cu.
#pragma once

namespace {

// ------------------------------------------------------------------ moduli
constexpr int CRT_NB = 15;     // bases; a configuration squares the first nsq and drops some of the last
constexpr int CRT_WORDS = 5;   // 32-bit words of M, at most
constexpr int CRT_NG = 7;      // groups of moduli in the reconstruction: pairs, and the last three
constexpr int CRT_CFGS = 48;
constexpr int CRT_KC = 8192;   // terms per accumulation: 2 * 8192 * 32 * 32 = 2^24
__host__ __device__ constexpr int crt_base(int i) {
    // pairwise coprime; the large ones first, as the order in which they are squared
    constexpr int b[CRT_NB] = {49, 47, 43, 41, 37, 32, 31, 29, 27, 25, 23, 19, 17, 13, 11};
    return b[i];
}

// Residue weights of the eight bytes of Y + 2^60: 256^i = wh b + wl (mod b^2),
// packed for dp4a.  The two sums start at kl and kh, the bits of floats 2^23 +
// k0 and 2^23 + k1, so each is a float without a conversion; k0 and k1 make
// the 2^23 and the 2^60 vanish modulo b (and b^2 for the two together).
struct CrtMod {
    uint32_t wl[2] = {0, 0}, wh[2] = {0, 0};
    uint32_t kl = 0, kh = 0;
    alignas(8) float nb[2] = {0, 0};  // -b and 1 / b, twice for the paired arithmetic
    alignas(8) float inv[2] = {0, 0};
};
struct CrtMods {
    CrtMod m[CRT_NB] = {};
    constexpr CrtMods() {
        for (int i = 0; i < CRT_NB; i++) {
            const uint32_t b = (uint32_t)crt_base(i), p = b * b;
            uint32_t pw = 1;
            for (int u = 0; u < 8; u++) {
                m[i].wl[u / 4] |= (pw % b) << (8 * (u % 4));
                m[i].wh[u / 4] |= (pw / b) << (8 * (u % 4));
                pw = pw * 256 % p;
            }
            uint32_t c = 8388608u % p, c60 = 1;
            for (int u = 0; u < 60; u++) c60 = c60 * 2 % p;
            c = (c + c60) % p;
            const uint32_t k0 = (b - c % b) % b;          // 2^23 + 2^60 + k0 = g b (mod b^2)
            const uint32_t g = (c + k0) % p / b;
            const uint32_t k1 = (2 * b - g - 8388608u % b) % b;  // 2^23 + k1 = -g (mod b)
            m[i].kl = 0x4B000000u + k0;
            m[i].kh = 0x4B000000u + k1;
            m[i].nb[0] = m[i].nb[1] = -(float)b;
            m[i].inv[0] = m[i].inv[1] = 1.0f / (float)b;
        }
    }
};
__constant__ CrtMods c_crt{};

// One configuration: which moduli, and the constants of the reconstruction.
struct CrtCfg {
    int nmod, nsq;   // moduli; the first nsq are squares (nmod + 2 nsq FP8 products)
    int words;       // words of the reconstruction: 4 while M < 2^127, else 5
    float bits;      // log2 M
    int sh;          // the words below hold 2^sh times their number: 2^sh M in [2^(32 words - 2), 2^(32 words - 1))
    float qinv;      // 2^(32 words - 18) / (2^sh M), for the quotient by M
    float p[CRT_NB], invp[CRT_NB], u[CRT_NB];  // modulus, 1 / p, (M / p)^-1 mod p (balanced)
    int32_t c[CRT_NB];                         // P / p, P the product of the group's moduli
    int32_t z0[CRT_NG];                        // 2 P: makes a group's sum positive, and vanishes modulo M
    uint32_t W[CRT_NG][CRT_WORDS];             // M / P
    uint32_t NM[CRT_WORDS];                    // 2^(32 words) - M
};
__host__ __device__ constexpr int crt_group(int l) { return l / 2 < CRT_NG ? l / 2 : CRT_NG - 1; }

// Every configuration worth having, by rising cost in FP8 products: squares of the
// first nsq bases, the last `drop` bases left out.  Built by the compiler, for the
// host and as a constant of the device code: no kernel can meet it half written, and
// no product's first call allocates or copies for it.  Exact arithmetic on 32-bit
// words: M and M / P are products of the other moduli.
struct CrtTable {
    CrtCfg cfg[CRT_CFGS] = {};
    int n = 0;

    static constexpr void mul(uint32_t (&a)[CRT_WORDS], uint32_t m) {
        uint64_t carry = 0;
        for (int j = 0; j < CRT_WORDS; j++) {
            const uint64_t t = (uint64_t)a[j] * m + carry;
            a[j] = (uint32_t)t;
            carry = t >> 32;
        }
    }
    // log2 x, x >= 1: the integer part by halving, the rest as 2 / ln 2 times the
    // series of artanh at (f - 1) / (f + 1) <= 1/3
    static constexpr double log2_of(double x) {
        int e = 0;
        while (x >= 2.0) x *= 0.5, e++;
        const double t = (x - 1.0) / (x + 1.0);
        double sum = 0, pw = t;
        for (int i = 1; i < 40; i += 2, pw *= t * t) sum += pw / i;
        return e + 2.0 * 1.44269504088896340736 * sum;
    }
    static constexpr int inverse(int r, int p) {  // r^-1 mod p, coprime
        int a = r % p, b = p, u = 1, v = 0;
        while (a > 1) {
            const int q = b / a, b1 = b - q * a, v1 = v - q * u;
            b = a, a = b1, v = u, u = v1;
        }
        return u < 0 ? u + p : u;
    }

    constexpr CrtTable() {
        double best = 0;
        for (int cost = 9; cost <= 3 * CRT_NB; cost++) {
            int bj = -1, bd = 0;
            double bbits = 0;
            for (int d = 0; d <= 6; d++) {
                const int nmod = CRT_NB - d, j2 = cost - nmod;
                if (j2 < 0 || j2 % 2 || j2 / 2 > nmod) continue;
                double bits = 0;
                for (int i = 0; i < nmod; i++) bits += (i < j2 / 2 ? 2 : 1) * log2_of(crt_base(i));
                if (bits > bbits) bbits = bits, bj = j2 / 2, bd = d;
            }
            if (bj < 0 || bbits <= best || n >= CRT_CFGS) continue;
            best = bbits;
            fill(cfg[n++], CRT_NB - bd, bj, bbits);
        }
    }
    static constexpr void fill(CrtCfg& c, int nmod, int nsq, double bits) {
        c.nmod = nmod;
        c.nsq = nsq;
        c.bits = (float)bits;
        c.words = bits < 127.0 ? 4 : 5;
        int p[CRT_NB] = {};
        for (int l = 0; l < nmod; l++) p[l] = l < nsq ? crt_base(l) * crt_base(l) : crt_base(l);
        uint32_t M[CRT_WORDS] = {1};
        for (int l = 0; l < nmod; l++) {
            mul(M, (uint32_t)p[l]);
            int r = 1, cl = 1;
            for (int i = 0; i < nmod; i++) {
                if (i == l) continue;
                r = (int)((int64_t)r * p[i] % p[l]);  // M / p mod p
                if (crt_group(i) == crt_group(l)) cl *= p[i];
            }
            const int inv = inverse(r, p[l]);
            c.p[l] = (float)p[l];
            c.invp[l] = 1.0f / (float)p[l];
            c.u[l] = (float)(2 * inv > p[l] ? inv - p[l] : inv);
            c.c[l] = cl;
        }
        c.sh = 0;
        while (!(M[c.words - 1] >> 30)) mul(M, 2), c.sh++;
        uint64_t borrow = 1;  // two's complement over `words` words
        double frac = 0;      // 2^sh M / 2^(32 words)
        for (int j = 0; j < c.words; j++) {
            const uint64_t t = (uint64_t)(uint32_t)~M[j] + borrow;
            c.NM[j] = (uint32_t)t;
            borrow = t >> 32;
            frac = (frac + M[j]) / 4294967296.0;
        }
        c.qinv = (float)(1.0 / 262144.0 / frac);  // 2^-18 / frac
        for (int g = 0; 2 * g < nmod && g < CRT_NG; g++) {  // without a modulus: z stays 0
            uint32_t W[CRT_WORDS] = {1};
            int P = 1;
            for (int i = 0; i < nmod; i++) {
                if (crt_group(i) == g) P *= p[i];
                else mul(W, (uint32_t)p[i]);
            }
            for (int i = 0; i < c.sh; i++) mul(W, 2);
            c.z0[g] = 2 * P;
            for (int j = 0; j < CRT_WORDS; j++) c.W[g][j] = W[j];
        }
    }
};
constexpr CrtTable crt_host{};
__device__ const CrtTable crt_dev{};

constexpr float CRT_MAGIC = 12582912.0f;  // 1.5 * 2^23: x + CRT_MAGIC rounds |x| < 2^22 to an integer

// ------------------------------------------------------------------ residue planes
typedef unsigned long long f32x2;  // two floats in a register pair
__device__ __forceinline__ f32x2 pack2(uint32_t a, uint32_t b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ f32x2 dup2(float a) { return pack2(__float_as_uint(a), __float_as_uint(a)); }
__device__ __forceinline__ void unpack2(f32x2 v, uint32_t& a, uint32_t& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Eight digits, |d| <= 16, as E4M3 bytes.
__device__ __forceinline__ uint2 crt_e4m3(const f32x2 (&f)[4]) {
    uint32_t w[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        uint32_t x0, x1;
        uint16_t h;
        unpack2(f[u], x0, x1);
        asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(h) : "f"(__uint_as_float(x1)), "f"(__uint_as_float(x0)));
        w[u] = h;
    }
    return make_uint2(__byte_perm(w[0], w[1], 0x5410), __byte_perm(w[2], w[3], 0x5410));
}

// Eight digits as bytes d + 64.
__device__ __forceinline__ uint2 crt_bytes64(const f32x2 (&f)[4]) {
    uint32_t x[8], h[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        unpack2(add2(f[u], dup2(CRT_MAGIC + 64.0f)), x[2 * u], x[2 * u + 1]);
        h[u] = __byte_perm(x[2 * u], x[2 * u + 1], 0x0040);
    }
    return make_uint2(__byte_perm(h[0], h[1], 0x5410), __byte_perm(h[2], h[3], 0x5410));
}

// Four bytes g = d + 64, |d| <= 26: an odd d beyond 16 is not an E4M3 number
// and becomes the even d -+ b; up / down flag those bytes (d above 16: up).
__device__ __forceinline__ uint32_t crt_even(uint32_t g, uint32_t b, uint32_t& up, uint32_t& down) {
    up = ((g + 0x2F2F2F2Fu) >> 7) & g & 0x01010101u;    // g >= 81, odd
    down = ((0xAFAFAFAFu - g) >> 7) & g & 0x01010101u;  // g <= 47, odd
    return g + down * b - up * b;
}

// Four bytes d + 64 as E4M3 bytes, by way of halves 1024 + (d + 64).
__device__ __forceinline__ uint32_t crt_e4m3_of64(uint32_t g) {
    uint32_t a = __byte_perm(g, 0x64646464u, 0x4140), c = __byte_perm(g, 0x64646464u, 0x4342);
    const uint32_t off = 0xE440E440u;  // -1088, twice
    uint16_t h0, h1;
    asm("add.rn.f16x2 %0, %0, %1;" : "+r"(a) : "r"(off));
    asm("add.rn.f16x2 %0, %0, %1;" : "+r"(c) : "r"(off));
    asm("cvt.rn.satfinite.e4m3x2.f16x2 %0, %1;" : "=h"(h0) : "r"(a));
    asm("cvt.rn.satfinite.e4m3x2.f16x2 %0, %1;" : "=h"(h1) : "r"(c));
    return __byte_perm((uint32_t)h0, (uint32_t)h1, 0x5410);
}

struct CrtDst {
    uint8_t* a;   // first copy
    uint8_t* b;   // second copy, or null
    uint32_t xb;  // xor of the second copy's bytes (0x80808080: negated)
};

__device__ __forceinline__ void crt_store(const CrtDst& d, int64_t off, uint2 v) {
    *reinterpret_cast<uint2*>(d.a + off) = v;
    if (d.b) *reinterpret_cast<uint2*>(d.b + off) = make_uint2(v.x ^ d.xb, v.y ^ d.xb);
}

// The residue digits of eight integers Yb = Y + 2^60 (lo, hi words), plane i at
// d + i * plane.
__device__ __forceinline__ void crt_digits8(const uint32_t (&lo)[8], const uint32_t (&hi)[8], int nmod, int nsq,
                                            const CrtDst& d, int64_t plane) {
    const f32x2 magic = dup2(CRT_MAGIC), unmagic = dup2(-CRT_MAGIC);
    // unrolled: the weights are constant-bank operands and the kinds of moduli
    // compile-time (a rolled loop spent an eighth of its instructions on loading
    // them)
#pragma unroll
    for (int i = 0; i < CRT_NB; i++) {
        if (i >= nmod) break;
        const CrtMod& c = c_crt.m[i];
        const f32x2 nb = *reinterpret_cast<const f32x2*>(c.nb), inv = *reinterpret_cast<const f32x2*>(c.inv);
        const bool wide = crt_base(i) > 33;
        const uint32_t bi = (uint32_t)crt_base(i);
        f32x2 f[4], q[4];
        uint2 up = make_uint2(0, 0), down = make_uint2(0, 0);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const f32x2 t = pack2(__dp4a(hi[2 * j], c.wl[1], __dp4a(lo[2 * j], c.wl[0], c.kl)),
                                  __dp4a(hi[2 * j + 1], c.wl[1], __dp4a(lo[2 * j + 1], c.wl[0], c.kl)));
            q[j] = add2(fma2(t, inv, magic), unmagic);
            f[j] = fma2(nb, q[j], t);
        }
        if (wide) {
            uint2 g = crt_bytes64(f);
            g.x = crt_even(g.x, bi, up.x, down.x);
            g.y = crt_even(g.y, bi, up.y, down.y);
            crt_store(d, (int64_t)i * plane, make_uint2(crt_e4m3_of64(g.x), crt_e4m3_of64(g.y)));
        } else {
            crt_store(d, (int64_t)i * plane, crt_e4m3(f));
        }
        if (i < nsq) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const f32x2 t = add2(pack2(__dp4a(hi[2 * j], c.wh[1], __dp4a(lo[2 * j], c.wh[0], c.kh)),
                                           __dp4a(hi[2 * j + 1], c.wh[1], __dp4a(lo[2 * j + 1], c.wh[0], c.kh))),
                                     q[j]);
                f[j] = fma2(nb, add2(fma2(t, inv, magic), unmagic), t);
            }
            if (wide) {  // the first digit's d -+ b leaves +-1 for this one
                uint2 g = crt_bytes64(f);
                g.x = g.x + up.x - down.x;
                g.y = g.y + up.y - down.y;
                g.x = crt_even(g.x, bi, up.x, down.x);
                g.y = crt_even(g.y, bi, up.y, down.y);
                crt_store(d, (int64_t)(nmod + i) * plane, make_uint2(crt_e4m3_of64(g.x), crt_e4m3_of64(g.y)));
            } else {
                crt_store(d, (int64_t)(nmod + i) * plane, crt_e4m3(f));
            }
        }
    }
}

// One operand: planes[i] is rows_out x Kp bytes at out + i * rows_out * Kp.
//   real, and A of a complex product (role 0): as k_split writes its planes
//   B of a complex product (role 1): out[r][q] = re, out[r][Kh+q] = -im,
//     out[half+r][q] = im, out[half+r][Kh+q] = re
struct CrtOperand {
    const double* X;
    int64_t scols;
    int transposed, conj, role;
    int64_t targets, rows_out, half;
    const int* e_t;
    uint8_t* out;
};

template <bool CPLX>
__device__ __forceinline__ void crt_planes_body(const CrtOperand& o, int64_t klen, int64_t Kh, int64_t Kp,
                                                int s, int nmod, int nsq, double (*sre)[SP_TQ + 1],
                                                double (*sim)[SP_TQ + 1]) {
    const int64_t q0 = (int64_t)blockIdx.x * SP_TQ;
    const int F = 4 + 5 * (s - 1);
    const int rr = threadIdx.x / 8, qs = (threadIdx.x % 8) * 8;
    const int64_t plane = o.rows_out * Kp;
    const bool staged = CPLX || o.transposed;
    for (int by = blockIdx.y; (int64_t)by * SP_TR < o.targets; by += gridDim.y) {
        const int64_t r0 = (int64_t)by * SP_TR;
        if (staged) {
            for (int e = threadIdx.x; e < SP_TR * SP_TQ; e += 256) {
                int tr, tq;
                if (!o.transposed) { tr = e / SP_TQ; tq = e % SP_TQ; }
                else { tq = e / SP_TR; tr = e % SP_TR; }
                const int64_t r = r0 + tr, q = q0 + tq;
                double re = 0, im = 0;
                if (r < o.targets && q < klen) {
                    const int64_t idx = o.transposed ? (q * o.scols + r) : (r * o.scols + q);
                    if constexpr (CPLX) {
                        re = o.X[2 * idx];
                        im = o.X[2 * idx + 1];
                        if (o.conj) im = -im;
                    } else {
                        re = o.X[idx];
                    }
                }
                sre[tr][tq] = re;
                if constexpr (CPLX) sim[tr][tq] = im;
            }
            __syncthreads();
        }
        const int64_t r = r0 + rr;
        if (r < o.targets) {
            const int e = o.e_t[r];
#pragma unroll 1
            for (int part = 0; part < (CPLX ? 2 : 1); part++) {
                uint32_t lo[8], hi[8];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    double v;
                    if (staged) {
                        v = sre[rr][qs + j];
                        if constexpr (CPLX) v = part ? sim[rr][qs + j] : v;
                    } else {
                        v = q0 + qs + j < klen ? __ldg(o.X + r * o.scols + q0 + qs + j) : 0.0;
                    }
                    const unsigned long long y = (unsigned long long)(fixed_of(v, e, F) + (1ll << 60));
                    lo[j] = (uint32_t)y;
                    hi[j] = (uint32_t)(y >> 32);
                }
                CrtDst d{o.out + r * Kp + q0 + qs, nullptr, 0};
                if constexpr (CPLX) {
                    if (o.role == 0) {
                        if (part) d.a += Kh;
                    } else if (part == 0) {
                        d.b = d.a + o.half * Kp + Kh;
                    } else {
                        d.b = d.a + Kh;
                        d.xb = 0x80808080u;
                        d.a += o.half * Kp;
                    }
                }
                crt_digits8(lo, hi, nmod, nsq, d, plane);
            }
        }
        if (staged) __syncthreads();
    }
}

// Both operands' residue planes in one launch (blockIdx.z picks the operand).
// Bound by instruction issue (78 % of the slots at 4096^3, 264 instructions an
// element for 23 to 25 digits): dp4a sums of the bytes of Y, reductions in float
// pairs, the parity fix on four digits a word.  8192^3, both operands: 1.04 ms
// (1.40 with scalar floats and a compare per digit, 1.22 with the moduli in a
// rolled loop); its 4.2 GB take 0.62.
template <bool CPLX>
__global__ void __launch_bounds__(256, 4) k_crt_planes(const CrtOperand a, const CrtOperand b, int64_t klen,
                                                       int64_t Kh, int64_t Kp,
                                                       const SplitPlan* __restrict__ plan) {
    __shared__ double sre[SP_TR][SP_TQ + 1];
    __shared__ double sim[CPLX ? SP_TR : 1][SP_TQ + 1];
    chain_wait();
    chain_trigger();
    if (plan->nonfinite) return;
    const int s = plan->s, nmod = crt_dev.cfg[plan->crt].nmod, nsq = crt_dev.cfg[plan->crt].nsq;
    if (blockIdx.z == 0) crt_planes_body<CPLX>(a, klen, Kh, Kp, s, nmod, nsq, sre, sim);
    else crt_planes_body<CPLX>(b, klen, Kh, Kp, s, nmod, nsq, sre, sim);
}

// ------------------------------------------------------------------ GEMM
constexpr int CG_T = 256;                   // output tile of a CTA pair; each CTA holds 128 rows of A, 128 of B
constexpr int CG_BK = 128;                  // K bytes per ring slot (one 128-byte swizzle row)
constexpr int CG_TILE = 128 * CG_BK;        // 16 KB
constexpr int CG_SLOT = 2 * CG_TILE;        // an A tile and a B tile
constexpr int CG_RING = 7;
constexpr int CG_THREADS = 384;             // warp 0 TMA, warp 1 MMA, two idle, warps 4..11 epilogue
// Registers a thread: all start with 168; the first warpgroup gives up what the
// epilogue warpgroups take, 128 x 40 + 256 x 232 = 384 x 168.
constexpr int CG_REGS_LOAD = 40, CG_REGS_EPI = 232;
constexpr int CG_KB = CRT_KC / CG_BK;       // K blocks per accumulation
constexpr int CG_GROUP_M = 8;

struct CrtGemmParams {
    int M, N, nkb;          // rows of A, (padded) rows of B^T, K blocks of CG_BK bytes
    int tm0, tm1, tn0, tn1; // tile rows and columns of C the launch covers
    int row0, rows;         // rows of C in y: [row0, row0 + rows)
    int64_t ldy;            // columns of y (multiple of 16, >= N)
    int16_t* y;             // [nmod][rows][ldy]
    int* status;
    const SplitPlan* plan;
};

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of the same variable in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t cluster_map(const void* p, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// mbar_wait for a barrier that threads of the other CTA arrive on
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, int* status, int code) {
    if (mbar_try_wait_cluster(bar, parity)) return true;
    const uint64_t t0 = f4j_globaltimer_ns();
    for (uint32_t it = 0; it < F4J_WAIT_LIMIT; ++it) {
        if (mbar_try_wait_cluster(bar, parity)) return true;
        if ((it & 255) == 255 && f4j_globaltimer_ns() - t0 > F4J_WAIT_NS) break;
    }
    if (status) atomicExch(status, code);
    return false;
}
__device__ __forceinline__ void tma_load_3d_pair(void* dst, const CUtensorMap* map, uint32_t bar, int c0, int c1,
                                                 int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 "
        "[%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
// D (+)= A B^T over one 128-byte K block: four K = 32 steps on the CTA pair.
__device__ __forceinline__ void umma2_f8_k128(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc,
                                              uint32_t acc) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
            "setp.ne.b32 p, %5, 0;\n\t"
            "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
            "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], da, db, %4, p;\n\t}" ::"r"(d),
            "r"(a_lo + 2 * k), "r"(b_lo + 2 * k), "r"(hi), "r"(idesc), "r"(k == 0 ? acc : 1u)
            : "memory");
    }
}
// One K block of a square's three products: x += a0 b0, y += a0 b1 + a1 b0.  The
// tile a0 is read from shared memory once for its two products of a K = 32 step
// (the MMA's A collector): the MMAs read 64 bytes a clock and the loads write 45
// of an SM's 128, and the MMAs took 580 clocks a K block for the 512 they take
// alone.  GEMM at 4096^3 1303 -> 1264 us, 8192^3 10.9 -> 10.5 ms.  Not unrolled:
// the kernel starts with a cold instruction cache (1024^3: 1.5 us).
__device__ __forceinline__ void umma2_f8_square(uint32_t x, uint32_t y, uint32_t a0, uint32_t b0, uint32_t a1,
                                                uint32_t b1, uint32_t hi, uint32_t idesc) {
#pragma unroll 1
    for (int k = 0; k < 4; k++) {
        asm volatile(
            "{\n\t.reg .pred t;\n\t.reg .b64 a0, b0, a1, b1;\n\tsetp.eq.b32 t, 0, 0;\n\t"
            "mov.b64 a0, {%2, %6};\n\tmov.b64 b0, {%3, %6};\n\t"
            "mov.b64 a1, {%4, %6};\n\tmov.b64 b1, {%5, %6};\n\t"
            "tcgen05.mma.cta_group::2.kind::f8f6f4.collector::a::fill [%0], a0, b0, %7, t;\n\t"
            "tcgen05.mma.cta_group::2.kind::f8f6f4.collector::a::lastuse [%1], a0, b1, %7, t;\n\t"
            "tcgen05.mma.cta_group::2.kind::f8f6f4 [%1], a1, b0, %7, t;\n\t}" ::"r"(x),
            "r"(y), "r"(a0 + 2 * k), "r"(b0 + 2 * k), "r"(a1 + 2 * k), "r"(b1 + 2 * k), "r"(hi), "r"(idesc)
            : "memory");
    }
}
// Arrive on the barrier of both CTAs once this thread's MMAs have completed.
__device__ __forceinline__ void umma2_commit(uint64_t* bar) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
            smem_u32(bar)),
        "h"((uint16_t)3)
        : "memory");
}

// Tile `t` of a tiles_m x tiles_n block, bands of CG_GROUP_M tile rows,
// column-major inside a band (see tile_origin).
__device__ __forceinline__ void crt_tile(int t, int tiles_m, int tiles_n, int& tm, int& tn) {
    const int per = CG_GROUP_M * tiles_n;
    const int g = t / per, first = g * CG_GROUP_M;
    const int gm = tiles_m - first < CG_GROUP_M ? tiles_m - first : CG_GROUP_M;
    const int r = t - g * per;
    tm = first + r % gm;
    tn = r / gm;
}

// Balanced x mod p for integers |x| <= 2^24 (a pair; p and 1 / p twice).
__device__ __forceinline__ f32x2 crt_mod2(f32x2 x, f32x2 np, f32x2 invp) {
    const f32x2 q = add2(fma2(x, invp, dup2(CRT_MAGIC)), dup2(-CRT_MAGIC));
    return fma2(np, q, x);
}
// Two integers |x| < 2^15 as 16-bit halves x + 2^15, and back.
__device__ __forceinline__ uint32_t crt_halves(f32x2 x) {
    uint32_t a, b;
    unpack2(add2(x, dup2(8388608.0f + 32768.0f)), a, b);
    return __byte_perm(a, b, 0x5410);
}
__device__ __forceinline__ f32x2 crt_floats(uint32_t h) {
    return add2(pack2(__byte_perm(h, 0x4B000000u, 0x7610), __byte_perm(h, 0x4B000000u, 0x7632)),
                dup2(-8388608.0f - 32768.0f));
}

// A unit is one modulus of one 256 x 256 tile: squares first (modulus-major,
// so the pairs running together share operand tiles in L2), then the singles.
// Ring slots carry (A digit, B digit) tile pairs: one per K block of a single
// modulus, (A0, B0) and (A1, B1) of a square.  TMEM holds two accumulators of
// 256 columns: X (x0 y0) and Y (x0 y1 + x1 y0) of a square, in turn the
// singles'.  X's products run two K blocks ahead of Y's at the start and the end of
// a square, so X is drained under Y's last products and Y under the next
// unit's first.  In between the three products of a K block go together
// (umma2_f8_square).  Epilogue warps with 232 registers read an accumulator whole
// before they reduce it; with 168 and a copy of the code for each kind of modulus
// the GEMM took, us, 49.7 for 47.8 at 1024^3, 56 / 54.7 at 1500 x 900 x 700, 355 /
// 344 at 2048 x 2048 x 4096.
__global__ void __launch_bounds__(CG_THREADS, 1) __cluster_dims__(2, 1, 1)
    k_crt_gemm(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               const __grid_constant__ CrtGemmParams p) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* ring = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full[CG_RING], empty[CG_RING], accfull[2], accempty[2], mma_done;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const uint32_t rank = cluster_rank();
    const int tiles_m = p.tm1 - p.tm0, tiles_n = p.tn1 - p.tn0, ntiles = tiles_m * tiles_n;
    const int pair = blockIdx.x / 2, npairs = gridDim.x / 2;

    if (threadIdx.x == 0) {
        for (int i = 0; i < CG_RING; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&accfull[i], 1);
            mbar_init(&accempty[i], 16);  // eight epilogue warps in each CTA
        }
        mbar_init(&mma_done, 1);
        abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 0 && lane == 0) {
        prefetch_tmap(&tmA);
        prefetch_tmap(&tmB);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    chain_wait();  // the setup above runs under the planes kernel's last blocks
    chain_trigger();
    // nonfinite: the gated plain path computes this product
    const bool off = p.plan->nonfinite != 0;
    const CrtCfg* __restrict__ cfg = crt_dev.cfg + (off ? 0 : p.plan->crt);
    const int nmod = cfg->nmod, nsq = cfg->nsq;
    const int nunits = off ? 0 : ntiles * nmod;

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(CG_REGS_LOAD));
        if (warp == 0) {
            // ---------------- TMA producer: lane 0 loads the slot's A tile, lane 1 its B tile
            int s = 0, round = 0;  // next slot, and how often the ring has been filled
            bool ok = true;
            const uint32_t full0 = cluster_map(&full[0], 0);
            const CUtensorMap* map = lane == 0 ? &tmA : &tmB;
            for (int u = pair; u < nunits && ok; u += npairs) {
                const int l = u / ntiles;
                int tm, tn;
                crt_tile(u - l * ntiles, tiles_m, tiles_n, tm, tn);
                const int row = (lane == 0 ? p.tm0 + tm : p.tn0 + tn) * CG_T + (int)rank * 128;
                const int nd = l < nsq ? 2 : 1;
                for (int kb = 0; kb < p.nkb && ok; kb++) {
                    for (int d = 0; d < nd; d++) {
                        if (lane == 0) {
                            if (round > 0)
                                ok = mbar_wait(&empty[s], (round & 1) ^ 1, p.status, 21) && !*(volatile int*)&abort_flag;
                            if (!ok) abort_flag = 1;
                            else if (rank == 0) mbar_arrive_expect_tx(&full[s], 2 * CG_SLOT);
                        }
                        ok = __shfl_sync(0xffffffffu, ok, 0);
                        if (!ok) break;
                        if (lane < 2)
                            tma_load_3d_pair(ring + s * CG_SLOT + lane * CG_TILE, map, full0 + 8 * s, kb * CG_BK, row,
                                             d ? nmod + l : l);
                        if (++s == CG_RING) s = 0, round++;
                    }
                }
            }
            // copies still in flight signal the first CTA's barriers: it waits for them (bounded), and the
            // cluster barrier below keeps both CTAs until then
            if (rank == 0 && lane == 0)
                for (int q = 0; q < CG_RING; q++) {
                    const int fills = round + (q < s ? 1 : 0);
                    if (fills) mbar_wait(&full[q], (fills - 1) & 1, nullptr, 0);
                }
        } else if (warp == 1) {
            // ---------------- MMA issuer: one thread of the pair's first CTA.  The
            // tensor pipe queues only a couple of MMAs, so what this thread does
            // between them (waits, slot arithmetic, commits) shows as idle pipe: ring
            // cursors instead of divisions, one barrier test per slot on the fast path.
            if (rank == 0 && lane == 0 && pair < nunits) {
                const uint64_t desc0 = umma_desc_sw128(ring);
                const uint32_t hi = (uint32_t)(desc0 >> 32), lo0 = (uint32_t)desc0;
                const uint32_t idesc = umma_idesc_e4m3_f32(256, 256);
                constexpr uint32_t SLOT16 = CG_SLOT >> 4, TILE16 = CG_TILE >> 4;
                struct Cursor {
                    uint32_t s = 0, par = 0;
                    __device__ __forceinline__ void next() {
                        if (++s == CG_RING) s = 0, par ^= 1;
                    }
                };
                Cursor cur;  // first slot not yet consumed
                uint32_t turn = 0, fill0 = 0, fill1 = 0;
                bool ok = true;
                auto acquire = [&](uint32_t a, uint32_t fills) {  // the epilogue has drained accumulator a
                    if (fills > 0) ok = ok && mbar_wait_cluster(&accempty[a], (fills - 1) & 1, p.status, 22);
                    tc_fence_after();
                };
                auto landed = [&](const Cursor& c) {
                    if (!mbar_try_wait(&full[c.s], c.par)) {
                        ok = ok && mbar_wait(&full[c.s], c.par, p.status, 23) && !*(volatile int*)&abort_flag;
                    }
                };
                auto mma = [&](uint32_t acc, uint32_t sa, uint32_t sb, bool first) {
                    umma2_f8_k128(tmem + acc * 256, lo0 + sa * SLOT16, lo0 + sb * SLOT16 + TILE16, hi, idesc,
                                  first ? 0u : 1u);
                };
                for (int u = pair; u < nunits && ok; u += npairs) {
                    const int l = u / ntiles;
                    for (int k0 = 0; k0 < p.nkb && ok; k0 += CG_KB) {
                        const int nk = p.nkb - k0 < CG_KB ? p.nkb - k0 : CG_KB;
                        if (l < nsq) {
                            acquire(0, fill0);
                            Cursor cx = cur;
                            int x = 0;  // K blocks of X issued
                            for (int kb = 0; kb < nk && ok; kb++) {
                                // X ahead of Y by two K blocks at the start and the end only: in between a
                                // K block's slots are freed at once, so more of the ring is loads in flight
                                const int lead = kb == 0 ? (nk < 3 ? nk : 3) : (kb + 2 < nk ? 0 : nk);
                                if (x < lead) {
                                    for (; x < lead; x++) {
                                        landed(cx);
                                        if (!ok) break;
                                        mma(0, cx.s, cx.s, x == 0);
                                        cx.next();
                                        cx.next();
                                    }
                                    if (!ok) break;
                                    if (x == nk) umma2_commit(&accfull[0]);
                                    if (kb == 0) acquire(1, fill1);
                                }
                                const uint32_t s0 = cur.s;
                                if (x == kb) landed(cur);
                                cur.next();
                                landed(cur);
                                if (!ok) break;
                                if (x == kb) {  // the middle
                                    const uint32_t a0 = lo0 + s0 * SLOT16, a1 = lo0 + cur.s * SLOT16;
                                    umma2_f8_square(tmem, tmem + 256, a0, a0 + TILE16, a1, a1 + TILE16, hi, idesc);
                                    x++;
                                    cx = cur;
                                    cx.next();
                                } else {
                                    mma(1, s0, cur.s, kb == 0);
                                    mma(1, cur.s, s0, false);
                                }
                                umma2_commit(&empty[s0]);
                                umma2_commit(&empty[cur.s]);
                                cur.next();
                            }
                            if (!ok) break;
                            umma2_commit(&accfull[1]);
                            fill0++;
                            fill1++;
                        } else {
                            acquire(turn, turn ? fill1 : fill0);
                            for (int kb = 0; kb < nk; kb++) {
                                landed(cur);
                                if (!ok) break;
                                mma(turn, cur.s, cur.s, kb == 0);
                                umma2_commit(&empty[cur.s]);
                                cur.next();
                            }
                            if (!ok) break;
                            umma2_commit(&accfull[turn]);
                            if (turn) fill1++;
                            else fill0++;
                            turn ^= 1;
                        }
                    }
                }
                if (!ok) abort_flag = 1;
                umma2_commit(&mma_done);
                mbar_wait_cluster(&mma_done, 0, p.status, 24);
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(CG_REGS_EPI));
        // ---------------- epilogue warps: lane quarter q of the CTA's 128 rows, column half h
        const int q = warp % 4, h = warp / 4 - 1;
        const uint32_t tq = tmem + ((uint32_t)(32 * q) << 16) + h * 128;
        uint32_t filled = 0;  // parity of accumulator a's fills so far in bit a
        int turn = 0;
        bool ok = true;
        const uint32_t empty_addr[2] = {cluster_map(&accempty[0], 0), cluster_map(&accempty[1], 0)};
        auto wait_full = [&](int a) {
            bool w = true;
            if (lane == 0) w = mbar_wait_cluster(&accfull[a], filled >> a & 1, p.status, 25);
            filled ^= 1u << a;
            ok = __shfl_sync(0xffffffffu, w, 0) && !*(volatile int*)&abort_flag;
            if (!ok) abort_flag = 1;
            tc_fence_after();
        };
        auto release = [&](int a) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(empty_addr[a]);
        };
        // The warp's 128 columns of accumulator a, reduced mod the p in (np, ip), to
        // halves.  TMEM is released once they are in registers: the next unit's
        // products do not wait for the arithmetic.
        auto drain = [&](int a, uint32_t (&r)[64], f32x2 np, f32x2 ip) {
            uint32_t v[4][32];
#pragma unroll
            for (int part = 0; part < 4; part++) tmem_ld32(tq + a * 256 + part * 32, v[part]);
            tmem_ld_wait();
            release(a);
#pragma unroll
            for (int part = 0; part < 4; part++)
#pragma unroll
                for (int i = 0; i < 16; i++)
                    r[part * 16 + i] = crt_halves(crt_mod2(pack2(v[part][2 * i], v[part][2 * i + 1]), np, ip));
        };
        for (int u = pair; u < nunits && ok; u += npairs) {
            const int l = u / ntiles;
            int tm, tn;
            crt_tile(u - l * ntiles, tiles_m, tiles_n, tm, tn);
            const int row = (p.tm0 + tm) * CG_T + (int)rank * 128 + 32 * q + lane;
            const int col0 = (p.tn0 + tn) * CG_T + h * 128;
            const f32x2 np = dup2(-cfg->p[l]), ip = dup2(cfg->invp[l]), uw = dup2(cfg->u[l]);
            int16_t* yrow = p.y + ((int64_t)l * p.rows + (row - p.row0)) * p.ldy + col0;
            // sixteen reduced values times the weight, plus what earlier K chunks
            // left, mod p, to columns c16 .. c16 + 15 of y: one whole 32-byte
            // sector a lane (two 16-byte stores each touched half a sector)
            auto put = [&](int c16, const f32x2 (&c)[8], bool add) {
                if (row >= p.M || col0 + c16 >= p.ldy) return;
                int16_t* dst = yrow + c16;
                f32x2 sum[8];
#pragma unroll
                for (int i = 0; i < 8; i++) sum[i] = 0ull;
                if (add) {
                    const uint4 o0 = reinterpret_cast<const uint4*>(dst)[0], o1 = reinterpret_cast<const uint4*>(dst)[1];
                    const uint32_t old[8] = {o0.x, o0.y, o0.z, o0.w, o1.x, o1.y, o1.z, o1.w};
#pragma unroll
                    for (int i = 0; i < 8; i++)  // signed halves: flip the top bit for the unsigned form
                        sum[i] = crt_floats(old[i] ^ 0x80008000u);
                }
                uint32_t w[8];
#pragma unroll
                for (int i = 0; i < 8; i++) w[i] = crt_halves(crt_mod2(fma2(c[i], uw, sum[i]), np, ip));
                asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst),
                             "r"(w[0] ^ 0x80008000u), "r"(w[1] ^ 0x80008000u), "r"(w[2] ^ 0x80008000u),
                             "r"(w[3] ^ 0x80008000u), "r"(w[4] ^ 0x80008000u), "r"(w[5] ^ 0x80008000u),
                             "r"(w[6] ^ 0x80008000u), "r"(w[7] ^ 0x80008000u)
                             : "memory");
            };
            const bool square = l < nsq;
            const f32x2 nb = dup2(c_crt.m[l].nb[0]), b = dup2(-c_crt.m[l].nb[0]), ib = dup2(c_crt.m[l].inv[0]);
            for (int k0 = 0; k0 < p.nkb && ok; k0 += CG_KB) {
                // both accumulators are reduced to halves first, so TMEM is free again early
                uint32_t xr[64], yr[64];
                const int a = square ? 0 : turn;
                wait_full(a);
                if (!ok) break;
                drain(a, xr, np, ip);
                if (square) {
                    wait_full(1);
                    if (!ok) break;
                    drain(1, yr, nb, ib);
                } else {
                    turn ^= 1;
                }
#pragma unroll
                for (int g = 0; g < 8; g++) {
                    f32x2 c[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) c[i] = crt_floats(xr[g * 8 + i]);
                    if (square) {
#pragma unroll
                        for (int i = 0; i < 8; i++) c[i] = fma2(b, crt_floats(yr[g * 8 + i]), c[i]);
                    }
                    put(g * 16, c, k0 > 0);
                }
                __syncwarp();  // rows past M skip their stores; the TMEM reads are warp-wide
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// ------------------------------------------------------------------ reconstruction
// round(sign mag 2^X) of a 128-bit magnitude (w1, w0), to nearest even.
__device__ __forceinline__ double crt_round(unsigned long long w1, unsigned long long w0, bool neg, int X) {
    if (!w1) {
        if (!w0) return 0.0;
        w1 = w0;
        w0 = 0;
        X -= 64;
    }
    const int z = __clzll((long long)w1);
    const unsigned long long top = z ? (w1 << z) | (w0 >> (64 - z)) : w1;
    const bool sticky = (w0 << z) != 0;
    unsigned long long m = top >> 11;  // 53 bits
    const uint32_t rem = ((uint32_t)top & 0x7FFu) << 1 | (sticky ? 1u : 0u);
    m += rem > 0x800u || (rem == 0x800u && (m & 1ull));
    // value = m 2^(X + 64 - z + 11), m in [2^52, 2^53]
    const int E = X + 75 - z + 1075 - 1;  // biased exponent - 1 of m = 2^52..: the hidden bit adds 1
    if (E >= 0 && E < 2045) {
        const unsigned long long bits = ((unsigned long long)E << 52) + m;
        return __longlong_as_double((long long)(bits | (neg ? 1ull << 63 : 0ull)));
    }
    const double v = (double)m;
    return scale_pow2(neg ? -v : v, X + 75 - z);
}

// The value of one entry from its sum S = C' + q M (words a, each a 64-bit sum
// of the products at its place; scaled by 2^sh): q = round(S / M) from the top
// (0 < S < 25 M: an error of 2^-16 M is far inside what |C'| < 0.497 M leaves),
// C' = S - q M modulo 2^(32 L), rounded once.
template <int L>
__device__ __forceinline__ double crt_value(unsigned long long (&a)[L], const CrtCfg& c, int X) {
    const unsigned long long t = a[L - 1] + (a[L - 2] >> 32);
    const float tf = __uint_as_float(0x4B000000u + (uint32_t)(t >> 14)) - 8388608.0f;
    const uint32_t q = __float_as_uint(__fmaf_rn(tf, c.qinv, 8388608.0f)) - 0x4B000000u;
    uint32_t x[L];
#pragma unroll
    for (int j = 0; j < L; j++) a[j] += (unsigned long long)q * c.NM[j];
#pragma unroll
    for (int j = 0; j < L; j++) {
        x[j] = (uint32_t)a[j];
        if (j + 1 < L) a[j + 1] += a[j] >> 32;
    }
    const bool neg = (int)x[L - 1] < 0;
    if (neg) {
        uint32_t carry = 1;
#pragma unroll
        for (int j = 0; j < L; j++) {
            x[j] = ~x[j] + carry;
            carry = carry && x[j] == 0;
        }
    }
    if (x[L - 1] == 0)  // much cancellation, or zero
        return crt_round((unsigned long long)x[3] << 32 | x[2], (unsigned long long)x[1] << 32 | x[0], neg, X);
    // top 64 bits, 53 of them to nearest even
    const int z = __clz((int)x[L - 1]);
    const uint32_t y3 = __funnelshift_l(x[L - 2], x[L - 1], z), y2 = __funnelshift_l(x[L - 3], x[L - 2], z);
    uint32_t below = (x[L - 3] << z) | x[L - 4];
    if (L == 5) below |= x[0];
    unsigned long long m = ((unsigned long long)y3 << 32 | y2) >> 11;
    const uint32_t rem = (y2 & 0x7FFu) << 1 | (below ? 1u : 0u);
    m += (rem + ((uint32_t)m & 1u)) > 0x800u;  // above half, or half and odd
    const int Y = X + 32 * (L - 2) - z + 11;   // value = m 2^Y, m in [2^52, 2^53]
    const int E = Y + 1074;                    // its exponent field less one (m's top bit adds it)
    if (E >= 0 && E < 2045)
        return __longlong_as_double((long long)((((unsigned long long)E << 52) + m) | (neg ? 1ull << 63 : 0ull)));
    const double v = (double)m;
    return scale_pow2(neg ? -v : v, Y);
}

struct CrtCombineParams {
    int yrow0, row0;     // the first row in y; y's first row in C
    int rows, yrows;     // rows to combine; rows of a plane of y
    int c0, c1, n;       // columns [c0, c1) of C's n (complex: complex columns)
    int64_t half, ldy;   // complex: column of the imaginary half in y
    const int16_t* y;
    const int* ea;
    const int* eb;
    double* C;
    const SplitPlan* plan;
};

// Two adjacent entries of C (X: exponent of the row's unit, eb: the columns').
template <int L>
__device__ __forceinline__ void crt_two(const int16_t* __restrict__ src, int64_t plane, const CrtCfg& c, int X, int eb0,
                                        int eb1, double& out0, double& out1) {
    const int nmod = c.nmod;
    int v[CRT_NB];
#pragma unroll
    for (int l = 0; l < CRT_NB; l++) {
        v[l] = 0;
        if (l < nmod) v[l] = __ldg(reinterpret_cast<const int*>(src));
        src += plane;
    }
    unsigned long long a0[L], a1[L];
#pragma unroll
    for (int j = 0; j < L; j++) a0[j] = a1[j] = 0;
    // a group's residues first become one number modulo P (0 < z < 2^25), so the
    // wide multiplies are per group: 7 x L of them instead of 15 x L
#pragma unroll
    for (int g = 0; g < CRT_NG; g++) {
        int z0 = c.z0[g], z1 = z0;
#pragma unroll
        for (int l = 2 * g; l < (g + 1 < CRT_NG ? 2 * g + 2 : CRT_NB); l++) {
            z0 += (int)(int16_t)(v[l] & 0xffff) * c.c[l];
            z1 += (v[l] >> 16) * c.c[l];
        }
#pragma unroll
        for (int j = 0; j < L; j++) {
            a0[j] += (unsigned long long)(uint32_t)z0 * c.W[g][j];
            a1[j] += (unsigned long long)(uint32_t)z1 * c.W[g][j];
        }
    }
    out0 = crt_value<L>(a0, c, X + eb0);
    out1 = crt_value<L>(a1, c, X + eb1);
}

// Entries j0, j0 + 1 of a row (complex: both parts).
template <int L, bool CPLX>
__device__ __forceinline__ void crt_combine_body(const CrtCombineParams& p, const CrtCfg& c, int row, int j0,
                                                 int ubits, int eb0, int eb1) {
    const int64_t plane = (int64_t)p.yrows * p.ldy;
    const int16_t* src = p.y + (int64_t)(p.yrow0 + row) * p.ldy + j0;
    const int64_t r = p.row0 + p.yrow0 + row;
    const int X = ubits + __ldg(p.ea + r) - c.sh;
    const bool two = j0 + 1 < p.c1;
    if constexpr (!CPLX) {
        double v0, v1;
        crt_two<L>(src, plane, c, X, eb0, eb1, v0, v1);
        double* dst = p.C + r * p.n + j0;
        if (two && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
            *reinterpret_cast<double2*>(dst) = make_double2(v0, v1);
        } else {
            dst[0] = v0;
            if (two) dst[1] = v1;
        }
    } else {
        double2 u0{0, 0}, u1{0, 0};
#pragma unroll 1  // one copy of the code, in 64 registers
        for (int part = 0; part < 2; part++) {
            u0.x = u0.y, u1.x = u1.y;
            crt_two<L>(src + part * p.half, plane, c, X, eb0, eb1, u0.y, u1.y);
        }
        double2* dst = reinterpret_cast<double2*>(p.C) + r * p.n + j0;  // complex buffers are 16-byte aligned
        dst[0] = u0;
        if (two) dst[1] = u1;
    }
}

// Between instruction issue (56 %) and HBM (its nmod int16 planes in, C out): the
// residues go in seven groups, so the wide multiply-adds are 7 instead of 15 per
// word, on 32-bit words without carry shifts.  8192^2: 0.55 ms (2.1 with a wide
// term and a 64-bit division per residue, 0.75 and then 0.68 with 64-bit limbs);
// its 2.5 GB take 0.37.  Two entries a thread fit 64 registers.
// Blocks of blockDim.x x blockDim.y = 256 threads over (columns, rows), two
// entries each along a row of C; blocks stride over the rows.
template <bool CPLX>
__global__ void __launch_bounds__(256, 4) k_crt_combine(const __grid_constant__ CrtCombineParams p) {
    __shared__ CrtCfg c;
    chain_wait();
    chain_trigger();
    if (p.plan->nonfinite) return;
    {
        const int* src = reinterpret_cast<const int*>(crt_dev.cfg + p.plan->crt);
        for (int i = threadIdx.y * blockDim.x + threadIdx.x; i < (int)(sizeof(CrtCfg) / 4); i += 256)
            reinterpret_cast<int*>(&c)[i] = src[i];
    }
    __syncthreads();
    const int ubits = -2 * (4 + 5 * (p.plan->s - 1));
    const int j0 = p.c0 + (int)(blockIdx.x * blockDim.x + threadIdx.x) * 2;
    if (j0 >= p.c1) return;
    const int eb0 = __ldg(p.eb + j0), eb1 = j0 + 1 < p.c1 ? __ldg(p.eb + j0 + 1) : 0;
    for (int row = blockIdx.y * blockDim.y + threadIdx.y; row < p.rows; row += gridDim.y * blockDim.y) {
        if (c.words == 4) crt_combine_body<4, CPLX>(p, c, row, j0, ubits, eb0, eb1);
        else crt_combine_body<5, CPLX>(p, c, row, j0, ubits, eb0, eb1);
    }
}

// ------------------------------------------------------------------ host side
// The cheapest configuration that holds a sum of klen products of F-bit
// integers with its sign (|C'| <= klen 2^(2F) < M / 2), or -1.
static int crt_config(int s, int64_t klen) {
    const CrtTable& T = crt_host;
    const double need = 2.0 * (4 + 5 * (s - 1)) + log2((double)(klen > 1 ? klen : 1)) + 1.01;
    for (int i = 0; i < T.n; i++)
        if (T.cfg[i].bits >= need) return i;
    return -1;
}
}  // namespace
