// tile_fft.cuh - on-chip transforms of any length whose radices are at most
// 16, register to register: the kernel behind every strided ("column") pass
// and every contiguous row of a length without a compile-time build.
//
// A CTA takes a TILE of W transforms, T threads each, and a thread holds up
// to 16 elements.  The first pass loads its butterflies' inputs straight
// from HBM into registers (all of them in flight at once), the last pass
// stores its outputs straight to HBM; between passes the tile is exchanged
// through shared memory.  So a transform of two or three radices costs one
// or two exchanges, and shared memory holds only the exchange buffer.
//
//   columns: consecutive threads take consecutive columns (W >= 4: 32-byte
//            segments at least), element i of column c at (pad(i)*W + c);
//   rows:    consecutive threads walk along a row, element i of row c at
//            (c*pitch + pad(i)).
//
// pad(i) = i + (i >> s) with 2^s the first radix when that is a power of
// two, no padding when it is odd: the first pass writes R0 consecutive
// elements per thread, so its threads' addresses step by R0 + 1 (or by an
// odd R0) and hit different banks, and because every later radix' input
// stride L/R and output stride ns are multiples of R0 the padded addresses
// of one butterfly's elements are again an arithmetic sequence: one add per
// element, whatever the length.
//
// What bounds it: latency, hidden by resident threads.  64 registers a
// thread (no spills) keep 1024 threads per SM, 128 KB of loads when all of
// them load, in CTAs small enough that one's loads overlap another's passes.
// Measured (GB300, share of the measured copy bandwidth, 128 -> 64
// registers): 256 x 263168 columns 232 -> 168 us (0.945), 2310 x 4096 rows
// 53.1 -> 37.5 us (0.594); at 48 registers, with spills, 195 and 36.2 us.
// Against the kernels these sizes used before: 387 and 74 us; 512^3 3D
// 1823 -> 1342 us.  Three radices cost 45 instructions an element, a third
// of them addresses, and run at 0.6-0.88; two radices at 0.85-0.97.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "butterfly.cuh"
#include "kernel_args.h"
#include "pdl.cuh"
#include "stockham.cuh"

namespace gfft {

constexpr int kTileMaxThreads = 512;  // per CTA; two such CTAs per SM, 64 registers a thread

// n / d for n < 2^31 (host-made, see tile_div)
struct TileDiv {
    uint32_t d, mul, shift;
};
inline TileDiv tile_div(int64_t d)
{
    TileDiv f{(uint32_t)d, 1u, 0u};
    while ((int64_t(1) << f.shift) < d) ++f.shift;
    f.mul = (uint32_t)((((uint64_t(1) << f.shift) - (uint64_t)d) << 32) / (uint64_t)d + 1);
    return f;
}
__device__ __forceinline__ uint32_t tdiv(uint32_t n, const TileDiv& f) { return (__umulhi(n, f.mul) + n) >> f.shift; }

struct TileArgs {
    InnerPlan ip;
    const float2* tw;
    const float2* post;      // W_N^k, k <= L/2 (even real modes)
    const float2* otw;       // columns: W_{ons*L}^{i*jm} at i*ons + jm, or nullptr
    const float2* otw_hi;    // columns: the same as a product of two tables, or nullptr
    const float2* otw_lo;
    const void* in;
    void* out;
    uint32_t ncols;
    TileDiv cpi, in_split, out_split, tw_div, ons, T;
    int64_t in_st8, out_st8;  // bytes between a transform's elements
    int64_t in_dist, in_hi, in_lo;  // elements
    int64_t out_dist, out_hi, out_lo;
    int32_t W, wshift;   // transforms per tile; columns: log2 W
    int32_t rows;        // 1: rows, 0: columns
    int32_t emul, cmul;  // shared index of element i of transform c: pad(i)*emul + c*cmul
    int32_t pshift;
    int32_t bufsz;       // float2 per exchange buffer
    int32_t nbuf;        // exchange buffers (1: one more barrier per inner pass)
    int32_t staged_out;  // columns: output of column c is out + c*L + k
    int32_t spitch;      // staged_out: shared pitch of one column
    int32_t otw_shift;
    int32_t conj_in, conj_out, weight, nreal;
    float scale;
};

struct TileCtx {
    int L, T, tid, ps, em;
    bool ok;
    const char* gi;  // the transform's input and output
    char* go;
    unsigned jm;  // columns: outer twiddle index of the column
    int c;
};

// Data accesses at a byte offset: plain loads, not the read-only path, since
// in-place passes write what they read and a dependent launch may start
// before its producer ends.
template <class OFF>
__device__ __forceinline__ float2 tld(const void* base, OFF off)
{
    return *reinterpret_cast<const float2*>(static_cast<const char*>(base) + off);
}
template <class OFF>
__device__ __forceinline__ float tld1(const void* base, OFF off)
{
    return *reinterpret_cast<const float*>(static_cast<const char*>(base) + off);
}
template <class OFF>
__device__ __forceinline__ void tst(void* base, OFF off, float2 x)
{
    *reinterpret_cast<float2*>(static_cast<char*>(base) + off) = x;
}

// One pass: radix R, up to 16 / R butterflies per thread, all their inputs
// in registers before any output is written.
template <int R, int IO, class OFF, bool FIRST, bool LAST>
__device__ __forceinline__ void tile_pass(const TileArgs& A, const TileCtx& c, int p, const float2* src, float2* dst,
                                          bool mid_sync, bool to_global)
{
    constexpr int NB = R >= 16 ? 1 : 16 / R;
    const PassDesc& pd = A.ip.pass[p];
    const int nbf = c.L / R;
    const int ns = pd.ns;
    float2 v[NB * R];
    if constexpr (FIRST) {
        if constexpr (IO == IO_R2C_ODD) {
            sfor<NB>([&](auto bb) {
                constexpr int b = decltype(bb)::value;
                const int j = c.tid + b * c.T;
                if (c.ok && j < nbf) {
                    sfor<R>([&](auto rr) {
                        constexpr int r = decltype(rr)::value;
                        v[b * R + r] = make_float2(tld1(c.gi, 4u * (j + r * nbf)), 0.f);
                    });
                }
            });
        } else if constexpr (IO == IO_C2R_ODD) {
            // Hermitian expansion of bins 0..N/2, conjugated
            const int h = c.L >> 1;
            const bool half = A.weight == WEIGHT_LOAD_HALF;
            sfor<NB>([&](auto bb) {
                constexpr int b = decltype(bb)::value;
                const int j = c.tid + b * c.T;
                if (c.ok && j < nbf) {
                    sfor<R>([&](auto rr) {
                        constexpr int r = decltype(rr)::value;
                        const int i = j + r * nbf;
                        v[b * R + r] = tld(c.gi, 8u * (i <= h ? i : c.L - i));
                    });
                    sfor<R>([&](auto rr) {
                        constexpr int r = decltype(rr)::value;
                        const int i = j + r * nbf;
                        const float s = half && i != 0 ? 0.5f : 1.f;
                        v[b * R + r] = pmul(v[b * R + r], make_float2(s, i <= h ? -s : s));
                    });
                }
            });
        } else {
            const OFF st = (OFF)nbf * (OFF)A.in_st8;
            sfor<NB>([&](auto bb) {
                constexpr int b = decltype(bb)::value;
                const int j = c.tid + b * c.T;
                if (c.ok && j < nbf) {
                    const OFF g = (OFF)j * (OFF)A.in_st8;
                    sfor<R>([&](auto rr) {
                        constexpr int r = decltype(rr)::value;
                        v[b * R + r] = tld(c.gi, g + r * st);
                    });
                }
            });
            if (A.conj_in) {
                sfor<NB * R>([&](auto ii) {
                    constexpr int i = decltype(ii)::value;
                    v[i].y = -v[i].y;
                });
            }
            if (A.otw) {
                const int64_t ws = (int64_t)nbf * A.ons.d;
                sfor<NB>([&](auto bb) {
                    constexpr int b = decltype(bb)::value;
                    const int j = c.tid + b * c.T;
                    if (c.ok && j < nbf) {
                        const float2* w = A.otw + (c.jm + (int64_t)j * A.ons.d);
                        sfor<R>([&](auto rr) {
                            constexpr int r = decltype(rr)::value;
                            v[b * R + r] = cmul(v[b * R + r], ldg2(w + r * ws));
                        });
                    }
                });
            } else if (A.otw_hi) {
                const unsigned mask = (1u << A.otw_shift) - 1u;
                sfor<NB>([&](auto bb) {
                    constexpr int b = decltype(bb)::value;
                    const int j = c.tid + b * c.T;
                    if (c.ok && j < nbf) {
                        sfor<R>([&](auto rr) {
                            constexpr int r = decltype(rr)::value;
                            const unsigned m = c.jm * (unsigned)(j + r * nbf);
                            v[b * R + r] =
                                cmul(v[b * R + r], cmul(ldg2(A.otw_hi + (m >> A.otw_shift)), ldg2(A.otw_lo + (m & mask))));
                        });
                    }
                });
            }
        }
    } else {
        const int rs = (nbf + (nbf >> c.ps)) * c.em;
        sfor<NB>([&](auto bb) {
            constexpr int b = decltype(bb)::value;
            // clamped, not guarded: a value left undefined in some threads
            // would be carried around the loop over the passes, for every
            // radix (1.4 KB of stack a thread)
            const int j = min(c.tid + b * c.T, nbf - 1);
            const float2* s = src + (j + (j >> c.ps)) * c.em;
            sfor<R>([&](auto rr) {
                constexpr int r = decltype(rr)::value;
                v[b * R + r] = s[r * rs];
            });
        });
        if (mid_sync) __syncthreads();
    }
    sfor<NB>([&](auto bb) {
        constexpr int b = decltype(bb)::value;
        const int j = c.tid + b * c.T;
        if (c.ok && j < nbf) {
            int q = j, k = 0;
            if (ns > 1) {
                q = fdiv(j, pd);
                k = j - q * ns;
                const float2* w = A.tw + pd.tw_off + k;
                sfor<R - 1>([&](auto rr) {
                    constexpr int r = decltype(rr)::value + 1;
                    v[b * R + r] = cmul(v[b * R + r], ldg2(w + r * ns));
                });
            }
            DFT<R>::run(&v[b * R]);
            if (!LAST || !to_global) {
                int base, ws;
                if (LAST && A.staged_out) {
                    base = c.c * A.spitch + j - c.c;  // dst already points at column c
                    ws = ns;
                } else {
                    const int i0 = q * ns * R + k;
                    base = (i0 + (i0 >> c.ps)) * c.em;
                    ws = (ns == 1 ? 1 : ns + (ns >> c.ps)) * c.em;
                }
                sfor<R>([&](auto rr) {
                    constexpr int r = decltype(rr)::value;
                    dst[base + r * ws] = v[b * R + r];
                });
            } else if constexpr (IO == IO_R2C_ODD) {
                const int h = c.L >> 1;
                sfor<R>([&](auto rr) {
                    constexpr int r = decltype(rr)::value;
                    const int i = j + r * ns;
                    if (i <= h)
                        tst(c.go, 8u * i,
                            cscale(v[b * R + r], (A.weight == WEIGHT_STORE_X2 && i != 0) ? 2.f * A.scale : A.scale));
                });
            } else if constexpr (IO == IO_C2R_ODD) {
                sfor<R>([&](auto rr) {
                    constexpr int r = decltype(rr)::value;
                    *reinterpret_cast<float*>(c.go + 4 * (j + r * ns)) =
                        v[b * R + r].x * A.scale;
                });
            } else {
                const OFF g = (OFF)j * (OFF)A.out_st8;
                const OFF st = (OFF)ns * (OFF)A.out_st8;
                const float2 sc = make_float2(A.scale, A.conj_out ? -A.scale : A.scale);
                sfor<R>([&](auto rr) {
                    constexpr int r = decltype(rr)::value;
                    tst(c.go, g + r * st, pmul(v[b * R + r], sc));
                });
            }
        }
    });
}

#define GFFT_TILE_CASE(RV, P, FIRST, LAST, DST, MID) \
    case RV: tile_pass<RV, IO, OFF, FIRST, LAST>(A, c, P, src, DST, MID, direct); break;
#define GFFT_TILE_SWITCH(P, FIRST, LAST, DST, MID)   \
    switch (A.ip.pass[P].radix) {                    \
        GFFT_TILE_CASE(1, P, FIRST, LAST, DST, MID) \
        GFFT_TILE_CASE(2, P, FIRST, LAST, DST, MID) \
        GFFT_TILE_CASE(3, P, FIRST, LAST, DST, MID) \
        GFFT_TILE_CASE(4, P, FIRST, LAST, DST, MID) \
        GFFT_TILE_CASE(5, P, FIRST, LAST, DST, MID) \
        GFFT_TILE_CASE(6, P, FIRST, LAST, DST, MID) \
        GFFT_TILE_CASE(7, P, FIRST, LAST, DST, MID) \
        GFFT_TILE_CASE(8, P, FIRST, LAST, DST, MID) \
        GFFT_TILE_CASE(9, P, FIRST, LAST, DST, MID) \
        GFFT_TILE_CASE(10, P, FIRST, LAST, DST, MID) \
        GFFT_TILE_CASE(11, P, FIRST, LAST, DST, MID) \
        GFFT_TILE_CASE(12, P, FIRST, LAST, DST, MID) \
        GFFT_TILE_CASE(13, P, FIRST, LAST, DST, MID) \
        GFFT_TILE_CASE(14, P, FIRST, LAST, DST, MID) \
        GFFT_TILE_CASE(15, P, FIRST, LAST, DST, MID) \
        GFFT_TILE_CASE(16, P, FIRST, LAST, DST, MID) \
    default: break;                                  \
    }

// OFF: byte offsets within one transform, 32 bits (one add per access) unless
// its span needs 64 (columns more than 4 GB long).
template <int MAXT, int MINB, int IO, class OFF = uint32_t>
__global__ void __launch_bounds__(MAXT, MINB) tile_kernel(const __grid_constant__ TileArgs A)
{
    extern __shared__ __align__(16) float2 tsm[];
    TileCtx c;
    c.L = A.ip.L;
    c.T = A.ip.nthr;
    c.ps = A.pshift;
    c.em = A.emul;
    if (A.rows) {
        c.c = (int)tdiv(threadIdx.x, A.T);
        c.tid = threadIdx.x - c.c * c.T;
    } else {
        c.c = threadIdx.x & (A.W - 1);
        c.tid = threadIdx.x >> A.wshift;
    }
    const uint32_t c0 = blockIdx.x * (uint32_t)A.W;
    const uint32_t col = c0 + (uint32_t)c.c;
    c.ok = c.c < A.W && c.tid < c.T && col < A.ncols;
    if (!c.ok) c.c = 0;
    const uint32_t cl = c.ok ? col : 0u;
    c.jm = 0;
    if (A.rows) {
        c.gi = static_cast<const char*>(A.in) + cl * A.in_dist * (IO == IO_R2C_ODD ? 4 : 8);
        c.go = static_cast<char*>(A.out) + cl * A.out_dist * (IO == IO_C2R_ODD ? 4 : 8);
    } else {
        const uint32_t item = tdiv(cl, A.cpi);
        const uint32_t j = cl - item * A.cpi.d;
        const uint32_t jh = tdiv(j, A.in_split), oh = tdiv(j, A.out_split);
        c.gi = static_cast<const char*>(A.in) + 8 * (item * A.in_dist + jh * A.in_hi + (j - jh * A.in_split.d) * A.in_lo);
        c.go = static_cast<char*>(A.out) + 8 * (item * A.out_dist + oh * A.out_hi + (j - oh * A.out_split.d) * A.out_lo);
        if (A.ons.d > 1) {
            const uint32_t jd = tdiv(j, A.tw_div);
            c.jm = jd - tdiv(jd, A.ons) * A.ons.d;
        }
    }
    pdl_wait();  // every access below may touch the caller's buffers
    const int off = c.c * A.cmul;
    const int np = A.ip.npass;
    const bool direct = IO != IO_R2C_EVEN && !A.staged_out;  // the last pass stores to HBM
    float2* src = tsm + off;
    float2* alt = tsm + (A.nbuf == 2 ? A.bufsz : 0) + off;
    if constexpr (IO == IO_C2R_EVEN) {
        // Hermitian pre-process into the exchange buffer, every bin loaded
        // once (see codelet_kernel); the passes then all run from it
        if (c.ok) {
            const bool half = A.weight == WEIGHT_LOAD_HALF;
            constexpr int U = 4;  // pairs in flight
            for (int k0 = c.tid; k0 <= (c.L >> 1); k0 += U * c.T) {
                float2 xa[U], xb[U], w[U];
                sfor<U>([&](auto uu) {
                    constexpr int u = decltype(uu)::value;
                    const int k = min(k0 + u * c.T, c.L >> 1);
                    xa[u] = tld(c.gi, 8u * k);
                    xb[u] = tld(c.gi, 8u * (c.L - k));
                    w[u] = ldg2(A.post + k);
                });
                sfor<U>([&](auto uu) {
                    constexpr int u = decltype(uu)::value;
                    const int k = k0 + u * c.T;
                    if (k == 0) {
                        // imaginary parts of DC and Nyquist ignored
                        src[0] = make_float2(xa[u].x + xb[u].x, -(xa[u].x - xb[u].x));
                    } else if (k <= (c.L >> 1)) {
                        const int n = c.L - k;
                        float2 a = xa[u], b = xb[u];
                        if (half) {
                            a = cscale(a, 0.5f);
                            b = cscale(b, 0.5f);
                        }
                        const float2 bc = cconj(b);
                        const float2 e = cadd(a, bc);
                        const float2 o = cmulc(csub(a, bc), w[u]);
                        src[k + (k >> c.ps)] = cconj(make_float2(e.x - o.y, e.y + o.x));
                        if (n != k) src[n + (n >> c.ps)] = cconj(make_float2(e.x + o.y, -e.y + o.x));
                    }
                });
            }
        }
        __syncthreads();
        if (np == 1) {
            GFFT_TILE_SWITCH(0, false, true, alt, false)
            return;
        }
        GFFT_TILE_SWITCH(0, false, false, alt, A.nbuf == 1)
        __syncthreads();
        float2* t = src;
        src = alt;
        alt = t;
    } else if (np == 1) {
        GFFT_TILE_SWITCH(0, true, true, src, false)
        if (!direct) __syncthreads();
    } else {
        GFFT_TILE_SWITCH(0, true, false, src, false)
        __syncthreads();
    }
    if (IO == IO_C2R_EVEN || np > 1) {
        for (int p = 1; p + 1 < np; ++p) {
            // opaque per pass: otherwise every radix' loop-invariant address
            // arithmetic is computed ahead of the loop (40 instructions an
            // element)
            asm volatile("" : "+r"(c.L), "+r"(c.T), "+r"(c.tid), "+r"(c.em), "+r"(c.ps));
            GFFT_TILE_SWITCH(p, false, false, alt, A.nbuf == 1)
            __syncthreads();
            float2* t = src;
            src = alt;
            alt = t;
        }
        GFFT_TILE_SWITCH(np - 1, false, true, alt, A.nbuf == 1 && !direct)
        if (!direct) __syncthreads();
        src = alt;
    }
    if constexpr (IO == IO_C2C) {
        if (A.staged_out) {
            // the tile's outputs are one contiguous block: consecutive
            // threads write consecutive bins, two at a time where aligned
            const float2* s = src - off;
            float2* g = static_cast<float2*>(A.out) + (int64_t)c0 * c.L;
            const int ncol = (int)min((uint32_t)A.W, A.ncols - c0);
            const float2 sc = make_float2(A.scale, A.conj_out ? -A.scale : A.scale);
            if ((reinterpret_cast<uintptr_t>(g) & 15) == 0 && (c.L & 1) == 0) {
                for (int q = 0; q < ncol; ++q) {
                    for (int k = 2 * threadIdx.x; k < c.L; k += 2 * blockDim.x) {
                        const float2 x = pmul(s[q * A.spitch + k], sc), y = pmul(s[q * A.spitch + k + 1], sc);
                        *reinterpret_cast<float4*>(g + q * c.L + k) = make_float4(x.x, x.y, y.x, y.y);
                    }
                }
            } else {
                for (int q = 0; q < ncol; ++q)
                    for (int k = threadIdx.x; k < c.L; k += blockDim.x)
                        g[q * c.L + k] = pmul(s[q * A.spitch + k], sc);
            }
        }
    }
    if constexpr (IO == IO_R2C_EVEN) {
        // even/odd post-process (see codelet_kernel)
        if (c.ok) {
            const float sc = A.scale;
            const float s2 = A.weight == WEIGHT_STORE_X2 ? 2.f * sc : sc;
            constexpr int U = 4;  // pairs in flight
            for (int k0 = c.tid; k0 <= (c.L >> 1); k0 += U * c.T) {
                float2 za[U], zb[U], w[U];
                sfor<U>([&](auto uu) {
                    constexpr int u = decltype(uu)::value;
                    const int k = min(k0 + u * c.T, c.L >> 1);
                    const int n = k ? c.L - k : 0;
                    w[u] = ldg2(A.post + k);
                    za[u] = src[k + (k >> c.ps)];
                    zb[u] = src[n + (n >> c.ps)];
                });
                sfor<U>([&](auto uu) {
                    constexpr int u = decltype(uu)::value;
                    const int k = k0 + u * c.T;
                    if (k == 0) {
                        const float2 z0 = za[u];
                        tst(c.go, 0u, make_float2((z0.x + z0.y) * sc, 0.f));
                        tst(c.go, 8u * c.L, make_float2((z0.x - z0.y) * sc, 0.f));
                    } else if (k <= (c.L >> 1)) {
                        const int n = c.L - k;
                        const float2 zk = za[u], zc = cconj(zb[u]);
                        const float2 e = make_float2(0.5f * (zk.x + zc.x), 0.5f * (zk.y + zc.y));
                        const float2 o = make_float2(0.5f * (zk.y - zc.y), 0.5f * (zc.x - zk.x));
                        const float2 wo = cmul(w[u], o);
                        tst(c.go, 8u * k, cscale(cadd(e, wo), s2));
                        if (n != k) tst(c.go, 8u * n, cscale(cconj(csub(e, wo)), s2));
                    }
                });
            }
        }
    }
}
#undef GFFT_TILE_CASE
#undef GFFT_TILE_SWITCH

}  // namespace gfft
