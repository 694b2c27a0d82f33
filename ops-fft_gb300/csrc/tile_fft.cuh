// tile_fft.cuh - on-chip transforms of any length whose radices are at most
// 16, register to register: the kernel behind every strided ("column") pass
// and every contiguous row of device memory.  Common lengths are compiled in
// (TileSpec, tile_list.h), any other runs on the same code with its length,
// threads and radices as arguments.
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
// thread (no spills but in the odd real modes: 540 bytes of loads R2C, 368 C2R)
// keep 1024 threads per SM, 128 KB of loads when all of
// them load, in CTAs small enough that one's loads overlap another's passes.
// Measured (GB300, share of the measured copy bandwidth, 128 -> 64
// registers): 256 x 263168 columns 232 -> 168 us (0.945), 2310 x 4096 rows
// 53.1 -> 37.5 us (0.594); at 48 registers, with spills, 195 and 36.2 us.
// Against the kernels these sizes used before: 387 and 74 us; 512^3 3D
// 1823 -> 1342 us.  With lengths as arguments two radices cost 46
// instructions a point, three 64, a third of them addresses; compiled in, a
// quarter fewer: 512^3 1033 us (0.92 of the copy rate over its three passes),
// 4096 x 4096 rows 44 us (0.90), 3000 x 4096 R2C 23.2 us (0.63: odd radices,
// the post-process; shared-memory pipe 69 %, issue 40 %).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "butterfly.cuh"
#include "kernel_args.h"
#include "pdl.cuh"
#include "stockham.cuh"

namespace gfft {

// Template mode of an argument-driven kernel for C2C and the even real modes in
// one; TileArgs::io tells which.  Plans whose launches differ in mode (rows and
// columns, the two passes of a long real transform) take it: a launch then
// finds the passes that the one before it ran in the instruction caches, where
// kernels of one mode each are cold every time (us, kernel a mode / this, and
// before the tiles: 2D R2C 115 x 21 x 120 11.0 / 8.8, 9.8; 1 x 875 x 750 16.5 /
// 13.0, 14.7; 3D R2C 32 x 30 x 40 13.4 / 10.8, 11.7; R2C 17150 x 4 14.2 / 10.4,
// 11.3; 100000 x 240 143 / 133, 317).  A lone mode is 2 to 6 % faster on a
// kernel of its own (C2C 360 x 90000 111 / 115, R2C 2100 x 16384 76 / 80).
constexpr int IO_TILE = -1;
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
    // columns, outer twiddle W_{ons*L}^{jm*i} of sample i = j + r*L/R:
    // otw[j*ons + jm] * otw_lo[r*ons + jm], or without otw
    // otw_hi[m >> shift] * otw_lo[m & mask] with m = jm*i, or none
    const float2* otw;
    const float2* otw_hi;
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
    int32_t staged_out;  // columns: the L outputs of a column are contiguous
    int32_t spitch;      // staged_out: shared pitch of one column
    uint32_t M;          // paired columns: columns of an item (see tile_pair)
    int32_t otw_shift;
    int32_t conj_in, conj_out, weight;
    int32_t io;  // IO_TILE: the mode
    float scale;
    const float* wl;     // even C2R rows: per-bin input weights (row c at c*wdist), or nullptr
    int64_t wdist;
};

extern __shared__ __align__(16) float2 tsm[];  // the exchange buffer

struct TileCtx {
    int L, T, tid, ps, em;
    int off;  // of the transform in the exchange buffer
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

// Compile-time shape of a tile (csrc/tile_list.h); TileDyn, L = 0, leaves it
// to the arguments.
struct TileDyn {
    static constexpr int L = 0, T = 0, W = 0, NP = 0;
    static constexpr bool ROWS = false;
    __host__ __device__ static constexpr int ns(int) { return 0; }
    __host__ __device__ static constexpr int nb(int R) { return R >= 16 ? 1 : 16 / R; }
};
template <int L_, int T_, int W_, bool ROWS_, int... Rs>
struct TileSpec {
    static constexpr int L = L_, T = T_, W = W_, NP = sizeof...(Rs);
    static constexpr bool ROWS = ROWS_;
    static constexpr int R[NP] = {Rs...};
    __host__ __device__ static constexpr int ns(int p)
    {
        int n = 1;
        for (int i = 0; i < p; ++i) n *= R[i];
        return n;
    }
    __host__ __device__ static constexpr int nb(int R) { return (L / R + T - 1) / T; }  // butterflies a thread
    __host__ __device__ static constexpr int shift()
    {
        int k = 0;
        while ((1 << k) < R[0]) ++k;
        return NP > 1 && (1 << k) == R[0] ? k : 30;
    }
};

// One pass: radix R, up to 16 / R butterflies per thread, all their inputs
// in registers before any output is written.
template <int R, int IO, class OFF, bool FIRST, bool LAST, class S = TileDyn, int P = 0>
__device__ __forceinline__ void tile_pass(const TileArgs& A, const TileCtx& c, int p, bool to_global)
{
    constexpr int NB = S::nb(R);
    constexpr bool ST = S::L > 0;
    const PassDesc& pd = A.ip.pass[p];
    const int nbf = c.L / R;
    const int ns = ST ? S::ns(P) : pd.ns;
    const bool staged = !(ST && S::ROWS) && A.staged_out;
    const int64_t in_st8 = ST && S::ROWS ? 8 : A.in_st8, out_st8 = ST && S::ROWS ? 8 : A.out_st8;
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
            const OFF st = (OFF)nbf * (OFF)in_st8;
            sfor<NB>([&](auto bb) {
                constexpr int b = decltype(bb)::value;
                const int j = c.tid + b * c.T;
                if (c.ok && j < nbf) {
                    const OFF g = (OFF)j * (OFF)in_st8;
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
            if (!(ST && S::ROWS) && A.otw) {
                sfor<NB>([&](auto bb) {
                    constexpr int b = decltype(bb)::value;
                    const int j = c.tid + b * c.T;
                    if (c.ok && j < nbf) {
                        const float2 wa = ldg2(A.otw + c.jm + (int64_t)j * A.ons.d);
                        const float2* wb = A.otw_lo + c.jm;
                        v[b * R] = cmul(v[b * R], wa);
                        sfor<R - 1>([&](auto rr) {
                            constexpr int r = decltype(rr)::value + 1;
                            v[b * R + r] = cmul(v[b * R + r], cmul(wa, ldg2(wb + r * A.ons.d)));
                        });
                    }
                });
            } else if (!(ST && S::ROWS) && A.otw_hi) {
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
            const int s = c.off + (j + (j >> c.ps)) * c.em;
            sfor<R>([&](auto rr) {
                constexpr int r = decltype(rr)::value;
                v[b * R + r] = tsm[s + r * rs];
            });
        });
        if (!LAST || !to_global) __syncthreads();  // in place: every read precedes any write
    }
    sfor<NB>([&](auto bb) {
        constexpr int b = decltype(bb)::value;
        const int j = c.tid + b * c.T;
        if (c.ok && j < nbf) {
            int q = j, k = 0;
            if (ns > 1) {
                q = ST ? j / ns : fdiv(j, pd);
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
                if (LAST && staged) {
                    base = c.c * A.spitch + j;
                    ws = ns;
                } else {
                    const int i0 = q * ns * R + k;
                    base = c.off + (i0 + (i0 >> c.ps)) * c.em;
                    ws = (ns == 1 ? 1 : ns + (ns >> c.ps)) * c.em;
                }
                sfor<R>([&](auto rr) {
                    constexpr int r = decltype(rr)::value;
                    tsm[base + r * ws] = v[b * R + r];
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
                const OFF g = (OFF)j * (OFF)out_st8;
                const OFF st = (OFF)ns * (OFF)out_st8;
                const float2 sc = make_float2(A.scale, A.conj_out ? -A.scale : A.scale);
                sfor<R>([&](auto rr) {
                    constexpr int r = decltype(rr)::value;
                    tst(c.go, g + r * st, pmul(v[b * R + r], sc));
                });
            }
        }
    });
}

#define GFFT_TILE_CASE(RV, P, FIRST, LAST) \
    case RV: tile_pass<RV, IO, OFF, FIRST, LAST>(A, c, P, direct); break;
#define GFFT_TILE_SWITCH(P, FIRST, LAST)         \
    switch (A.ip.pass[P].radix) {                \
        GFFT_TILE_CASE(1, P, FIRST, LAST) \
        GFFT_TILE_CASE(2, P, FIRST, LAST) \
        GFFT_TILE_CASE(3, P, FIRST, LAST) \
        GFFT_TILE_CASE(4, P, FIRST, LAST) \
        GFFT_TILE_CASE(5, P, FIRST, LAST) \
        GFFT_TILE_CASE(6, P, FIRST, LAST) \
        GFFT_TILE_CASE(7, P, FIRST, LAST) \
        GFFT_TILE_CASE(8, P, FIRST, LAST) \
        GFFT_TILE_CASE(9, P, FIRST, LAST) \
        GFFT_TILE_CASE(10, P, FIRST, LAST) \
        GFFT_TILE_CASE(11, P, FIRST, LAST) \
        GFFT_TILE_CASE(12, P, FIRST, LAST) \
        GFFT_TILE_CASE(13, P, FIRST, LAST) \
        GFFT_TILE_CASE(14, P, FIRST, LAST) \
        GFFT_TILE_CASE(15, P, FIRST, LAST) \
        GFFT_TILE_CASE(16, P, FIRST, LAST) \
    default: break;                              \
    }

// Columns of the even real modes come in pairs: a tile holds W/2 neighbouring
// columns u of an item's M and, in its other half, the columns M - u that
// hold their mirror bins, so the even/odd post-process of the last pass (R2C)
// and the Hermitian pre-process of the first one (C2R) happen on chip.  The
// columns 0 and M/2 are their own mirrors and leave theirs empty.
__device__ __forceinline__ bool tile_pair(const TileArgs& A, uint32_t q, uint32_t& item, uint32_t& u, uint32_t& j)
{
    const uint32_t W2 = (uint32_t)A.W >> 1;
    const uint32_t cu = blockIdx.x * W2 + (q & (W2 - 1));
    if (cu >= A.ncols) return false;
    item = tdiv(cu, A.cpi);
    u = cu - item * A.cpi.d;
    if (q < W2) {
        j = u;
        return true;
    }
    j = A.M - u;
    return u != 0 && 2 * u != A.M;
}

template <class S>
struct TileShift {
    static constexpr int value = S::shift();
};

// OFF: byte offsets within one transform, 32 bits (one add per access) unless
// its span needs 64 (columns more than 4 GB long).
template <int MAXT, int MINB, int IO, class OFF = uint32_t, class S = TileDyn>
__global__ void __launch_bounds__(MAXT, MINB) tile_kernel(const __grid_constant__ TileArgs A)
{
    constexpr bool ST = S::L > 0;
    const bool rows = ST ? S::ROWS : A.rows != 0;
    TileCtx c;
    if constexpr (ST) {
        c.L = S::L;
        c.T = S::T;
        c.ps = TileShift<S>::value;
        c.em = S::ROWS ? 1 : S::W;
        c.c = S::ROWS ? threadIdx.x / S::T : threadIdx.x % S::W;
        c.tid = S::ROWS ? threadIdx.x % S::T : threadIdx.x / S::W;
    } else {
        c.L = A.ip.L;
        c.T = A.ip.nthr;
        c.ps = A.pshift;
        c.em = A.emul;
        if (rows) {
            c.c = (int)tdiv(threadIdx.x, A.T);
            c.tid = threadIdx.x - c.c * c.T;
        } else {
            c.c = threadIdx.x & (A.W - 1);
            c.tid = threadIdx.x >> A.wshift;
        }
    }
    const uint32_t c0 = blockIdx.x * (uint32_t)A.W;
    const uint32_t col = c0 + (uint32_t)c.c;
    c.ok = c.c < A.W && c.tid < c.T && col < A.ncols;
    constexpr bool kAny = IO == IO_TILE;
    const int io = kAny ? A.io : IO;
    const bool paired = !rows && (io == IO_R2C_EVEN || io == IO_C2R_EVEN);
    uint32_t item = 0, pu = 0, pj = 0;
    if (paired) c.ok = tile_pair(A, (uint32_t)c.c, item, pu, pj) && c.tid < c.T;
    if (!c.ok) c.c = 0;
    const uint32_t cl = c.ok ? col : 0u;
    c.jm = 0;
    if (rows) {
        c.gi = static_cast<const char*>(A.in) + cl * A.in_dist * (IO == IO_R2C_ODD ? 4 : 8);
        c.go = static_cast<char*>(A.out) + cl * A.out_dist * (IO == IO_C2R_ODD ? 4 : 8);
    } else if (paired) {
        if (!c.ok) item = pj = 0;
        c.gi = static_cast<const char*>(A.in) + 8 * (item * A.in_dist + pj);
        c.go = static_cast<char*>(A.out) + 8 * (item * A.out_dist + pj);
        c.jm = pj;
    } else {
        item = tdiv(cl, A.cpi);
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
    c.off = c.c * A.cmul;
    const int np = ST ? S::NP : A.ip.npass;
    const bool direct = io != IO_R2C_EVEN && ((ST && S::ROWS) || !A.staged_out);  // the last pass stores to HBM
    if constexpr (IO == IO_C2R_EVEN || kAny) {
        // Hermitian pre-process into the exchange buffer, every bin loaded
        // once (see codelet_kernel); the passes then all run from it
        if (io != IO_C2R_EVEN) {
        } else if (!rows) {
            // column u's samples X[u + r*M] and their mirrors X[L - u - r*M]:
            // column M - u, sample Lq-1-r (column 0: its own sample Lq-r;
            // r = 0 pairs DC with Nyquist)
            const uint32_t W2 = (uint32_t)A.W >> 1;
            const uint32_t cu = threadIdx.x & (W2 - 1);
            uint32_t it2 = 0, u = 0, j = 0;
            if (tile_pair(A, cu, it2, u, j)) {
                const bool half = A.weight == WEIGHT_LOAD_HALF;
                const bool self = 2 * u == A.M;
                const int Lq = c.L, M = (int)A.M;
                const int rn = u == 0 ? Lq / 2 + 1 : (self ? (Lq + 1) / 2 : Lq);
                const int n = Lq * M;
                const float2* x = static_cast<const float2*>(A.in) + it2 * A.in_dist;
                const int rstep = (int)(blockDim.x / W2);
                // Z'[i] and Z'[n - i] from X[i] and X[n - i]: with W_N^i for
                // every i <= n the upper half needs no case of its own
                auto pre = [&](int r, int rm, uint32_t mo, float2 a, float2 b, float2 w) {
                    if (half) {
                        a = cscale(a, 0.5f);
                        b = cscale(b, 0.5f);
                    }
                    const float2 bc = cconj(b);
                    const float2 ev = cadd(a, bc);
                    const float2 o = cmulc(csub(a, bc), w);
                    float2* s0 = tsm + cu;
                    s0[(r + (r >> c.ps)) * c.em] = cconj(make_float2(ev.x - o.y, ev.y + o.x));
                    s0[(rm + (rm >> c.ps)) * c.em + mo] = cconj(make_float2(ev.x + o.y, -ev.y + o.x));
                };
                int r = (int)(threadIdx.x / W2);
                if (u != 0 && !self) {
                    constexpr int U = 4;  // pairs in flight
                    for (; r + (U - 1) * rstep < Lq; r += U * rstep) {
                        float2 xa[U], xb[U], w[U];
                        sfor<U>([&](auto uu) {
                            constexpr int e = decltype(uu)::value;
                            const uint32_t i = u + (uint32_t)((r + e * rstep) * M);
                            xa[e] = tld(x, 8u * i);
                            xb[e] = tld(x, 8u * (n - i));
                            w[e] = ldg2(A.post + i);
                        });
                        sfor<U>([&](auto uu) {
                            constexpr int e = decltype(uu)::value;
                            pre(r + e * rstep, Lq - 1 - r - e * rstep, W2, xa[e], xb[e], w[e]);
                        });
                    }
                    for (; r < Lq; r += rstep) {
                        const int i = (int)u + r * M;
                        pre(r, Lq - 1 - r, W2, x[i], x[n - i], ldg2(A.post + i));
                    }
                } else {
                    for (; r < rn; r += rstep) {
                        const int i = (int)u + r * M;
                        const float2 a = x[i], b = x[n - i];
                        if (i == 0) {
                            tsm[cu] = make_float2(a.x + b.x, -(a.x - b.x));
                        } else {
                            // (the middle sample is its own mirror: both stores
                            // write the same value, W_N^{n/2} = -i)
                            pre(r, u == 0 ? Lq - r : Lq - 1 - r, 0, a, b, ldg2(A.post + i));
                        }
                    }
                }
            }
        } else if (c.ok) {
            const bool half = A.weight == WEIGHT_LOAD_HALF;
            const float* wl = A.wl ? A.wl + cl * A.wdist : nullptr;
            constexpr int U = 4;  // pairs in flight
            for (int k0 = c.tid; k0 <= (c.L >> 1); k0 += U * c.T) {
                float2 xa[U], xb[U], w[U];
                sfor<U>([&](auto uu) {
                    constexpr int u = decltype(uu)::value;
                    const int k = min(k0 + u * c.T, c.L >> 1);
                    xa[u] = tld(c.gi, 8u * k);
                    xb[u] = tld(c.gi, 8u * (c.L - k));
                    w[u] = ldg2(A.post + k);
                    if (wl) {
                        xa[u] = cscale(xa[u], __ldg(wl + k));
                        xb[u] = cscale(xb[u], __ldg(wl + (c.L - k)));
                    }
                });
                sfor<U>([&](auto uu) {
                    constexpr int u = decltype(uu)::value;
                    const int k = k0 + u * c.T;
                    if (k == 0) {
                        // imaginary parts of DC and Nyquist ignored
                        tsm[c.off] = make_float2(xa[u].x + xb[u].x, -(xa[u].x - xb[u].x));
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
                        tsm[c.off + k + (k >> c.ps)] = cconj(make_float2(e.x - o.y, e.y + o.x));
                        if (n != k) tsm[c.off + n + (n >> c.ps)] = cconj(make_float2(e.x + o.y, -e.y + o.x));
                    }
                });
            }
        }
        if (io == IO_C2R_EVEN) __syncthreads();
    }
    if constexpr (ST) {
        sfor<S::NP>([&](auto pp) {
            constexpr int P = decltype(pp)::value;
            tile_pass<S::R[P], IO, OFF, P == 0 && IO != IO_C2R_EVEN, P == S::NP - 1, S, P>(A, c, P, direct);
            if (P + 1 < S::NP) __syncthreads();
        });
    } else {
        // the first pass of a C2R reads the exchange buffer, as the inner ones do
        int first = 1;
        if constexpr (IO == IO_C2R_EVEN || kAny) {
            if (io == IO_C2R_EVEN) first = 0;
        }
        if (first == 0) {
        } else if (np == 1) {
            GFFT_TILE_SWITCH(0, true, true)
        } else {
            GFFT_TILE_SWITCH(0, true, false)
        }
        if (np > first) {
            if (first) __syncthreads();
            for (int p = first; p + 1 < np; ++p) {
                // opaque per pass: otherwise every radix' loop-invariant
                // address arithmetic is computed ahead of the loop (40
                // instructions an element)
                asm volatile("" : "+r"(c.L), "+r"(c.T), "+r"(c.tid), "+r"(c.em), "+r"(c.ps));
                GFFT_TILE_SWITCH(p, false, false)
                __syncthreads();
            }
            GFFT_TILE_SWITCH(np - 1, false, true)
        }
    }
    if (direct) return;
    __syncthreads();
    if constexpr (IO == IO_C2C || IO == IO_C2R_EVEN || kAny) {
        if (A.staged_out) {
            // a column's outputs are contiguous: consecutive threads write
            // consecutive bins, two at a time where aligned
            const float2 sc = make_float2(A.scale, A.conj_out ? -A.scale : A.scale);
            const int lane = threadIdx.x & 31;
            for (int q = threadIdx.x >> 5; q < A.W; q += blockDim.x >> 5) {
                uint32_t it2 = 0, u = 0, j = 0;
                if (!paired) {
                    if (c0 + q >= A.ncols) break;
                    it2 = tdiv(c0 + q, A.cpi);
                    j = c0 + q - it2 * A.cpi.d;
                } else if (!tile_pair(A, (uint32_t)q, it2, u, j)) {
                    continue;
                }
                float2* g = static_cast<float2*>(A.out) + it2 * A.out_dist + (int64_t)j * c.L;
                const float2* sq = tsm + q * A.spitch;
                if ((reinterpret_cast<uintptr_t>(g) & 15) == 0 && (c.L & 1) == 0) {
#pragma unroll 4
                    for (int k = 2 * lane; k < c.L; k += 64) {
                        const float2 x = pmul(sq[k], sc), y = pmul(sq[k + 1], sc);
                        *reinterpret_cast<float4*>(g + k) = make_float4(x.x, x.y, y.x, y.y);
                    }
                } else {
#pragma unroll 4
                    for (int k = lane; k < c.L; k += 32) g[k] = pmul(sq[k], sc);
                }
            }
        }
    }
    if constexpr (IO == IO_R2C_EVEN || kAny) {
        // even/odd post-process (see codelet_kernel)
        if (io != IO_R2C_EVEN) {
        } else if (!rows) {
            // bins u + M*kk of column u and their mirrors: column M - u, bin
            // Lq-1-kk (column 0: its own bin Lq-kk; kk = 0 is DC and Nyquist)
            const uint32_t W2 = (uint32_t)A.W >> 1;
            const uint32_t cu = threadIdx.x & (W2 - 1);
            uint32_t it2 = 0, u = 0, j = 0;
            if (tile_pair(A, cu, it2, u, j)) {
                const float sc = A.scale;
                const float s2 = A.weight == WEIGHT_STORE_X2 ? 2.f * sc : sc;
                const bool self = 2 * u == A.M;
                const int Lq = c.L, M = (int)A.M;
                const int kn = u == 0 ? Lq / 2 + 1 : (self ? (Lq + 1) / 2 : Lq);
                const int n = Lq * M;
                float2* out = static_cast<float2*>(A.out) + it2 * A.out_dist;
                const float2* s = tsm + cu;
                const int kstep = (int)(blockDim.x / W2);
                auto post = [&](int k, float2 zk, float2 zn, float2 w) {
                    const float2 zc = cconj(zn);
                    const float2 ev = make_float2(0.5f * (zk.x + zc.x), 0.5f * (zk.y + zc.y));
                    const float2 o = make_float2(0.5f * (zk.y - zc.y), 0.5f * (zc.x - zk.x));
                    const float2 wo = cmul(w, o);
                    tst(out, 8u * k, cscale(cadd(ev, wo), s2));
                    if (2 * k != n) tst(out, 8u * (n - k), cscale(cconj(csub(ev, wo)), s2));
                };
                int kk = (int)(threadIdx.x / W2);
                if (u != 0 && !self) {
                    // with W_N^k for every k <= n the upper half needs no
                    // case of its own
                    constexpr int U = 4;  // pairs in flight
                    for (; kk + (U - 1) * kstep < Lq; kk += U * kstep) {
                        float2 za[U], zb[U], w[U];
                        sfor<U>([&](auto uu) {
                            constexpr int e = decltype(uu)::value;
                            const int q = kk + e * kstep, m = Lq - 1 - q;
                            za[e] = s[(q + (q >> c.ps)) * c.em];
                            zb[e] = s[(m + (m >> c.ps)) * c.em + W2];
                            w[e] = ldg2(A.post + (u + (uint32_t)(q * M)));
                        });
                        sfor<U>([&](auto uu) {
                            constexpr int e = decltype(uu)::value;
                            post((int)u + (kk + e * kstep) * M, za[e], zb[e], w[e]);
                        });
                    }
                    for (; kk < Lq; kk += kstep) {
                        const int m = Lq - 1 - kk, k = (int)u + kk * M;
                        post(k, s[(kk + (kk >> c.ps)) * c.em], s[(m + (m >> c.ps)) * c.em + W2], ldg2(A.post + k));
                    }
                } else {
                    for (; kk < kn; kk += kstep) {
                        const int m = u == 0 ? (kk ? Lq - kk : 0) : Lq - 1 - kk, k = (int)u + kk * M;
                        const float2 zk = s[(kk + (kk >> c.ps)) * c.em], zn = s[(m + (m >> c.ps)) * c.em];
                        if (k == 0) {
                            out[0] = make_float2((zk.x + zk.y) * sc, 0.f);
                            out[n] = make_float2((zk.x - zk.y) * sc, 0.f);
                        } else {
                            post(k, zk, zn, ldg2(A.post + k));
                        }
                    }
                }
            }
        } else if (c.ok) {
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
                    za[u] = tsm[c.off + k + (k >> c.ps)];
                    zb[u] = tsm[c.off + n + (n >> c.ps)];
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
