// dtile.cu - double-precision transforms that fit one CTA: a whole axis in one
// launch, register to register with exchanges through shared memory (the
// scheme of tile_fft.cuh on double2), with the even/odd post-process of a D2Z
// and the Hermitian pre-process of a Z2D on chip.
//
// What bounds it: GB300's FP64 pipe, a small fraction of its FP32 rate: 82 %
// busy (D2Z 3000 x 2048).  The one-launch-per-radix passes of dfft.cu kept it 78 %
// busy and wrote every intermediate to HBM.  Here a warp instruction's lanes are what counts:
// butterflies of several rows share warps (1000 points, 100 butterflies a
// pass: 3.2 warps' worth instead of 4).  Measured, one launch per radix ->
// this: Z2Z 4096 x 2048 912 -> 689 us, 1000 x 4096 415 -> 362 (398 with a row
// to every warp group), 300 x 1280 42 -> 33, D2Z 3000 x 2048 394 -> 320, Z2D
// 372 -> 333, Z2Z 1500 x 64 51 -> 27.  Registers and residency make no
// difference (80, 64 or 128 registers: 688, 691, 700 us), although 80 spill
// (272 bytes of stack, 2.3 KB of loads over all radices).  Columns: 2D Z2Z 1024^2
// 228 -> 165, 500 x 16 x 64 60 -> 48 (32 columns; 93 with 8).
#include <cuda_runtime.h>
#include <stdint.h>

#include "butterfly.cuh"
#include "kernel_args.h"
#include "launch_common.cuh"
#include "pdl.cuh"
#include "stockham.cuh"
#include "tile_fft.cuh"

namespace gfft {
namespace {

struct DTileArgs {
    DPassArgs a;
    TileDiv in_split, out_split, half;  // half: L/2 + 1 pairs of a row
    TileDiv nbf[kRagMaxPass];           // rows: butterflies of a row per pass
    int32_t wshift, emul, cmul;
};

extern __shared__ __align__(16) double2 dsm[];

struct DCtx {
    int L, T, ps, em;
    int nt;      // transforms of this CTA
    int64_t t0;  // the first of them
};

// Butterfly b of this thread in a pass: its transform's exchange offset and
// first elements, and its index j within the transform.  A warp instruction
// costs the FP64 pipe the same with 1 or 32 active lanes, so rows spread the
// butterflies of all of the CTA's rows over its threads.
struct DBf {
    bool act;
    int j, off;
    int64_t ib, ob;  // first element of the input and output (their units)
};

__device__ __forceinline__ DBf dbutterfly(const DTileArgs& A, const DCtx& c, int idx, const TileDiv& per)
{
    DBf f;
    int cc;
    if (A.a.t_fast) {
        cc = idx & (A.a.W - 1);
        f.j = idx >> A.wshift;
        f.act = cc < c.nt && f.j < (int)per.d;
        f.j = min(f.j, (int)per.d - 1);
    } else {
        cc = (int)tdiv((uint32_t)idx, per);
        f.j = idx - cc * (int)per.d;
        f.act = cc < c.nt;
    }
    if (cc >= c.nt) cc = 0;
    f.off = cc * A.cmul;
    const uint32_t tt = (uint32_t)(c.t0 + cc);
    const uint32_t th = tdiv(tt, A.in_split), oh = tdiv(tt, A.out_split);
    f.ib = th * A.a.in_hi + (tt - th * A.in_split.d) * A.a.in_lo;
    f.ob = oh * A.a.out_hi + (tt - oh * A.out_split.d) * A.a.out_lo;
    return f;
}

__device__ __forceinline__ void dstore(const DPassArgs& a, int64_t o, double2 e)
{
    if (a.io & DIO_PAIR_OUT) {
        double* y = static_cast<double*>(a.out) + 2 * o;
        y[0] = e.x;
        y[1] = e.y;
    } else {
        static_cast<double2*>(a.out)[o] = e;
    }
}

template <int R, bool FIRST, bool LAST>
__device__ __forceinline__ void dtile_pass(const DTileArgs& A, const DCtx& c, int p, bool to_global)
{
    const DPassArgs& a = A.a;
    constexpr int NB = R >= kDTileElems ? 1 : kDTileElems / R;
    const PassDesc& pd = a.ip.pass[p];
    const int nbf = c.L / R, ns = pd.ns;
    double2 v[NB * R];
    if constexpr (FIRST) {
        sfor<NB>([&](auto bb) {
            constexpr int b = decltype(bb)::value;
            const DBf f = dbutterfly(A, c, threadIdx.x + b * c.T, A.nbf[p]);
            const int j = f.j;
            if (f.act) {
                if (a.io & DIO_REAL_IN) {
                    const double* x = static_cast<const double*>(a.in) + f.ib;
                    sfor<R>([&](auto rr) {
                        constexpr int r = decltype(rr)::value;
                        v[b * R + r] = make_double2(x[(int64_t)(j + r * nbf) * a.in_stride], 0.0);
                    });
                } else if (a.io & DIO_HERM_IN) {
                    // conj of the Hermitian extension: conj(X[i]) for i <= n/2, X[n-i] above
                    const double2* x = static_cast<const double2*>(a.in) + f.ib;
                    sfor<R>([&](auto rr) {
                        constexpr int r = decltype(rr)::value;
                        const int i = j + r * nbf;
                        v[b * R + r] = (2 * i <= c.L) ? cconj(x[(int64_t)i * a.in_stride])
                                                      : x[(int64_t)(c.L - i) * a.in_stride];
                    });
                } else if (a.io & DIO_PAIR_IN) {
                    const double* x = static_cast<const double*>(a.in) + 2 * f.ib;
                    sfor<R>([&](auto rr) {
                        constexpr int r = decltype(rr)::value;
                        const int64_t e = 2 * (int64_t)(j + r * nbf);
                        v[b * R + r] = make_double2(x[e], x[e + 1]);
                    });
                } else {
                    const double2* x = static_cast<const double2*>(a.in) + f.ib;
                    sfor<R>([&](auto rr) {
                        constexpr int r = decltype(rr)::value;
                        const double2 e = x[(int64_t)(j + r * nbf) * a.in_stride];
                        v[b * R + r] = a.conj_in ? cconj(e) : e;
                    });
                }
            }
        });
    } else {
        const int rs = (nbf + (nbf >> c.ps)) * c.em;
        sfor<NB>([&](auto bb) {
            constexpr int b = decltype(bb)::value;
            // idle threads read a valid element, not nothing: see tile_pass
            const DBf f = dbutterfly(A, c, threadIdx.x + b * c.T, A.nbf[p]);
            const int s = f.off + (f.j + (f.j >> c.ps)) * c.em;
            sfor<R>([&](auto rr) {
                constexpr int r = decltype(rr)::value;
                v[b * R + r] = dsm[s + r * rs];
            });
        });
        if (!LAST || !to_global) __syncthreads();  // in place: every read precedes any write
    }
    sfor<NB>([&](auto bb) {
        constexpr int b = decltype(bb)::value;
        const DBf f = dbutterfly(A, c, threadIdx.x + b * c.T, A.nbf[p]);
        const int j = f.j;
        if (f.act) {
            int q = j, k = 0;
            if (ns > 1) {
                q = fdiv(j, pd);
                k = j - q * ns;
                const double2* tw = static_cast<const double2*>(a.tw);
                const int ks = k * (c.L / (ns * R));
                sfor<R - 1>([&](auto rr) {
                    constexpr int r = decltype(rr)::value + 1;
                    v[b * R + r] = cmul(v[b * R + r], __ldg(tw + r * ks));
                });
            }
            DFT<R>::run(&v[b * R]);
            if (!LAST || !to_global) {
                const int i0 = q * ns * R + k;
                const int base = f.off + (i0 + (i0 >> c.ps)) * c.em;
                const int ws = (ns == 1 ? 1 : ns + (ns >> c.ps)) * c.em;
                sfor<R>([&](auto rr) {
                    constexpr int r = decltype(rr)::value;
                    dsm[base + r * ws] = v[b * R + r];
                });
            } else if (a.io & DIO_REAL_OUT) {
                double* y = static_cast<double*>(a.out) + f.ob;
                sfor<R>([&](auto rr) {
                    constexpr int r = decltype(rr)::value;
                    y[(int64_t)(j + r * ns) * a.out_stride] = v[b * R + r].x * a.scale;
                });
            } else {
                const bool half = (a.io & DIO_HALF_OUT) != 0;
                sfor<R>([&](auto rr) {
                    constexpr int r = decltype(rr)::value;
                    const int o = j + r * ns;
                    if (!half || 2 * o <= c.L) {
                        double2 e = a.conj_out ? cconj(v[b * R + r]) : v[b * R + r];
                        if (a.scale != 1.0) e = cscale(e, a.scale);
                        dstore(a, f.ob + (int64_t)o * a.out_stride, e);
                    }
                });
            }
        }
    });
}

#define GFFT_DT_CASE(RV, P, FIRST, LAST) \
    case RV: dtile_pass<RV, FIRST, LAST>(A, c, P, direct); break;
#define GFFT_DT_SWITCH(P, FIRST, LAST)   \
    switch (a.ip.pass[P].radix) {        \
        GFFT_DT_CASE(1, P, FIRST, LAST) \
        GFFT_DT_CASE(2, P, FIRST, LAST) \
        GFFT_DT_CASE(3, P, FIRST, LAST) \
        GFFT_DT_CASE(4, P, FIRST, LAST) \
        GFFT_DT_CASE(5, P, FIRST, LAST) \
        GFFT_DT_CASE(6, P, FIRST, LAST) \
        GFFT_DT_CASE(7, P, FIRST, LAST) \
        GFFT_DT_CASE(8, P, FIRST, LAST) \
        GFFT_DT_CASE(9, P, FIRST, LAST) \
        GFFT_DT_CASE(10, P, FIRST, LAST) \
        GFFT_DT_CASE(11, P, FIRST, LAST) \
        GFFT_DT_CASE(12, P, FIRST, LAST) \
        GFFT_DT_CASE(13, P, FIRST, LAST) \
        GFFT_DT_CASE(14, P, FIRST, LAST) \
        GFFT_DT_CASE(15, P, FIRST, LAST) \
        GFFT_DT_CASE(16, P, FIRST, LAST) \
    default: break;                      \
    }

__global__ void __launch_bounds__(kDTileThreads, 3) dtile_kernel(const __grid_constant__ DTileArgs A)
{
    const DPassArgs& a = A.a;
    DCtx c;
    c.L = a.n;
    c.T = blockDim.x;
    c.ps = a.pshift;
    c.em = A.emul;
    c.t0 = (int64_t)blockIdx.x * a.W;
    c.nt = (int)(a.ntf - c.t0 < a.W ? a.ntf - c.t0 : a.W);
    pdl_wait();  // every access below may touch the caller's buffers
    const int np = a.ip.npass;
    const bool pre = (a.io & DIO_C2R_PRE) != 0, direct = !(a.io & DIO_R2C_POST);
    if (pre) {
        // Hermitian pre-process (see dreal_kernel) into the exchange buffer
        const double2* w = static_cast<const double2*>(a.post);
        for (int idx = threadIdx.x; idx < c.nt * (int)A.half.d; idx += blockDim.x) {
            const DBf f = dbutterfly(A, c, idx, A.half);
            const double2* x = static_cast<const double2*>(a.in) + f.ib;
            const int k = f.j, n = c.L - k;
            if (k == 0) {
                const double x0 = x[0].x, xl = x[n].x;
                dsm[f.off] = make_double2(x0 + xl, -(x0 - xl));
            } else {
                const double2 xa = x[k], xb = cconj(x[n]);
                const double2 e = cadd(xa, xb);
                const double2 o = cmulc(csub(xa, xb), __ldg(w + k));
                dsm[f.off + k + (k >> c.ps)] = cconj(make_double2(e.x - o.y, e.y + o.x));
                if (n != k) dsm[f.off + n + (n >> c.ps)] = cconj(make_double2(e.x + o.y, -e.y + o.x));
            }
        }
        __syncthreads();
        if (np == 1) {
            GFFT_DT_SWITCH(0, false, true)
        } else {
            GFFT_DT_SWITCH(0, false, false)
        }
    } else if (np == 1) {
        GFFT_DT_SWITCH(0, true, true)
    } else {
        GFFT_DT_SWITCH(0, true, false)
    }
    if (np > 1) {
        __syncthreads();
        for (int p = 1; p + 1 < np; ++p) {
            // opaque per pass, see tile_kernel
            asm volatile("" : "+r"(c.L), "+r"(c.T), "+r"(c.em), "+r"(c.ps));
            GFFT_DT_SWITCH(p, false, false)
            __syncthreads();
        }
        GFFT_DT_SWITCH(np - 1, false, true)
    }
    if (direct) return;
    __syncthreads();
    // even/odd post-process (see dreal_kernel)
    const double2* w = static_cast<const double2*>(a.post);
    const double sc = a.scale;
    for (int idx = threadIdx.x; idx < c.nt * (int)A.half.d; idx += blockDim.x) {
        const DBf f = dbutterfly(A, c, idx, A.half);
        double2* y = static_cast<double2*>(a.out) + f.ob;
        const int k = f.j, n = c.L - k;
        if (k == 0) {
            const double2 z0 = dsm[f.off];
            y[0] = make_double2((z0.x + z0.y) * sc, 0.0);
            y[n] = make_double2((z0.x - z0.y) * sc, 0.0);
        } else {
            const double2 zk = dsm[f.off + k + (k >> c.ps)], zc = cconj(dsm[f.off + n + (n >> c.ps)]);
            const double2 e = make_double2(0.5 * (zk.x + zc.x), 0.5 * (zk.y + zc.y));
            const double2 o = make_double2(0.5 * (zk.y - zc.y), 0.5 * (zc.x - zk.x));
            const double2 wo = cmul(__ldg(w + k), o);
            double2 xk = cadd(e, wo), xn = cconj(csub(e, wo));
            if (sc != 1.0) {
                xk = cscale(xk, sc);
                xn = cscale(xn, sc);
            }
            y[k] = xk;
            if (n != k) y[n] = xn;
        }
    }
}

}  // namespace
}  // namespace gfft

using namespace gfft;

extern "C" int gfft_launch_dtile(const DPassArgs* a, void* stream)
{
    static unsigned long long attr_mask = 0;
    const int threads = a->threads;
    if (a->W < 1 || threads < 32 || threads % 32 || threads > kDTileThreads || a->ip.npass > kRagMaxPass || a->ntf < 1 || a->ntf >= (int64_t(1) << 31) - 64 ||
        a->smem_bytes > kMaxSmemBytes || a->ip.L != a->n)
        return (int)cudaErrorInvalidValue;
    DTileArgs d{};
    d.a = *a;
    d.half = tile_div(a->n / 2 + 1);
    for (int p = 0; p < a->ip.npass; ++p) d.nbf[p] = tile_div(a->n / a->ip.pass[p].radix);
    // a split at or beyond the transforms never divides
    d.in_split = tile_div(a->in_split < a->ntf ? a->in_split : a->ntf);
    d.out_split = tile_div(a->out_split < a->ntf ? a->out_split : a->ntf);
    if (a->t_fast) {
        while ((1 << d.wshift) < a->W) ++d.wshift;
        if ((1 << d.wshift) != a->W) return (int)cudaErrorInvalidValue;
        d.emul = a->W;
        d.cmul = 1;
    } else {
        d.emul = 1;
        d.cmul = a->pitch;
    }
    const cudaError_t e = ensure_smem_attr(dtile_kernel, attr_mask, (size_t)a->smem_bytes);
    if (e != cudaSuccess) return (int)e;
    const unsigned grid = (unsigned)((a->ntf + a->W - 1) / a->W);
    return (int)launch_pdl(dtile_kernel, dim3(grid), dim3(threads), (size_t)a->smem_bytes,
                           static_cast<cudaStream_t>(stream), d);
}
