// ragged.cu - ragged batches of transforms in one persistent launch.
//
// Every CTA (512 threads, two per SM) loops over work items claimed from the
// queue head.  An item is a tile of the register-to-register scheme of
// tile_fft.cuh with its lengths, strides, radices and table offsets in a
// 240-byte record:
//
//   RAG_SINGLE  `count` same-length transforms, rows of the tile; even R2C
//               fuses the even/odd post-process, odd R2C reads reals and
//               stores bins k <= n/2;
//   RAG_P1      `count` adjacent columns of a long transform, staged so that
//               the workspace is written in one contiguous block;
//   RAG_P2      `count` adjacent columns of that block's transpose, with the
//               W_n'^{j*i} twiddle on the loads; loads and stores both touch
//               `count` neighbouring elements a row;
//   RAG_POST    a range of the even/odd post-process of a long even R2C.
//
// With eight items or more a CTA the index after the next one is claimed (one
// atomic) and the next record copied (cp.async) while an item is processed; a finished item is published
// after the next item's first barrier, when its stores have drained.  Claims
// ahead cannot deadlock: a CTA's claims increase, and every wait is on lower
// items, so the lowest unfinished item is always being processed.  Waits (P2
// on P1, POST on P2) are done by one thread with a clock bound.  Shorter
// queues are claimed item by item (a CTA that started early took two items
// and left others without: 163 transforms of up to 8192 points 26 -> 21 us),
// and when every item has a CTA and none waits, CTA b takes item b.
//
// What bounds it: issue and latency at 32 warps per SM (issue 30 % active,
// warps waiting on loads 5.9, at barriers 4.6 per issue).  10000 transforms
// of 16..32768 points: 977 -> 415 us against the staged shared-memory passes
// this replaced; 163 of up to 8192, one item a CTA with cold code, 17.0 -> 18.8.
// 64 registers spill (128 bytes of stack, 2.9 KB of loads over all radices).
// Measured and left out: the passes specialised by item kind, with a tenth of
// the spills, 163 transforms 26.7 us, 10000 653 (three copies of them); CTAs of 256 threads, four per SM
// (one length 10 % faster, mixed lengths 516 us); HBM reads started one round
// of the grid ahead with bulk L2 prefetches (515 us); one copy of each radix'
// code for first, inner and last passes (559 us).
#include <cuda_runtime.h>

#include <mutex>

#include "butterfly.cuh"
#include "kernel_args.h"
#include "pipe_ptx.cuh"
#include "stockham.cuh"

namespace gfft {
namespace {

constexpr int NT = 512;  // threads per CTA

struct RagCtx {
    int L, T, tid, ps, em;
    bool ok;
    const char* gi;
    char* go;
    uint32_t in_st, out_st;  // bytes
    int c;                   // transform of the tile
    unsigned jm;             // P2: column
    const float2* tw;
    bool conj_in, conj_out;
    float scale;
};

// One pass (see tile_pass): up to 16 / R butterflies a thread.
template <int R, bool FIRST, bool LAST>
__device__ __forceinline__ void rag_pass(const RagItem& q, const RagCtx& c, int p, float2* buf, bool to_global)
{
    constexpr int NB = R >= 16 ? 1 : 16 / R;
    const int nbf = c.L / R;
    const int ns = q.pass[p].ns;
    float2 v[NB * R];
    if constexpr (FIRST) {
        const uint32_t st = (uint32_t)nbf * c.in_st;
        sfor<NB>([&](auto bb) {
            constexpr int b = decltype(bb)::value;
            const int j = c.tid + b * c.T;
            const bool act = c.ok && j < nbf;
            const char* g = c.gi + (uint32_t)j * c.in_st;
            // zeros, not nothing, in idle threads: see the clamp below
            if ((q.flags & RAG_REAL_IN) && q.kind != RAG_P2) {
                sfor<R>([&](auto rr) {
                    constexpr int r = decltype(rr)::value;
                    v[b * R + r] = make_float2(0.f, 0.f);
                    if (act) v[b * R + r].x = *reinterpret_cast<const float*>(g + r * st);
                });
            } else {
                // past the L1: workspace lines are written by other CTAs
                sfor<R>([&](auto rr) {
                    constexpr int r = decltype(rr)::value;
                    v[b * R + r] = make_float2(0.f, 0.f);
                    if (act) v[b * R + r] = __ldcg(reinterpret_cast<const float2*>(g + r * st));
                });
            }
        });
        if (c.conj_in) {
            sfor<NB * R>([&](auto ii) {
                constexpr int i = decltype(ii)::value;
                v[i].y = -v[i].y;
            });
        }
        if (q.kind == RAG_P2) {
            if (q.otw_shift < 0) {
                // one table read like the data: entry i*La + j
                const float2* w = c.tw + q.hi_off + c.jm;
                sfor<NB>([&](auto bb) {
                    constexpr int b = decltype(bb)::value;
                    const int j = c.tid + b * c.T;
                    if (c.ok && j < nbf) {
                        sfor<R>([&](auto rr) {
                            constexpr int r = decltype(rr)::value;
                            v[b * R + r] = cmul(v[b * R + r], ldg2(w + (j + r * nbf) * q.stride));
                        });
                    }
                });
            } else {
                const float2* hi = c.tw + q.hi_off;
                const float2* lo = c.tw + q.lo_off;
                const int shift = q.otw_shift;
                const unsigned mask = (1u << shift) - 1u;
                sfor<NB>([&](auto bb) {
                    constexpr int b = decltype(bb)::value;
                    const int j = c.tid + b * c.T;
                    if (c.ok && j < nbf) {
                        sfor<R>([&](auto rr) {
                            constexpr int r = decltype(rr)::value;
                            const unsigned e = c.jm * (unsigned)(j + r * nbf);
                            v[b * R + r] = cmul(v[b * R + r], cmul(ldg2(hi + (e >> shift)), ldg2(lo + (e & mask))));
                        });
                    }
                });
            }
        }
    } else {
        const int rs = (nbf + (nbf >> c.ps)) * c.em;
        sfor<NB>([&](auto bb) {
            constexpr int b = decltype(bb)::value;
            const int j = min(c.tid + b * c.T, nbf - 1);  // clamped, not guarded: see tile_pass
            const float2* s = buf + (j + (j >> c.ps)) * c.em;
            sfor<R>([&](auto rr) {
                constexpr int r = decltype(rr)::value;
                v[b * R + r] = s[r * rs];
            });
        });
        if (!LAST || !to_global) __syncthreads();  // in place: every read precedes any write
    }
    sfor<NB>([&](auto bb) {
        constexpr int b = decltype(bb)::value;
        const int j = c.tid + b * c.T;
        if (c.ok && j < nbf) {
            int qq = j, k = 0;
            if (!FIRST) {
                qq = fdiv(j, q.pass[p]);
                k = j - qq * ns;
                const float2* w = c.tw + q.pass[p].tw_off + k;
                sfor<R - 1>([&](auto rr) {
                    constexpr int r = decltype(rr)::value + 1;
                    v[b * R + r] = cmul(v[b * R + r], ldg2(w + r * ns));
                });
            }
            DFT<R>::run(&v[b * R]);
            if (!LAST || !to_global) {
                int base, ws;
                if (LAST && q.kind == RAG_P1) {
                    base = c.c * q.pitch + j - c.c;  // buf already points at column c
                    ws = ns;
                } else {
                    const int i0 = qq * ns * R + k;
                    base = (i0 + (i0 >> c.ps)) * c.em;
                    ws = (FIRST ? 1 : ns + (ns >> c.ps)) * c.em;
                }
                sfor<R>([&](auto rr) {
                    constexpr int r = decltype(rr)::value;
                    buf[base + r * ws] = v[b * R + r];
                });
            } else {
                char* g = c.go + (uint32_t)j * c.out_st;
                const uint32_t st = (uint32_t)ns * c.out_st;
                if (q.flags & RAG_HALF_OUT) {
                    // bin of output r: P2 j' + stride*(j + r*ns), else j + r*ns
                    const int k0 = q.kind == RAG_P2 ? (int)c.jm + q.stride * j : j;
                    const int ks = q.kind == RAG_P2 ? q.stride * ns : ns;
                    sfor<R>([&](auto rr) {
                        constexpr int r = decltype(rr)::value;
                        if (k0 + r * ks <= q.nhalf) *reinterpret_cast<float2*>(g + r * st) = v[b * R + r];
                    });
                } else {
                    const float2 sc = make_float2(c.scale, c.conj_out ? -c.scale : c.scale);
                    sfor<R>([&](auto rr) {
                        constexpr int r = decltype(rr)::value;
                        *reinterpret_cast<float2*>(g + r * st) = pmul(v[b * R + r], sc);
                    });
                }
            }
        }
    });
}

#define GFFT_RAG_CASE(RV, P, FIRST, LAST) \
    case RV: rag_pass<RV, FIRST, LAST>(q, c, P, buf, direct); break;
#define GFFT_RAG_SWITCH(P, FIRST, LAST)   \
    switch (q.pass[P].radix) {            \
        GFFT_RAG_CASE(1, P, FIRST, LAST)  \
        GFFT_RAG_CASE(2, P, FIRST, LAST)  \
        GFFT_RAG_CASE(3, P, FIRST, LAST)  \
        GFFT_RAG_CASE(4, P, FIRST, LAST)  \
        GFFT_RAG_CASE(5, P, FIRST, LAST)  \
        GFFT_RAG_CASE(6, P, FIRST, LAST)  \
        GFFT_RAG_CASE(7, P, FIRST, LAST)  \
        GFFT_RAG_CASE(8, P, FIRST, LAST)  \
        GFFT_RAG_CASE(9, P, FIRST, LAST)  \
        GFFT_RAG_CASE(10, P, FIRST, LAST) \
        GFFT_RAG_CASE(11, P, FIRST, LAST) \
        GFFT_RAG_CASE(12, P, FIRST, LAST) \
        GFFT_RAG_CASE(13, P, FIRST, LAST) \
        GFFT_RAG_CASE(14, P, FIRST, LAST) \
        GFFT_RAG_CASE(15, P, FIRST, LAST) \
        GFFT_RAG_CASE(16, P, FIRST, LAST) \
    default: break;                       \
    }

// Even/odd post-process of an even-length R2C: bins k and L - k from Z[k]
// and Z[L - k], for k0, k0 + step, ... below k1 (k1 <= L/2 + 1), four pairs
// of loads in flight.
template <class GetZ>
__device__ __forceinline__ void r2c_post(GetZ getz, const float2* post, float2* out, int L, int k0, int k1, int step)
{
    constexpr int U = 4;
    for (int kk = k0; kk < k1; kk += U * step) {
        float2 za[U], zb[U], w[U];
        sfor<U>([&](auto uu) {
            constexpr int u = decltype(uu)::value;
            const int k = min(kk + u * step, k1 - 1);
            za[u] = getz(k);
            zb[u] = getz(k ? L - k : 0);
            w[u] = ldg2(post + k);
        });
        sfor<U>([&](auto uu) {
            constexpr int u = decltype(uu)::value;
            const int k = kk + u * step;
            if (k == 0) {
                out[0] = make_float2(za[u].x + za[u].y, 0.f);
                out[L] = make_float2(za[u].x - za[u].y, 0.f);
            } else if (k < k1) {
                const float2 zk = za[u], zc = cconj(zb[u]);
                const float2 e = make_float2(0.5f * (zk.x + zc.x), 0.5f * (zk.y + zc.y));
                const float2 o = make_float2(0.5f * (zk.y - zc.y), 0.5f * (zc.x - zk.x));
                const float2 wo = cmul(w[u], o);
                out[k] = cadd(e, wo);
                if (L - k != k) out[L - k] = cconj(csub(e, wo));
            }
        });
    }
}

// Bounded wait for a completion counter; the acquire load orders the
// caller's later reads (after a CTA barrier) behind the counted items.
__device__ __forceinline__ bool wait_count(int* ctr, int need, int* err, long long budget)
{
    if (budget <= 0) budget = 1ll << 31;
    const long long t0 = clock64();
    for (;;) {
        int v;
        asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
        if (v >= need) return true;
        if (*reinterpret_cast<volatile int*>(err) & 4) return false;
        __nanosleep(128);
        if (clock64() - t0 > budget) {
            atomicOr(err, 4);
            return false;
        }
    }
}

constexpr int kRecChunks = (int)(sizeof(RagItem) / 16);

__global__ void __launch_bounds__(NT, 2) ragged_kernel(const __grid_constant__ RagArgs A)
{
    extern __shared__ __align__(16) float2 tile[];
    __shared__ __align__(16) RagItem s_rec[2];
    __shared__ int s_claim[2];
    __shared__ int s_ok;
    const int t = threadIdx.x;
    if (t == 0) {
        s_claim[0] = A.claim == RAG_CLAIM_NONE ? (int)blockIdx.x : atomicAdd(A.queue, 1);
        s_claim[1] = A.claim == RAG_CLAIM_AHEAD ? atomicAdd(A.queue, 1) : A.nitems;
    }
    __syncthreads();
    int it = s_claim[0], nxt = s_claim[1];
    if (it < A.nitems && t < kRecChunks)
        reinterpret_cast<int4*>(&s_rec[0])[t] = __ldg(reinterpret_cast<const int4*>(A.items + it) + t);
    __syncthreads();
    int pending = -1;  // completed P1 / P2 item not yet published
    for (int cur = 0; it < A.nitems; cur ^= 1) {
        // run ahead: claim the item after the next one, fetch the next record
        int claimed = 0;
        if (t == NT - 1) claimed = A.claim == RAG_CLAIM_AHEAD ? atomicAdd(A.queue, 1) : A.nitems;
        if (t < kRecChunks && nxt < A.nitems)
            cp_async16(reinterpret_cast<unsigned char*>(&s_rec[cur ^ 1]) + 16 * t,
                       reinterpret_cast<const unsigned char*>(A.items + nxt) + 16 * t);
        cp_async_commit();
        const RagItem& q = s_rec[cur];
        bool run = true;
        // thread 0 publishes the previous item: before a wait, else after
        // this item's first barrier, when that item's stores have drained and
        // the fence is cheap
        auto publish = [&]() {
            if (t == 0 && pending >= 0) {
                __threadfence();
                atomicAdd(A.queue + 1 + pending, 1);
            }
            pending = -1;
        };
        if (q.kind >= RAG_P2) {
            publish();
            if (t == 0) s_ok = wait_count(A.queue + 1 + q.xform, q.need + A.need_bias, A.err, A.wait_cycles) ? 1 : 0;
            __syncthreads();
            run = s_ok != 0;
        }
        float2* const ws = static_cast<float2*>(A.ws);
        if (run && q.kind == RAG_POST) {
            const float2* z = ws + q.in_off;
            r2c_post([&](int k) { return __ldcg(z + k); }, static_cast<const float2*>(A.tw) + q.post_off,
                     reinterpret_cast<float2*>(static_cast<char*>(A.out) + q.out_off), q.L, q.first + t,
                     q.first + q.count, NT);
        } else if (run) {
            RagCtx c;
            c.L = q.L;
            c.T = q.T;
            c.ps = q.ps;
            c.tw = static_cast<const float2*>(A.tw);
            const int d = (int)((unsigned)t * q.wmagic >> 20);
            const bool rows = q.kind == RAG_SINGLE;
            if (rows) {
                c.c = d;
                c.tid = t - d * q.T;
                c.em = 1;
            } else {
                c.tid = d;
                c.c = t - d * q.W;
                c.em = q.W;
            }
            c.ok = c.tid < q.T && c.c < q.count;
            if (!c.ok) c.c = 0;
            const bool inv = A.inverse != 0;
            c.conj_in = inv && (q.flags & RAG_CONJ_IN);
            c.conj_out = inv && (q.flags & RAG_CONJ_OUT);
            c.scale = (q.flags & RAG_CONJ_OUT) ? A.scale_c2c : 1.f;
            c.jm = (unsigned)(q.first + c.c);
            const uint32_t ie = (q.flags & RAG_REAL_IN) && q.kind != RAG_P2 ? 4u : 8u;
            float2* buf = tile;
            if (rows) {
                const RagRow r = A.rows[q.first + c.c];
                c.gi = static_cast<const char*>(A.in) + r.in_off;
                c.go = static_cast<char*>(A.out) + r.out_off;
                c.in_st = ie;
                c.out_st = 8;
                buf += c.c * q.pitch;
            } else {
                const char* ib = q.kind == RAG_P1 ? static_cast<const char*>(A.in) + q.in_off
                                                  : reinterpret_cast<const char*>(ws + q.in_off);
                char* ob = (q.flags & RAG_WS_OUT) ? reinterpret_cast<char*>(ws + q.out_off)
                                                  : static_cast<char*>(A.out) + q.out_off;
                c.gi = ib + (size_t)c.jm * ie;
                c.go = ob + (size_t)c.jm * 8;
                c.in_st = (uint32_t)q.stride * ie;
                c.out_st = (uint32_t)q.stride * 8u;
                buf += c.c;
            }
            const bool direct = q.kind != RAG_P1 && !(q.flags & RAG_R2C_POST);
            const int np = q.np;
            if (np == 1) {
                GFFT_RAG_SWITCH(0, true, true)
            } else {
                GFFT_RAG_SWITCH(0, true, false)
                __syncthreads();
                publish();
                for (int p = 1; p + 1 < np; ++p) {
                    asm volatile("" : "+r"(c.L), "+r"(c.T), "+r"(c.tid), "+r"(c.em), "+r"(c.ps));
                    GFFT_RAG_SWITCH(p, false, false)
                    __syncthreads();
                }
                GFFT_RAG_SWITCH(np - 1, false, true)
            }
            if (!direct) __syncthreads();
            if (q.kind == RAG_P1) {
                // `count` columns of L outputs: one contiguous block
                float2* g = ws + q.out_off + (int64_t)q.first * q.L;
                if ((reinterpret_cast<uintptr_t>(g) & 15) == 0 && (q.L & 1) == 0) {
                    for (int w = t >> 5; w < q.count; w += NT / 32)
                        for (int k = 2 * (t & 31); k < q.L; k += 64) {
                            const float2 x = tile[w * q.pitch + k], y = tile[w * q.pitch + k + 1];
                            *reinterpret_cast<float4*>(g + w * q.L + k) = make_float4(x.x, x.y, y.x, y.y);
                        }
                } else {
                    for (int w = t >> 5; w < q.count; w += NT / 32)
                        for (int k = t & 31; k < q.L; k += 32) g[w * q.L + k] = tile[w * q.pitch + k];
                }
            } else if (q.flags & RAG_R2C_POST) {
                if (c.ok)
                    r2c_post([&](int k) { return buf[k + (k >> c.ps)]; }, c.tw + q.post_off,
                             reinterpret_cast<float2*>(c.go), c.L, c.tid, (c.L >> 1) + 1, c.T);
            }
        }
        cp_async_wait_all();
        if (t == NT - 1) s_claim[cur] = claimed;
        publish();
        if (run && (q.kind == RAG_P1 || q.kind == RAG_P2)) pending = q.xform;
        // every thread's stores precede thread 0's fence, which orders them
        // before the counter update; the tile, the record and the claim are
        // free or visible for the next item
        __syncthreads();
        it = nxt;
        nxt = s_claim[cur];
        if (A.claim == RAG_CLAIM_NONE) return;
        if (A.claim == RAG_CLAIM_NEXT) {
            publish();
            if (t == 0) s_claim[0] = atomicAdd(A.queue, 1);
            __syncthreads();
            it = s_claim[0];
            nxt = A.nitems;
            if (it < A.nitems && t < kRecChunks)
                reinterpret_cast<int4*>(&s_rec[cur ^ 1])[t] = __ldg(reinterpret_cast<const int4*>(A.items + it) + t);
            __syncthreads();
        }
    }
    if (t == 0 && pending >= 0) {
        __threadfence();
        atomicAdd(A.queue + 1 + pending, 1);
    }
    if (A.claim == RAG_CLAIM_NONE) return;
    // the last CTA clears the queue, instead of a memset ahead of every launch
    // (10000 transforms 438 -> 419 us); no CTA touches it after counting itself
    __syncthreads();
    if (t == 0) {
        __threadfence();
        s_ok = atomicAdd(A.queue + 1 + A.count, 1) == (int)gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (s_ok)
        for (int i = t; i < A.count + 2; i += NT) A.queue[i] = 0;
}

}  // namespace
}  // namespace gfft

using namespace gfft;

extern "C" int gfft_ragged_ctas(int smem_bytes)
{
    // the kernel's static shared memory counts against the opt-in limit, so
    // the attribute is a dynamic size actually launched with: the largest of
    // any plan on the device so far, since plans that asked for more are still
    // launched (set each time: a device reset forgets it)
    static std::mutex mu;
    static int limit[64] = {0};
    int occ = 0, dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) {
        std::lock_guard<std::mutex> lk(mu);
        int& most = limit[dev & 63];
        const int want = smem_bytes > most ? smem_bytes : most;
        e = cudaFuncSetAttribute(ragged_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, want);
        if (e == cudaSuccess) most = want;
    }
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, ragged_kernel, NT, (size_t)smem_bytes);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return -(int)e;
    }
    return occ;
}

extern "C" int gfft_launch_ragged(const RagArgs* a, void* stream)
{
    // stream-ordered work only (capturable): attributes and residency come
    // from gfft_ragged_ctas, called beforehand
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (a->nitems <= 0) return 0;
    if (a->smem_bytes <= 0 || a->smem_bytes > kMaxSmemBytes || a->ctas <= 0) return (int)cudaErrorInvalidValue;
    const int grid = a->ctas < a->nitems ? a->ctas : a->nitems;
    ragged_kernel<<<(unsigned)grid, NT, (size_t)a->smem_bytes, st>>>(*a);
    return (int)cudaGetLastError();
}
