// planner.cpp - see planner.h.
#include "planner.h"
#include "tile_list.h"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <functional>

namespace gfft {

namespace {

constexpr int kBigPrimes[] = {17, 19, 23, 29, 31, 37, 41, 43, 47};

int max_threads_for(int rmax) { return rmax <= 16 ? 512 : 256; }

int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

}  // namespace

std::vector<int64_t> prime_factors(int64_t n)
{
    std::vector<int64_t> f;
    if (n <= 1) return f;
    for (int64_t p = 2; p * p <= n; ++p) {
        while (n % p == 0) {
            f.push_back(p);
            n /= p;
        }
    }
    if (n > 1) f.push_back(n);
    return f;
}

bool all_primes_at_most(int64_t n, int64_t pmax)
{
    for (int64_t p : prime_factors(n))
        if (p > pmax) return false;
    return true;
}

bool length_supported(int64_t n) { return n >= 1 && all_primes_at_most(n, 47); }

std::vector<int> choose_radices(int L)
{
    if (L == 1) return {1};
    if (!all_primes_at_most(L, 47)) return {};
    std::vector<int> allowed;
    for (int r = 16; r >= 2; --r) allowed.push_back(r);
    for (int p : kBigPrimes)
        if (L % p == 0) allowed.insert(allowed.begin(), p);
    std::sort(allowed.begin(), allowed.end(), std::greater<int>());

    std::vector<int> best, cur;
    int best_pass = 1 << 30, best_min = 0, best_pow2 = -1;
    std::function<void(int, int)> dfs = [&](int rem, int maxr) {
        if ((int)cur.size() > best_pass || (int)cur.size() >= kMaxPass) return;
        if (rem == 1) {
            const int np = (int)cur.size();
            const int mn = *std::min_element(cur.begin(), cur.end());
            int pow2 = 0;
            for (int r : cur) pow2 += ((r & (r - 1)) == 0);
            if (np < best_pass || (np == best_pass && (mn > best_min || (mn == best_min && pow2 > best_pow2)))) {
                best = cur;
                best_pass = np;
                best_min = mn;
                best_pow2 = pow2;
            }
            return;
        }
        for (int r : allowed) {
            if (r > maxr || rem % r) continue;
            cur.push_back(r);
            dfs(rem / r, r);
            cur.pop_back();
        }
    };
    dfs(L, 1 << 30);
    return best;
}

int64_t TwiddleBuilder::add_outer(int64_t ns, int64_t rows, int64_t M)
{
    // layout [row][k]: entry row*ns + k = W_M^{row*k}
    for (const TwSeg& t : segs)
        if (t.kind == 2 && t.M == M && t.R_or_mult == ns && t.count >= rows * ns) return t.offset;
    const int64_t off = count;
    TwSeg s{};
    s.offset = off;
    s.count = ns * rows;
    s.M = M;
    s.R_or_mult = ns;
    s.kind = 2;
    segs.push_back(s);
    count += ns * rows;
    count += count & 1;
    return off;
}

// Pass table: consecutive butterflies (consecutive k) read consecutive entries.
int64_t TwiddleBuilder::add_pass_table(int64_t ns, int R) { return add_outer(ns, R, ns * R); }

int64_t TwiddleBuilder::add_linear(int64_t n, int64_t M, int64_t mult)
{
    for (const TwSeg& t : segs)
        if (t.kind == 1 && t.M == M && t.R_or_mult == mult && t.count >= n) return t.offset;
    const int64_t off = count;
    TwSeg s{};
    s.offset = off;
    s.count = n;
    s.M = M;
    s.R_or_mult = mult;
    s.kind = 1;
    segs.push_back(s);
    count += n;
    count += count & 1;
    return off;
}

int64_t TwiddleBuilder::add_dft_matrix(int R, int prec)
{
    for (const TwSeg& t : segs)
        if (t.kind == 3 && t.M == R && t.R_or_mult == prec) return t.offset;
    const int64_t n = gfft_tc_bmat_entries(R, prec);
    if (n <= 0) return -1;
    const int64_t off = count;
    TwSeg s{};
    s.offset = off;
    s.count = n;
    s.M = R;
    s.R_or_mult = prec;
    s.kind = 3;
    segs.push_back(s);
    count += n;
    count += count & 1;
    return off;
}

int64_t TwiddleBuilder::add_dtable(int64_t n)
{
    for (const auto& d : dsegs)
        if (d.second == n) return d.first;
    const int64_t off = count;
    dsegs.emplace_back(off, n);
    count += 2 * n;
    return off;
}

bool build_inner(int L, const std::vector<int>& radices, int nthr, TwiddleBuilder& tb, InnerPlan& ip)
{
    if (radices.empty() || (int)radices.size() > kMaxPass) return false;
    ip = InnerPlan{};
    ip.L = L;
    ip.npass = (int)radices.size();
    ip.nthr = nthr;
    ip.rmax = 16;
    int64_t ns = 1;
    for (int p = 0; p < ip.npass; ++p) {
        const int R = radices[p];
        if (R > 16) ip.rmax = 47;
        PassDesc& d = ip.pass[p];
        d.radix = R;
        d.ns = (int32_t)ns;
        d.ns_magic = ns > 1 ? (uint32_t)(((1ull << 32) + (uint64_t)ns - 1) / (uint64_t)ns) : 0u;
        d.tw_off = ns > 1 ? (int32_t)tb.add_pass_table(ns, R) : -1;
        ns *= R;
    }
    return ns == L;
}

namespace {

int pick_nthr(int L, const std::vector<int>& radices, int maxthr)
{
    int nbf_max = 1;
    for (int r : radices) nbf_max = std::max(nbf_max, L / r);
    if (nbf_max <= maxthr) return nbf_max;
    return (int)ceil_div(nbf_max, ceil_div(nbf_max, maxthr));
}

// Shared-memory buffers a row transform needs (see row_body in stockham.cuh).
int row_nbuf(int npass, int start, bool last_global)
{
    const int writes = npass - (last_global ? 1 : 0);
    if (start == 1) return writes >= 1 ? 2 : 1;
    return writes >= 2 ? 2 : 1;
}

}  // namespace

// Hints of the problem being planned (set by build_steps for its duration).
thread_local const PlanHints* t_hints = nullptr;

struct HintScope {
    explicit HintScope(const PlanHints* h) : prev(t_hints) { t_hints = h; }
    ~HintScope() { t_hints = prev; }
    const PlanHints* prev;
};

// Largest lengths accepted by the generic kernels (checked exactly below).
int row_max_length() { return 13312; }

bool codelets_enabled()
{
    static const bool on = [] {
        const char* v = std::getenv("OPS_FFT_CODELETS");
        return !(v && v[0] == '0');
    }();
    if (t_hints && t_hints->codelets == 0) return false;
    return on;
}
int col_max_length() { return 2048; }

bool clusters_enabled()
{
    static const bool on = [] {
        const char* v = std::getenv("OPS_FFT_CLUSTER");
        return !(v && v[0] == '0');
    }();
    if (t_hints && t_hints->cluster == 0) return false;
    return on;
}

namespace {

// ------------------------------------------------------------ tile kernel
// (csrc/tile_fft.cuh)
constexpr int kTileMaxThreads = 512;
constexpr int kTileElems = 16;  // elements a thread holds
constexpr int kSMs = 152;       // of a GB300: the rules for small batches count CTAs and threads per SM
constexpr int64_t kTileMaxCols = (int64_t(1) << 31) - 64;  // 32-bit column arithmetic

}  // namespace

int tile_threads(int L, const std::vector<int>& rad, int elems)
{
    int t = 1;
    for (int r : rad) {
        const int nb = r >= elems ? 1 : elems / r;
        t = std::max(t, (int)ceil_div(L / r, nb));
    }
    return t;
}

// Radices for the tile kernel: fewest passes, then fewest threads, then
// balanced; an odd radix (or a power of two) first, which keeps the shared
// addresses of a butterfly an arithmetic sequence, the others descending.
// c2r: the first pass reads the exchange buffer too (the Hermitian
// pre-process wrote it), so L/R0 has to be a multiple of a power-of-two R0.
std::vector<int> choose_tile_radices(int L, bool c2r, int max_threads, int elems)
{
    if (L == 1) return {1};
    std::vector<int> best, cur;
    int best_np = 1 << 30, best_t = 0, best_min = 0;
    std::function<void(int, int)> dfs = [&](int rem, int maxr) {
        if ((int)cur.size() > best_np || (int)cur.size() >= kMaxPass) return;
        if (rem == 1) {
            const int np = (int)cur.size(), t = tile_threads(L, cur, elems);
            if (t > max_threads) return;
            const int mn = *std::min_element(cur.begin(), cur.end());
            if (np < best_np || (np == best_np && (t < best_t || (t == best_t && mn > best_min)))) {
                best = cur;
                best_np = np;
                best_t = t;
                best_min = mn;
            }
            return;
        }
        for (int r = std::min(maxr, kTileElems); r >= 2; --r) {
            if (rem % r) continue;
            cur.push_back(r);
            dfs(rem / r, r);
            cur.pop_back();
        }
    };
    dfs(L, kTileElems);
    if (best.size() > 1) {
        auto pow2 = [&](int r) { return (r & (r - 1)) == 0 && (!c2r || (L / r) % r == 0); };
        size_t first = best.size();
        for (size_t i = 0; i < best.size() && first == best.size(); ++i)
            if (best[i] & 1) first = i;
        for (size_t i = 0; i < best.size() && first == best.size(); ++i)
            if (pow2(best[i])) first = i;
        if (first < best.size()) std::rotate(best.begin(), best.begin() + first, best.begin() + first + 1);
    }
    return best;
}

// log2 of the first radix when that is a power of two: the shared padding
int tile_pshift(int L, const std::vector<int>& rad, bool c2r)
{
    if (rad.size() < 2 || (rad[0] & (rad[0] - 1)) != 0 || (c2r && (L / rad[0]) % rad[0])) return 30;
    int s = 0;
    while ((1 << s) < rad[0]) ++s;
    return s;
}

namespace {

// Whether a tile is compiled in with its length, threads and radices.
bool tile_compiled(bool rows, int L, int T, int W, const std::vector<int>& rad)
{
#define GFFT_IS_ROW(ID, LL, TT, WW, ...) \
    if (rows && L == LL && T == TT && W == WW && rad == std::vector<int>{__VA_ARGS__}) return true;
#define GFFT_IS_COL(ID, LL, TT, WW, ...) \
    if (!rows && L == LL && T == TT && W == WW && rad == std::vector<int>{__VA_ARGS__}) return true;
    GFFT_TILE_ROWS(GFFT_IS_ROW)
    GFFT_TILE_COLS(GFFT_IS_COL)
#undef GFFT_IS_ROW
#undef GFFT_IS_COL
    return false;
}

// Whether any column tile of this length is compiled in.
bool column_tile_compiled(int L)
{
#define GFFT_IS_LEN(ID, LL, TT, WW, ...) \
    if (L == LL) return true;
    GFFT_TILE_COLS(GFFT_IS_LEN)
#undef GFFT_IS_LEN
    return false;
}

// Score bonus of a codelet configuration with a per-group work buffer
// (ping-pong passes) over the in-place one.
constexpr double kPingPongScore = 0.0;

// Codelet row step (see csrc/codelet.cuh for the execution model and the
// shared-memory layout).  Returns false when no codelet applies.
bool make_codelet_step(int L, int64_t ntf, int64_t in_dist, int64_t out_dist, int io_mode, int nreal, int weight,
                       TwiddleBuilder& tb, Step& st)
{
    if (!codelets_enabled()) return false;
    // OPS_FFT_CODELET_VARIANT=k selects the k-th entry of this length
    // (tuning experiments); unset or absent, the first one
    const char* env_var = std::getenv("OPS_FFT_CODELET_VARIANT");
    int want = env_var ? std::atoi(env_var) : 0;
    if (t_hints && t_hints->codelet_variant >= 0) want = t_hints->codelet_variant;
    int id = gfft_codelet_find(L, want);
    if (id < 0) id = gfft_codelet_find(L, 0);
    if (id < 0) return false;
    int cl = 0, cn = 0, cr[kMaxPass], cnr = 0, cmaxt = 0, cminb = 0;
    if (gfft_codelet_info(id, &cl, &cn, cr, &cnr, &cmaxt, &cminb) != 0 || cl != L) return false;
    const std::vector<int> rad(cr, cr + cnr);
    const bool even_mode = io_mode == IO_R2C_EVEN || io_mode == IO_C2R_EVEN;
    const bool staged = false;
    const int pshift = (rad[0] % 2 == 0) ? 4 : 30;
    const int maxidx = even_mode ? L : L - 1;
    int lpad = maxidx + (maxidx >> pshift) + 2;
    lpad += lpad & 1;
    const int esize = io_mode == IO_R2C_ODD ? 4 : 8;
    const int64_t row_bytes = in_dist * esize;
    TwiddleBuilder trial = tb;  // do not register tables unless the codelet is used
    st = Step{};
    st.kind = Step::ROW;
    RowArgs& a = st.row;
    if (!build_inner(L, rad, cn, trial, a.ip)) return false;
    int64_t lo = -1, hi = -1;
    for (int p = 0; p < a.ip.npass; ++p) {
        const PassDesc& d = a.ip.pass[p];
        if (d.ns <= 1) continue;
        lo = lo < 0 ? d.tw_off : std::min<int64_t>(lo, d.tw_off);
        hi = std::max<int64_t>(hi, d.tw_off + (int64_t)d.ns * d.radix);
    }
    const int64_t tw_cnt = lo < 0 ? 0 : hi - lo;
    const int64_t post_cnt = even_mode ? L / 2 + 1 : 0;
    int64_t post_off = -1;
    if (even_mode) post_off = trial.add_linear(L / 2 + 1, 2 * (int64_t)L, 1);
    auto align = [](int64_t x, int64_t a) { return (x + a - 1) / a * a; };
    const int64_t hdr = 128;
    // the tables arrive by bulk copies of their 16-byte aligned supersets
    // (a table starting 8 bytes into a 16-byte unit sits 8 bytes in): one
    // spare 16-byte unit each
    const int64_t tw_bytes = tw_cnt > 0 ? align(tw_cnt * 8 + 16, 16) : 0;
    const int64_t post_bytes = post_cnt > 0 ? align(post_cnt * 8 + 16, 16) : 0;
    const int tps = 1;
    // one transform per slot: raw row at offset src % 16 (< 16), padded work
    // layout from offset 16, both inside the slot
    const int64_t stage_bytes = align(std::max<int64_t>(row_bytes + 32, 16 + (int64_t)lpad * 8), 128);
    const int64_t cta_fixed = align(hdr + tw_bytes + post_bytes, 128);
    const int64_t nslots = (ntf + tps - 1) / tps;
    double best = -1e300;  // any configuration that fits beats none
    int best_ng = 0, best_ns = 0;
    int64_t best_gb = 0;
    // OPS_FFT_CODELET_NG / OPS_FFT_CODELET_NST pin the groups per CTA and
    // prefetch stages (tuning experiments); unset, the score below decides
    const char* env_ng = std::getenv("OPS_FFT_CODELET_NG");
    const char* env_ns = std::getenv("OPS_FFT_CODELET_NST");
    const int force_ng = (t_hints && t_hints->codelet_ng > 0) ? t_hints->codelet_ng : (env_ng ? std::atoi(env_ng) : 0);
    const int force_ns = (t_hints && t_hints->codelet_nst > 0) ? t_hints->codelet_nst : (env_ns ? std::atoi(env_ns) : 0);
    // a per-group work buffer (ping-pong passes, half the group barriers):
    // OPS_FFT_CODELET_PP=0/1 or the autotuner pin it; unset, the score decides
    const char* env_pp = std::getenv("OPS_FFT_CODELET_PP");
    const int force_pp = (t_hints && t_hints->codelet_pp >= 0) ? t_hints->codelet_pp : (env_pp ? std::atoi(env_pp) : -1);
    const int64_t work_bytes = align((int64_t)lpad * 8, 128);
    int best_pp = 0;
    for (int pp = 0; pp <= 1; ++pp)
    for (int nst = 2; nst <= 4; ++nst) {
        if (force_pp >= 0 && pp != force_pp) continue;
        if (force_ns ? nst != force_ns : nst > 3) continue;
        const int64_t gb = align(64 + nst * stage_bytes + (pp ? work_bytes : 0), 128);
        for (int ng = 1; ng <= 15 && ng * cn <= cmaxt; ++ng) {
            if (force_ng && ng != force_ng) continue;
            const int64_t smem = cta_fixed + ng * gb;
            if (smem > kMaxSmemBytes) break;
            const int64_t warps = (int64_t)ng * cn / 32;
            // registers: the launch bound caps each thread at 65536 / (MAXT * MINB);
            // they are allocated per warp in each of the 4 SM sub-partitions
            // (16384 registers each), so resident warps come in multiples of 4
            const int64_t reg_cap = std::min<int64_t>(255, (65536 / ((int64_t)cmaxt * cminb)) & ~(int64_t)7);
            const int64_t warps_by_regs = 4 * (16384 / (reg_cap * 32));
            const int64_t ctas = std::min<int64_t>(
                {(228 * 1024) / (smem + 1024), 64 / warps, 32, warps_by_regs / warps});
            if (ctas < 1) continue;
            int64_t groups_sm = ctas * ng;
            // a small batch cannot keep every group busy
            groups_sm = std::min<int64_t>(groups_sm, std::max<int64_t>(1, (nslots + 151) / 152));
            const double occ = (double)std::min<int64_t>(groups_sm * cn, 1536) / 1536.0;
            // bytes of input copies in flight per SM, saturating at 40 KB
            // (more stages beyond that measured slower: R2C, C2R and the
            // weighted R2C adjoint at N=3000, batch 4096, 4 groups per SM,
            // 2 stages 1-3 % faster than 3)
            const double infl =
                (double)std::min<int64_t>(groups_sm * (nst - 1) * tps * row_bytes, 40 * 1024) / (40 * 1024.0);
            const double score = occ + infl - 0.02 * nst + kPingPongScore * pp;
            // ties: more groups per CTA (up to 384 threads) share the CTA's
            // twiddle tables and hide each other's barriers (measured faster)
            const bool tie_better = score > best - 1e-9 && ng > best_ng && ng * cn <= 384;
            if (score > best + 1e-9 || tie_better) {
                best = score;
                best_ng = ng;
                best_ns = nst;
                best_gb = gb;
                best_pp = pp;
            }
        }
    }
    if (best_ng == 0) {
        // a tuned shape that this transform has no room for (it was timed on
        // another: the adjoint's slots are one bin longer): the score's choice
        if (!t_hints || (t_hints->codelet_ng <= 0 && t_hints->codelet_nst <= 0 && t_hints->codelet_pp < 0)) return false;
        PlanHints free = *t_hints;
        free.codelet_ng = free.codelet_nst = 0;
        free.codelet_pp = -1;
        const HintScope scope(&free);
        return make_codelet_step(L, ntf, in_dist, out_dist, io_mode, nreal, weight, tb, st);
    }
    tb = trial;
    st.post_off = post_off;
    a.ntf = ntf;
    a.in_dist = in_dist;
    a.out_dist = out_dist;
    a.tfpc = tps;
    a.lpad = lpad;
    a.nbuf = best_pp ? 2 : 1;
    a.io_mode = io_mode;
    a.weight = weight;
    a.nreal = nreal;
    a.staged = staged ? 1 : 0;
    a.scale = 1.f;
    a.conj_out = io_mode == IO_C2R_EVEN ? 1 : 0;
    a.nstage = best_ns;
    a.pshift = pshift;
    a.in_esize = esize;
    a.tw_lo = (int32_t)(lo < 0 ? 0 : lo);
    a.tw_cnt = (int32_t)tw_cnt;
    a.post_cnt = (int32_t)post_cnt;
    a.stage_bytes = (int32_t)stage_bytes;
    a.smem_tw = (int32_t)hdr;
    a.smem_post = (int32_t)(hdr + tw_bytes);
    a.smem_stage = (int32_t)cta_fixed;
    a.smem_work = best_pp ? (int32_t)(64 + best_ns * stage_bytes) : 0;  // group offset of the work buffer
    a.group_bytes = (int32_t)best_gb;
    a.ngroups = best_ng;
    a.smem_bytes = (int32_t)(cta_fixed + best_ng * best_gb);
    a.codelet = id;
    st.tw_off = 0;
    return true;
}

// A switch or a tuned choice that describes a codelet asks for that codelet.
bool codelet_asked(int io_mode)
{
    for (const char* name : {"OPS_FFT_CODELET_VARIANT", "OPS_FFT_CODELET_NG", "OPS_FFT_CODELET_NST", "OPS_FFT_CODELET_PP"})
        if (std::getenv(name)) return true;
    const char* fuse = std::getenv("OPS_FFT_FUSE_R2C");
    if (fuse && fuse[0] == '0' && io_mode == IO_R2C_EVEN) return true;
    return t_hints && (t_hints->codelet_variant >= 0 || t_hints->codelet_ng > 0 || t_hints->codelet_nst > 0 ||
                       t_hints->codelet_pp >= 0);
}

// Whether rows of a length with a codelet run on the tile kernel when their
// buffers are in device memory: at every batch, with the length's tile
// compiled in too (tile_list.h).  Measured (us, tile / codelet): C2C 128 x 8
// 2.3 / 3.3, 512 x 16 1.9 / 3.0, 1024 x 64 2.2 / 4.2, 2048 x 64 2.5 / 4.1,
// 4096 x 128 3.6 / 4.4, 1500 x 8192 35.6 / 42.2, 512 x 32768 43 / 56, 4096 x
// 4096 44 / 55; R2C 1024 x 64 2.4 / 3.5, 3000 x 64 3.2 / 3.9, 3000 x 4096 23.3
// / 27.7, 8192 x 4096 54 / 86; C2R 1024 x 64 2.7 / 3.4, 3000 x 4096 27.6 /
// 28.0, 8192 x 4096 61 / 88.  The codelets keep pinned host buffers used in
// place, chunked host calls, plans tuned to one of them (a tuned plan may also
// stay here) and 8192 points (C2R 16384: clusters below 1024 rows).
bool tile_beats_codelet(int L, int io_mode) { return L <= 4096 && !codelet_asked(io_mode); }

// Rows of any length with radices <= 16 on the tile kernel.
bool make_tile_row_step(int L, int64_t ntf, int64_t in_dist, int64_t out_dist, int io_mode, int nreal, int weight,
                        TwiddleBuilder& tb, Step& st)
{
    if (ntf >= kTileMaxCols) return false;
    const std::vector<int> rad = choose_tile_radices(L, io_mode == IO_C2R_EVEN);
    if (rad.empty()) return false;
    int T = tile_threads(L, rad);
    if (T > kTileMaxThreads) return false;
    // one thread per row reads 8 L bytes of its own: beyond 12 complex values
    // and 12 MB the row kernel's staged copies are faster (us, row kernel /
    // this: 16 x 2^20 100 / 129, x 131072 17.0 / 18.4, x 100000 16.0 / 15.1, x
    // 1000 4.3 / 2.9; 13 x 100000 11.3 / 9.7; 12 x 1.4M 81 / 84)
    if (T == 1 && L > 12 && io_mode == IO_C2C && ntf * L > 3 << 19) return false;
    // few rows: one butterfly a thread and pass (half the instructions on a
    // row's critical path when its radices are 8 or less) while that leaves
    // at most 256 threads on an SM
    int T1 = 1;
    for (int r : rad) T1 = std::max(T1, L / r);
    if (T1 <= kTileMaxThreads && ntf * T1 <= kSMs * 256) T = T1;
    TwiddleBuilder trial = tb;
    st = Step{};
    st.kind = Step::ROW;
    RowArgs& a = st.row;
    if (!build_inner(L, rad, T, trial, a.ip)) return false;
    const bool even_mode = io_mode == IO_R2C_EVEN || io_mode == IO_C2R_EVEN;
    if (even_mode) st.post_off = trial.add_linear(L / 2 + 1, 2 * (int64_t)L, 1);
    const int ps = tile_pshift(L, rad, io_mode == IO_C2R_EVEN);
    int pitch = L + (L >> ps) + 1;
    if (T < 16) {
        while (pitch % 16 != T % 16) ++pitch;
    } else {
        pitch += pitch & 1;
    }
    // two warps per CTA, more only for longer rows: small CTAs wait for
    // fewer threads at each barrier (100 x 131072: 36.4 us at 64 threads, 41
    // at 256; 1024 x 16384: 44.3 against 48.0).  With fewer rows than that a
    // compiled tile keeps its width and idles (one row, us: R2C 256 3.7 -> 2.1,
    // codelet 2.9; C2C 128 2.4 -> 1.5)
    const int full = std::max(1, 64 / T);
    const int W = tile_compiled(true, L, T, full, rad) ? full : (int)std::min<int64_t>(full, ntf);
    const int64_t one = (int64_t)W * pitch * 8;
    if (one > kMaxSmemBytes) return false;
    tb = trial;
    a.tile = 1;
    a.ntf = ntf;
    a.in_dist = in_dist;
    a.out_dist = out_dist;
    a.tfpc = W;
    a.lpad = pitch;
    a.nbuf = 1;
    a.io_mode = io_mode;
    a.weight = weight;
    a.nreal = nreal;
    a.scale = 1.f;
    a.conj_out = io_mode == IO_C2R_EVEN ? 1 : 0;
    a.nstage = 1;
    a.pshift = ps;
    a.in_esize = io_mode == IO_R2C_ODD ? 4 : 8;
    a.post_cnt = even_mode ? L / 2 + 1 : 0;
    a.smem_bytes = (int32_t)one;
    a.codelet = -1;
    st.tw_off = 0;
    return true;
}

// One on-chip transform per contiguous batch item (persistent row kernel,
// see csrc/row_pipe.cuh for the shared-memory layout).
bool make_row_step(int L, int64_t ntf, int64_t in_dist, int64_t out_dist, int io_mode, int nreal, int weight,
                   TwiddleBuilder& tb, Step& st)
{
    std::vector<int> rad = choose_radices(L);
    if (rad.empty()) return false;
    int rmax = *std::max_element(rad.begin(), rad.end()) > 16 ? 47 : 16;
    int maxthr = max_threads_for(rmax);
    int nthr = pick_nthr(L, rad, maxthr);
    int codelet = -1;
    if (make_codelet_step(L, ntf, in_dist, out_dist, io_mode, nreal, weight, tb, st)) {
        Step t;
        if (tile_beats_codelet(L, io_mode) &&
            make_tile_row_step(L, ntf, in_dist, out_dist, io_mode, nreal, weight, tb, t)) {
            st.dev = t.row;
            st.dev_post_off = t.post_off;
            st.has_dev = true;
        }
        return true;
    }
    // OPS_FFT_CODELETS=0, or a tuned choice of no codelets, asks for the kernel below
    if (codelets_enabled() && make_tile_row_step(L, ntf, in_dist, out_dist, io_mode, nreal, weight, tb, st)) return true;
    const bool even_mode = io_mode == IO_R2C_EVEN || io_mode == IO_C2R_EVEN;
    const bool staged = nthr < 32 && (io_mode == IO_C2C || io_mode == IO_R2C_EVEN);
    const int start = io_mode == IO_C2R_EVEN ? 1 : 0;
    const bool last_global = !(io_mode == IO_R2C_EVEN || (io_mode == IO_C2C && staged));
    const int nbuf = std::max(1, row_nbuf((int)rad.size(), start, last_global));
    const int pshift = (rad[0] % 2 == 0) ? 4 : 30;
    const int maxidx = even_mode ? L : L - 1;
    int lpad = maxidx + (maxidx >> pshift) + 2;
    lpad += lpad & 1;
    const int esize = io_mode == IO_R2C_ODD ? 4 : 8;
    const int64_t row_bytes = in_dist * esize;

    st = Step{};
    st.kind = Step::ROW;
    RowArgs& a = st.row;
    if (!build_inner(L, rad, nthr, tb, a.ip)) return false;
    // pass-table window (contiguous range of the blob used by this transform)
    int64_t lo = -1, hi = -1;
    for (int p = 0; p < a.ip.npass; ++p) {
        const PassDesc& d = a.ip.pass[p];
        if (d.ns <= 1) continue;
        const int64_t b0 = d.tw_off, b1 = d.tw_off + (int64_t)d.ns * d.radix;
        lo = lo < 0 ? b0 : std::min(lo, b0);
        hi = std::max(hi, b1);
    }
    const int64_t tw_cnt = lo < 0 ? 0 : hi - lo;
    const bool tw_in_smem = tw_cnt * 8 <= 72 * 1024;

    const int64_t post_cnt = even_mode ? L / 2 + 1 : 0;
    if (even_mode) st.post_off = tb.add_linear(L / 2 + 1, 2 * (int64_t)L, 1);

    auto align = [](int64_t x, int64_t a) { return (x + a - 1) / a * a; };
    const int64_t hdr = 128;
    const int64_t tw_bytes = tw_in_smem ? align(tw_cnt * 8, 16) : 0;
    const int64_t post_bytes = align(post_cnt * 8, 16);
    // tiles must keep the bulk copies 16-byte aligned when rows are not
    int tf_mult = 1;
    while ((row_bytes * tf_mult) % 16 != 0 && tf_mult < 16) tf_mult *= 2;
    const int64_t tmax = std::max<int64_t>(
        1, std::min<int64_t>({(int64_t)maxthr / nthr, std::max<int64_t>(1, (48 * 1024) / row_bytes), ntf}));
    // keep at least ~one tile per SM for small batches
    const int64_t tcap = std::max<int64_t>(1, (ntf + 151) / 152);
    double best = -1;
    int best_tf = 1, best_ns = 1;
    int64_t best_smem = 0;
    for (int ns_ = 1; ns_ <= 3; ++ns_) {
        for (int64_t tf = std::min(tmax, std::max<int64_t>(tcap, 1)); tf >= 1; --tf) {
            const int64_t stage = align(tf * row_bytes, 128);
            const int64_t work = tf * nbuf * (int64_t)lpad * 8;
            const int64_t smem = hdr + tw_bytes + post_bytes + ns_ * stage + work;
            if (smem > kMaxSmemBytes) continue;
            const int64_t threads = tf * nthr;
            const int64_t warps = (threads + 31) / 32;
            const int64_t ctas = std::min<int64_t>({(228 * 1024) / (smem + 1024), 64 / std::max<int64_t>(warps, 1), 32});
            if (ctas < 1) continue;
            const double thr_sm = (double)std::min<int64_t>(ctas * threads, 1024) / 1024.0;
            const double infl = (double)std::min<int64_t>(ctas * (ns_ - 1) * tf * row_bytes, 96 * 1024) / (96 * 1024.0);
            double score = thr_sm + infl + (tf % tf_mult == 0 ? 0.5 : 0.0) + 0.01 * ns_;
            if (score > best) {
                best = score;
                best_tf = (int)tf;
                best_ns = ns_;
                best_smem = smem;
            }
        }
    }
    if (best < 0) return false;
    a.ntf = ntf;
    a.in_dist = in_dist;
    a.out_dist = out_dist;
    a.tfpc = best_tf;
    a.lpad = lpad;
    a.nbuf = nbuf;
    a.io_mode = io_mode;
    a.weight = weight;
    a.nreal = nreal;
    a.staged = staged ? 1 : 0;
    a.scale = 1.f;
    a.conj_out = io_mode == IO_C2R_EVEN ? 1 : 0;
    a.nstage = best_ns;
    a.pshift = pshift;
    a.in_esize = esize;
    a.tw_lo = (int32_t)(lo < 0 ? 0 : lo);
    a.tw_cnt = tw_in_smem ? (int32_t)tw_cnt : 0;
    a.post_cnt = (int32_t)post_cnt;
    a.stage_bytes = (int32_t)align(best_tf * row_bytes, 128);
    a.smem_tw = (int32_t)hdr;
    a.smem_post = (int32_t)(hdr + tw_bytes);
    a.smem_stage = (int32_t)align(hdr + tw_bytes + post_bytes, 128);
    a.smem_work = (int32_t)(a.smem_stage + (int64_t)best_ns * a.stage_bytes);
    a.smem_bytes = (int32_t)(a.smem_work + (int64_t)best_tf * nbuf * lpad * 8);
    a.codelet = codelet;
    a.ngroups = 0;
    a.group_bytes = 0;
    (void)best_smem;
    st.tw_off = 0;
    return a.smem_bytes <= kMaxSmemBytes;
}

// Whether the launcher has a compiled instance of an even real column tile.
bool pair_compiled(bool r2c, int L, int T, int W, const std::vector<int>& rad)
{
    return tile_compiled(false, L, T, W, rad) && (r2c ? W == 16 || L == 1024 : W == 8);
}

// Turns the column pass described by st.col (addresses filled in) into tiles
// of the tile kernel; false when it does not apply.
bool make_tile_col(int64_t S, int Lq, int64_t Ns, bool staged_out, TwiddleBuilder& tb, Step& st)
{
    ColArgs& a = st.col;
    if (a.ncols >= kTileMaxCols) return false;
    const std::vector<int> rad = choose_tile_radices(Lq);
    if (rad.empty()) return false;
    int T = tile_threads(Lq, rad);
    // strided axes: 16 columns (128-byte row segments) where the threads
    // allow it (512-point axes of 512^3: 1283 us against 1489 at 8 columns;
    // 256 x 263168: 169 against 313); passes of a long row, whose segments
    // are neighbours in memory, take 8 and smaller CTAs (131072 x 128: 121
    // against 127 us).  At least 4: narrower segments waste sectors.
    int W = S > 1 ? 16 : 8;
    while (W > 4 && W * T > kTileMaxThreads) W >>= 1;
    if (T * W > kTileMaxThreads) return false;
    // few columns: narrower tiles until two CTAs per SM are there, but not
    // below the narrowest compiled one (us, 4 columns argument-driven / compiled:
    // 2D R2C 25 x 128 x 30 8.0 / 5.4, C2R 10 x 256 x 256 12.2 / 8.2, 1 x 512 x 256
    // 11.3 / 7.6, C2C 22 x 512 x 100 13.8 / 11.4)
    auto compiled = [&](int w) { return tile_compiled(false, Lq, T, w, rad); };
    while (W > 4 && a.ncols / W < 2 * kSMs && (!compiled(W) || compiled(W / 2))) W >>= 1;
    // and, as for rows, a thread for every butterfly while that leaves at most
    // 256 threads on an SM (us, without / with: 32 x 30 2D 7.1 / 5.3, 32 x 30 x
    // 40 12.3 / 9.9)
    int T1 = 1;
    for (int r : rad) T1 = std::max(T1, Lq / r);
    if (!compiled(W) && T1 * W <= kTileMaxThreads && a.ncols * T1 <= kSMs * 256) T = T1;
    TwiddleBuilder trial = tb;
    InnerPlan ip;
    if (!build_inner(Lq, rad, T, trial, ip)) return false;
    const int ps = tile_pshift(Lq, rad);
    const int Lp = Lq + (Lq >> ps);
    int spitch = 0;
    int64_t buf = (int64_t)W * Lp;
    if (staged_out) {
        spitch = Lq;
        while (spitch % 16 != 16 / W % 16) ++spitch;
        buf = std::max<int64_t>(buf, (int64_t)W * spitch);
    }
    // one exchange buffer and two barriers a pass: two buffers and one
    // barrier leave fewer CTAs per SM (512 x 65536 in 64 KB tiles: 161 us
    // against 116)
    const int64_t smem = buf * 8;
    if (smem > kMaxSmemBytes) return false;
    if (Ns > 1) {
        const int64_t M = Ns * Lq;
        // the outer twiddle W_M^{j*i} of a first-pass butterfly (samples i =
        // jb + r*Lq/R) is W_M^{j*jb} * W_{Ns*R}^{j*r}: two tables whose rows
        // of Ns entries are read like the data's, small enough that a tile's
        // part stays in the L1 (one table of all M entries, read beside the
        // data, doubled the L2 reads of the pass: 131072 x 128 125 -> 110 us)
        const int64_t rows = Lq / rad[0];
        if ((rows + rad[0]) * Ns <= (int64_t)1 << 20) {
            a.otw2d = 1;
            st.hi_off = trial.add_outer(Ns, rows, M);
            st.lo_off = trial.add_pass_table(Ns, rad[0]);
        } else {
            int shift = 0;
            while ((int64_t(1) << (2 * shift)) < M) ++shift;
            a.otw_shift = shift;
            st.lo_off = trial.add_linear(int64_t(1) << shift, M, 1);
            st.hi_off = trial.add_linear(ceil_div(M, int64_t(1) << shift), M, int64_t(1) << shift);
        }
    }
    tb = trial;
    a.ip = ip;
    a.tile = 1;
    a.tfpc = W;
    a.tfp = W;
    a.pshift = ps;
    a.nbuf = 1;
    a.wsize = (int32_t)buf;
    a.spitch = spitch;
    a.smem_bytes = (int32_t)smem;
    return true;
}

bool make_col_step(int64_t n, int64_t S, int64_t items, int64_t D, int Lq, int64_t Ns, TwiddleBuilder& tb, Step& st,
                   bool column_kernel = false);

// The two column passes of a long even real transform (complex length L = Lq
// * Ns) with the even/odd packing on chip: the last pass of an R2C and the
// first of a C2R run on tiles of paired columns.  Both passes read and write
// HBM once; the packing as a third pass was a third of the traffic (R2C
// 262144 x 128 162 -> 149 us, C2R 162 -> 156).  src -> mid -> dst, rows of the
// middle buffer mid_dist apart.  False when a pass has no tile.
bool make_pair_steps(int64_t L, int64_t batch, bool r2c, int weight, int src, int mid, int64_t mid_dist, int dst,
                     const std::vector<int>& fac, TwiddleBuilder& tb, std::vector<Step>& out)
{
    TwiddleBuilder trial = tb;
    const int64_t nb = L + 1;
    Step a, b;
    if (!make_col_step(L, 1, batch, L, fac[0], 1, trial, a) || !make_col_step(L, 1, batch, L, fac[1], fac[0], trial, b))
        return false;
    if (!a.col.tile || !b.col.tile) return false;
    // the paired pass: half a tile of neighbouring columns each way (R2C 16
    // columns, 149 us against 164 with 8; C2R 8, 156 against 160 with 16)
    Step& ps = r2c ? b : a;
    ColArgs& c = ps.col;
    const int Lq = c.ip.L;
    const std::vector<int> rad = choose_tile_radices(Lq, !r2c);
    int T = tile_threads(Lq, rad);
    int W = r2c ? 16 : 8;
    while (W > 8 && W * T > kTileMaxThreads) W >>= 1;
    if (W * T > kTileMaxThreads) return false;
    // few pairs, as for few columns in make_tile_col: half the width, a thread
    // for every butterfly (R2C, us: 30000 x 4 11.7 -> 10.4, 36000 x 1 11.9 -> 10.2)
    const int64_t pairs = batch * (L / Lq / 2 + 1);
    if (!pair_compiled(r2c, Lq, T, W, rad)) {
        while (W > 8 && pairs / (W / 2) < 2 * kSMs) W >>= 1;
        int T1 = 1;
        for (int r : rad) T1 = std::max(T1, Lq / r);
        if (T1 * W <= kTileMaxThreads && 2 * pairs * T1 <= kSMs * 256) T = T1;
    }
    if (!build_inner(Lq, rad, T, trial, c.ip)) return false;
    c.pshift = tile_pshift(Lq, rad, !r2c);
    c.pair_m = (int32_t)(L / Lq);
    c.tfpc = W;
    c.tfp = W;
    c.io_mode = r2c ? IO_R2C_EVEN : IO_C2R_EVEN;
    c.weight = weight;
    c.cpi = c.pair_m / 2 + 1;
    c.ncols = batch * c.cpi;
    if (c.ncols * 2 >= kTileMaxCols) return false;
    c.in_split = c.out_split = c.cpi;
    int64_t buf = (int64_t)W * (Lq + (Lq >> c.pshift));
    c.spitch = 0;
    if (!r2c) {
        c.spitch = Lq;
        while (c.spitch % 16 != 16 / W % 16) ++c.spitch;
        buf = std::max<int64_t>(buf, (int64_t)W * c.spitch);
    }
    c.wsize = (int32_t)buf;
    c.smem_bytes = (int32_t)(buf * 8);
    if (c.smem_bytes > kMaxSmemBytes) return false;
    ps.post_off = trial.add_linear(L + 1, 2 * L, 1);
    a.col.in_dist = r2c ? L : nb;
    a.col.out_dist = b.col.in_dist = mid_dist;
    b.col.out_dist = r2c ? nb : L;
    if (!r2c) b.col.conj_out = 1;
    a.src = src;
    a.dst = b.src = mid;
    b.dst = dst;
    tb = trial;
    out.push_back(a);
    out.push_back(b);
    return true;
}

// One column pass over an axis of length n (stride S between samples, S
// independent columns per item, `items` items `D` apart).  The pass runs the
// q-th factor Lq of the axis decomposition after a product Ns of earlier
// factors (outer Stockham pass); Ns == 1 and Lq == n is a plain strided
// transform.  column_kernel: not on tiles (see build_steps; and the allocation-
// free path, whose twiddles live in a fixed array).
bool make_col_step(int64_t n, int64_t S, int64_t items, int64_t D, int Lq, int64_t Ns, TwiddleBuilder& tb, Step& st,
                   bool column_kernel)
{
    std::vector<int> rad = choose_radices(Lq);
    if (rad.empty()) return false;
    const int rmax = *std::max_element(rad.begin(), rad.end()) > 16 ? 47 : 16;
    const int maxthr = max_threads_for(rmax);
    const bool staged_out = (S == 1 && Ns == 1 && Lq != n);
    const int writes = (int)rad.size() - (staged_out ? 0 : 1);
    const int nbuf = writes >= 2 ? 2 : 1;
    const int64_t cpi = (n / Lq) * S;
    // widest column group that fits
    int tf = 16;
    int nthr = 1;
    for (; tf >= 1; tf >>= 1) {
        const int tfp = tf + 1;
        if ((int64_t)nbuf * Lq * tfp * 8 > kMaxSmemBytes) continue;
        nthr = pick_nthr(Lq, rad, std::max(1, maxthr / tf));
        if (nthr * tf > maxthr) continue;
        if ((int64_t)nbuf * Lq * tfp * 8 > 110 * 1024 && tf > 4) continue;
        break;
    }
    if (tf < 1) return false;
    st = Step{};
    st.kind = Step::COL;
    ColArgs& a = st.col;
    a.ncols = items * cpi;
    a.cpi = cpi;
    a.in_dist = D;
    a.in_split = cpi;
    a.in_hi = 0;
    a.in_lo = 1;
    a.in_stride = (n / Lq) * S;
    a.out_dist = D;
    a.out_split = Ns * S;
    a.out_hi = Ns * Lq * S;
    a.out_lo = 1;
    a.out_stride = Ns * S;
    a.ons = Ns;
    a.tw_div = S;
    a.tfpc = tf;
    a.tfp = tf + 1;
    a.nbuf = nbuf;
    a.staged_out = staged_out ? 1 : 0;
    a.scale = 1.f;
    st.tw_off = 0;
    if (!column_kernel && make_tile_col(S, Lq, Ns, staged_out, tb, st)) return true;
    if (!build_inner(Lq, rad, nthr, tb, a.ip)) return false;
    if (Ns > 1) {
        const int64_t M = Ns * Lq;
        int shift = 0;
        while ((int64_t(1) << (2 * shift)) < M) ++shift;  // 2^shift >= sqrt(M)
        a.otw_shift = shift;
        st.lo_off = tb.add_linear(int64_t(1) << shift, M, 1);
        st.hi_off = tb.add_linear(ceil_div(M, int64_t(1) << shift), M, int64_t(1) << shift);
    }
    return true;
}

// Whole batched transform on thread-block clusters (one cluster per
// transform, see csrc/cluster_fft.cuh): a C2C of length n (io_mode IO_C2C)
// or an even R2C / C2R of real length 2n with the packing fused
// (IO_R2C_EVEN / IO_C2R_EVEN).  False when no configuration exists.
bool make_cluster_step(int64_t n, int64_t batch, TwiddleBuilder& tb, Step& st, int io_mode = IO_C2C,
                       int weight = WEIGHT_NONE)
{
    if (!clusters_enabled() || n > 0x7fffffff) return false;
    const char* env_c = std::getenv("OPS_FFT_CLUSTER_C");
    const int want_c = (t_hints && t_hints->cluster_c > 0) ? t_hints->cluster_c : (env_c ? std::atoi(env_c) : 0);
    int C = 0, Q = 0, P = 0, Q0 = 0, P0 = 0, nt = 0, smem = 0;
    const int kid = gfft_cluster_lookup(n, want_c, &C, &Q, &P, &Q0, &P0, &nt, &smem);
    if (kid < 0) return false;
    st = Step{};
    st.kind = Step::CLUSTER;
    ClusterArgs& a = st.cl;
    a.kid = kid;
    a.csize = C;
    a.ntf = batch;
    a.in_dist = io_mode == IO_C2R_EVEN ? n + 1 : n;
    a.out_dist = io_mode == IO_R2C_EVEN ? n + 1 : n;
    a.io_mode = io_mode;
    a.weight = weight;
    a.conj_out = io_mode == IO_C2R_EVEN ? 1 : 0;
    a.post_off = io_mode == IO_C2C ? 0 : tb.add_linear(n + 1, 2 * n, 1);
    a.twq_off = tb.add_pass_table(Q0, Q / Q0);
    a.twp_off = tb.add_pass_table(P0, P / P0);
    a.outer_off = tb.add_linear(n, n, 1);
    a.scale = 1.f;
    a.smem_bytes = smem;
    a.clusters = 0;
    a.length = (int32_t)n;
    st.tw_off = 0;
    return true;
}

// Lengths that a row kernel holds in one thread group (n <= 4096) run on a
// cluster only for batches of at most OPS_FFT_CLUSTER_MAXBATCH transforms
// (default 0: never) or when the autotuner chose it; longer lengths always
// prefer a cluster.  Measured C2C 4096 (us, cluster vs row codelet): b = 8
// 3.57 / 3.62, 64 4.50 / 3.70, 256 7.04 / 5.22, 1024 18.5 / 16.1; R2C 8192
// b = 64 5.44 / 4.17, 256 9.16 / 7.02.
bool cluster_for_batch(int64_t n, int64_t batch)
{
    if (n > 4096) return true;
    if (t_hints && t_hints->cluster == 1) return true;
    const char* v = std::getenv("OPS_FFT_CLUSTER_MAXBATCH");
    return batch <= (v ? (int64_t)std::atoll(v) : (int64_t)0);
}

// Nothing asks for a cluster or for another row kernel.
bool row_tile_beats_cluster(int io_mode)
{
    return clusters_enabled() && codelets_enabled() && !codelet_asked(io_mode) && !std::getenv("OPS_FFT_CLUSTER_C") &&
           !std::getenv("OPS_FFT_CLUSTER_MAXBATCH") && !(t_hints && (t_hints->cluster >= 0 || t_hints->cluster_c > 0));
}

// Strided-axis transform as a list of column passes with buffer routing.
bool make_axis_steps(int64_t n, int64_t S, int64_t items, int64_t D, int src, int dst, int spare, int cap,
                     TwiddleBuilder& tb, std::vector<Step>& out, bool& needs_spare, bool column_kernel = false)
{
    std::vector<int> fac = split_axis(n, cap);
    if (fac.empty()) return false;
    const int Q = (int)fac.size();
    // routing: pass q reads b[q] and writes b[q+1].  Only the last pass may
    // run in place (its read set equals its write set); every other pass
    // must write a buffer different from the one it reads, and `src` may be
    // reused as scratch only after the first pass consumed it.
    std::vector<int> b(Q + 1);
    b[0] = src;
    b[Q] = dst;
    if (Q >= 2) {
        b[Q - 1] = dst;
        for (int q = Q - 2; q >= 1; --q) b[q] = (b[q + 1] == dst) ? spare : dst;
        if (b[1] == src) {
            if (Q != 2) return false;
            b[1] = spare;
        }
    }
    needs_spare = false;
    int64_t Ns = 1;
    for (int q = 0; q < Q; ++q) {
        Step st;
        if (!make_col_step(n, S, items, D, fac[q], Ns, tb, st, column_kernel)) return false;
        st.src = b[q];
        st.dst = b[q + 1];
        if (st.src == spare || st.dst == spare) needs_spare = true;
        out.push_back(st);
        Ns *= fac[q];
    }
    return true;
}

bool row_feasible(int L, int io_mode)
{
    TwiddleBuilder scratch;
    Step st;
    const bool even = io_mode == IO_R2C_EVEN || io_mode == IO_C2R_EVEN;
    const int64_t in_dist = io_mode == IO_C2R_EVEN ? L + 1 : (io_mode == IO_C2R_ODD ? L / 2 + 1 : L);
    const int64_t out_dist = io_mode == IO_R2C_EVEN ? L + 1 : (io_mode == IO_R2C_ODD ? L / 2 + 1 : L);
    return make_row_step(L, 1, in_dist, out_dist, io_mode, even ? 2 * L : L, WEIGHT_NONE, scratch, st);
}

}  // namespace

std::vector<int> split_axis(int64_t n, int cap)
{
    if (!length_supported(n)) return {};
    if (n <= cap) return {(int)n};
    // smallest number of factors; balanced (closest to n^(1/Q))
    std::vector<int64_t> divs;
    for (int64_t d = 2; d <= cap && d < n; ++d)
        if (n % d == 0) divs.push_back(d);
    for (int Q = 2; Q <= 4; ++Q) {
        const double target = std::pow((double)n, 1.0 / Q);
        std::vector<int> best;
        double best_score = 1e300;
        std::vector<int> cur;
        std::function<void(int64_t, int)> dfs = [&](int64_t rem, int left) {
            if (left == 1) {
                if (rem > cap || rem < 2) return;
                cur.push_back((int)rem);
                double score = 0;
                for (int f : cur) score += std::fabs(std::log((double)f / target));
                if (score < best_score) {
                    best_score = score;
                    best = cur;
                }
                cur.pop_back();
                return;
            }
            for (int64_t d : divs) {
                if (rem % d || rem / d < 2) continue;
                cur.push_back((int)d);
                dfs(rem / d, left - 1);
                cur.pop_back();
            }
        };
        dfs(n, Q);
        if (!best.empty()) {
            // largest factor first: the first pass writes contiguous blocks
            std::sort(best.begin(), best.end(), std::greater<int>());
            return best;
        }
    }
    return {};
}

bool build_scratch_c2c_steps(int64_t n, int64_t batch, TwiddleBuilder& tb, std::vector<Step>& out)
{
    out.clear();
    if (n < 2 || batch < 1 || !length_supported(n)) return false;
    const std::vector<int> fac = split_axis(n, col_max_length());
    if (fac.size() != 2) return false;
    Step first, second;
    if (!make_col_step(n, 1, batch, n, fac[0], 1, tb, first, true) ||
        !make_col_step(n, 1, batch, n, fac[1], fac[0], tb, second, true))
        return false;
    first.src = BUF_IN;
    first.dst = BUF_WS;
    second.src = BUF_WS;
    second.dst = BUF_OUT;
    out.push_back(first);
    out.push_back(second);
    return true;
}

namespace {

// One tensor-core pass over sequences q = b*S + s of length L = R*R.
Step tc_step(int L, int prec, int64_t nseq, int64_t S, int64_t in_dist, int64_t in_s, int64_t in_n,
             int64_t out_dist, int64_t out_s, int64_t out_n, int64_t outer_n, TwiddleBuilder& tb)
{
    const int R = L == 256 ? 16 : 8;
    const int TS = 128 / R;
    Step st;
    st.kind = Step::TC;
    TcArgs& a = st.tc;
    a.R = R;
    a.prec = prec;
    a.nseq = nseq;
    a.S = S;
    a.in_dist = in_dist;
    a.in_s = in_s;
    a.in_n = in_n;
    a.out_dist = out_dist;
    a.out_s = out_s;
    a.out_n = out_n;
    a.scale = 1.0f;
    auto mode = [&](int64_t dist, int64_t ss, int64_t sn) {
        // interleaved: side-by-side sequences, whole 16-byte pairs per tile
        if (ss == 1 && S % TS == 0 && nseq % TS == 0 && dist % 2 == 0 && sn % 2 == 0) return (int)TC_IO_INTERLEAVED;
        if (sn == 1 && ss % 2 == 0 && dist % 2 == 0) return (int)TC_IO_CONTIG;
        return (int)TC_IO_GENERIC;
    };
    a.in_mode = mode(in_dist, in_s, in_n);
    a.out_mode = mode(out_dist, out_s, out_n);
    st.bmat_off = tb.add_dft_matrix(R, prec);
    st.tw_off = tb.add_linear(L, L, 1);
    if (outer_n > 1) {
        // W_N^e = hi[e >> sh] * lo[e & mask], e < N
        int sh = 0;
        while ((int64_t(1) << (2 * sh)) < outer_n) ++sh;
        a.otw_shift = sh;
        a.otw_lo_n = 1 << sh;
        a.otw_hi_n = (int)(((outer_n - 1) >> sh) + 1);
        st.hi_off = tb.add_linear(a.otw_hi_n, outer_n, int64_t(1) << sh);
        st.lo_off = tb.add_linear(a.otw_lo_n, outer_n, 1);
    }
    return st;
}

}  // namespace

bool build_tc_c2c_steps(int64_t n, int64_t batch, int prec, bool inplace, TwiddleBuilder& tb, std::vector<Step>& out,
                        int64_t& ws_bytes)
{
    if (prec != TC_PREC_TF32X3 && prec != TC_PREC_BF16X3) return false;
    if (batch < 1) return false;
    const int IN = inplace ? BUF_OUT : BUF_IN;
    ws_bytes = 0;
    out.clear();
    if (n == 64 || n == 256) {
        // one pass: sequence b contiguous; S = batch so every tile is one batch item
        Step st = tc_step((int)n, prec, batch, batch, 0, n, 1, 0, n, 1, 1, tb);
        st.src = IN;
        st.dst = BUF_OUT;
        out.push_back(st);
        return true;
    }
    int64_t L1 = 0;
    for (int64_t c : {int64_t(256), int64_t(64)})
        if (n % c == 0 && (n / c == 64 || n / c == 256)) {
            L1 = c;
            break;
        }
    if (!L1) return false;
    const int64_t L2 = n / L1;  // = S of the first pass
    // pass 1: x[b*n + s + L2*n1] -> W_n^{s*k1} * X1 at ws[b*n + s + L2*k1]
    Step p1 = tc_step((int)L1, prec, batch * L2, L2, n, 1, L2, n, 1, L2, n, tb);
    p1.src = IN;
    p1.dst = BUF_WS;
    // pass 2: ws[b*n + k1*L2 + n2] -> out[b*n + k1 + L1*k2]
    Step p2 = tc_step((int)L2, prec, batch * L1, L1, n, L2, 1, n, 1, L1, 1, tb);
    p2.src = BUF_WS;
    p2.dst = BUF_OUT;
    out.push_back(p1);
    out.push_back(p2);
    ws_bytes = n * batch * 8;
    return true;
}

namespace {

// Element addressing of one side of a double-precision pass (see DPassArgs).
struct DLayout {
    int64_t split = 1, hi = 0, lo = 0, stride = 1;
};

// One launch for ntf double-precision transforms of length n (csrc/dtile.cu);
// false when n needs more than one CTA or a radix above 16.  c2r: with the
// Hermitian pre-process.
bool make_dtile(int64_t n, int64_t ntf, bool t_fast, bool c2r, DPassArgs& a)
{
    if (n > 8192 || ntf >= kTileMaxCols) return false;
    const std::vector<int> rad = choose_tile_radices((int)n, c2r, kDTileThreads, kDTileElems);
    if (rad.empty()) return false;
    TwiddleBuilder scratch;  // the tables of ip are FP32 and unused
    const int T = tile_threads((int)n, rad, kDTileElems);
    if ((int)rad.size() > kRagMaxPass || !build_inner((int)n, rad, T, scratch, a.ip)) return false;
    const int ps = tile_pshift((int)n, rad, c2r);
    const int64_t lp = n + (n >> ps);
    int W = 1, threads = 0;
    // work of a CTA of w transforms in units of a full warp's, and the threads it needs
    auto cost = [&](int w, int64_t& need) {
        int64_t c = 0;
        need = 32;
        for (int r : rad) {
            const int64_t nb = r >= kDTileElems ? 1 : kDTileElems / r, bf = w * (n / r);
            need = std::max(need, ceil_div(bf, nb));
            c += ceil_div(bf, 32) * r;
        }
        need = ceil_div(need, 32) * 32;
        return (double)c / w;
    };
    int64_t need = 0;
    if (t_fast) {
        // 8 columns (128-byte segments) where the threads allow it, more while
        // they fill the lanes of their warps better: short axes have few
        // butterflies a column (us, one launch a radix / 8 columns / this: 2D
        // Z2Z 500 x 16 x 64 61 / 93 / 48, 100 x 24 x 100 49 / 42 / 35, Z2D
        // 1551 x 9 x 64 62 / 86 / 46, 49 x 16 x 1305 173 / 218 / 174; 100 x
        // 48 x 60 stays at 8: 51 / 35, 16 columns 36)
        W = 8;
        while (W > 1 && W * T > kDTileThreads) W >>= 1;
        double best = cost(W, need);
        threads = (int)need;
        for (int w = 2 * W; W >= 8 && w <= 32 && ntf / w >= 2 * kSMs && w * lp * 16 <= 72 * 1024; w *= 2) {
            const double c = cost(w, need);
            if (need > kDTileThreads) break;
            if (c < 0.95 * best) {
                best = c;
                W = w;
                threads = (int)need;
            }
        }
    } else {
        // the rows per CTA whose passes fill the lanes of their warps best
        // (a tie goes to fewer; few transforms keep one row a CTA)
        double best = 0;
        for (int w = 1; w * T <= kDTileThreads + 31 && w <= 64 && w * (lp | 1) * 16 <= 72 * 1024; ++w) {
            const double c = cost(w, need);
            if (need > kDTileThreads) break;
            if (threads == 0 || c < 0.98 * best) {
                best = c;
                W = w;
                threads = (int)need;
            }
            if (ntf / w < 2 * kSMs) break;
        }
        if (threads == 0) return false;
    }
    const int64_t pitch = t_fast ? 1 : lp | 1;
    const int64_t smem = (t_fast ? W * lp : W * pitch) * 16;
    if (smem > kMaxSmemBytes) return false;
    a.tile = 1;
    a.n = (int32_t)n;
    a.radix = 1;
    a.ns = 1;
    a.ntf = ntf;
    a.t_fast = t_fast ? 1 : 0;
    a.W = W;
    a.threads = threads;
    a.pshift = ps;
    a.pitch = (int32_t)pitch;
    a.smem_bytes = (int32_t)smem;
    a.scale = 1.0;
    return true;
}

// Double precision: every axis that fits one CTA in one launch
// (csrc/dtile.cu), the others as global-memory Stockham passes
// (csrc/dfft.cu).  A pass never writes the buffer it reads: the passes of an
// axis go src -> WS / WS2 (alternating) -> ... -> OUT, one launch per radix.
bool build_dsteps(const Problem& p, bool inplace, TwiddleBuilder& tb, StepList& out, int64_t& ws_bytes,
                  int64_t& ws2_bytes)
{
    auto unsupported = [&](const char* why) {
        out.supported = false;
        out.why = why;
        return true;
    };
    if (p.weight != WEIGHT_NONE) return unsupported("double precision has no adjoint entries");
    const int IN = inplace ? BUF_OUT : BUF_IN;
    int cur = IN;
    // one axis: ntf transforms of length n; `src` / `dst` the layouts of the
    // first pass's input and the last pass's output, `mid` the layout of the
    // intermediates; io bits of the first and the last pass
    // (in_ws: the last pass writes a workspace instead of the output, for a
    // step that follows; `cur` then names that workspace)
    auto axis = [&](int64_t n, int64_t ntf, DLayout src, DLayout mid, DLayout dst, int io_first, int io_last,
                    bool t_fast, bool in_ws = false, bool c2r = false) -> bool {
        const std::vector<int> rad = choose_radices((int)n);
        if (rad.empty()) return false;
        const int k = (int)rad.size();
        const int64_t toff = tb.add_dtable(n);
        {
            // one launch; in place only where both sides are laid out alike
            Step st;
            st.kind = Step::DPASS;
            const int to = in_ws ? (cur == BUF_WS ? BUF_WS2 : BUF_WS) : BUF_OUT;
            const DLayout& lo = in_ws ? mid : dst;
            const bool alike = src.split == lo.split && src.hi == lo.hi && src.lo == lo.lo && src.stride == lo.stride &&
                               io_first == 0 && io_last == 0;
            if ((cur != to || alike) && make_dtile(n, ntf, t_fast, c2r, st.dp)) {
                DPassArgs& a = st.dp;
                a.io = io_first | io_last;
                a.in_split = src.split;
                a.in_hi = src.hi;
                a.in_lo = src.lo;
                a.in_stride = src.stride;
                a.out_split = lo.split;
                a.out_hi = lo.hi;
                a.out_lo = lo.lo;
                a.out_stride = lo.stride;
                st.dtw_off = toff;
                st.src = cur;
                st.dst = to;
                out.steps.push_back(st);
                cur = to;
                return true;
            }
        }
        int from = cur;
        int next_ws = (from == BUF_WS) ? BUF_WS2 : BUF_WS;
        int64_t ns = 1;
        for (int i = 0; i < k; ++i) {
            const bool last = i + 1 == k;
            int to = (last && !in_ws) ? BUF_OUT : next_ws;
            if (last && from == BUF_OUT) to = next_ws;  // a one-pass axis on the output: via a workspace
            Step st;
            st.kind = Step::DPASS;
            DPassArgs& a = st.dp;
            a.ntf = ntf;
            a.n = (int32_t)n;
            a.radix = rad[i];
            a.ns = (int32_t)ns;
            a.io = (i == 0 ? io_first : 0) | (last ? io_last : 0);
            a.t_fast = t_fast ? 1 : 0;
            a.scale = 1.0;
            const DLayout& li = i == 0 ? src : mid;
            const DLayout& lo = (last && to == BUF_OUT) ? dst : mid;
            a.in_split = li.split;
            a.in_hi = li.hi;
            a.in_lo = li.lo;
            a.in_stride = li.stride;
            a.out_split = lo.split;
            a.out_hi = lo.hi;
            a.out_lo = lo.lo;
            a.out_stride = lo.stride;
            st.dtw_off = toff;
            st.src = from;
            st.dst = to;
            out.steps.push_back(st);
            if (to != BUF_OUT) next_ws = (to == BUF_WS) ? BUF_WS2 : BUF_WS;
            from = to;
            ns *= rad[i];
        }
        if (in_ws) {
            cur = from;
            return true;
        }
        if (from != BUF_OUT) {  // the axis ended in a workspace laid out like the output
            Step cp;
            cp.kind = Step::COPY;
            cp.src = from;
            cp.dst = BUF_OUT;
            out.steps.push_back(cp);
        }
        cur = BUF_OUT;
        return true;
    };

    if (p.kind == Kind::C2C) {
        const int nd = p.rank;
        const int64_t dims[3] = {p.n0, nd >= 2 ? p.n1 : 1, nd == 3 ? p.n2 : 1};
        int64_t total = p.batch * std::max<int64_t>(p.stride, 1);
        for (int a = 0; a < nd; ++a) total *= dims[a];
        for (int a = 0; a < nd; ++a)
            if (!length_supported(dims[a])) return unsupported("length has a prime factor > 47");
        for (int a = nd - 1; a >= 0; --a) {
            const int64_t n = dims[a];
            int64_t S = (nd == 1) ? std::max<int64_t>(p.stride, 1) : 1;
            for (int b = a + 1; b < nd; ++b) S *= dims[b];
            if (n == 1) continue;
            DLayout l;
            l.split = S;
            l.hi = n * S;
            l.lo = 1;
            l.stride = S;
            if (!axis(n, total / n, l, l, l, 0, 0, S > 1)) return unsupported("length not decomposable");
        }
        if (out.steps.empty() && IN != BUF_OUT) {
            Step cp;
            cp.kind = Step::COPY;
            cp.src = IN;
            cp.dst = BUF_OUT;
            out.steps.push_back(cp);
        }
        for (Step& s : out.steps)
            if (s.kind == Step::COPY) s.copy_bytes = total * 16;
        ws_bytes = ws2_bytes = total * 16;
        return true;
    }
    if (p.stride > 1) return unsupported("double-precision real transforms are horizontal");
    const bool d2z = p.kind == Kind::R2C;
    const int nd = p.rank;
    const int64_t dims[3] = {p.n0, nd >= 2 ? p.n1 : 1, nd == 3 ? p.n2 : 1};
    const int64_t n = dims[nd - 1], nb = n / 2 + 1;
    int64_t rows = p.batch;  // rows along the fastest axis
    for (int a = 0; a + 1 < nd; ++a) rows *= dims[a];
    for (int a = 0; a < nd; ++a)
        if (!length_supported(dims[a])) return unsupported("length has a prime factor > 47");
    auto need = [&](int64_t a, int64_t b) {
        ws_bytes = std::max(ws_bytes, a);
        ws2_bytes = std::max(ws2_bytes, b);
    };
    // the slower axes: transforms down the columns of the half spectrum,
    // element stride S = the faster axes' extent (the fastest as nb bins)
    auto col_axis = [&](int a, bool in_ws) -> bool {
        int64_t S = nb;
        for (int b = a + 1; b + 1 < nd; ++b) S *= dims[b];
        DLayout l;
        l.split = S;
        l.hi = dims[a] * S;
        l.lo = 1;
        l.stride = S;
        return axis(dims[a], rows * nb / dims[a], l, l, l, 0, 0, true, in_ws);
    };
    if (!d2z) {
        // Z2D: the backward column transforms first, into a workspace
        const size_t c0 = out.steps.size();
        for (int a = nd - 2; a >= 0; --a)
            if (dims[a] > 1 && !col_axis(a, true)) return unsupported("length not decomposable");
        if (out.steps.size() > c0) {
            out.steps[c0].dp.conj_in = 1;
            out.steps.back().dp.conj_out = 1;
            need(rows * nb * 16, rows * nb * 16);
        }
    }
    const int src = cur;  // the input, or the workspace holding the column result
    const int64_t in_bytes = d2z ? rows * n * 8 : rows * nb * 16;
    if (n % 2 == 0) {
        // even N: the real row is an L = N/2 complex row; an L-point
        // transform and the even/odd post-process (D2Z), or the Hermitian
        // pre-process and an L-point transform (Z2D), as in the FP32 path
        const int64_t L = n / 2;
        DLayout rowL;
        rowL.hi = L;
        const int64_t toff = tb.add_dtable(n);  // W_N^k for the pre/post-process
        Step pp;
        pp.kind = Step::DPASS;
        DPassArgs& a = pp.dp;
        a.ntf = rows;
        a.n = (int32_t)n;
        a.radix = 1;
        a.ns = 1;
        a.scale = 1.0;
        a.in_split = a.out_split = 1;
        a.in_stride = a.out_stride = 1;
        pp.dtw_off = toff;
        // packing and transform in one launch when it fits and nothing is
        // overwritten that is still to be read (rows of both sides differ)
        Step one;
        one.kind = Step::DPASS;
        if (src != BUF_OUT && make_dtile(L, rows, false, !d2z, one.dp)) {
            DPassArgs& f = one.dp;
            f.io = d2z ? DIO_PAIR_IN | DIO_R2C_POST : DIO_C2R_PRE | DIO_PAIR_OUT;
            f.in_split = f.out_split = 1;
            f.in_stride = f.out_stride = 1;
            f.in_hi = d2z ? L : nb;
            f.out_hi = d2z ? nb : L;
            f.conj_out = d2z ? 0 : 1;
            one.dtw_off = tb.add_dtable(L);
            one.post_off = toff;
            one.src = src;
            one.dst = BUF_OUT;
            out.steps.push_back(one);
            cur = BUF_OUT;
        } else if (d2z) {
            if (!axis(L, rows, rowL, rowL, rowL, DIO_PAIR_IN, 0, false, true))
                return unsupported("length not decomposable");
            a.io = DIO_R2C_POST;
            a.in_hi = L;
            a.out_hi = nb;
            pp.src = cur;
            pp.dst = BUF_OUT;
            out.steps.push_back(pp);
        } else {
            a.io = DIO_C2R_PRE;
            a.in_hi = nb;
            a.out_hi = L;
            pp.src = src;
            pp.dst = src == BUF_WS2 ? BUF_WS : BUF_WS2;
            out.steps.push_back(pp);
            cur = pp.dst;
            if (!axis(L, rows, rowL, rowL, rowL, 0, DIO_PAIR_OUT, false, false, true)) return unsupported("length not decomposable");
            out.steps.back().dp.conj_out = 1;  // the backward transform as a forward one
        }
        need(rows * std::max<int64_t>(L, nb) * 16, rows * std::max<int64_t>(L, nb) * 16);
    } else {
        if (src == BUF_OUT) {
            // in place: input and output rows have different pitches, the
            // input moves to the second workspace first
            Step cp;
            cp.kind = Step::COPY;
            cp.copy_bytes = in_bytes;
            cp.src = BUF_OUT;
            cp.dst = BUF_WS2;
            out.steps.push_back(cp);
            cur = BUF_WS2;
        }
        DLayout full, half, real;
        full.hi = n;
        half.hi = nb;
        real.hi = n;
        if (!axis(n, rows, d2z ? real : half, full, d2z ? half : real, d2z ? DIO_REAL_IN : DIO_HERM_IN,
                  d2z ? DIO_HALF_OUT : DIO_REAL_OUT, false))
            return unsupported("length not decomposable");
        need(rows * n * 16, std::max<int64_t>(rows * n * 16, in_bytes));
    }
    // (the rows start from the input, its copy or the column result in a
    // workspace, never from the output, so their last pass writes the output
    // directly: a copy could not change the row pitch)
    for (const Step& s : out.steps)
        if (s.kind == Step::COPY && s.dst == BUF_OUT) return false;
    if (d2z) {
        // D2Z: the forward column transforms last, over the half spectrum
        cur = BUF_OUT;
        for (int a = nd - 2; a >= 0; --a)
            if (dims[a] > 1 && !col_axis(a, false)) return unsupported("length not decomposable");
        for (Step& s : out.steps)
            if (s.kind == Step::COPY && s.dst == BUF_OUT) s.copy_bytes = rows * nb * 16;
        if (nd > 1) need(rows * nb * 16, rows * nb * 16);
    }
    return true;
}

}  // namespace

bool build_steps(const Problem& p, bool inplace, TwiddleBuilder& tb, StepList& out, int64_t& ws_bytes,
                 int64_t& ws2_bytes)
{
    if (p.dbl) {
        const HintScope hints(&p.hints);
        out = StepList{};
        ws_bytes = 0;
        ws2_bytes = 0;
        return build_dsteps(p, inplace, tb, out, ws_bytes, ws2_bytes);
    }
    const HintScope hints(&p.hints);
    out = StepList{};
    ws_bytes = 0;
    ws2_bytes = 0;
    auto unsupported = [&](const char* why) {
        out.supported = false;
        out.why = why;
        return true;
    };
    const int cap = col_max_length();
    const int IN = inplace ? BUF_OUT : BUF_IN;
    auto need_ws = [&](int64_t bytes) { ws_bytes = std::max(ws_bytes, bytes); };
    auto need_ws2 = [&](int64_t bytes) { ws2_bytes = std::max(ws2_bytes, bytes); };

    if (p.rank == 2 || p.rank == 3) {
        const int nd = p.rank;
        const int64_t dims[3] = {p.n0, p.n1, p.rank == 3 ? p.n2 : 1};
        for (int a = 0; a < nd; ++a)
            if (!length_supported(dims[a])) return unsupported("multi-dimensional length has a prime factor > 47");
        const int64_t last = dims[nd - 1];
        int64_t outer = p.batch;  // rows along the fastest axis
        for (int a = 0; a + 1 < nd; ++a) outer *= dims[a];
        // beside rows with a prime above 16, on the generic row kernel, the
        // strided axes of few points stay on the column kernel: a tile's code is
        // cold after that kernel's, and the passes are too short to make up for
        // it.  All axes or none (kernels of three kinds are colder still), none
        // where a compiled tile or an axis of 16 points, one pass without an
        // exchange, waits, and of 2D transforms those of 17 to 90 points (us,
        // tiles / column kernel: 3D 60 x 21 x 19 19.0 / 16.1, 32 x 30 x 41 24.9 /
        // 22.2, 21 x 125 x 41 27.7 / 25.6, 200 x 60 x 41 30.5 / 28.2, 8 x 21 x 38 17.1
        // / 15.1, but 16 x 96 x 38 20.9 / 22.8, 135 x 16 x 38 18.0 / 20.1; 2D 470 x
        // 20 x 41 23.3 / 21.7, 2 x 80 x 86 20.3 / 18.9, but 1 x 75 x 34 15.4 / 16.1,
        // 1 x 16 x 205 20.1 / 21.3, 1 x 300 x 86 25.5 / 26.3)
        const int64_t row_len = p.kind == Kind::C2C || last % 2 ? last : last / 2;
        const std::vector<int> row_rad = row_len <= row_max_length() ? choose_radices((int)row_len) : std::vector<int>{};
        bool column_kernel = !row_rad.empty() && *std::max_element(row_rad.begin(), row_rad.end()) > 16 &&
                             outer * (p.kind == Kind::C2C ? last : last / 2 + 1) <= (int64_t)1 << 18;
        int strided = 0;
        for (int a = 0; a + 1 < nd; ++a) strided += dims[a] > 1;
        for (int a = 0; a + 1 < nd && column_kernel; ++a) {
            const int64_t n = dims[a];
            if (n > 1 && (n > cap || n == 16 || column_tile_compiled((int)n) || (strided == 1 && (n < 16 || n > 90))))
                column_kernel = false;
        }

        if (p.kind == Kind::C2C) {
            // one transform per axis, fastest first: the first pass reads the
            // input, every later pass works on the output (strided columns)
            const int64_t bytes = outer * last * 8;
            int cur = IN;
            int64_t S = 1;
            for (int a = nd - 1; a >= 0; --a) {
                const int64_t n = dims[a];
                const int64_t items = outer * last / (n * S);
                bool spare = false;
                if (n > 1) {
                    if (S == 1 && n <= row_max_length() && row_feasible((int)n, IO_C2C)) {
                        Step st;
                        if (!make_row_step((int)n, items, n, n, IO_C2C, 0, WEIGHT_NONE, tb, st)) return false;
                        st.src = cur;
                        st.dst = BUF_OUT;
                        out.steps.push_back(st);
                    } else if (!make_axis_steps(n, S, items, n * S, cur, BUF_OUT, BUF_WS, cap, tb, out.steps, spare,
                                                S > 1 && column_kernel)) {
                        return unsupported("multi-dimensional axis length not decomposable");
                    }
                    cur = BUF_OUT;
                }
                if (spare) need_ws(bytes);
                S *= n;
            }
            if (out.steps.empty() && IN != BUF_OUT) {  // every length 1: a copy
                Step cp;
                cp.kind = Step::COPY;
                cp.copy_bytes = bytes;
                cp.src = IN;
                cp.dst = BUF_OUT;
                out.steps.push_back(cp);
            }
            return true;
        }

        // real 2D / 3D: rows along the fastest axis through the 1D real
        // planner, the slower axes as column passes over the half spectrum
        // (element stride: the product of the faster axes, the fastest
        // counted as last/2 + 1 bins)
        const int64_t nb = last / 2 + 1;
        const int64_t half_bytes = outer * nb * 8;
        auto col_stride = [&](int a) {
            int64_t S = nb;
            for (int b = a + 1; b + 1 < nd; ++b) S *= dims[b];
            return S;
        };
        auto col_items = [&](int a) {
            int64_t it = p.batch;
            for (int b = 0; b < a; ++b) it *= dims[b];
            return it;
        };
        Problem rows;
        rows.hints = p.hints;
        rows.kind = p.kind;
        rows.n0 = last;
        rows.batch = outer;
        rows.weight = p.weight;
        StepList sub;
        int64_t sub_ws = 0, sub_ws2 = 0;
        bool spare = false;
        if (p.kind == Kind::R2C) {
            if (!build_steps(rows, inplace, tb, sub, sub_ws, sub_ws2)) return false;
            if (!sub.supported) return unsupported(sub.why.c_str());
            out.steps = sub.steps;
            need_ws(sub_ws);
            need_ws2(sub_ws2);
            for (int a = nd - 2; a >= 0; --a) {
                const int64_t n = dims[a], S = col_stride(a);
                if (n == 1) continue;
                if (!make_axis_steps(n, S, col_items(a), n * S, BUF_OUT, BUF_OUT, BUF_WS, cap, tb, out.steps, spare,
                                     column_kernel))
                    return unsupported("column length not decomposable");
                if (spare) need_ws(half_bytes);
            }
            return true;
        }
        // C2R: backward column transforms of the half spectrum into the
        // second work area (the input stays intact), then the real rows
        bool cols = false;
        for (int a = 0; a + 1 < nd; ++a) cols |= dims[a] > 1;
        if (!build_steps(rows, cols ? false : inplace, tb, sub, sub_ws, sub_ws2)) return false;
        if (!sub.supported) return unsupported(sub.why.c_str());
        if (cols) {
            int from = IN;
            for (int a = nd - 2; a >= 0; --a) {
                const int64_t n = dims[a], S = col_stride(a);
                if (n == 1) continue;
                if (!make_axis_steps(n, S, col_items(a), n * S, from, BUF_WS2, BUF_WS, cap, tb, out.steps, spare,
                                     column_kernel))
                    return unsupported("column length not decomposable");
                if (spare) need_ws(half_bytes);
                from = BUF_WS2;
            }
            out.steps.front().col.conj_in = 1;
            out.steps.back().col.conj_out = 1;
            need_ws2(half_bytes);
            for (Step& s : sub.steps) {
                if (s.src == BUF_WS2 || s.dst == BUF_WS2)
                    return unsupported("C2R rows of this length need a second work area of their own");
                if (s.src == BUF_IN) s.src = BUF_WS2;
            }
        }
        out.steps.insert(out.steps.end(), sub.steps.begin(), sub.steps.end());
        need_ws(sub_ws);
        need_ws2(sub_ws2);
        return true;
    }

    const int64_t N = p.n0;
    if (!length_supported(N)) return unsupported("length has a prime factor > 47");

    if (p.kind == Kind::C2C) {
        if (p.prec != 0 && p.stride == 1) {
            int64_t ws = 0;
            std::vector<Step> tc;
            if (build_tc_c2c_steps(N, p.batch, p.prec, inplace, tb, tc, ws)) {
                out.steps = tc;
                need_ws(ws);
                return true;
            }
        }
        bool spare = false;
        if (p.stride > 1) {
            // VERTICAL: transforms down the columns of [N][stride]
            if (!make_axis_steps(N, p.stride, 1, N * p.stride, IN, BUF_OUT, BUF_WS, cap, tb, out.steps, spare))
                return unsupported("vertical length not decomposable");
            if (spare) need_ws(N * p.stride * 8);
            return true;
        }
        // 8192 points also fit one CTA: from 64 rows faster than a cluster of
        // four (us: 16 rows 5.5 / 4.7, 64 5.5 / 6.0, 128 7.2 / 8.7, 512 18.9 /
        // 19.1, 8192 208 / 237)
        if (N == 8192 && p.batch >= 64 && row_tile_beats_cluster(IO_C2C)) {
            Step st;
            if (make_tile_row_step((int)N, p.batch, N, N, IO_C2C, 0, WEIGHT_NONE, tb, st)) {
                st.src = IN;
                st.dst = BUF_OUT;
                out.steps.push_back(st);
                return true;
            }
        }
        if (cluster_for_batch(N, p.batch)) {
            Step st;
            if (make_cluster_step(N, p.batch, tb, st)) {
                st.src = IN;
                st.dst = BUF_OUT;
                out.steps.push_back(st);
                return true;
            }
        }
        if (N <= row_max_length() && row_feasible((int)N, IO_C2C)) {
            Step st;
            if (!make_row_step((int)N, p.batch, N, N, IO_C2C, 0, WEIGHT_NONE, tb, st)) return false;
            st.src = IN;
            st.dst = BUF_OUT;
            out.steps.push_back(st);
            return true;
        }
        if (!make_axis_steps(N, 1, p.batch, N, IN, BUF_OUT, BUF_WS, cap, tb, out.steps, spare))
            return unsupported("length not decomposable");
        if (spare) need_ws(N * p.batch * 8);
        return true;
    }

    if (p.stride > 1) return unsupported("VERTICAL layout is not supported for R2C/C2R");
    const bool r2c = p.kind == Kind::R2C;
    const int64_t nb = N / 2 + 1;
    const int64_t in_bytes = r2c ? N * p.batch * 4 : nb * p.batch * 8;
    // A single fused kernel reads rows of one pitch and writes rows of
    // another, so an in-place call first copies the input to the workspace.
    auto single = [&](int io_mode, int L, int64_t in_dist, int64_t out_dist, bool tile = false) {
        Step st;
        if (tile ? !make_tile_row_step(L, p.batch, in_dist, out_dist, io_mode, (int)N, p.weight, tb, st)
                 : !make_row_step(L, p.batch, in_dist, out_dist, io_mode, (int)N, p.weight, tb, st))
            return false;
        int src = IN;
        if (inplace) {
            Step cp;
            cp.kind = Step::COPY;
            cp.copy_bytes = in_bytes;
            cp.src = BUF_OUT;
            cp.dst = BUF_WS;
            out.steps.push_back(cp);
            need_ws(in_bytes);
            src = BUF_WS;
        }
        st.src = src;
        st.dst = BUF_OUT;
        out.steps.push_back(st);
        return true;
    };
    if (N % 2 == 0) {
        const int64_t L = N / 2;
        const int mode = r2c ? IO_R2C_EVEN : IO_C2R_EVEN;
        const bool row_ok = L <= row_max_length() && row_feasible((int)L, mode);
        // 8192 points also fit one CTA: rows from the batches where its waves
        // fill the chip, clusters below (us, rows / clusters: R2C 16384 x 64
        // 6.8 / 7.3, 128 8.2 / 11.4, 4096 129 / 183; C2R 64 7.3 / 6.3, 512
        // 24.3 / 22.5, 1024 40.9 / 41.5, 4096 144 / 152)
        if (row_ok && L == 8192 && p.batch >= (r2c ? 64 : 1024) && row_tile_beats_cluster(mode)) {
            if (single(mode, (int)L, r2c ? L : nb, r2c ? nb : L, true)) return true;
        }
        if (row_ok && !cluster_for_batch(L, p.batch)) {
            if (!single(mode, (int)L, r2c ? L : nb, r2c ? nb : L)) return false;
            return true;
        }
        // two passes over HBM beat a 16-CTA cluster from 8 rows (us, 131072:
        // R2C x 1 8.9 / 8.6, x 8 10.4 / 11.7, x 64 33 / 46, x 512 223 / 316;
        // C2R x 512 242 / 323); 65536: R2C 114 / 118, C2R 125 / 123.  Out of
        // place the middle result sits in the output, in place in the workspace
        // (which the plan holds for both) that the cluster's copy needs too.
        if (L == 65536 && p.batch >= 8 && row_tile_beats_cluster(mode)) {
            const std::vector<int> fac = split_axis(L, cap);
            if (fac.size() == 2 && make_pair_steps(L, p.batch, r2c, p.weight, IN, inplace ? BUF_WS : BUF_OUT,
                                                   r2c && !inplace ? nb : L, BUF_OUT, fac, tb, out.steps)) {
                if (inplace) need_ws(L * p.batch * 8);
                return true;
            }
        }
        // long real transforms (and short ones in small batches) on a
        // cluster, packing fused (an in-place call first copies the input to
        // the workspace: input and output rows have different pitches)
        {
            Step cl;
            if (cluster_for_batch(L, p.batch) && make_cluster_step(L, p.batch, tb, cl, mode, p.weight)) {
                int src = IN;
                if (inplace) {
                    Step cp;
                    cp.kind = Step::COPY;
                    cp.copy_bytes = in_bytes;
                    cp.src = BUF_OUT;
                    cp.dst = BUF_WS;
                    out.steps.push_back(cp);
                    need_ws(in_bytes);
                    src = BUF_WS;
                }
                cl.src = src;
                cl.dst = BUF_OUT;
                out.steps.push_back(cl);
                return true;
            }
        }
        if (row_ok) return single(mode, (int)L, r2c ? L : nb, r2c ? nb : L);
        // long real transforms: two passes with the packing on chip, the middle
        // result in a workspace
        {
            const std::vector<int> fac = split_axis(L, cap);
            if (fac.size() == 2 &&
                make_pair_steps(L, p.batch, r2c, p.weight, IN, BUF_WS, L, BUF_OUT, fac, tb, out.steps)) {
                need_ws(L * p.batch * 8);
                return true;
            }
        }
        // longer ones: separate packing around a multi-pass C2C
        Step pk;
        pk.kind = Step::PACK;
        pk.pack.L = (int)L;
        pk.pack.ntf = p.batch;
        pk.pack.c2r = r2c ? 0 : 1;
        pk.pack.weight = p.weight;
        pk.pack.scale = 1.f;
        pk.post_off = tb.add_linear(L / 2 + 1, N, 1);
        bool spare = false;
        Step cl;
        const bool use_cluster = make_cluster_step(L, p.batch, tb, cl);
        if (r2c) {
            // input (float2 view) -> ... -> WS, then pack WS -> out
            if (use_cluster) {
                cl.src = IN;
                cl.dst = BUF_WS;
                out.steps.push_back(cl);
            } else if (!make_axis_steps(L, 1, p.batch, L, IN, BUF_WS, BUF_WS2, cap, tb, out.steps, spare)) {
                return unsupported("length not decomposable");
            }
            pk.pack.in_dist = L;
            pk.pack.out_dist = nb;
            pk.src = BUF_WS;
            pk.dst = BUF_OUT;
            out.steps.push_back(pk);
        } else {
            pk.pack.in_dist = nb;
            pk.pack.out_dist = L;
            pk.src = IN;
            pk.dst = BUF_WS;
            out.steps.push_back(pk);
            if (use_cluster) {
                cl.src = BUF_WS;
                cl.dst = BUF_OUT;
                cl.cl.conj_out = 1;
                out.steps.push_back(cl);
            } else {
                if (!make_axis_steps(L, 1, p.batch, L, BUF_WS, BUF_OUT, BUF_WS2, cap, tb, out.steps, spare))
                    return unsupported("length not decomposable");
                out.steps.back().col.conj_out = 1;
            }
        }
        need_ws(L * p.batch * 8);
        if (spare) need_ws2(L * p.batch * 8);
        return true;
    }
    // odd N: full-length complex transform inside one CTA
    const int mode = r2c ? IO_R2C_ODD : IO_C2R_ODD;
    if (N <= row_max_length() && row_feasible((int)N, mode)) {
        if (!single(mode, (int)N, r2c ? N : nb, r2c ? nb : N)) return false;
        return true;
    }
    return unsupported("odd real-data length beyond one CTA");
}

// Argument-driven tiles of different modes in one list share a kernel (IO_TILE
// in csrc/tile_fft.cuh).
void share_tiles(std::vector<Step>& steps)
{
    auto rad = [](const InnerPlan& ip) {
        std::vector<int> r;
        for (int p = 0; p < ip.npass; ++p) r.push_back(ip.pass[p].radix);
        return r;
    };
    auto driven = [&](Step& s, int& io) -> int32_t* {
        if (s.kind == Step::ROW) {
            RowArgs& a = s.has_dev ? s.dev : s.row;
            io = a.io_mode;
            return a.tile && io <= IO_C2R_EVEN && !tile_compiled(true, a.ip.L, a.ip.nthr, a.tfpc, rad(a.ip)) ? &a.tile : nullptr;
        }
        if (s.kind != Step::COL || !s.col.tile) return nullptr;
        ColArgs& a = s.col;
        io = a.io_mode;
        const bool compiled = io == IO_C2C ? tile_compiled(false, a.ip.L, a.ip.nthr, a.tfpc, rad(a.ip))
                                           : pair_compiled(io == IO_R2C_EVEN, a.ip.L, a.ip.nthr, a.tfpc, rad(a.ip));
        return compiled ? nullptr : &a.tile;
    };
    int modes = 0, io = 0;
    for (Step& s : steps)
        if (driven(s, io)) modes |= 1 << io;
    if ((modes & (modes - 1)) == 0) return;
    for (Step& s : steps)
        if (int32_t* tile = driven(s, io)) *tile = 2;
}

}  // namespace gfft
