// ragged.cpp - ragged batches: many 1D transforms of different lengths and
// kinds executed by one persistent launch (aclfftRagged* extension).
//
// Plan creation groups the transforms into classes (kind, length), builds
// each class's on-chip plan - one Stockham transform, or a two-step split
// L = La * Lb for lengths beyond one CTA - and the work-item table the
// persistent kernel consumes (csrc/ragged.cu).  Item order: the long
// transforms in groups, a group's second steps (which wait on counters for
// its first steps) one group later, then the on-chip items by decreasing
// cost, so that the launch ends on short items.
//
// Autotuning: per class, candidate radix orders are timed in isolation on
// scratch buffers and the fastest is kept; choices are
// cached process-wide (and in a text file when OPS_FFT_TUNE_CACHE names
// one) keyed by (kind, length), as the radices of the one or two transforms:
// radices that are no candidate of a length any more are tuned again.
//
// Execution: the kernel launch (its last CTA leaves the queue cleared for the
// next one), captured once per (input, output, direction) into a CUDA graph
// on a plan-owned stream and replayed on the caller's stream; when the
// caller's stream is itself being captured, the launch is issued directly
// into that capture.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <fstream>
#include <map>
#include <mutex>
#include <new>
#include <sstream>
#include <string>
#include <type_traits>
#include <vector>

#include "handle.h"

namespace {

using namespace gfft;

constexpr int kThreads = 512;
constexpr int kSmemBudget = 110 * 1024;  // per CTA (two CTAs per SM)
constexpr int kMaxSingle = 4096;         // longest on-chip complex length
constexpr int64_t kMaxLength = 1 << 24;
constexpr int kOuterTable = 1 << 16;     // longest length with a whole outer-twiddle table (512 KB)
constexpr int kPostPairs = 4096;         // bin pairs of one post-process item
constexpr int kResident = 2 * 152;       // CTAs at once: two on each SM of a GB300
// workspace of one group of long transforms: the next group's first steps
// are queued between a group's first and second steps, so the workspace in
// flight is two groups and stays in the L2
constexpr int64_t kGroupBytes = 24 << 20;

enum RagType : int { RAG_C2C = 0, RAG_R2C = 1 };
enum RagMode : int { RAG_MODE_SINGLE = 0, RAG_MODE_LONG = 1 };

// One on-chip transform of length L on the tile scheme.
struct TilePlan {
    int L = 0, T = 0, ps = 30, np = 0;
    PassDesc pass[kRagMaxPass] = {};
    int padded() const { return L + (L >> ps); }
};

// A transform class: one kind and length.
struct RagClass {
    TilePlan p1, p2;   // single: the whole transform (p1); long: La and Lb points
    int n = 0, type = 0, mode = 0;
    int L = 0;         // complex length transformed (n for C2C and odd R2C, n/2 for even R2C)
    int La = 0, Lb = 0;  // long: L = La * Lb
    int group = 0;     // single: transforms per item; long: columns per P1 item
    int group2 = 0;    // long: columns per P2 item
    int pitch = 0;     // single: shared pitch of a row; long: of a staged P1 column
    int otw_shift = 0;
    int64_t post_off = -1, hi_off = -1, lo_off = -1;
    bool even_r2c() const { return type == RAG_R2C && !(n & 1); }
    bool odd_r2c() const { return type == RAG_R2C && (n & 1); }
};

bool primes_le_13(int64_t n)
{
    for (int p : {2, 3, 5, 7, 11, 13})
        while (n % p == 0) n /= p;
    return n == 1;
}

// Candidate radix sequences of length L: the tile planner's choice, the row
// planner's, and the first one's reverse.
std::vector<std::vector<int>> candidates(int L)
{
    std::vector<std::vector<int>> out;
    auto add = [&](const std::vector<int>& r) {
        if (r.empty() || (int)r.size() > kRagMaxPass || tile_threads(L, r) > kThreads) return;
        if (*std::max_element(r.begin(), r.end()) > 16) return;
        if (std::find(out.begin(), out.end(), r) == out.end()) out.push_back(r);
    };
    const std::vector<int> base = choose_tile_radices(L, false, kThreads);
    add(base);
    add(choose_radices(L));
    add(std::vector<int>(base.rbegin(), base.rend()));
    return out;
}

TilePlan tile_plan(int L, const std::vector<int>& rad, TwiddleBuilder& tb)
{
    TilePlan t;
    InnerPlan ip;
    if (!build_inner(L, rad, 1, tb, ip) || ip.npass > kRagMaxPass) return t;
    t.L = L;
    t.T = tile_threads(L, rad);
    t.ps = tile_pshift(L, rad);
    t.np = ip.npass;
    for (int q = 0; q < t.np; ++q) t.pass[q] = ip.pass[q];
    return t;
}

struct Key {
    int type, n;
    bool operator<(const Key& o) const { return type != o.type ? type < o.type : n < o.n; }
};

// Tuned choice per class: variant indices of the first and second transform.
struct Choice {
    int v1 = 0, v2 = 0;
};

std::mutex g_tune_mu;
std::map<Key, std::string> g_tuned;  // tuned radices, see radices_text
bool g_tune_file_loaded = false;

// File lines: "r <kind> <length> <radices>", e.g. "r 0 8192 16.8+8.8"; any
// other line is ignored.
void load_tune_file()
{
    if (g_tune_file_loaded) return;
    g_tune_file_loaded = true;
    const char* path = std::getenv("OPS_FFT_TUNE_CACHE");
    if (!path || !*path) return;
    std::ifstream f(path);
    std::string line;
    while (std::getline(f, line)) {
        std::istringstream is(line);
        std::string tag, radices;
        int t, n;
        if ((is >> tag >> t >> n >> radices) && tag == "r") g_tuned[{t, n}] = radices;
    }
}

void save_tune_file()
{
    const char* path = std::getenv("OPS_FFT_TUNE_CACHE");
    if (!path || !*path) return;
    std::ofstream f(path, std::ios::trunc);
    for (auto& kv : g_tuned) f << "r " << kv.first.type << ' ' << kv.first.n << ' ' << kv.second << '\n';
}

struct ClassPlan {
    RagClass dev{};
    std::vector<TilePlan> cand1, cand2;
    Choice choice;
    bool tuned = false;
    int split = 1;             // long: least items a step is cut into, see split_steps
    std::vector<int> members;  // transform indices
};

}  // namespace

struct aclfftRaggedPlan_t {
    int count = 0;
    std::vector<int> len, type;
    std::vector<int64_t> in_off, out_off;
    std::vector<ClassPlan> classes;
    std::vector<int> cls;         // class of each transform
    std::vector<int64_t> ws_off;  // long transforms: float2 offset of their workspace
    std::vector<RagRow> rows;     // the rows of the single items, in item order
    std::vector<int> row_xf;      // their transforms
    std::vector<RagItem> items;
    TwiddleBuilder tb;
    int64_t ws_floats2 = 0;
    int smem = 0;
    int ctas = 0;  // persistent CTAs for `smem` (0: not computed yet)
    int ctas_smem = -1;
    int nlong = 0;
    int64_t in_min = 0, out_min = 0;
    bool autotune = true, use_graph = true, tuned = false;
    long long wait_cycles = 1ll << 31;  // bound of each dependency wait
    int need_bias = 0;                  // test hook: unreachable dependency counts
    cudaStream_t stream = nullptr;
    // device state
    bool dev_ready = false;
    int device = -1;
    void* tw = nullptr;
    RagRow* d_rows = nullptr;
    RagItem* d_items = nullptr;
    int* d_queue = nullptr;
    int* d_err = nullptr;
    float2* d_ws = nullptr;
    cudaStream_t s_cap = nullptr;
    cudaGraphExec_t gexec = nullptr;
    void* g_in = nullptr;
    void* g_out = nullptr;
    int g_inv = -1;
    cudaStream_t g_stream = nullptr;
};

namespace {

void free_device(aclfftRaggedPlan_t* p)
{
    if (p->gexec) cudaGraphExecDestroy(p->gexec);
    if (p->s_cap) cudaStreamDestroy(p->s_cap);
    for (void* q : {(void*)p->tw, (void*)p->d_rows, (void*)p->d_items, (void*)p->d_queue, (void*)p->d_err, (void*)p->d_ws})
        if (q) cudaFree(q);
    p->gexec = nullptr;
    p->s_cap = nullptr;
    p->tw = nullptr;
    p->d_rows = nullptr;
    p->d_items = nullptr;
    p->d_queue = nullptr;
    p->d_err = nullptr;
    p->d_ws = nullptr;
    p->dev_ready = false;
}

int ctas_for(aclfftRaggedPlan_t* p, int smem);

// The captured graph bakes in the kernel arguments: settings that change
// them force a new capture at the next exec.
void drop_graph(aclfftRaggedPlan_t* p)
{
    if (p->gexec) cudaGraphExecDestroy(p->gexec);
    p->gexec = nullptr;
    p->g_in = p->g_out = nullptr;
    p->g_inv = -1;
}

// Shared memory an item of the class needs with the chosen variants: one
// exchange buffer, for P1 also the staged columns.
int class_smem(const RagClass& c)
{
    if (c.mode == RAG_MODE_SINGLE) return c.group * c.pitch * 8;
    return std::max({c.group * c.p1.padded(), c.group * c.pitch, c.group2 * c.p2.padded()}) * 8;
}

// Spreads m transforms (or columns) evenly over the items they need, W each,
// and gives each the threads that are left, up to one for every butterfly:
// fewer instructions on an item's critical path (10000 transforms, most
// classes with less than a tile of them: 515 -> 444 us).
int spread_tile(TilePlan& t, int W, int64_t m)
{
    int T1 = 1;
    for (int p = 0; p < t.np; ++p) T1 = std::max(T1, t.L / t.pass[p].radix);
    const int64_t items = (m + W - 1) / W;
    W = (int)((m + items - 1) / items);
    t.T = std::max(t.T, std::min(T1, kThreads / W));
    return W;
}

// Tile of an on-chip class with `members` transforms.
void shape_single(RagClass& c, int64_t members)
{
    auto pitch = [&] {
        c.pitch = c.p1.padded() + 1;
        while (c.p1.T < 16 && c.pitch % 16 != c.p1.T % 16) ++c.pitch;
    };
    pitch();
    c.group = std::max(1, std::min(kThreads / c.p1.T, kSmemBudget / (c.pitch * 8)));
    if (members < 1) return;
    c.group = spread_tile(c.p1, c.group, members);
    pitch();
}

// Applies candidate choice ch to the class's plan.
bool apply_choice(ClassPlan& cp, Choice ch)
{
    RagClass& c = cp.dev;
    if (ch.v1 < 0 || ch.v1 >= (int)cp.cand1.size()) return false;
    c.p1 = cp.cand1[ch.v1];
    if (c.mode == RAG_MODE_SINGLE) {
        shape_single(c, (int64_t)cp.members.size());
        c.group2 = 0;
    } else {
        if (ch.v2 < 0 || ch.v2 >= (int)cp.cand2.size()) return false;
        c.p2 = cp.cand2[ch.v2];
        c.pitch = c.La | 1;  // consecutive columns in different banks
        auto cut = [&](int cols) { return (cols + cp.split - 1) / cp.split; };
        c.group = spread_tile(c.p1, std::min(kThreads / c.p1.T, cut(c.Lb)), c.Lb);
        c.group2 = spread_tile(c.p2, std::min(kThreads / c.p2.T, cut(c.La)), c.La);
    }
    cp.choice = ch;
    return class_smem(c) <= kSmemBudget;
}

// The radices of a choice: "16.16.16", of a long transform "16.8+8.8".
std::string radices_text(const ClassPlan& cp, Choice ch)
{
    std::ostringstream os;
    auto put = [&](const TilePlan& t) {
        for (int q = 0; q < t.np; ++q) os << (q ? "." : "") << t.pass[q].radix;
    };
    put(cp.cand1[ch.v1]);
    if (cp.dev.mode == RAG_MODE_LONG) {
        os << '+';
        put(cp.cand2[ch.v2]);
    }
    return os.str();
}

// Applies the choice with these radices; false when there is none any more.
bool apply_radices(ClassPlan& cp, const std::string& radices)
{
    const int n2 = cp.dev.mode == RAG_MODE_LONG ? (int)cp.cand2.size() : 1;
    for (int a = 0; a < (int)cp.cand1.size(); ++a)
        for (int b = 0; b < n2; ++b)
            if (radices_text(cp, {a, b}) == radices) return apply_choice(cp, {a, b});
    return false;
}

double class_cost(const RagClass& c) { return (double)c.L * std::log2((double)std::max(c.L, 2)); }

RagItem tile_item(int kind, const TilePlan& t, int W, int count, int first)
{
    RagItem it{};
    it.kind = kind;
    it.L = t.L;
    it.T = t.T;
    it.W = W;
    it.count = count;
    it.np = t.np;
    it.ps = t.ps;
    it.first = first;
    const int d = kind == RAG_SINGLE ? t.T : W;
    it.wmagic = (uint32_t)(((1 << 20) + d - 1) / d);
    for (int q = 0; q < t.np; ++q) it.pass[q] = t.pass[q];
    return it;
}

void build_items(aclfftRaggedPlan_t* p)
{
    p->items.clear();
    p->rows.clear();
    p->row_xf.clear();
    std::vector<std::pair<double, RagItem>> singles;
    struct Long {
        std::vector<RagItem> p1, p2, post;
    };
    std::vector<Long> groups(1);
    int64_t group_bytes = 0;
    for (int ci = 0; ci < (int)p->classes.size(); ++ci) {
        ClassPlan& cp = p->classes[ci];
        if (cp.dev.mode == RAG_MODE_SINGLE) {
            cp.dev.p1 = cp.cand1[cp.choice.v1];
            shape_single(cp.dev, (int64_t)cp.members.size());
        }
        const RagClass& c = cp.dev;
        const int c2c = c.type == RAG_C2C ? RAG_CONJ_IN : 0;
        if (c.mode == RAG_MODE_SINGLE) {
            for (size_t i = 0; i < cp.members.size(); i += c.group) {
                const int count = (int)std::min<size_t>(c.group, cp.members.size() - i);
                RagItem it = tile_item(RAG_SINGLE, c.p1, c.group, count, (int)p->rows.size());
                it.pitch = c.pitch;
                it.flags = c2c ? RAG_CONJ_IN | RAG_CONJ_OUT : (c.odd_r2c() ? RAG_REAL_IN | RAG_HALF_OUT : RAG_R2C_POST);
                it.nhalf = c.n / 2;
                it.post_off = (int32_t)c.post_off;
                for (int k = 0; k < count; ++k) {
                    const int x = cp.members[i + k];
                    p->rows.push_back({p->in_off[x], p->out_off[x]});
                    p->row_xf.push_back(x);
                }
                singles.push_back({class_cost(c) * count, it});
            }
            continue;
        }
        for (int x : cp.members) {
            const int64_t bytes = (c.even_r2c() ? 2 : 1) * (int64_t)c.L * 8;
            if (group_bytes > 0 && group_bytes + bytes > kGroupBytes) {
                groups.emplace_back();
                group_bytes = 0;
            }
            group_bytes += bytes;
            Long& g = groups.back();
            const int64_t ws = p->ws_off[x];
            int np1 = 0, np2 = 0;
            for (int j = 0; j < c.Lb; j += c.group, ++np1) {
                RagItem it = tile_item(RAG_P1, c.p1, c.group, std::min(c.group, c.Lb - j), j);
                it.xform = x;
                it.pitch = c.pitch;
                it.flags = c2c | (c.odd_r2c() ? RAG_REAL_IN : 0);
                it.stride = c.Lb;
                it.in_off = p->in_off[x];
                it.out_off = ws;
                g.p1.push_back(it);
            }
            for (int j = 0; j < c.La; j += c.group2, ++np2) {
                RagItem it = tile_item(RAG_P2, c.p2, c.group2, std::min(c.group2, c.La - j), j);
                it.xform = x;
                it.need = np1;
                it.flags = c2c ? RAG_CONJ_OUT : (c.odd_r2c() ? RAG_HALF_OUT : RAG_WS_OUT);
                it.nhalf = c.n / 2;
                it.stride = c.La;
                it.in_off = ws;
                it.out_off = c.even_r2c() ? ws + c.L : p->out_off[x];
                it.otw_shift = c.otw_shift;
                it.hi_off = (int32_t)c.hi_off;
                it.lo_off = (int32_t)c.lo_off;
                g.p2.push_back(it);
            }
            for (int k = 0; c.even_r2c() && k <= c.L / 2; k += kPostPairs) {
                RagItem it{};
                it.kind = RAG_POST;
                it.L = c.L;
                it.xform = x;
                it.need = np1 + np2;
                it.first = k;
                it.count = std::min(kPostPairs, c.L / 2 + 1 - k);
                it.in_off = ws + c.L;
                it.out_off = p->out_off[x];
                it.post_off = (int32_t)c.post_off;
                g.post.push_back(it);
            }
        }
    }
    std::stable_sort(singles.begin(), singles.end(),
                     [](const std::pair<double, RagItem>& a, const std::pair<double, RagItem>& b) {
                         return a.first > b.first;
                     });
    auto put = [&](const std::vector<RagItem>& v) { p->items.insert(p->items.end(), v.begin(), v.end()); };
    // group g's second steps one group after its first steps, its
    // post-process one more later; the on-chip items last, longest first, so
    // that the launch ends on short ones
    const size_t ng = groups.size();
    for (size_t g = 0; g < ng + 2; ++g) {
        if (g < ng) put(groups[g].p1);
        if (g >= 1 && g - 1 < ng) put(groups[g - 1].p2);
        if (g >= 2) put(groups[g - 2].post);
    }
    for (auto& s : singles) p->items.push_back(s.second);
    p->smem = 16;
    for (auto& cp : p->classes) p->smem = std::max(p->smem, class_smem(cp.dev));
}

// Items of a plan that leaves CTAs idle: each step of its long transforms is cut
// into at least four (else two) items while all still have a CTA of their own.
// One 512-thread tile holds a whole step of 8192 points, and the two steps wait
// for each other (us, uncut / cut, and before the tiles: 163 transforms of up to
// 8192 points 20.7 / 18.8, 17.1; 10 of them 15.9 / 14.8, 14.8; 20 of 8192 19.6 /
// 16.5, 16.7; 250 22.6 / 18.8, 18.5; into eight: 20 of 8192 19.3, 60 of up to
// 32768 23.2 against 21.2 uncut).
void split_steps(aclfftRaggedPlan_t* p)
{
    auto build = [&](int split) {
        for (auto& cp : p->classes) {
            if (cp.dev.mode != RAG_MODE_LONG) continue;
            cp.split = split;
            apply_choice(cp, cp.choice);
        }
        build_items(p);
    };
    build_items(p);
    const bool any = std::any_of(p->classes.begin(), p->classes.end(),
                                 [](const ClassPlan& cp) { return cp.dev.mode == RAG_MODE_LONG; });
    if (!any || (int)p->items.size() >= kResident) return;
    for (int split : {4, 2, 1}) {
        build(split);
        if ((int)p->items.size() <= kResident) return;
    }
}

template <class T>
bool upload(T*& d, const std::vector<T>& h)
{
    if (d) cudaFree(d);
    d = nullptr;
    const size_t bytes = std::max<size_t>(h.size(), 1) * sizeof(T);
    if (gfft::dev_alloc(reinterpret_cast<void**>(&d), bytes) != cudaSuccess) {
        cudaGetLastError();
        d = nullptr;
        return false;
    }
    if (!h.empty() && cudaMemcpy(d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return true;
}

bool upload_tables(aclfftRaggedPlan_t* p)
{
    return upload(p->d_rows, p->rows) && upload(p->d_items, p->items);
}

aclfftResult device_setup(aclfftRaggedPlan_t* p)
{
    if (p->dev_ready) return ACLFFT_SUCCESS;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return ACLFFT_SETUP_FAILED;
    }
    const size_t twb = (size_t)std::max<int64_t>(p->tb.count, 2) * 8;
    if (gfft::dev_alloc(&p->tw, twb) != cudaSuccess || gfft::dev_alloc(reinterpret_cast<void**>(&p->d_queue),
                                                             (size_t)(p->count + 2) * sizeof(int)) != cudaSuccess ||
        cudaMemset(p->d_queue, 0, (size_t)(p->count + 2) * sizeof(int)) != cudaSuccess ||
        gfft::dev_alloc(reinterpret_cast<void**>(&p->d_err), sizeof(int)) != cudaSuccess ||
        cudaMemset(p->d_err, 0, sizeof(int)) != cudaSuccess ||
        (p->ws_floats2 > 0 &&
         gfft::dev_alloc(reinterpret_cast<void**>(&p->d_ws), (size_t)p->ws_floats2 * sizeof(float2)) != cudaSuccess) ||
        cudaStreamCreateWithFlags(&p->s_cap, cudaStreamNonBlocking) != cudaSuccess) {
        cudaGetLastError();
        free_device(p);
        gfft::set_last_error("ragged plan: device allocation failed");
        return ACLFFT_ALLOC_FAILED;
    }
    if (!p->tb.segs.empty() && (gfft_gen_twiddles(p->tw, p->tb.segs.data(), (int)p->tb.segs.size(), nullptr) != 0 ||
                                cudaDeviceSynchronize() != cudaSuccess)) {
        cudaGetLastError();
        free_device(p);
        gfft::set_last_error("ragged plan: twiddle generation failed");
        return ACLFFT_SETUP_FAILED;
    }
    if (!upload_tables(p)) {
        free_device(p);
        gfft::set_last_error("ragged plan: table upload failed");
        return ACLFFT_ALLOC_FAILED;
    }
    p->device = dev;
    p->ctas = ctas_for(p, p->smem);
    p->ctas_smem = p->smem;
    if (p->ctas <= 0) {
        free_device(p);
        return ACLFFT_SETUP_FAILED;
    }
    p->dev_ready = true;
    return ACLFFT_SUCCESS;
}

// Persistent CTAs for a shared-memory size (attribute calls: not inside a
// stream capture).
int ctas_for(aclfftRaggedPlan_t* p, int smem)
{
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, p->device < 0 ? 0 : p->device) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    const int per_sm = gfft_ragged_ctas(smem);
    if (per_sm <= 0) {
        gfft::set_last_error(std::string("ragged kernel setup: ") +
                             (per_sm < 0 ? cudaGetErrorString((cudaError_t)(-per_sm)) : "no CTA fits an SM"));
        return 0;
    }
    return per_sm * sms;
}

RagArgs make_args(aclfftRaggedPlan_t* p, const RagItem* items, int nitems, int smem, const void* in, void* out,
                  bool inverse)
{
    RagArgs a{};
    a.rows = p->d_rows;
    a.items = items;
    a.nitems = nitems;
    a.smem_bytes = smem;
    a.ctas = smem == p->ctas_smem ? p->ctas : ctas_for(p, smem);
    // (claims ahead, 4 items a CTA or more / fewer: equal within 1 %; all
    // 14000 items of the 10000-transform batch claimed one by one: 554 against
    // 515 us)
    bool deps = false;
    for (auto& cp : p->classes) deps |= cp.dev.mode == RAG_MODE_LONG;
    a.claim = nitems <= a.ctas && !deps ? RAG_CLAIM_NONE
              : nitems < 8 * a.ctas     ? RAG_CLAIM_NEXT
                                        : RAG_CLAIM_AHEAD;
    a.queue = p->d_queue;
    a.count = p->count;
    a.err = p->d_err;
    a.tw = p->tw;
    a.in = in;
    a.out = out;
    a.ws = p->d_ws;
    a.inverse = inverse ? 1 : 0;
    a.scale_c2c = 1.f;
    a.wait_cycles = p->wait_cycles;
    a.need_bias = p->need_bias;
    return a;
}

int launch(aclfftRaggedPlan_t* p, const RagArgs& a, cudaStream_t st)
{
    return gfft_launch_ragged(&a, st);
}

// Times every candidate of every class on its own trial batch: m copies of
// the class's transform (m * n ~ 2^20 points, so a trial launch runs
// several waves like the real batch does) in scratch buffers, with their
// own queue, transform table and workspace.  The fastest candidate is kept
// and cached by (kind, length).
aclfftResult autotune(aclfftRaggedPlan_t* p)
{
    std::lock_guard<std::mutex> lk(g_tune_mu);
    load_tune_file();
    constexpr int64_t kTrialPoints = 1 << 20;
    auto trial_m = [&](const RagClass& c) { return (int)std::min<int64_t>(2048, std::max<int64_t>(4, kTrialPoints / c.n)); };
    auto ws_per = [](const RagClass& c) -> int64_t {
        if (c.mode != RAG_MODE_LONG) return 0;
        return c.even_r2c() ? 2 * (int64_t)c.L : c.L;
    };
    int64_t scratch = 16, wsmax = 1;
    int maxm = 1;
    for (auto& cp : p->classes) {
        const int m = trial_m(cp.dev);
        maxm = std::max(maxm, m);
        scratch = std::max<int64_t>(scratch, (int64_t)m * ((int64_t)cp.dev.n + 2) * 8);
        wsmax = std::max<int64_t>(wsmax, (int64_t)m * ws_per(cp.dev));
    }
    void *sin = nullptr, *sout = nullptr;
    int* squeue = nullptr;
    float2* sws = nullptr;
    RagRow* srows = nullptr;
    RagItem* sitems = nullptr;
    size_t cap_rows = 0, cap_items = 0;
    bool ok = gfft::dev_alloc(&sin, (size_t)scratch) == cudaSuccess && gfft::dev_alloc(&sout, (size_t)scratch) == cudaSuccess &&
              cudaMemset(sin, 0, (size_t)scratch) == cudaSuccess &&
              gfft::dev_alloc(reinterpret_cast<void**>(&squeue), (size_t)(maxm + 2) * sizeof(int)) == cudaSuccess &&
              gfft::dev_alloc(reinterpret_cast<void**>(&sws), (size_t)wsmax * sizeof(float2)) == cudaSuccess;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    ok = ok && cudaEventCreate(&e0) == cudaSuccess && cudaEventCreate(&e1) == cudaSuccess;
    for (int ci = 0; ci < (int)p->classes.size() && ok; ++ci) {
        ClassPlan& cp = p->classes[ci];
        const Key key{cp.dev.type, cp.dev.n};
        auto hit = g_tuned.find(key);
        if (hit != g_tuned.end() && apply_radices(cp, hit->second)) {
            cp.tuned = true;
            continue;
        }
        const int n1 = (int)cp.cand1.size();
        const int n2 = cp.dev.mode == RAG_MODE_LONG ? (int)cp.cand2.size() : 1;
        if (n1 * n2 <= 1) continue;
        const int m = trial_m(cp.dev);
        // the trial batch: one class (index 0), m transforms packed in scratch
        aclfftRaggedPlan_t tmp;
        tmp.count = m;
        tmp.in_off.resize(m);
        tmp.ws_off.resize(m);
        for (int k = 0; k < m; ++k) {
            tmp.in_off[k] = (int64_t)k * ((int64_t)cp.dev.n + 2) * 8;
            tmp.ws_off[k] = (int64_t)k * ws_per(cp.dev);
        }
        tmp.out_off = tmp.in_off;
        double best = 1e30;
        Choice bestc;
        for (int a1 = 0; a1 < n1 && ok; ++a1)
            for (int a2 = 0; a2 < n2 && ok; ++a2) {
                if (!apply_choice(cp, {a1, a2})) continue;
                tmp.classes.assign(1, cp);
                tmp.classes[0].members.resize(m);
                for (int k = 0; k < m; ++k) tmp.classes[0].members[k] = k;
                build_items(&tmp);
                // trial tables: reallocated only when they grow
                auto put = [&](auto*& d, size_t& cap, const auto& h) {
                    using T = typename std::decay_t<decltype(h)>::value_type;
                    if (h.size() > cap) {
                        if (d) cudaFree(d);
                        d = nullptr;
                        cap = 0;
                        if (gfft::dev_alloc(reinterpret_cast<void**>(&d), h.size() * sizeof(T)) != cudaSuccess) return false;
                        cap = h.size();
                    }
                    return h.empty() ||
                           cudaMemcpy(d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice) == cudaSuccess;
                };
                if (!put(srows, cap_rows, tmp.rows) || !put(sitems, cap_items, tmp.items)) {
                    ok = false;
                    break;
                }
                RagArgs ra{};
                ra.rows = srows;
                ra.items = sitems;
                ra.nitems = (int)tmp.items.size();
                ra.smem_bytes = tmp.smem;
                ra.ctas = ctas_for(p, tmp.smem);
                ra.claim = RAG_CLAIM_AHEAD;
                ra.queue = squeue;
                ra.count = m;
                ra.err = p->d_err;
                ra.tw = p->tw;
                ra.in = sin;
                ra.out = sout;
                ra.ws = sws;
                ra.scale_c2c = 1.f;
                ra.wait_cycles = 1ll << 31;  // trials never use the plan's test settings
                ra.need_bias = 0;
                if (ra.ctas <= 0) {
                    ok = false;
                    break;
                }
                float tbest = 1e30f;
                for (int rep = 0; rep < 3 && ok; ++rep) {
                    ok = cudaMemsetAsync(squeue, 0, (size_t)(m + 2) * sizeof(int), p->s_cap) == cudaSuccess &&
                         cudaEventRecord(e0, p->s_cap) == cudaSuccess && gfft_launch_ragged(&ra, p->s_cap) == 0 &&
                         cudaEventRecord(e1, p->s_cap) == cudaSuccess && cudaEventSynchronize(e1) == cudaSuccess;
                    float ms = 0;
                    if (ok) cudaEventElapsedTime(&ms, e0, e1);
                    if (rep > 0) tbest = std::min(tbest, ms);
                }
                // the planner's choice (the first) stays unless another is 5 %
                // faster: one length alone is not the mixed batch
                if (tbest < (bestc.v1 == 0 && bestc.v2 == 0 && best < 1e30 ? 0.95 * best : best)) {
                    best = tbest;
                    bestc = {a1, a2};
                }
            }
        if (!ok) break;
        apply_choice(cp, bestc);
        cp.tuned = true;
        g_tuned[key] = radices_text(cp, bestc);
    }
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    for (void* q : {(void*)sin, (void*)sout, (void*)squeue, (void*)sws, (void*)srows, (void*)sitems})
        if (q) cudaFree(q);
    if (!ok) {
        cudaGetLastError();
        for (auto& cp : p->classes) {
            apply_choice(cp, {0, 0});
            cp.tuned = false;
        }
    } else {
        save_tune_file();
        p->tuned = true;
    }
    build_items(p);
    if (p->gexec) {
        cudaGraphExecDestroy(p->gexec);
        p->gexec = nullptr;
    }
    p->ctas = ctas_for(p, p->smem);
    p->ctas_smem = p->smem;
    if (!upload_tables(p)) return ACLFFT_ALLOC_FAILED;
    if (!ok) {
        gfft::set_last_error("ragged autotune: a trial launch failed");
        return ACLFFT_EXEC_FAILED;
    }
    return ACLFFT_SUCCESS;
}

// Device memory of device `dev` (any device when dev < 0) or managed
// memory; another GPU's memory would be dereferenced as a peer address.
bool device_pointer(const void* ptr, int dev)
{
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, ptr) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (at.type == cudaMemoryTypeManaged) return true;
    return at.type == cudaMemoryTypeDevice && (dev < 0 || at.device == dev);
}

// On-chip plans of a class: one tile, or two factors of at most kMaxSingle
// points.
bool plan_class(ClassPlan& cp, TwiddleBuilder& tb, std::map<int, double>& memo)
{
    RagClass& c = cp.dev;
    auto plans = [&](int L) {
        std::vector<TilePlan> v;
        for (auto& r : candidates(L)) v.push_back(tile_plan(L, r, tb));
        return v;
    };
    if (c.L <= kMaxSingle) {
        cp.cand1 = plans(c.L);
        if (!cp.cand1.empty()) {
            c.mode = RAG_MODE_SINGLE;
            return true;
        }
    }
    c.mode = RAG_MODE_LONG;
    // the factors whose steps cost least: items of W * len points, each
    // costing its passes plus about 1.5 for its loads and stores (30000 as
    // 240 x 125 instead of the balanced 200 x 150: five passes either way,
    // fuller tiles); a negative entry of the memo marks a length without a plan
    auto cost = [&](int len) {
        auto it = memo.find(len);
        if (it != memo.end()) return it->second;
        const std::vector<int> r = choose_tile_radices(len, false, kThreads);
        double v = -1;
        if (!r.empty() && (int)r.size() <= kRagMaxPass) {
            const int W = kThreads / tile_threads(len, r);
            v = ((double)r.size() + 1.5) / ((double)W * len);
        }
        memo[len] = v;
        return v;
    };
    int Lb = 0;
    double best = 0;
    for (int d = 2; (int64_t)d * d <= c.L; ++d) {
        if (c.L % d || c.L / d > kMaxSingle) continue;
        const double a = cost(d), b = cost(c.L / d);
        if (a < 0 || b < 0) continue;
        if (Lb == 0 || a + b <= best) {
            best = a + b;
            Lb = d;
        }
    }
    if (Lb == 0) return false;
    c.Lb = Lb;
    c.La = c.L / Lb;
    cp.cand1 = plans(c.La);
    cp.cand2 = plans(c.Lb);
    if (c.L <= kOuterTable) {
        c.otw_shift = -1;
        c.hi_off = tb.add_pass_table(c.La, c.Lb);
        return true;
    }
    int sh = 0;
    while ((int64_t(1) << (2 * sh)) < c.L) ++sh;
    c.otw_shift = sh;
    c.hi_off = tb.add_linear(((c.L - 1) >> sh) + 1, c.L, int64_t(1) << sh);
    c.lo_off = tb.add_linear(int64_t(1) << sh, c.L, 1);
    return true;
}

}  // namespace

extern "C" {

ACLFFT_API aclfftResult aclfftRaggedPlanCreate(aclfftRaggedPlan* plan, int count, const int* lengths,
                                               const aclfftType* types, const long long* inOffsets,
                                               const long long* outOffsets)
{
    ACLFFT_CHECK_NULL(plan);
    *plan = nullptr;
    ACLFFT_CHECK_PARAM(count >= 1, ACLFFT_INVALID_SIZE);
    ACLFFT_CHECK_NULL(lengths);
    ACLFFT_CHECK_NULL(types);
    ACLFFT_CHECK_NULL(inOffsets);
    ACLFFT_CHECK_NULL(outOffsets);
    for (int i = 0; i < count; ++i) {
        ACLFFT_CHECK_PARAM(types[i] == ACLFFT_C2C || types[i] == ACLFFT_R2C, ACLFFT_INVALID_TYPE);
        ACLFFT_CHECK_PARAM(lengths[i] >= 2 && lengths[i] <= kMaxLength, ACLFFT_INVALID_SIZE);
        ACLFFT_CHECK_PARAM(inOffsets[i] >= 0 && outOffsets[i] >= 0, ACLFFT_INVALID_VALUE);
        ACLFFT_CHECK_PARAM(inOffsets[i] % 8 == 0 && outOffsets[i] % 8 == 0, ACLFFT_INVALID_VALUE);
        if (!primes_le_13(lengths[i])) {
            gfft::set_last_error("ragged batches take lengths whose prime factors are <= 13");
            return ACLFFT_NOT_SUPPORTED;
        }
    }
    auto* p = new (std::nothrow) aclfftRaggedPlan_t();
    if (!p) return ACLFFT_ALLOC_FAILED;
    p->count = count;
    p->len.assign(lengths, lengths + count);
    p->in_off.assign(inOffsets, inOffsets + count);
    p->out_off.assign(outOffsets, outOffsets + count);
    p->type.resize(count);
    p->cls.resize(count);
    p->ws_off.resize(count);
    std::map<Key, int> cidx;
    std::map<int, double> memo;
    for (int i = 0; i < count; ++i) {
        const int t = types[i] == ACLFFT_C2C ? RAG_C2C : RAG_R2C;
        p->type[i] = t;
        const int n = lengths[i];
        const Key k{t, n};
        auto f = cidx.find(k);
        int ci;
        if (f == cidx.end()) {
            ci = (int)p->classes.size();
            cidx[k] = ci;
            ClassPlan cp;
            RagClass& c = cp.dev;
            c.n = n;
            c.type = t;
            c.L = (t == RAG_R2C && !(n & 1)) ? n / 2 : n;
            c.post_off = -1;
            c.hi_off = c.lo_off = -1;
            if (!plan_class(cp, p->tb, memo)) {
                delete p;
                gfft::set_last_error("ragged batches: length does not split into two on-chip factors");
                return ACLFFT_NOT_SUPPORTED;
            }
            if (c.even_r2c()) c.post_off = p->tb.add_linear(c.L / 2 + 1, n, 1);
            if (cp.cand1.empty() || (c.mode == RAG_MODE_LONG && cp.cand2.empty()) || !apply_choice(cp, {0, 0})) {
                delete p;
                gfft::set_last_error("ragged batches: no on-chip plan for a length");
                return ACLFFT_NOT_SUPPORTED;
            }
            p->classes.push_back(cp);
        } else {
            ci = f->second;
        }
        p->classes[ci].members.push_back(i);
        p->cls[i] = ci;
        p->ws_off[i] = -1;
        const RagClass& c = p->classes[ci].dev;
        if (c.mode == RAG_MODE_LONG) {
            // 128-byte aligned: contiguous blocks are written 16 bytes a thread
            p->ws_off[i] = p->ws_floats2;
            p->ws_floats2 += ((c.even_r2c() ? 2 : 1) * (int64_t)c.L + 15) / 16 * 16;
        }
        if (c.L > kMaxSingle) ++p->nlong;
        const int64_t in_b = t == RAG_C2C ? (int64_t)n * 8 : (int64_t)n * 4;
        const int64_t out_b = t == RAG_C2C ? (int64_t)n * 8 : ((int64_t)n / 2 + 1) * 8;
        p->in_min = std::max(p->in_min, (int64_t)inOffsets[i] + in_b);
        p->out_min = std::max(p->out_min, (int64_t)outOffsets[i] + out_b);
    }
    if (p->tb.count > 0x7fffffff) {  // 32-bit table offsets in the items
        delete p;
        gfft::set_last_error("ragged batches: twiddle tables too large");
        return ACLFFT_NOT_SUPPORTED;
    }
    split_steps(p);
    *plan = p;
    return ACLFFT_SUCCESS;
}

ACLFFT_API aclfftResult aclfftRaggedSetStream(aclfftRaggedPlan plan, cudaStream_t stream)
{
    ACLFFT_CHECK_PARAM(plan != nullptr, ACLFFT_INVALID_PLAN);
    plan->stream = stream;
    return ACLFFT_SUCCESS;
}

ACLFFT_API aclfftResult aclfftRaggedSetOptions(aclfftRaggedPlan plan, int autotune_on, int use_graph)
{
    ACLFFT_CHECK_PARAM(plan != nullptr, ACLFFT_INVALID_PLAN);
    plan->autotune = autotune_on != 0;
    plan->use_graph = use_graph != 0;
    return ACLFFT_SUCCESS;
}

ACLFFT_API aclfftResult aclfftRaggedAutotune(aclfftRaggedPlan plan)
{
    ACLFFT_CHECK_PARAM(plan != nullptr, ACLFFT_INVALID_PLAN);
    const aclfftResult r = device_setup(plan);
    if (r != ACLFFT_SUCCESS) return r;
    return autotune(plan);
}

ACLFFT_API aclfftResult aclfftRaggedExec(aclfftRaggedPlan plan, void* idata, void* odata, int direction)
{
    ACLFFT_CHECK_PARAM(plan != nullptr, ACLFFT_INVALID_PLAN);
    ACLFFT_CHECK_NULL(idata);
    ACLFFT_CHECK_NULL(odata);
    ACLFFT_CHECK_PARAM(direction == ACLFFT_FORWARD || direction == ACLFFT_BACKWARD, ACLFFT_INVALID_VALUE);
    if (!device_pointer(idata, -1) || !device_pointer(odata, -1)) {
        gfft::set_last_error("ragged exec takes device pointers");
        return ACLFFT_INVALID_VALUE;
    }
    aclfftResult r = device_setup(plan);
    if (r != ACLFFT_SUCCESS) return r;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev != plan->device) {
        cudaGetLastError();
        return ACLFFT_INVALID_DEVICE;
    }
    if (!device_pointer(idata, dev) || !device_pointer(odata, dev)) {
        gfft::set_last_error("ragged exec takes device pointers of the plan's device");
        return ACLFFT_INVALID_VALUE;
    }
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(plan->stream, &cs) != cudaSuccess) {
        cudaGetLastError();
        return ACLFFT_EXEC_FAILED;
    }
    const bool capturing = cs != cudaStreamCaptureStatusNone;
    if (plan->autotune && !plan->tuned && !capturing) {
        r = autotune(plan);
        if (r != ACLFFT_SUCCESS) return r;
    }
    const bool inv = direction == ACLFFT_BACKWARD;
    const RagArgs a = make_args(plan, plan->d_items, (int)plan->items.size(), plan->smem, idata, odata, inv);
    auto fail = [&](const char* what, int rc) {
        gfft::set_last_error(std::string("ragged exec: ") + what + ": " + cudaGetErrorString((cudaError_t)rc));
        cudaGetLastError();
        return ACLFFT_EXEC_FAILED;
    };
    if (!plan->use_graph || capturing) {
        const int rc = launch(plan, a, plan->stream);
        return rc == 0 ? ACLFFT_SUCCESS : fail("launch", rc);
    }
    if (!plan->gexec || plan->g_in != idata || plan->g_out != odata || plan->g_inv != (int)inv) {
        if (plan->gexec) cudaGraphExecDestroy(plan->gexec);
        plan->gexec = nullptr;
        cudaGraph_t g = nullptr;
        const cudaError_t eb = cudaStreamBeginCapture(plan->s_cap, cudaStreamCaptureModeThreadLocal);
        if (eb != cudaSuccess) return fail("begin capture", (int)eb);
        const int lrc = launch(plan, a, plan->s_cap);
        const cudaError_t ec = cudaStreamEndCapture(plan->s_cap, &g);
        const cudaError_t ei = (lrc == 0 && ec == cudaSuccess) ? cudaGraphInstantiate(&plan->gexec, g, 0) : cudaSuccess;
        if (lrc != 0 || ec != cudaSuccess || ei != cudaSuccess) {
            if (g) cudaGraphDestroy(g);
            plan->gexec = nullptr;
            return fail("graph capture", lrc != 0 ? lrc : (ec != cudaSuccess ? (int)ec : (int)ei));
        }
        cudaGraphDestroy(g);
        plan->g_in = idata;
        plan->g_out = odata;
        plan->g_inv = (int)inv;
    }
    const cudaError_t el = cudaGraphLaunch(plan->gexec, plan->stream);
    if (el != cudaSuccess) return fail("graph launch", (int)el);
    return ACLFFT_SUCCESS;
}

ACLFFT_API aclfftResult aclfftRaggedGetInfo(aclfftRaggedPlan plan, aclfftRaggedInfo* info)
{
    ACLFFT_CHECK_PARAM(plan != nullptr, ACLFFT_INVALID_PLAN);
    ACLFFT_CHECK_NULL(info);
    std::memset(info, 0, sizeof(*info));
    info->transforms = plan->count;
    info->classes = (int)plan->classes.size();
    info->long_transforms = plan->nlong;
    info->items = (int)plan->items.size();
    for (auto& cp : plan->classes) info->tuned_classes += cp.tuned ? 1 : 0;
    info->workspace_bytes = (size_t)plan->ws_floats2 * 8;
    info->in_bytes_min = (size_t)plan->in_min;
    info->out_bytes_min = (size_t)plan->out_min;
    info->graph = plan->gexec ? 1 : 0;
    info->smem_bytes = plan->smem;
    info->twiddle_entries = plan->tb.count;
    return ACLFFT_SUCCESS;
}

ACLFFT_API aclfftResult aclfftRaggedGetError(aclfftRaggedPlan plan, int* flags)
{
    ACLFFT_CHECK_PARAM(plan != nullptr, ACLFFT_INVALID_PLAN);
    ACLFFT_CHECK_NULL(flags);
    *flags = 0;
    if (!plan->dev_ready) return ACLFFT_SUCCESS;
    // ordered after the plan's launches: the read is queued on the plan's
    // stream (which may be a non-blocking stream the legacy default stream
    // does not wait for) and that stream is synchronised
    int v = 0;
    if (cudaMemcpyAsync(&v, plan->d_err, sizeof(int), cudaMemcpyDeviceToHost, plan->stream) != cudaSuccess ||
        cudaStreamSynchronize(plan->stream) != cudaSuccess) {
        cudaGetLastError();
        gfft::set_last_error("ragged: reading the device error word failed");
        return ACLFFT_EXEC_FAILED;
    }
    *flags = v;
    if (v == 0) return ACLFFT_SUCCESS;
    if (cudaMemsetAsync(plan->d_err, 0, sizeof(int), plan->stream) != cudaSuccess ||
        cudaStreamSynchronize(plan->stream) != cudaSuccess)
        cudaGetLastError();
    gfft::set_last_error("ragged: a dependency wait ran out of time; the output is incomplete");
    return ACLFFT_EXEC_FAILED;
}

ACLFFT_API aclfftResult aclfftRaggedSetWaitLimit(aclfftRaggedPlan plan, long long cycles)
{
    ACLFFT_CHECK_PARAM(plan != nullptr, ACLFFT_INVALID_PLAN);
    ACLFFT_CHECK_PARAM(cycles > 0, ACLFFT_INVALID_VALUE);
    if (plan->wait_cycles != cycles) drop_graph(plan);
    plan->wait_cycles = cycles;
    return ACLFFT_SUCCESS;
}

ACLFFT_API aclfftResult aclfftRaggedDebugHoldDependencies(aclfftRaggedPlan plan, int extra)
{
    ACLFFT_CHECK_PARAM(plan != nullptr, ACLFFT_INVALID_PLAN);
    ACLFFT_CHECK_PARAM(extra >= 0, ACLFFT_INVALID_VALUE);
    if (plan->need_bias != extra) drop_graph(plan);
    plan->need_bias = extra;
    return ACLFFT_SUCCESS;
}

ACLFFT_API aclfftResult aclfftRaggedDestroy(aclfftRaggedPlan plan)
{
    ACLFFT_CHECK_PARAM(plan != nullptr, ACLFFT_INVALID_PLAN);
    free_device(plan);
    delete plan;
    return ACLFFT_SUCCESS;
}

// Host replay of every item's accesses: input/output extents per transform,
// workspace ranges, table ranges, thread and shared-memory limits, and the
// queue order of dependent items.
ACLFFT_API int aclfftRaggedDebugCheck(aclfftRaggedPlan plan, char* msg, int msglen)
{
    auto report = [&](const std::string& s, int rc) {
        if (msg && msglen > 0) std::snprintf(msg, (size_t)msglen, "%s", s.c_str());
        return rc;
    };
    if (!plan) return report("no plan", -1);
    const int64_t twn = plan->tb.count;
    std::vector<int> done1(plan->count, 0), done2(plan->count, 0);
    // bytes of a transform's input and output, columns seen per step
    auto in_bytes = [&](const RagClass& c) { return (int64_t)c.n * (c.type == RAG_C2C ? 8 : 4); };
    auto out_bytes = [&](const RagClass& c) { return c.type == RAG_C2C ? (int64_t)c.n * 8 : ((int64_t)c.n / 2 + 1) * 8; };
    std::vector<int64_t> cols1(plan->count, 0), cols2(plan->count, 0), pairs(plan->count, 0), rows_seen(plan->count, 0);
    for (const RagItem& it : plan->items) {
        if (plan->smem > kSmemBudget) return report("shared memory", 2);
        if (it.kind != RAG_POST) {
            int64_t ns = 1;
            if (it.np < 1 || it.np > kRagMaxPass || it.T < 1 || it.W < 1) return report("passes", 3);
            auto pad = [&](int i) { return i + (i >> it.ps); };
            for (int q = 0; q < it.np; ++q) {
                const PassDesc& d = it.pass[q];
                const int R = d.radix, nbf = it.L / (R > 0 ? R : 1), nb = R >= 16 ? 1 : 16 / (R > 0 ? R : 16);
                if (R < 1 || R > 16 || it.L % R || d.ns != ns || (int64_t)nb * it.T < nbf) return report("pass", 3);
                if (ns > 1 && (d.tw_off < 0 || d.tw_off + ns * R > twn)) return report("pass tables", 3);
                for (int j = 0; j < nbf; ++j) {
                    const int qq = ns > 1 ? (int)(((uint64_t)(unsigned)j * d.ns_magic) >> 32) : j;
                    if (qq != j / ns) return report("magic division", 3);
                    const int i0 = (int)(j / ns * ns * R + j % ns), ws = ns == 1 ? 1 : (int)(ns + (ns >> it.ps));
                    for (int r = 0; r < R; ++r) {
                        if (q > 0 && pad(j) + r * (nbf + (nbf >> it.ps)) != pad(j + r * nbf)) return report("read stride", 3);
                        if (q + 1 < it.np && pad(i0) + r * ws != pad(i0 + r * (int)ns)) return report("write stride", 3);
                    }
                }
                ns *= R;
            }
            if (ns != it.L) return report("radix product", 3);
            if (it.T * it.W > kThreads || it.count < 1 || it.count > it.W) return report("tile threads", 4);
            const int d = it.kind == RAG_SINGLE ? it.T : it.W;
            for (int t = 0; t < kThreads; ++t)
                if ((int)((unsigned)t * it.wmagic >> 20) != t / d) return report("thread division", 4);
            const int64_t tile = it.kind == RAG_SINGLE ? (int64_t)it.W * it.pitch : (int64_t)it.W * (pad(it.L - 1) + 1);
            if (tile * 8 > plan->smem || (it.kind == RAG_SINGLE && it.pitch < pad(it.L - 1) + 1))
                return report("exchange buffer", 4);
        }
        if (it.kind == RAG_SINGLE) {
            if (it.first < 0 || it.first + it.count > (int)plan->rows.size()) return report("row range", 4);
            for (int k = 0; k < it.count; ++k) {
                const int x = plan->row_xf[it.first + k];
                const RagClass& c = plan->classes[plan->cls[x]].dev;
                const RagRow& r = plan->rows[it.first + k];
                if (c.mode != RAG_MODE_SINGLE || c.L != it.L) return report("row class", 4);
                if (r.in_off != plan->in_off[x] || r.out_off != plan->out_off[x]) return report("row offsets", 4);
                if ((it.flags & RAG_R2C_POST) && (it.post_off < 0 || it.post_off + it.L / 2 + 1 > twn))
                    return report("post table", 4);
                const int want = c.type == RAG_C2C ? RAG_CONJ_IN | RAG_CONJ_OUT
                                                   : (c.odd_r2c() ? RAG_REAL_IN | RAG_HALF_OUT : RAG_R2C_POST);
                if (it.flags != want || it.nhalf != c.n / 2) return report("row mode", 4);
                ++rows_seen[x];
            }
            continue;
        }
        if (it.xform < 0 || it.xform >= plan->count) return report("xform", 5);
        const int x = it.xform;
        const RagClass& c = plan->classes[plan->cls[x]].dev;
        const int64_t ws = plan->ws_off[x], wsn = (c.even_r2c() ? 2 : 1) * (int64_t)c.L;
        if (c.mode != RAG_MODE_LONG || ws < 0 || ws + wsn > plan->ws_floats2) return report("workspace", 5);
        if (it.kind == RAG_P1) {
            const int64_t e = (it.flags & RAG_REAL_IN) ? 4 : 8;
            if (it.L != c.La || it.stride != c.Lb || it.first + it.count > c.Lb) return report("p1 range", 6);
            if (it.in_off != plan->in_off[x] || (int64_t)c.L * e > in_bytes(c)) return report("p1 input", 6);
            if (it.out_off != ws) return report("p1 workspace", 6);
            if (it.pitch < it.L || (int64_t)it.W * it.pitch * 8 > plan->smem) return report("p1 staging", 6);
            if (done2[x]) return report("p1 queued late", 6);
            ++done1[x];
            cols1[x] += it.count;
        } else if (it.kind == RAG_P2) {
            if (it.L != c.Lb || it.stride != c.La || it.first + it.count > c.La) return report("p2 range", 7);
            if (it.need != done1[x] || cols1[x] != c.Lb) return report("p2 queued before its p1 items", 7);
            if (it.otw_shift < 0 ? it.hi_off < 0 || it.hi_off + (int64_t)c.L > twn
                                 : it.hi_off < 0 || it.hi_off + ((c.L - 1) >> it.otw_shift) + 1 > twn || it.lo_off < 0 ||
                                       it.lo_off + (1 << it.otw_shift) > twn || (int64_t)(c.La - 1) * (c.Lb - 1) >= c.L)
                return report("outer twiddles", 7);
            if (it.in_off != ws) return report("p2 workspace", 7);
            const bool wsout = (it.flags & RAG_WS_OUT) != 0;
            if (wsout != c.even_r2c() || it.out_off != (wsout ? ws + c.L : plan->out_off[x])) return report("p2 output", 7);
            if (!wsout && !(it.flags & RAG_HALF_OUT) && (int64_t)c.L * 8 > out_bytes(c)) return report("p2 extent", 7);
            if ((it.flags & RAG_HALF_OUT) && ((int64_t)it.nhalf + 1) * 8 > out_bytes(c)) return report("p2 extent", 7);
            ++done2[x];
            cols2[x] += it.count;
        } else {
            if (it.need != done1[x] + done2[x] || cols2[x] != c.La) return report("post queued early", 8);
            if (it.first < 0 || it.count < 1 || it.first + it.count > c.L / 2 + 1 || it.L != c.L || !c.even_r2c())
                return report("post range", 8);
            if (it.in_off != ws + c.L || it.out_off != plan->out_off[x] || it.post_off < 0 ||
                it.post_off + c.L / 2 + 1 > twn)
                return report("post tables", 8);
            pairs[x] += it.count;
        }
    }
    for (int x = 0; x < plan->count; ++x) {
        const RagClass& c = plan->classes[plan->cls[x]].dev;
        if (c.mode == RAG_MODE_SINGLE ? rows_seen[x] != 1
                                      : cols1[x] != c.Lb || cols2[x] != c.La || (c.even_r2c() && pairs[x] != c.L / 2 + 1))
            return report("a transform is not covered once", 9);
    }
    return report("ok", 0);
}

}  // extern "C"
