// Per-shape algorithm and tile choice (CONV2D_ALGO_AUTO).
//
// The reference picks F(2x3) fused / F(2x3) / F(4x3) with fixed size rules
// (src/conv2d.cpp:83-114).  Here every candidate (algorithm x GEMM channel
// tile, plus the row-Winograd F(4x3) kernel this operator adds) is planned on
// scratch output memory and timed on the device the first time a shape is seen; the winner is cached per shape and, when
// WG_CONV2D_TUNE_FILE names a file, persisted there so later processes make
// the same choice without measuring.  The reference selection wins unless
// another candidate is more than 3% faster, and of candidates that the
// measurement does not tell apart the more accurate one (pick_tuned), so noise
// between nearly equal candidates seldom flips the choice from run to run.  The
// direct kernel is timed as well: where it is faster than the winner, calls run
// it.  Times are weighed by accuracy (accuracy_weight).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "wg_plan.h"

namespace wg {

namespace {

using Key = std::tuple<unsigned, unsigned, unsigned, unsigned, unsigned, unsigned, unsigned, int, int, int>;

struct Choice {
    int algo;      // among the Winograd algorithms
    int bn;
    float ms;
    bool direct;   // the direct kernel ran faster
};

// Operations per second, padding included, that the direct kernel holds under
// the board's power cap: 32 x 256 x 56^2 -> 256 takes 70 us in the first
// milliseconds, as it is timed here, and 82.5 us (1,487 TFLOP/s) once calls
// have run back to back for some tenths of a second; the Winograd paths, with
// 0.25-0.5 of its products, keep their times (101.7 us).  32 x 512 x 28^2 ->
// 512, 70.5 us here against F(4x3)'s 65.5, would be 80 us in earnest.
constexpr double kSustainedFlops = 1.48e15;

// Candidates within a few percent of one another change places with every
// measurement; the more accurate one then wins.  Relative errors against 64
// bits (fp16 tensors): direct 2.1e-4, F(2x3) 6.4e-4, row F(4x3) 9.5e-4, F(4x3)
// 2.0e-3.
float accuracy_weight(int algo) {
    return algo == CONV2D_ALGO_4X3_NON_FUSED ? 1.08f : algo == CONV2D_ALGO_4X3_ROW ? 1.04f : 1.f;
}

// A candidate this close, in ms, to the fastest one counts as equal to it, so that
// near ties go the same way in every plan.  By the best of 8 single calls
// 4x512x28^2 -> 256 (direct 15.5 us, F(4x3) 14.2, weighed 15.3) ran the direct
// kernel in 6 of 10 plans and F(4x3), ten times its error, in 4; 2x512x28^2 -> 128
// (F(2x3) 12.8, F(4x3) 12.1, weighed 13.1) F(2x3) in 2 and F(4x3) in 8.  Now the
// first runs direct in 10 of 10, the second F(2x3).
constexpr float kTieMs = 0.7e-3f;

// In the tune file the algorithm's number carries the direct kernel's flag.
constexpr int kDirectFlag = 16;

std::mutex g_mu;
std::map<Key, Choice> g_cache;
bool g_loaded = false;

Key key_of(const problem_t& pr, const conv2d_options_t& opt) {
    return Key(pr.n, pr.c, pr.h, pr.w, pr.k, pr.p, pr.q,
               opt.operand_bf16 + 2 * opt.io_bf16 + 4 * opt.layout_nhwc + 8 * opt.m_fp32,
               opt.f4_points, opt.tile_scaling);
}

const char* tune_file() {
    const char* f = std::getenv("WG_CONV2D_TUNE_FILE");
    return (f && *f) ? f : nullptr;
}

void load_file_locked() {
    if (g_loaded) return;
    g_loaded = true;
    const char* path = tune_file();
    if (!path) return;
    FILE* fp = std::fopen(path, "r");
    if (!fp) return;
    unsigned n, c, h, w, k, p, q;
    int bf, f4, sc, algo, bn;
    float ms;
    while (std::fscanf(fp, "%u %u %u %u %u %u %u %d %d %d %d %d %f", &n, &c, &h, &w, &k, &p, &q, &bf, &f4, &sc, &algo,
                       &bn, &ms) == 13)
        g_cache[Key(n, c, h, w, k, p, q, bf, f4, sc)] = Choice{algo & ~kDirectFlag, bn, ms, (algo & kDirectFlag) != 0};
    std::fclose(fp);
}

void append_file_locked(const Key& kk, const Choice& ch) {
    const char* path = tune_file();
    if (!path) return;
    FILE* fp = std::fopen(path, "a");
    if (!fp) return;
    std::fprintf(fp, "%u %u %u %u %u %u %u %d %d %d %d %d %.5f\n", std::get<0>(kk), std::get<1>(kk), std::get<2>(kk),
                 std::get<3>(kk), std::get<4>(kk), std::get<5>(kk), std::get<6>(kk), std::get<7>(kk), std::get<8>(kk),
                 std::get<9>(kk), ch.algo | (ch.direct ? kDirectFlag : 0), ch.bn, ch.ms);
    std::fclose(fp);
}

// Device time of one call of a candidate plan, or a negative value when the
// candidate cannot be planned: after a warm-up four times 8 calls back to back
// (once, if they take over 10 ms), the mean of the faster two.  Event times go in
// steps of about 1 us: the best of 8 single calls of 20 us came out up to 2 us
// apart from one plan to the next, and held the launch of the first kernel, which
// calls in a program overlap (4x512x28^2 -> 256 direct 21-22 us by itself, 15.5 among
// others; F(4x3), of three kernels, 19-20 and 14.2).
float time_candidate(const problem_t& pr, conv2d_options_t opt, int algo, int bn, void* scratch_out,
                     cudaStream_t s) {
    problem_t p = pr;
    p.out = scratch_out;
    opt.algo = algo;
    opt.gemm_bn = bn;
    Plan pl;
    if (pl.build(&p, &opt) != CONV2D_OK || pl.algo != algo) return -1.f;
    if (pl.run(s) != CONV2D_OK) return -1.f;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    constexpr int kCalls = 8;
    std::vector<float> times;
    bool ok = true;
    for (int rep = 0; rep < 4 && ok; ++rep) {
        ok = cudaEventRecord(a, s) == cudaSuccess;
        for (int i = 0; i < kCalls && ok; ++i) ok = pl.run(s) == CONV2D_OK;
        ok = ok && cudaEventRecord(b, s) == cudaSuccess && cudaEventSynchronize(b) == cudaSuccess;
        float ms = 0.f;
        ok = ok && cudaEventElapsedTime(&ms, a, b) == cudaSuccess;
        if (ok) times.push_back(ms / kCalls);
        if (ms > 10.f) break;
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaStreamSynchronize(s);
    if (times.empty()) return -1.f;
    std::sort(times.begin(), times.end());
    return times.size() == 1 ? times[0] : (times[0] + times[1]) / 2;
}

}  // namespace

void pick_tuned(const TunedTime* t, int n, int fallback, float direct_ms, double direct_flops, TunedTime* best, bool* direct) {
    *best = TunedTime{fallback, 0, -1.f};
    *direct = false;
    TunedTime ref{fallback, 0, -1.f};
    float least = -1.f;   // of the weighed times
    const auto weighed = [](const TunedTime& x) { return x.ms * accuracy_weight(x.algo); };
    for (int i = 0; i < n; ++i) {
        if (least < 0.f || weighed(t[i]) < least) least = weighed(t[i]);
        if (t[i].algo == fallback && (ref.ms < 0.f || t[i].ms < ref.ms)) ref = t[i];
    }
    if (n == 0) return;
    // the most accurate of those as fast as the fastest, the fastest of these
    for (int i = 0; i < n; ++i) {
        if (weighed(t[i]) > least + kTieMs) continue;
        const float wi = accuracy_weight(t[i].algo), wb = accuracy_weight(best->algo);
        if (best->ms < 0.f || wi < wb || (wi == wb && t[i].ms < best->ms)) *best = t[i];
    }
    // the reference rule's pick unless it is more than 3% slower or the less accurate
    if (ref.ms > 0.f && accuracy_weight(fallback) <= accuracy_weight(best->algo) && weighed(*best) > weighed(ref) / 1.03f) *best = ref;
    if (direct_ms <= 0.f) return;
    const double sustained_ms = direct_flops / kSustainedFlops * 1e3;
    *direct = std::max(static_cast<double>(direct_ms), sustained_ms) < std::max(least + kTieMs, weighed(*best));
}

int autotune_choose(const problem_t& pr, const conv2d_options_t& opt, int fallback, int* algo_out, int* bn_out,
                    bool* direct_out) {
    const Key kk = key_of(pr, opt);
    {
        std::lock_guard<std::mutex> lk(g_mu);
        load_file_locked();
        auto it = g_cache.find(kk);
        if (it != g_cache.end()) {
            *algo_out = it->second.algo;
            *bn_out = it->second.bn;
            *direct_out = it->second.direct;
            return CONV2D_OK;
        }
    }
    const size_t out_bytes = static_cast<size_t>(pr.n) * pr.k * (pr.h + 2 * pr.p - 2) * (pr.w + 2 * pr.q - 2) * 2;
    void* scratch = nullptr;
    if (cudaMalloc(&scratch, out_bytes) != cudaSuccess) {
        cudaGetLastError();
        *algo_out = fallback;
        *bn_out = 0;
        *direct_out = false;
        return CONV2D_ERR_NOMEM;
    }
    cudaStream_t s;
    cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
    struct Cand {
        int algo, bn;
    };
    std::vector<Cand> cands;
    cands.push_back({CONV2D_ALGO_2X3_FUSED, 0});
    cands.push_back({CONV2D_ALGO_4X3_ROW, 0});
    const int bn0 = default_bn(static_cast<int>(pr.k));
    for (int a : {CONV2D_ALGO_2X3_NON_FUSED, CONV2D_ALGO_4X3_NON_FUSED}) {
        cands.push_back({a, bn0});
        if (pr.k > 128) cands.push_back({a, bn0 == 256 ? 128 : 256});
    }
    std::vector<TunedTime> times;
    for (const Cand& cd : cands) {
        const float ms = time_candidate(pr, opt, cd.algo, cd.bn, scratch, s);
        if (ms >= 0.f) times.push_back({cd.algo, cd.bn, ms});
    }
    const float direct_ms = times.empty() ? -1.f : time_candidate(pr, opt, CONV2D_ALGO_DIRECT, 0, scratch, s);
    cudaStreamDestroy(s);
    cudaFree(scratch);
    // the kernel multiplies whole rows with their padding, 16 channels and 32 filters at a time
    const double positions = pr.n * (pr.h + std::max<double>(pr.p, 2.0 * pr.p - 2)) * (pr.w + std::max<double>(pr.q, 2.0 * pr.q - 2));
    const double flops = 18.0 * positions * ((pr.c + 15) / 16 * 16) * ((pr.k + 31) / 32 * 32);
    TunedTime pick;
    bool direct = false;
    pick_tuned(times.data(), static_cast<int>(times.size()), fallback, direct_ms, flops, &pick, &direct);
    const Choice best{pick.algo, pick.bn, std::max(pick.ms, 0.f), direct};
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (g_cache.find(kk) == g_cache.end()) {
            g_cache[kk] = best;
            append_file_locked(kk, best);
        }
    }
    *algo_out = best.algo;
    *bn_out = best.bn;
    *direct_out = best.direct;
    return CONV2D_OK;
}

void autotune_clear() {
    std::lock_guard<std::mutex> lk(g_mu);
    g_cache.clear();
    g_loaded = false;
}

}  // namespace wg
