// Per-shape algorithm and tile choice (CONV2D_ALGO_AUTO).
//
// The reference picks F(2x3) fused / F(2x3) / F(4x3) with fixed size rules
// (src/conv2d.cpp:83-114).  Here every candidate (algorithm x GEMM channel
// tile, plus the row-Winograd F(4x3) kernel this operator adds) is planned on
// scratch output memory and timed on the device the first time a shape is seen; the winner is cached per shape and, when
// WG_CONV2D_TUNE_FILE names a file, persisted there so later processes make
// the same choice without measuring.  The reference selection wins unless
// another candidate is more than 3% faster, so noise between nearly equal
// candidates cannot flip the choice from run to run.  The direct kernel is
// timed as well: where it is faster than the winner, calls run it.  Times are
// weighed by accuracy (accuracy_weight).
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

// Device time of one call of a candidate plan (best of 8 after a warm-up; with
// the best of 3 a choice now and then took a GEMM tile a fifth slower), or a
// negative value when the candidate cannot be planned.
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
    float best = -1.f;
    for (int rep = 0; rep < 8; ++rep) {
        cudaEventRecord(a, s);
        if (pl.run(s) != CONV2D_OK) break;
        cudaEventRecord(b, s);
        if (cudaEventSynchronize(b) != cudaSuccess) break;
        float ms = 0.f;
        cudaEventElapsedTime(&ms, a, b);
        if (best < 0.f || ms < best) best = ms;
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaStreamSynchronize(s);
    return best;
}

}  // namespace

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
    Choice best{fallback, 0, -1.f, false};
    float ref_ms = -1.f;
    int ref_bn = 0;
    for (const Cand& cd : cands) {
        const float ms = time_candidate(pr, opt, cd.algo, cd.bn, scratch, s);
        if (ms < 0.f) continue;
        const float weighed = ms * accuracy_weight(cd.algo);
        if (cd.algo == fallback && (ref_ms < 0.f || weighed < ref_ms)) {
            ref_ms = weighed;
            ref_bn = cd.bn;
        }
        if (best.ms < 0.f || weighed < best.ms) best = Choice{cd.algo, cd.bn, weighed, false};
    }
    const float direct_ms = best.ms < 0.f ? -1.f : time_candidate(pr, opt, CONV2D_ALGO_DIRECT, 0, scratch, s);
    cudaStreamDestroy(s);
    cudaFree(scratch);
    if (ref_ms > 0.f && best.ms > 0.f && best.ms > ref_ms / 1.03f) best = Choice{fallback, ref_bn, ref_ms, false};
    if (best.ms < 0.f) best = Choice{fallback, 0, 0.f, false};
    // the kernel multiplies whole rows with their padding, 16 channels and 32 filters at a time
    const double positions = pr.n * (pr.h + std::max<double>(pr.p, 2.0 * pr.p - 2)) * (pr.w + std::max<double>(pr.q, 2.0 * pr.q - 2));
    const double flops = 18.0 * positions * ((pr.c + 15) / 16 * 16) * ((pr.k + 31) / 32 * 32);
    best.direct = direct_ms > 0.f && std::max(static_cast<double>(direct_ms), flops / kSustainedFlops * 1e3) < best.ms;
    best.ms /= accuracy_weight(best.algo);
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
