// Plan persistence: the Winograd-domain filter U of a plan written to a file
// together with what it was made for, and read back into a plan of the same
// layer, so a restarted process skips the filter transform (and, with the
// autotuner's WG_CONV2D_TUNE_FILE, the tuning runs).  The reference has no
// counterpart (it transforms the filter on every call).
//
// File: a fixed header (magic, version, the layer's C, K, padding, the
// transform, operand type and padded sizes, the byte count and an FNV-1a
// checksum of the payload) followed by U exactly as it lies in device memory:
// U[E][Cp/8][Kp][8] in the operand type, or for the row F(4x3) kernel
// U1[18][Cp16/8][Kp64][8] fp16, for the direct kernel U9[9][Cp/8][Kp][8] in the
// tensors' type (each with its own transform code in the header).
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/conv2d.h"
#include "wg_plan.h"

namespace wg {

namespace {

constexpr char kPlanMagic[8] = {'W', 'G', 'C', 'P', 'L', 'A', 'N', '1'};

struct PlanFileHeader {
    char magic[8];
    uint32_t version;
    uint32_t c, k, p, q;
    int32_t xform, op;
    uint32_t e, cp, kp;
    uint64_t u_bytes;
    uint64_t checksum;
};

uint64_t fnv1a(const unsigned char* p, size_t n) {
    uint64_t h = 1469598103934665603ull;
    for (size_t i = 0; i < n; ++i) {
        h ^= p[i];
        h *= 1099511628211ull;
    }
    return h;
}

constexpr int32_t kDirectXform = 32;   // U9[9][Cp/8][Kp][8], the filter itself

bool same_layer(const PlanFileHeader& a, const PlanFileHeader& b) {
    return a.c == b.c && a.k == b.k && a.xform == b.xform && a.op == b.op && a.e == b.e && a.cp == b.cp && a.kp == b.kp &&
           a.u_bytes == b.u_bytes;
}

PlanFileHeader header_of(const Plan& pl) {
    PlanFileHeader h;
    std::memset(&h, 0, sizeof(h));
    std::memcpy(h.magic, kPlanMagic, 8);
    h.version = 1;
    h.c = pl.prob.c;
    h.k = pl.prob.k;
    h.p = pl.prob.p;
    h.q = pl.prob.q;
    h.xform = static_cast<int32_t>(pl.xf) + (pl.algo == CONV2D_ALGO_4X3_ROW ? 16 : 0);   // row F(4x3): own layout
    h.op = static_cast<int32_t>(pl.op);
    h.e = static_cast<uint32_t>(pl.g.alpha * pl.g.alpha);
    if (pl.run_direct) {
        h.xform = kDirectXform;
        h.e = 9;
    }
    h.cp = static_cast<uint32_t>(pl.g.cp);
    h.kp = static_cast<uint32_t>(pl.g.kp);
    h.u_bytes = static_cast<uint64_t>(pl.u_bytes);
    return h;
}

// The plan of the Winograd algorithm that a tuned plan running the direct
// kernel stands for: its filter files are that algorithm's, as they are where
// the direct kernel is not the faster.
int winograd_plan(const Plan& pl, bool filter_only, std::unique_ptr<Plan>& out) {
    conv2d_options_t o = pl.opt;
    o.algo = pl.algo;
    out.reset(new Plan());
    return out->build(&pl.prob, &o, filter_only);
}

}  // namespace

}  // namespace wg

using namespace wg;

extern "C" {

int conv2d_plan_save(const void* param, const char* path) {
    Plan* pl = plan_of(param);
    if (!pl || !path) return set_last_error(CONV2D_ERR_INVALID, "param blob not set up, or null path");
    DeviceGuard dg(pl->device);
    if (!pl->filter_ready || pl->opt.filter_policy == 1) {
        const int st = pl->filter(nullptr);
        if (st) return st;
    }
    std::unique_ptr<Plan> winograd;
    if (pl->run_direct && pl->algo != CONV2D_ALGO_DIRECT) {
        // from the plan's own copy of the filter: the caller's may have changed or be gone
        void* w = nullptr;
        if (const int st = winograd_plan(*pl, true, winograd)) return st;
        if (cudaMalloc(&w, static_cast<size_t>(pl->prob.k) * pl->prob.c * 18) != cudaSuccess) {
            cudaGetLastError();
            return set_last_error(CONV2D_ERR_NOMEM, "workspace of the filter transform");
        }
        winograd->prob.weight = w;
        const bool ok = launch_direct_unfilter(pl->U, w, pl->g.k, pl->g.c, nullptr) == cudaSuccess &&
                        winograd->filter(nullptr) == CONV2D_OK && cudaDeviceSynchronize() == cudaSuccess;
        cudaFree(w);
        if (!ok) return set_last_error(CONV2D_ERR_CUDA, "filter transform failed");
        pl = winograd.get();
    }
    PlanFileHeader h = header_of(*pl);
    std::vector<unsigned char> u(h.u_bytes);
    if (cudaDeviceSynchronize() != cudaSuccess || cudaMemcpy(u.data(), pl->U, h.u_bytes, cudaMemcpyDeviceToHost) != cudaSuccess)
        return set_last_error(CONV2D_ERR_CUDA, "copy of the transformed filter failed");
    h.checksum = fnv1a(u.data(), u.size());
    FILE* f = std::fopen(path, "wb");
    if (!f) return set_last_error(CONV2D_ERR_INVALID, "cannot open the plan file for writing");
    const bool ok = std::fwrite(&h, sizeof(h), 1, f) == 1 && std::fwrite(u.data(), 1, u.size(), f) == u.size();
    if (std::fclose(f) != 0 || !ok) return set_last_error(CONV2D_ERR_INVALID, "plan file write failed");
    return CONV2D_OK;
}

int conv2d_plan_load(const void* param, const char* path) {
    Plan* owner = blob_plan(param);
    if (!owner || !path) return set_last_error(CONV2D_ERR_INVALID, "param blob not set up, or null path");
    std::lock_guard<std::mutex> lock(owner->loading);
    Plan* pl = plan_of(param);
    FILE* f = std::fopen(path, "rb");
    if (!f) return set_last_error(CONV2D_ERR_INVALID, "cannot open the plan file");
    PlanFileHeader h;
    std::vector<unsigned char> u;
    bool ok = std::fread(&h, sizeof(h), 1, f) == 1;
    DeviceGuard dg(pl->device);
    // a tuned plan that runs the direct kernel: the file's filter is that of the
    // Winograd algorithm, which gets a plan of its own once the file is read
    const bool tuned = pl->run_direct && pl->algo != CONV2D_ALGO_DIRECT;
    std::unique_ptr<Plan> winograd;
    if (tuned)
        if (const int st = winograd_plan(*pl, true, winograd)) {
            std::fclose(f);
            return st;
        }
    const PlanFileHeader want = header_of(tuned ? *winograd : *pl);
    if (ok && (std::memcmp(h.magic, kPlanMagic, 8) != 0 || h.version != 1)) {
        std::fclose(f);
        return set_last_error(CONV2D_ERR_INVALID, "not a plan file");
    }
    if (ok && !same_layer(h, want)) {
        std::fclose(f);
        return set_last_error(CONV2D_ERR_INVALID,
                              "plan file was made for another layer, transform or operand type");
    }
    if (ok) {
        u.resize(h.u_bytes);
        ok = std::fread(u.data(), 1, u.size(), f) == u.size();
    }
    std::fclose(f);
    if (!ok) return set_last_error(CONV2D_ERR_INVALID, "plan file truncated");
    if (fnv1a(u.data(), u.size()) != h.checksum) return set_last_error(CONV2D_ERR_INVALID, "plan file checksum mismatch");
    if (tuned)
        if (const int st = winograd_plan(*pl, false, winograd)) return st;
    Plan* to = tuned ? winograd.get() : pl;
    // U may still be read by work queued earlier on any stream
    if (cudaDeviceSynchronize() != cudaSuccess || cudaMemcpy(to->U, u.data(), u.size(), cudaMemcpyHostToDevice) != cudaSuccess)
        return set_last_error(CONV2D_ERR_CUDA, "copy of the transformed filter failed");
    to->filter_ready = true;
    if (tuned) set_loaded(const_cast<void*>(param), winograd.release());
    return CONV2D_OK;
}

}  // extern "C"
