// vs_resident.cu -- launch plan and launches of the resident kernel
// (vs_resident.cuh).  Its variants are compiled in one file each
// (vs_resident_fast.cu and so on), which build side by side.
#include <algorithm>
#include <functional>
#include <queue>
#include <vector>

#include "vs_resident.cuh"

namespace vsb {
namespace {

ResidentFn resident_fn(const ResidentPlan& p, bool hist) {
    if (p.tmm) return p.fast ? resident_fast_tmm(hist) : resident_exact_tmm(hist);
    return p.fast ? resident_fast(hist) : resident_exact(hist);
}

void cluster_launch(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, const ResidentPlan& p) {
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = p.ctas;
    attr->val.clusterDim.y = 1;
    attr->val.clusterDim.z = 1;
    cfg->gridDim = dim3(p.ctas, (unsigned)p.order.size());
    cfg->blockDim = dim3(p.threads);
    cfg->dynamicSmemBytes = p.smem;
    cfg->attrs = attr;
    cfg->numAttrs = 1;
}

}  // namespace

bool resident_plan(const TubeGrid* grids, int n, int npairs, bool fast, ResidentPlan* out) {
    *out = ResidentPlan{};
    if (npairs < 1 || npairs > kMaxPairs || n > 65535) return false;      // a tube per row of the grid
    int dev = 0, optin = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return false;
    // The cluster size with the shortest batch.  A step of a tube takes about
    // 0.5 us (the exchange and two barriers) plus 0.013 us per row of each of
    // the CTA's warps; the clusters that fit at once take the tubes longest
    // first (a cluster needs its CTAs in one GPC, so about 0.9 of the SMs serve
    // clusters of 3 to 6 CTAs and 0.8 larger ones).  Measured, us per step:
    // 256 vowel tubes with 2 CTAs 9.6 (8.4 longest first), 3 CTAs 10.6, 4 CTAs
    // 10.8 (two-step strips 17.4); one 55 x 253 tube with 16 CTAs 0.69, 8 CTAs
    // 0.81, 2 CTAs 1.9 (two-step strips 2.5).
    bool tmm = false;
    for (int i = 0; i < n; ++i) tmm = tmm || grids[i].tmm;
    const int warps = kMaxWarps - (tmm ? 1 : 0);     // a warp for the two-mass model
    std::vector<int> idx((size_t)n);
    std::vector<double> t((size_t)n);
    double best = 1e300;
    for (int C : {1, 2, 3, 4, 6, 8, 16}) {
        ResidentPlan p;
        p.ctas = C;
        p.fast = fast;
        p.tmm = tmm;
        bool ok = true;
        for (int i = 0; i < n && ok; ++i) {
            const int NR = grids[i].H - 2, nwx = (grids[i].W - 2) / kTileCols + 1;
            if (NR < C || nwx > warps) { ok = false; break; }
            const int nrow = (NR + C - 1) / C, ng = std::min(warps / nwx, nrow), R = (nrow + ng - 1) / ng;
            p.warps = std::max(p.warps, ng * nwx);
            ok = R <= kMaxRows;
            t[(size_t)i] = 0.5 + (fast ? 0.013 : 0.02) * R * ng * nwx;
        }
        if (!ok) continue;
        for (int i = 0; i < n; ++i) {
            const int NR = grids[i].H - 2, nwx = (grids[i].W - 2) / kTileCols + 1;
            p.smem = std::max(p.smem, res_layout(nwx, p.warps / nwx, (NR + C - 1) / C, !fast).bytes);
            idx[(size_t)i] = i;
        }
        if (p.smem > optin) continue;
        std::stable_sort(idx.begin(), idx.end(), [&](int a, int b) { return t[(size_t)a] > t[(size_t)b]; });
        p.order = idx;
        p.threads = 32 * (p.warps + (tmm ? 1 : 0));
        const int slots = std::max(1, (int)(sms * (C <= 2 ? 1.0 : C <= 6 ? 0.9 : 0.8)) / C);
        std::priority_queue<double, std::vector<double>, std::greater<double>> free_at;
        double end = 0.0;
        for (int i : idx) {
            double start = 0.0;
            if ((int)free_at.size() == slots) {
                start = free_at.top();
                free_at.pop();
            }
            free_at.push(start + t[(size_t)i]);
            end = std::max(end, start + t[(size_t)i]);
        }
        if (end < best) {
            best = end;
            *out = p;
        }
    }
    if (out->order.empty()) return false;
    for (const bool hist : {false, true}) {
        const void* fn = (const void*)resident_fn(*out, hist);
        if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin) != cudaSuccess ||
            cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
            cudaGetLastError();
            *out = ResidentPlan{};
            return false;
        }
    }
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[1];
    cluster_launch(&cfg, attr, *out);
    int resident = 0;
    if (cudaOccupancyMaxActiveClusters(&resident, (const void*)resident_fn(*out, true), &cfg) != cudaSuccess ||
        resident < 1) {
        cudaGetLastError();
        *out = ResidentPlan{};
        return false;
    }
    return true;
}

cudaError_t launch_resident_run(const TubeDev* tubes, RunState* rs, const int* order, int64_t steps,
                                const ResidentPlan& plan, cudaStream_t stream, bool hist) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[1];
    cluster_launch(&cfg, attr, plan);
    cfg.stream = stream;
    cudaError_t e = cudaSuccess;
    while (steps > 0 && e == cudaSuccess) {
        const int k = (int)std::min<int64_t>(steps, 1 << 30);
        e = cudaLaunchKernelEx(&cfg, resident_fn(plan, hist), tubes, rs, order, k, plan.warps);
        // the step counter advances after every cluster has run: a cluster
        // that starts later reads RunState::step then
        if (e == cudaSuccess) e = launch_advance(rs, k, stream);
        steps -= k;
    }
    return e;
}

}  // namespace vsb
