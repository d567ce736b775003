// vpmc_work.cuh -- the working set of one single-instance grid (vorticity
// queries, the RBF product and the RBF solves), carved from a scratch slot.
#pragma once

#include "vpmc_grid.cuh"

namespace vpmc {

struct Work {
    GridInst plan;
    GridBufs g;
    ItemBufs it;
    QueryBufs q;
    QRec* self = nullptr;
    double* vec[8] = {};
};

inline int work_blocks(long n) {
    long b = (n + 255) / 256;
    if (b < 1) b = 1;
    if (b > 65535L * 8) b = 65535L * 8;
    return int(b);
}

// k: walk cells per h_w the caller would like (0: the default walk's).
inline int setup_work(vpmc_context* ctx, int slot, long N, float hw, float Lx, float Ly, int periodic, long M, int nvec,
                      Work* w, int k = 0, float cover = 1.f, bool deformed = false, int rows = 1) {
    InstDesc d{Lx, Ly, hw, periodic, 0, int(N), cover, k};
    const long nb = grid_plan(&d, 1, 0, 1, &w->plan);
    if (nb < 0) return int(-nb);
    const long nq = M > N ? M : N;
    auto carve_all = [&](Carver& c) {
        carve_grid(c, N, nb, 1, &w->g, deformed, rows);
        carve_items(c, nb, nq, &w->it);
        if (M > 0) carve_queries(c, nb, M, &w->q);
        w->self = c.take<QRec>(size_t(N < 1 ? 1 : N));
        for (int i = 0; i < nvec; ++i) w->vec[i] = c.take<double>(size_t(N < 1 ? 1 : N));
    };
    Carver dry;
    carve_all(dry);
    char* base = nullptr;
    VPMC_TRY(scratch(ctx, slot, dry.off, &base));
    Carver c{base, 0};
    carve_all(c);
    VPMC_CUDA(cudaMemcpyAsync(w->g.inst, &w->plan, sizeof(GridInst), cudaMemcpyHostToDevice, ctx->stream));
    return VPMC_OK;
}

}  // namespace vpmc
