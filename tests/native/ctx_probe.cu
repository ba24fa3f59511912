// ctx_probe.cu -- a context's device arrays by name, for tests that look at a pass and not at the whole call
#include <cstring>

#include "engine.h"

extern "C" size_t probe_array(pimd_ctx *ctx, const char *name, void *out, size_t bytes) {
    const pimd::KP &kp = ctx->E.kp;
    const size_t P = kp.P, S = kp.S, N = kp.N, nk = kp.nk, nd = ctx->E.dm.nd, ndp = ctx->E.dm.ndp;
    struct {
        const char *name;
        const void *p;
        size_t bytes;
    } const a[] = {
        {"pos", kp.pos, P * S * 32},        {"F", kp.F, P * S * 32},            {"dip", kp.dip, P * S * 24},
        {"Efdr", kp.Efdr, P * S * 24},      {"dipf", kp.dipf, P * S * 16},      {"Sq", kp.Sq, P * nk * 16},
        {"Sm", kp.Sm, P * nk * 16},         {"Sdip", kp.Sdip, P * nk * 48},     {"kinfo", kp.kinfo, nk * 32},
        {"Tself", kp.Tself, P * N * 144},   {"M", ctx->E.dm.M, P * nd * 6 * ndp * (ctx->E.precision ? 4 : 8)},
    };
    for (const auto &x : a) {
        if (strcmp(x.name, name) || !x.p) continue;
        if (out && (bytes != x.bytes || cudaDeviceSynchronize() != cudaSuccess ||
                    cudaMemcpy(out, x.p, bytes, cudaMemcpyDeviceToHost) != cudaSuccess))
            return 0;
        return x.bytes;
    }
    return 0;
}
