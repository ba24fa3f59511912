// reinit_probe.cu -- the buffers of a context's accelerators set up again (with alloc_fail.c: where memory is short)
#include "engine.h"

extern "C" int probe_dg_init(pimd_ctx *ctx) { return pimd::dg_init(ctx->E); }
extern "C" void probe_dm_init(pimd_ctx *ctx) { pimd::dm_init(ctx->E); }
extern "C" int probe_dg_keeps_exy(pimd_ctx *ctx) { return ctx->E.dg.exyc != nullptr; }
extern "C" int probe_dg_x_of_all_beads(pimd_ctx *ctx) { return ctx->E.dg_xall; }
