// mdx_resident.cuh -- host interface of the on-chip red-black runs
// (k_sor_resident.cu).
#pragma once

#include "mdx_internal.cuh"
#include "mdx_cell32.cuh"
#include "mdx_pot.cuh"

// Whether the grid's whole state fits the SMs in that form (and the stream is
// not being captured: a replay would repeat the words' sequence numbers).
bool mdx_res_pot_ok(mdx_ctx_t* ctx);
bool mdx_res_face32_ok(mdx_ctx_t* ctx);
bool mdx_res_face64_ok(mdx_ctx_t* ctx);
// `iters` red-black iterations in one launch on, respectively, Phi, the FP32
// corrections and the FP64 fields.  MDX_RES_REFUSED: the device did not take
// the cooperative launch (a stream that has part of the SMs only) or has no
// memory left for the inboxes; nothing ran,
// the caller sweeps with its other kernels, and the functions above say no from
// then on, until the solver is set up again or the stream changes.
enum { MDX_RES_REFUSED = -1 };
int mdx_res_pot_run(mdx_ctx_t* ctx, const pot_geom& L, int iters);
int mdx_res_face32_run(mdx_ctx_t* ctx, const mixed_params& P, int iters);
struct mdx_sor_params;
int mdx_res_face64_run(mdx_ctx_t* ctx, const mdx_sor_params& p, int iters);
void mdx_res_free(mdx_ctx_t* ctx);
