// bpc_kernels.h -- launcher interface between the C ABI (bpc_api.cu) and the
// sm_100a kernels (bpc_kernels.cu).
#pragma once
#include <cuda_runtime.h>

#include "bpc_core.cuh"

namespace bpc {

constexpr int kWarps = 4;  // warps (codeblocks) per CTA
// CTAs per SM the register budget is sized for.  Decoder: 7 x 4 warps at 72
// registers, of which the 4-warp forms spill 16-40 bytes and the one-warp 64x64
// forms none (a 16384x16384 3-pass decode at 6 / 7 / 8 CTAs: 5.17 / 4.87 / 4.81
// ms, but a 4096x4096 one, one wave, 0.384 / 0.390 / 0.404 ms).  Encoder: 5 x 4
// warps, a budget of 102 registers (64x64 takes 96, 32x32 80 and 90; no spills;
// 4 / 5 / 6 CTAs: 4.48 / 4.13 / 4.06 ms at 16384x16384, 0.160 / 0.160 / 0.182 ms
// at 2048x2048, where the 6-CTA form's spills lengthen the serial chain of the
// heaviest codeblock).
#ifndef DEC_MIN_CTAS
#define DEC_MIN_CTAS 7
#endif
#ifndef ENC_MIN_CTAS
#define ENC_MIN_CTAS 5
#endif
constexpr int kMinCtasDec = DEC_MIN_CTAS;
constexpr int kMinCtasEnc = ENC_MIN_CTAS;

// Input alignment the kernels' vector loads need: the encoder reads each
// lane's two coefficients with one 8-byte load, the decoder reads the slot
// stream with 16-byte loads.  Entry points refuse other pointers (a misaligned
// vector load would fault and lose the CUDA context).
constexpr unsigned kEncInAlign = 8, kDecInAlign = 16;
inline bool aligned_to(const void *p, unsigned a) { return ((uintptr_t)p & (uintptr_t)(a - 1)) == 0; }

// Longest LUT a launch takes; entries past Params::tab_n are range-checked only.
// The longest table a mode has, 16 levels and 3 passes, is 19,845 entries.
constexpr int kMaxLut = 230144;

// Warps of one-warp decoder CTAs resident at once: each CTA keeps its own copy
// of the table, so shared memory (smem_sm per SM, of which a CTA takes smem_cta
// and kReservedSmem) may hold fewer of them than the registers do.
constexpr long long kReservedSmem = 1024;
inline long long one_warp_resident(int sms, long long smem_sm, long long smem_cta) {
    const long long n = smem_sm / (smem_cta + kReservedSmem), regs = kMinCtasDec * kWarps;
    return sms * (n < regs ? n : regs);
}
// Whether a plain decode of `warps` warps runs one-warp CTAs and the latency
// form of the step, given the warps resident at once in 4-warp CTAs and in
// one-warp ones.  One-warp CTAs go to different SMs one after another, so the
// heaviest codeblocks (the coarse subbands, neighbours in raster order) do not
// share one, and no SM gets a whole CTA more than another.  One-warp / 4-warp,
// us, images of noise amplitude 30 and 60:
//   more than a wave of 4-warp CTAs: 5760x5760 568 / 550
//   64x64, 3 passes: 2560x2560 310 / 376 and 312 / 383, 3456x3456 342 / 414 and
//     353 / 396; with deeper tables at 1.8 waves of one-warp CTAs 371 / 415 and
//     394 / 395, at 2.0 403 / 418 and 416 / 418, at 2.2 408 / 413 and 432 / 405, at
//     2.7 443 / 414 and 477 / 394: up to two waves
//   32x32, 3 passes: 1024x1024 196 / 206 and 191 / 200, 2304x2304 (0.92 of a
//     one-warp wave) 214 / 216 and 206 / 210, 2752x2752 (1.32) 229 / 229 and 244 /
//     222: up to one
//   32x32, 2 passes: 1024x1024 136 / 138 and 134 / 136, 1536x1536 (0.28 of a
//     4-warp wave) 141 / 140 and 139 / 138, 2560x2560 153 / 150 and 163 / 157,
//     2880x2880 179 / 157 and 186 / 171: up to a quarter of a 4-warp wave
inline bool one_warp_pays(int passes, int cbs, long long warps, long long resident4, long long resident1) {
    if (warps > resident4) return false;
    if (cbs == 64) return warps <= 2 * resident1;
    return passes == 3 ? warps <= resident1 : 4 * warps <= resident4 && warps <= resident1;
}

// Launch the encoder (enc) or decoder over p.ncb codeblocks.  grid <= 0 picks
// one CTA per kWarps codeblocks; a positive grid runs persistent CTAs that
// walk the codeblocks grid-stride.  latency_forms lets a decode take one-warp
// CTAs and the latency form of the step (one_warp_pays; the heavy launch of an
// isolated decode runs it too), which finish a launch alone on the GPU sooner
// but execute more instructions; callers that run many launches at once pass
// false.
cudaError_t launch_code(bool enc, int passes, int cbs, const Params &p, int grid, cudaStream_t st,
                        bool latency_forms = true);

// One plain (sched null) or work-ordered launch over codeblocks
// [cb_begin, cb_end) (cb_end < 0: all) after the C ABI's argument checks
// (bpc_api.cu); returns a BPC_* code.
int code_device(bool enc, const int *in, int *out, int X, int Y, const int *d_lut, int lut_n, int passes, int levels,
                int cb, int *d_status, int *d_counts, int grid, void *stream, int cb_begin = 0, int cb_end = -1,
                int *sched = nullptr, bool latency_forms = true);

// Work order for a whole-image launch (bpc_order.cu): with scratch `sched` of
// sched_ints(ncb, cbs) ints, queue the kernels that sort the image's work
// units by expected cost, heaviest first, and set p.order.  Images of more than
// two waves are sorted for a balanced last wave; decodes of 64x64 codeblocks
// between nine tenths of a wave and two waves are sorted for an isolated launch
// (launch_code) when `isolate` allows it, which also sets p.ctr to the bulk
// launch's queue counter in the scratch.  Other images keep raster order
// (p.order and p.ctr stay null).
long long sched_ints(int ncb, int cbs);
// SMs of device `dev`, its opt-in shared memory per block and its shared memory
// per SM (cached)
int sm_count(int dev);
int shared_optin(int dev);
int shared_per_sm(int dev);
// warps of the plain coder resident at once on device `dev` (-1: current)
int resident_warps(bool enc, int dev);
// more than two waves on device `dev` (-1: the current device)
bool order_pays(bool enc, int ncb, int cbs, int dev = -1);
cudaError_t plan_order(bool enc, int cbs, Params &p, int *sched, cudaStream_t st, bool isolate);
// heavy CTAs of an isolated decode (kWarps codeblocks each)
constexpr int kIsoCtas = 6;

// LUT training: add, per LUT entry, [2k] symbols coded and [2k+1] symbols
// equal to 1 over p.ncb codeblocks of p.in (planes 0..14) to stats.
cudaError_t launch_stats(int passes, int cbs, const Params &p, unsigned long long *stats, cudaStream_t st);

}  // namespace bpc
