// Kernel-selection overrides carried in the `flags` argument of the launch entries, for tests
// and A/B timing only: every choice computes the same result, the default heuristics pick among
// them by shape.  Private to this library and its tests (not part of the C ABI contract).
#pragma once
#define MIORI_TUNE_GEMM_NARROW 0x100u   // GEMM: 128x128 tiles
#define MIORI_TUNE_GEMM_WIDE 0x200u     // GEMM: 128x256 tiles, one CTA per tile
#define MIORI_TUNE_GEMM_PAIR 0x4000u    // GEMM: two-CTA (cta_group::2) kernel
#define MIORI_TUNE_GEMM_NOPAIR 0x8000u  // GEMM: never the two-CTA kernel
#define MIORI_TUNE_GEMM_SPLIT_SHIFT 16  // GEMM: bits 16..19 = forced K split count (1..15; needs the workspace for it)
#define MIORI_TUNE_GEMM_MASK 0xFC300u       // GEMM: any of the above
