// launch_rules.h - rules of the launchers that need no CUDA header (the CPU
// tests compile them by themselves).
#pragma once

namespace scb {

// Row splits of a backward-weight launch of `groups` M-tile groups over
// `chunks` 64-row chunks, where `ctas` CTAs run at once.  A split's chunks are
// one chain of additions in the TMEM accumulator, and the chain's length sets
// dW's error (norm against FP64, 60k voxels, C = K = 128: 45 chunks 1.74e-6, 43
// 1.66e-6, 23 0.85e-6).  So it is never longer than with the splits that fill
// the CTAs, rounded up.  Where those leave a second wave of a few CTAs, two
// whole waves are taken instead: half the chain, and no empty SMs.  One wave
// of the splits rounded down is faster by a second prologue and dW reduction,
// but its chain is longer.  us, rounded up / two waves / rounded down: 60k
// voxels, C = K = 128 185 / 122 / 110, C = K = 256 541 / 355 / 351; 200k, C = K =
// 128 509 / 304 / 298; two CTAs per SM, 60k, C = 128, K = 64 95 / 83 / 73; 40k, C =
// 512, K = 256 708 / 458 / 552.
inline int wgrad_row_splits(int chunks, int groups, int ctas) {
  auto up = [](int a, int b) { return (a + b - 1) / b; };
  auto clamp = [&](int s) { return up(chunks, up(chunks, s < chunks ? s : chunks)); };
  const int filled = up(ctas, groups);
  const int one = clamp(filled);
  if (static_cast<long long>(one) * groups <= ctas) return one;
  const int two = 2 * ctas / groups;
  return two > filled ? clamp(two) : one;
}

// fp32 forward / backward-input: 64 output columns a block instead of 32 where
// the 64-row blocks alone are two per SM.
inline bool simt_wide_columns(long long rows, int columns, int sms) { return columns > 32 && rows >= 64ll * 2 * sms; }

// fp32 backward-weight: rows per block, in whole chunks, for about six blocks
// per SM; at least four chunks, at most `range` rows.
inline long long simt_wgrad_rows(long long rows, int tiles, int sms, int chunk, int range) {
  long long r = (rows * tiles + sms * 6 - 1) / (sms * 6);
  r = (r + chunk - 1) / chunk * chunk;
  if (r < 4 * chunk) r = 4 * chunk;
  return r > range ? range : r;
}

}  // namespace scb
