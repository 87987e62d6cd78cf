// Which GEMM kernel a shape gets. Plain C++, so that the rule can be looked at without a GPU.
#pragma once

namespace zx {

// Width of the CTA pair's tile, or 0 for the single-CTA kernel: the least of three estimates in microseconds, each launch
// + waves * (tile + per 1000 of K), with constants fitted to 100 shapes (M 256 to 16384, N 512 to 11264, K 512 to 5640) run
// with each kernel in turn. Over those shapes the choice costs 0.3 % against the best of the three on average and 4 % at
// most; the kernels differ by up to 35 %. For example (single / 128 / 256 wide): 256 x 2048 x 4096 22.7 / 18.1 / 23.6 us,
// 8192 x 2048 x 512 20.6 / 23.2 / 24.2, 3000 x 2056 x 5640 136 / 97 / 108, 4096 x 11264 x 4096 279 / 312 / 238.
// One row block (M <= 128) leaves half of a pair idle.
inline int gemm_choose_tile(int M, int N, int K, int sm_count) {
  if (M <= 128 || sm_count < 2) return 0;
  auto waves = [](int rows, int n_rows, int cols, int n_cols, int units) {
    const long long tiles = (long long)((rows + n_rows - 1) / n_rows) * ((cols + n_cols - 1) / n_cols);
    return (double)((tiles + units - 1) / units);
  };
  const double k = K * 1e-3;
  const double single = 2.4 + waves(M, 128, N, 256, sm_count) * (1.8 + 5.1 * k);
  const double narrow = 4.0 + waves(M, 256, N, 128, sm_count / 2) * (1.1 + 3.2 * k);
  const double wide = 3.4 + waves(M, 256, N, 256, sm_count / 2) * (1.8 + 4.85 * k);
  if (single <= wide && single <= narrow) return 0;
  return wide <= narrow ? 256 : 128;
}

}  // namespace zx
