// The launch shape and table placement fitted to a call (test
// infrastructure): csrc/bgt_launch_fit.h on its own.
//
//   launch_fit_check THREADS PER_SM MODE TABLE_BYTES COMPACT N N ...
//                                  a call with groups of N, N, ... particles;
//                                  prints the fitted THREADS PER_SM MODE
#include <stdio.h>
#include <stdlib.h>

#include <vector>

#include "../bmad-ecosystem_b200/csrc/bgt_launch_fit.h"

int main(int argc, char** argv) {
  bgt_tuning t{};
  t.threads_per_block = atoi(argv[1]);
  t.blocks_per_sm = atoi(argv[2]);
  t.table_mode = atoi(argv[3]);
  const size_t table = strtoull(argv[4], nullptr, 10);
  t.compact_every = atoi(argv[5]);
  std::vector<int64_t> groups;
  for (int k = 6; k < argc; k++) groups.push_back(atoll(argv[k]));
  t = bgt::fit_tuning(
      t, 148, 224 * 1024,
      [&](int block) {
        int64_t n = 0;
        for (int64_t g : groups) n += (g + block - 1) / block;
        return n;
      },
      [&](int block) { return table + (t.compact_every ? 9 * 8 : 0) * block + 2 * 13 * 8 * block; },
      [](int block, int per_sm, int tmode) {  // bgt_track_kernels.cu
        if (block == 64) return tmode == 0 && (per_sm == 8 || per_sm == 10 || per_sm == 12 || per_sm == 16);
        if (block == 128) return tmode == 0 ? per_sm == 4 || per_sm == 5 || per_sm == 6 || per_sm == 8
                                            : per_sm >= 3 && per_sm <= 5;
        return per_sm == 2 || per_sm == 3 || (tmode == 0 && per_sm == 4);
      });
  printf("%d %d %d\n", t.threads_per_block, t.blocks_per_sm, t.table_mode);
}
