// The largest front and the number of levels of a 2-D grid's subdomain with and without a
// limit on joined fronts, for test_join_limit.py
#include <cstdio>
#include <cstdlib>

#include "host/mf_symbolic.hpp"

int main(int argc, char **argv) {
  const int k = std::atoi(argv[1]), limit = std::atoi(argv[2]), thin = std::atoi(argv[3]);
  dg::Csr A;
  A.nrows = k * k;
  A.ptr.push_back(0);
  for (int i = 0; i < k; i++)
    for (int j = 0; j < k; j++) {
      const int nb[5][2] = {{i - 1, j}, {i, j - 1}, {i, j}, {i, j + 1}, {i + 1, j}};
      for (auto &q : nb)
        if (q[0] >= 0 && q[0] < k && q[1] >= 0 && q[1] < k) {
          A.col.push_back(q[0] * k + q[1]);
          A.val.push_back(1.0);
        }
      A.ptr.push_back((int64_t)A.col.size());
    }
  dg::MfOptions opt;
  opt.leaf = 8;
  opt.thin = thin;
  if (limit > 0) opt.max_rows = limit;
  dg::MfBatch B;
  dg::mf_build_single(A, opt, B);
  std::printf("%d %d\n", B.max_m, B.nlevels);
}
