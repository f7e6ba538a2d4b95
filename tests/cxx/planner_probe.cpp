// Prints the planner's splits for the cases on stdin, one per line:
//   ranges N cost...           -> even_ranges: N + 1 bounds
//   shares SMS K (work npass)* -> sm_shares: K shares
#include <cstdio>
#include <iostream>
#include <sstream>
#include <string>

#include "layout.hpp"

int main() {
  std::string line, kind;
  while (std::getline(std::cin, line)) {
    std::istringstream in(line);
    in >> kind;
    if (kind == "ranges") {
      int n;
      in >> n;
      std::vector<int64_t> cost;
      for (int64_t c; in >> c;) cost.push_back(c);
      for (int32_t b : hmvm::even_ranges(cost, n)) std::printf("%d ", b);
    } else {
      int sms, k;
      in >> sms >> k;
      std::vector<double> work(k);
      std::vector<int> npass(k);
      for (int i = 0; i < k; i++) in >> work[i] >> npass[i];
      for (int s : hmvm::sm_shares(work, npass, sms)) std::printf("%d ", s);
    }
    std::printf("\n");
  }
  return 0;
}
