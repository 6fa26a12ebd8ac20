// Prints AutoSegment (csrc/fvs_launch_rule.h) for sweeps given one per line on
// standard input as name=value words.
#include <cstdio>
#include <iostream>
#include <sstream>
#include <string>

#include "fvs_launch_rule.h"

int main() {
  std::string line;
  while (std::getline(std::cin, line)) {
    fvs::SweepShape q;
    std::istringstream words(line);
    std::string w;
    while (words >> w) {
      const size_t eq = w.find('=');
      const std::string key = w.substr(0, eq);
      const long long v = std::stoll(w.substr(eq + 1));
      if (key == "rank") q.rank = int(v);
      else if (key == "cells") q.cells = v;
      else if (key == "n") q.n = int(v);
      else if (key == "exact") q.exact = v != 0;
      else if (key == "mixed") q.mixed = v != 0;
      else if (key == "cut_cells") q.cut_cells = v != 0;
      else if (key == "family") q.family = static_cast<fvs::SweepFamily>(v);
      else if (key == "variant") q.variant = int(v);
      else return 2;
    }
    std::printf("%d\n", fvs::AutoSegment(q));
  }
  return 0;
}
