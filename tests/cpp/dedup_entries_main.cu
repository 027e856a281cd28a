// Prints dedup_entries(n) of each argument (host code only).
#include <cstdio>
#include <cstdlib>

#include "bxg_internal.h"

int main(int argc, char** argv) {
  for (int i = 1; i < argc; ++i)
    std::printf("%u\n", bxg::dedup_entries(std::strtoull(argv[i], nullptr, 10)));
}
