// Prints launch shapes chosen by the library's host code (compiled with
// csrc/geometry.cpp, no GPU needed).
//
//   shape_probe slices              ny, CTAs per half, slots, columns, slices of the complex128 line product
#include "internal.h"

#include <cstdio>
#include <cstring>

using namespace lsw;

int main(int argc, char** argv) {
  if (argc == 2 && !std::strcmp(argv[1], "slices")) {
    for (int ny = 5; ny <= 192; ++ny)
      for (int cl : {1, 2, 4})
        for (int r : {1, 2, 4, 8}) {
          const int columns = (ny + cl - 1) / cl;
          std::printf("%d %d %d %d %d\n", ny, cl, r, columns, fp64_slices(ny, columns, r, 384));
        }
    return 0;
  }
  std::fprintf(stderr, "usage: shape_probe slices\n");
  return 2;
}
