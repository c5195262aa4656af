// The balance's check of its node list (dg_nodes.cuh, node_follows) on the
// host: argv[1] a file of 128-bit keys (low word first), argv[2] the level Lm of
// the paths.  Prints the first index that may not stand where it does, or -1,
// for 128-bit keys and, where the keys fit, for 64-bit keys.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../dendro_gb300/csrc/dg_nodes.cuh"

namespace dg {
void check_device_flags(Context &, const char *) {}
}  // namespace dg

template <typename W>
static long first_bad(const std::vector<W> &k, unsigned Lm) {
  for (size_t i = 0; i < k.size(); i++)
    if (!dg::node_follows<W>(i > 0, i ? k[i - 1] : (W)0, k[i], Lm)) return (long)i;
  return -1;
}

int main(int argc, char **argv) {
  if (argc != 3) return 2;
  FILE *f = std::fopen(argv[1], "rb");
  if (!f) return 2;
  std::vector<dg::u128> wide;
  std::vector<uint64_t> narrow;
  uint64_t w[2];
  bool fits = true;
  while (std::fread(w, sizeof(uint64_t), 2, f) == 2) {
    wide.push_back((dg::u128)w[1] << 64 | w[0]);
    narrow.push_back(w[0]);
    fits = fits && w[1] == 0;
  }
  std::fclose(f);
  const unsigned Lm = (unsigned)std::atoi(argv[2]);
  std::printf("%ld", first_bad(wide, Lm));
  if (fits) std::printf(" %ld", first_bad(narrow, Lm));
  std::printf("\n");
  return 0;
}
