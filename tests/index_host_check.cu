// Host-side check of the device index arithmetic (bc_kernels.cuh), compiled by
// tests/test_index_logic.py with nvcc and run on the CPU.  Reads cases from
// stdin and prints results for comparison with Python integers.
#include <cstdio>
#include "bc_kernels.cuh"
using namespace bc;
int main() {
  char op[16];
  while (scanf("%15s", op) == 1) {
    if (op[0] == 'P') {  // P n b -> limb words below digit n
      int n, b;
      if (scanf("%d %d", &n, &b) != 2) return 1;
      printf("%d\n", words_below(n, b));
    } else if (op[0] == 'N') {  // N M -> run records of a transform
      int M;
      if (scanf("%d", &M) != 1) return 1;
      printf("%llu\n", run_records(M));
    } else if (op[0] == 'Q') {  // Q bit0 nbits h0 h1 h2 next -> "word value" of each word that starts in the run
      unsigned long long bit0, h0, h1, h2;
      int nbits;
      unsigned next;
      if (scanf("%llu %d %llx %llx %llx %x", &bit0, &nbits, &h0, &h1, &h2, &next) != 6) return 1;
      const U192 h = {{h0, h1, h2}};
      run_words(bit0, nbits, h, next, [](unsigned long long w, uint32_t x) { printf("%llu %x ", w, x); });
      printf("\n");
    }
  }
  return 0;
}
