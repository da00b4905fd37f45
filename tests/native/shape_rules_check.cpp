// Prints what the direct sum's rules (shape_rules.h) choose, a line per line of input:
//   ordered <targets> <SMs>            -> targets per CTA of the ordered FP64 kernel
//   mixed <sources> <targets> <SMs>    -> 1 for small tiles
#include <stdio.h>
#include <string.h>

#include "../../gravhopper_gb300/csrc/shape_rules.h"

int main() {
  char kind[32];
  long long a, b, c;
  while (scanf("%31s %lld %lld", kind, &a, &b) == 3) {
    if (!strcmp(kind, "ordered")) printf("%d\n", gh::ordered_targets(a, (int)b));
    if (!strcmp(kind, "mixed") && scanf("%lld", &c) == 1) printf("%d\n", gh::small_tiles(a, b, (int)c));
  }
  return 0;
}
