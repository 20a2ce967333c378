// Prints, for each SM count, ray count and (block, smem_stack) of the command
// line, the launch form and the rays a warp takes (obvhs_gb300/csrc/traverse_form.h).
// usage: traverse_form_check SMS N BLOCK SMEM [SMS N BLOCK SMEM ...]
#include <stdio.h>
#include <stdlib.h>

#include "traverse_form.h"

int main(int argc, char** argv) {
  for (int i = 1; i + 3 < argc; i += 4) {
    const int form = trav_form_index((uint32_t)strtoul(argv[i + 2], 0, 10), atoi(argv[i + 3]));
    printf("%d %u\n", form, form < 0 ? 0u : trav_rays_per_warp((uint32_t)strtoul(argv[i + 1], 0, 10), atoi(argv[i]), form));
  }
  return 0;
}
