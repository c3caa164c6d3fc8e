// The rule of gw_stage_shape.h: argv = groups sms warps advance.
#include <stdio.h>
#include <stdlib.h>

#include "gw_stage_shape.h"

int main(int, char** argv) {
  const gw::StageShape s = gw::stage_shape(atoi(argv[1]), atoi(argv[2]), atoi(argv[3]), atoi(argv[4]) != 0);
  printf("%d %d %d\n", s.dense, s.wide, s.fpw);
  return 0;
}
