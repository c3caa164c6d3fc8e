// wait_number (gw_wait.h) against stand-ins of the stream query: the number
// arrives while the work runs, with its end, and not at all.
#include <stdio.h>

#include "gw_wait.h"

int main() {
  unsigned long long slot = 6;
  int asked = 0;
  bool r = gw::wait_number(&slot, 6, [&] { return asked++, true; });
  printf("there %d %d\n", r, asked);
  r = gw::wait_number(&slot, 7, [&] {
    if (++asked == 3) slot = 7;
    return true;
  });
  printf("while running %d %d\n", r, asked);
  r = gw::wait_number(&slot, 8, [&] { return slot = 8, false; });
  printf("with the end %d\n", r);
  r = gw::wait_number(&slot, 9, [&] { return false; });
  printf("never %d\n", r);
  printf("next %u %u %u\n", gw::next_number(0), gw::next_number(7), gw::next_number(0xffffffffu));
  return 0;
}
