// Reserves the marcher's list of tail rays in a fresh context (host code).
#include "rm_internal.h"

extern "C" int tail_probe() {
  rm::Ctx c;
  try {
    rm::reserve_tail(c);
  } catch (const std::exception&) {
    return -1;
  }
  const bool got = c.tail.cap > 0;
  c.tail.release();
  return got ? 1 : 0;
}
