// csrc/drain.h for ctypes
#include "drain.h"
extern "C" int host_drain_first(int n0, int n1, int ring) { return mpsa::drain_first(n0, n1, ring); }
extern "C" int host_drain_end(int n0, int n1) { return mpsa::drain_end(n0, n1); }
extern "C" int host_drain_step(int u, int n0, int n1) { return mpsa::drain_step(u, n0, n1); }
