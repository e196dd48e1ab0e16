// PbHostRanges for tests/test_host_ranges_cpu.py, as C calls
#include "../../pyre_b200/csrc/pb_host_ranges.h"

static PbHostRanges r;
extern "C" {
void hr_add(uint64_t p, uint64_t n) { r.add((const void*)(uintptr_t)p, (size_t)n); }
void hr_drop(uint64_t p) { r.drop((const void*)(uintptr_t)p); }
int hr_inside(uint64_t p, uint64_t n) { return r.inside((const void*)(uintptr_t)p, (size_t)n); }
}
