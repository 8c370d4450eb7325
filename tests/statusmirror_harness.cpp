// Host-side harness for epblas-parallel_gb300/csrc/statusmirror.h, compiled with
// g++ by tests/test_status_mirror.py.
#include "../epblas-parallel_gb300/csrc/statusmirror.h"

extern "C" {

void *watch_new() { return new mw::StatusWatch; }
void watch_begin(void *w, uint64_t now) { static_cast<mw::StatusWatch *>(w)->begin(now); }
int watch_check(void *w, uint64_t now) { return static_cast<mw::StatusWatch *>(w)->check(now); }

}
