// Host build of cg_hostcopy.h, for tests/test_host_copy.py.
#include "../../cachegen_b200/csrc/cg_hostcopy.h"

extern "C" int hc_uses_x86() { return CG_HOST_X86; }
extern "C" void hc_copy(uint8_t *d, const uint8_t *s, int64_t n) { cg::copy_piece(d, s, n); }
extern "C" void hc_pause() { cg::spin_pause(); }
extern "C" void hc_touch(uint8_t *p, int64_t n) {
    for (int64_t k = 0; k < n; k += 4096) cg::touch_page(p + k);
}
