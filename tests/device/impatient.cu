// The library with waits of the tcgen05 screen that run out within microseconds: a limit from zero up, by
// CTA, and tests of the phase that do not suspend.  Waits for what is in flight then are a thousand times as
// long as a product or a copy takes.
// Built by tests/device/__init__.py.
#define CFM_SCREEN_WAIT_NS ((blockIdx.x + 3 * blockIdx.y) % 8 * 400u)
#define CFM_SCREEN_DRAIN_NS 2000000u
#define CFM_SCREEN_WAIT "test_wait"
#include "cfm_reader.cu"
