// C entry of tests/test_pad_host.py: the padding rule of the complex64 state.
#include "../marie-tools_gb300/csrc/embed.h"

extern "C" int shim_pad_dims(const int* n, int C, int* m) { return marie::embed::pad_dims(n, C, m) ? 1 : 0; }
