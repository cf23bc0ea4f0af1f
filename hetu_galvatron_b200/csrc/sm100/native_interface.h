// Version of what host/torch_ops.cpp takes from the kernel library: the argument lists of the entry points that it calls by
// address, and the structs that it hands them.  Both sides export it; raise it with any change of those.
#pragma once

constexpr int kHgNativeInterface = 7;
