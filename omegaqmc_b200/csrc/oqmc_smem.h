// Dynamic shared memory that a launch above 48 KB opts its kernel in to: all a
// CTA can have (no kernel here has static shared memory), not the launch's own
// size.  The limit belongs to the kernel on its device and is shared by every
// host thread, and the size of one kernel's launches varies with the walker
// count: a smaller call between another thread's opt-in and its launch would
// lower the limit under it and make the launch fail.  Raised to the one value,
// it can only be set again to the same.
#pragma once

constexpr int OQ_SMEM_OPTIN = 227 * 1024;
