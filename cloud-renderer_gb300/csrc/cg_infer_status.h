// cg_infer_status.h -- how inference launches report a bounded wait that ran out.
#pragma once

// Two words of the context's status block that no launch clears: a launch that
// failed ORs its bits into one (1: a wait ran out, 2: and the drain after it) and
// raises the other to its number (numbers grow with every call).  Launches need no
// order among themselves or towards a clear: a report stays until the host has taken
// it, and a call that waits for its own launch knows whether that one failed.
struct InferStatus {
    unsigned long long bits;    // of every launch since the last report was taken
    unsigned long long launch;  // the latest launch that failed (0: none)
};

inline bool infer_failed(const InferStatus& s, unsigned long long launch) {
    return s.launch == launch;
}
