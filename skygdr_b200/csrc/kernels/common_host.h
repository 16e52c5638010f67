// Definitions shared by device code and by host code that never sees nvcc.
#pragma once

namespace sky {

// Per-launch status block in device memory. The host sets it to "unset"
// (status 0, cursor and t_start all ones) before a launch and reads it after.
struct LaunchStatus {
    unsigned int status;            // SkyStatus; first non-OK code wins
    unsigned int detail;            // code-specific (chunk index low bits, barrier id, ...)
    unsigned long long cursor;      // smallest chunk index NOT done; ~0ull = everything done
    unsigned long long chunks_done;
    unsigned long long bytes_done;
    unsigned long long stall_ns;    // summed over CTAs: time waiting for credit
    unsigned long long t_start_ns;  // globaltimer of the first CTA to start
    unsigned long long t_end_ns;    // globaltimer of the last CTA to finish
    unsigned int ctas_done;
    unsigned int work_counter;      // dynamic chunk scheduler
};

// What the CTAs of a launch know of their flow's credit page, in device memory behind the working status block. Reads of the page
// itself are round trips to host memory that do not overlap (they name the same line): one CTA at a time reads it, for all.
struct SkyGrantCache {
    unsigned long long granted;     // largest grant read so far (0: none yet)
    unsigned int unlimited;         // the last read found the flow unpaced
    unsigned int lock;              // 1: some CTA is reading the page, or waiting for credit on behalf of all
};

// Working block of a flow's transfer launches: status, then grant cache.
struct FlowWork {
    LaunchStatus status;
    SkyGrantCache grant;
};

}  // namespace sky
