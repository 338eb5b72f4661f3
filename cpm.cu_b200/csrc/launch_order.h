// Which launches of the stream have surely ended when the next one starts.  Host only.
//
// With programmatic launches (launch_kernel) a grid may start as soon as every CTA of its predecessor has executed griddepcontrol.launch_dependents
// or left.  A launch that executes it first thing tells its successor nothing new: what has ended by the successor's start is what had
// ended by its own.  A launch that executes it after its griddepcontrol.wait ("holds its successor back") has its predecessor, and with
// it everything before, behind it by then.  Launches without the instruction, events and copies between launches only make the order stricter.
//
// The producer's launcher says held() where its kernel does so; a consumer that leaves its own wait out, or to its end, asks ended() for the
// launch that wrote what it reads, instead of knowing it from the caller's order of calls.
#pragma once

struct LaunchOrder {
    long issued = 0;   // number of the last launch, counted from 1, never reset
    long done = 0;     // launches 1 .. done have ended when launch issued + 1 starts
    void launched() { ++issued; }
    void held() { done = issued - 1; }
    bool ended(long launch) const { return launch > 0 && launch <= done; }
};
