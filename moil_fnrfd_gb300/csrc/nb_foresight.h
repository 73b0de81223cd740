// nb_foresight.h -- when the host foresees the list rebuilds of MD steps, and when it leaves them to the
// device (host code without CUDA).
//
// With a list period the host knows which steps rebuild, unless a site outruns the lists before: such
// a run of steps is dropped and redone with the device's decision, and so are the next runs, more of
// them each time lists are outrun again (2, 6, 14, 30, 62, then 64) and half as many after each run that
// kept its schedule.  A new system starts afresh.
#pragma once

struct ListForesight {
    int left = 0;       // runs still left to the device
    int backoff = 0;
    bool host(bool periods) const { return periods && left == 0; }
    void begin() { if (left > 0) --left; }                        // a run starts
    void kept() { backoff /= 2; }                                 // a foreseen run kept its schedule
    void outrun() { left = backoff = 2 * backoff + 2 < 64 ? 2 * backoff + 2 : 64; }
    void reset() { left = backoff = 0; }
};
