// ahead.cuh — steps that are queued without a wait between them, and when the caller looks whether one of them has failed.  Plain arithmetic (compiled by the host
// compiler in tests/test_ahead_host.py).
#pragma once

// A mark is a copy of 32 bytes and an event between two tokens, 9 us: 300 int8-cache tokens of a 0.5B model's two layers took 28.7 ms without marks, 29.4 with one
// behind every fourth token (a wait behind every token: 37.5); every eighth is half of that.
constexpr int kAheadGroup = 8;

// step(i) queues step i.  mark(j) queues a copy of the error words behind the steps so far; look(j) waits for that copy and returns its error.  Marks stand behind every
// kAheadGroup steps and are looked at kAheadGroup steps later, so that the device always has steps to go on with while the host waits, and at most 2 kAheadGroup - 1
// steps follow one that failed: a step whose wait for a peer runs out takes a second or more, and so does every step behind it.  A mark that nobody would look at is not made
// (prompts of up to 2 kAheadGroup tokens have none).  Returns the first error of any of them.
template <typename Step, typename Mark, typename Look> inline int run_ahead(int n, Step step, Mark mark, Look look) {
    for (int i = 0; i < n; i++) {
        const int g = i / kAheadGroup, k = i % kAheadGroup;
        if (k == 0 && g >= 2)
            if (const int rc = look(g & 1)) return rc;
        if (const int rc = step(i)) return rc;
        if (k == kAheadGroup - 1 && (g + 2) * kAheadGroup < n)
            if (const int rc = mark(g & 1)) return rc;
    }
    return 0;
}
