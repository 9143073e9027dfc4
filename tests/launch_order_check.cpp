// Which launches csrc/cuda/launch_order.h lets run beside the ones before them, for sequences of launches of which each
// names the memory that it touches.  A launch that depends on one that may still be running must be told to wait.
#include "launch_order.h"
#include <stdio.h>
#include <stdlib.h>
#include <initializer_list>

using boatcu::LaunchOrder;

static char W[64], X[64], Y[64], Z[64], dW[64], dX[64];
static int stream_a, stream_b;

static void expect(bool ok, const char* what) {
    if (ok) return;
    printf("wrong: %s\n", what);
    exit(1);
}

typedef std::initializer_list<const char*> List;

static bool launch(LaunchOrder& o, LaunchOrder::Place at, List reads, List writes) {
    o.begin(at);
    for (const char* p : reads) o.name(p, 64, false);
    for (const char* p : writes) o.name(p, 64, true);
    const bool beside = o.beside();
    o.end(true);
    return beside;
}

static void launch_unnamed(LaunchOrder& o, LaunchOrder::Place at) {
    o.begin(at);
    o.end(true);
}

static void within_a_sequence() {
    LaunchOrder o;
    const LaunchOrder::Place at = {1, &stream_a, false, 0};
    expect(!launch(o, at, {X, Y}, {dW}), "the first launch of a sequence waits");
    expect(launch(o, at, {Y, W}, {dX}), "what depends on nothing that runs goes beside");
    expect(!launch(o, at, {dX}, {Z}), "read after write");
    expect(launch(o, at, {W}, {dW}), "the one that waited lets go of those before it");
    expect(!launch(o, at, {Y}, {W}), "write after read");
    launch_unnamed(o, at);
    expect(!launch(o, at, {X}, {Y}), "behind a launch that names nothing");
    o.interrupt();
    expect(!launch(o, at, {X}, {Z}), "behind a copy");
    for (int i = 0; i < 200; ++i) launch(o, at, {W}, {X + i % 8});
    expect(!launch(o, at, {W}, {X}), "more ranges than the table holds");
}

// The program updates the weights with a kernel of its own between a backward and the next forward: the table sees the
// library's launches alone, in which nothing writes W.
static void a_kernel_of_the_program_between_two_calls() {
    LaunchOrder o;
    launch(o, {1, &stream_a, false, 0}, {Y, W}, {dX});
    expect(!launch(o, {2, &stream_a, false, 0}, {X, W}, {Z}), "the first launch of the next call");
    launch(o, {0, &stream_a, false, 0}, {Y, W}, {dX});
    expect(!launch(o, {0, &stream_a, false, 0}, {X, W}, {Z}), "calls outside a sequence");
    launch(o, {0, &stream_a, false, 0}, {Y, W}, {dX});
    expect(!launch(o, {3, &stream_a, false, 0}, {X, W}, {Z}), "a sequence behind such a call");
}

// A sum over the ranks on the library stream, which the table does not see, then a step on the summed gradients.
static void a_collective_between_two_calls() {
    LaunchOrder o;
    launch(o, {1, &stream_a, false, 0}, {X, Y}, {dW});
    launch(o, {1, &stream_a, false, 0}, {Y, W}, {dX});
    launch(o, {1, &stream_a, false, 0}, {Z}, {Y});
    expect(!launch(o, {0, &stream_a, false, 0}, {dW}, {W}), "a step on gradients that were just summed");
}

// Two threads, whose launches go to one stream or, on the per-thread default stream, to two under one handle: B writes Y,
// A's launches take B's out of the table, B reads Y.
static void two_threads_take_turns(bool per_thread) {
    LaunchOrder o;
    const LaunchOrder::Place a = {1, &stream_a, per_thread, 0}, b = {2, &stream_a, per_thread, 0};
    launch(o, b, {X}, {Y});
    expect(!launch(o, a, {W}, {dW}), "A behind B");
    expect(!launch(o, a, {dW}, {dX}), "A behind itself");
    expect(!launch(o, b, {Y}, {Z}), "B behind A");
    expect(launch(o, b, {W}, {dX}) == !per_thread, "beside, but on no per-thread stream");
}

static void another_stream() {
    LaunchOrder o;
    launch(o, {1, &stream_a, false, 0}, {X}, {Y});
    expect(!launch(o, {1, &stream_b, false, 0}, {W}, {Z}), "the first launch on another stream");
}

// The stream goes into a capture and out of it: what is launched in between goes into a graph and does not run now.
static void a_capture_begins_or_ends() {
    LaunchOrder o;
    const LaunchOrder::Place eager = {1, &stream_a, false, 0}, captured = {1, &stream_a, false, 7}, next = {1, &stream_a, false, 8};
    launch(o, eager, {X}, {Y});
    expect(!launch(o, captured, {W}, {Z}), "the first launch of a capture");
    expect(launch(o, captured, {W}, {dX}), "beside another of the capture");
    expect(!launch(o, eager, {Y}, {dW}), "the first launch behind a capture");
    launch(o, captured, {X}, {Y});
    expect(!launch(o, next, {W}, {Z}), "the first launch of the next capture");
}

// A launch that fails - of which nothing runs - takes no place in the table, and the launches before it may still be running.
static void a_launch_that_fails() {
    LaunchOrder o;
    const LaunchOrder::Place at = {1, &stream_a, false, 0};
    launch(o, at, {X}, {Y});
    o.begin(at);
    o.name(Y, 64, false);
    o.name(Z, 64, true);
    expect(!o.beside(), "what depends on the one before");
    o.end(false);
    expect(!launch(o, at, {Y}, {dX}), "the first launch behind one that failed");
    launch(o, at, {X}, {Y});
    o.begin(at);
    o.end(false);                                   // a turn that ends before its launch
    expect(!launch(o, at, {Y}, {dX}), "the first launch behind none");
}

int main() {
    within_a_sequence();
    a_kernel_of_the_program_between_two_calls();
    a_collective_between_two_calls();
    two_threads_take_turns(false);
    two_threads_take_turns(true);
    another_stream();
    a_capture_begins_or_ends();
    a_launch_that_fails();
    printf("ok\n");
    return 0;
}
