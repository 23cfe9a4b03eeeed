// graph_rule.h -- when a plan's execute is captured into a CUDA graph (molints_plan_set_graph).
#pragma once

namespace molints {

// The second of two executes in a row into an output is captured; an execute into the captured output
// launches the graph.  The first runs uncaptured: capture and instantiation cost more than they save one
// execute (8 polarised atoms on B200: 1.1 ms, against 0.12 ms for an uncaptured execute and 0.09 for a
// launch), and a program that takes two outputs in turn never captures for the one that has no graph.
struct GraphRule {
    enum Step { EAGER, CAPTURE, LAUNCH };
    const void *last = nullptr;  // the last execute's output
    Step next(const void *out, bool captured) {
        const bool again = last == out;
        last = out;
        return captured ? LAUNCH : again ? CAPTURE : EAGER;
    }
};

}  // namespace molints
