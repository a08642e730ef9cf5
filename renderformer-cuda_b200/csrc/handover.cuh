// The words of the attention's workspace: through one the two pieces of a handed-over unit agree who does what, through another the pieces
// of a cut unit which of them merges it; and each is zero again for the next launch whatever becomes of a piece. Every transition is one atomic step on the word; the steps are plain functions, which the
// host's test runs in every order.
#pragma once

namespace rfk {
namespace handover {

enum Word : int {
    kIdle = 0,    // before the first piece is done, and once both pieces are done with the word
    kReady = 1,   // the first piece has left its state
    kFailed = 2,  // the first piece gave up: there is no state
    kTaken = 3,   // the second piece has taken all of the unit; the first piece, when it is done, clears the word
};
enum Act : int {
    kGo = 0,      // the second piece takes up the state
    kWait = 1,    // it goes on waiting
    kWhole = 2,   // it takes all of the unit
};
struct Step { int next, act; };   // what the word becomes, and what the party does

// the first piece is done: `ok` with its state in the workspace
__host__ __device__ constexpr Step give(int word, bool ok) { return {word == kTaken ? kIdle : ok ? kReady : kFailed, kGo}; }
// the second piece looks whether its wait is over, and does not change the word
__host__ __device__ constexpr Step look(int word) { return {word, word == kReady ? kGo : word == kIdle ? kWait : kWhole}; }
// the second piece is past its wait: it has seen the first piece done, or has run out of time
__host__ __device__ constexpr Step settle(int word) {
    return word == kReady ? Step{kIdle, kGo} : Step{word == kFailed ? kIdle : kTaken, kWhole};
}

// Units whose keys are cut into pieces that nobody waits for: a counter of the pieces that have arrived, in the upper half of those that
// gave up. The last one zeroes it for the next launch, and merges the pieces if all have left their shares.
__host__ __device__ constexpr int piece(bool failed) { return failed ? 0x10001 : 1; }   // what a piece adds
struct Arrival { bool last, merge; };
__host__ __device__ constexpr Arrival arrive(int before, bool failed, int pieces) {
    const bool last = (before & 0xffff) == pieces - 1;
    return {last, last && !failed && before < 0x10000};
}

}  // namespace handover
}  // namespace rfk
