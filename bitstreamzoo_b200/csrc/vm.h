// Device-side interpreter ("VM") for short streams (see vm.cu): straight-line
// segments, and whole programs with their if/while control flow.
#pragma once

#include <cstdint>
#include <vector>

#include "device.h"

namespace bsz {

// One instruction, 16 bytes.
//
// Segment mode: operands and destinations are value locations: v >= 0 is
// slot v of the slot file (v * n_words words in), v < 0 is entry -1 - v of
// the external pointer table (bound inputs, constants, and buffers that
// outlive the segment).
//
// Program mode adds control flow and device-side state: every stream value
// is a slot with a tail bit (tails[slot]); ints live in 64-bit registers;
// per-class op counters reproduce the dynamic op count and op mix.
enum VmCode : uint8_t {
  kVmNot = 0, kVmAnd, kVmOr, kVmXor,
  kVmAndNot,   // a & ~b, bits at and above the bit length cleared as ~ clears them
  kVmAdd, kVmShl, kVmShr, kVmPop,
  kVmCopy,     // dst <- a (words and tail)
  kVmFill,     // dst <- constant `fill`: 0 ZERO, 1 the N-bit mask (ONES operand), 2 all ones, tail 1
  kVmLoad,     // slot dst <- the device words at pointer (b << 32 | a), tail = fill
  kVmStore,    // the device words at pointer (b << 32 | dst) <- slot a
  // program mode only
  kVmJz,       // if slot a is zero (no stored bit and tail 0): jump to instruction b
  kVmJmp,      // jump to instruction b
  kVmPopI,     // ireg[dst] <- popcount(slot a); error 1 if tail(a) = 1
  kVmIConst,   // ireg[dst] <- (uint32)a | (int64)b << 32
  kVmIAdd, kVmISub, kVmIMul,   // ireg[dst] <- ireg[a] op ireg[b]
  kVmTick,     // ireg[dst] += 1; error 2 if it exceeds 10000 (while-loop limit)
  kVmInc,      // ireg[dst] += 1 (entries of a conditional region, for the op counts)
  kVmErr       // error a
};

// Error codes written by program mode; the host raises the reference
// interpreter's messages for 1-3.  kVmErrBudget: the program executed more
// than kVmMaxExecuted instructions (nested while loops multiply their
// 10,000-iteration limits); the host then runs it with the host-driven walk
// instead, which is exact because program mode writes only its own slots and
// output buffers.
enum VmError : uint32_t { kVmOk = 0, kVmErrNegPop = 1, kVmErrWhile = 2, kVmErrNegShift = 3, kVmErrBudget = 4 };
constexpr int64_t kVmMaxExecuted = int64_t(1) << 27;

// VmOp::flags.
enum VmFlag : uint8_t {
  kVmBar = 1,     // the threads synchronise before this instruction (vm_finish)
  kVmTrack = 2,   // program mode: dst's tail may be 1 somewhere in the program, so it is written
  kVmTailA = 4,   // program mode: a's tail may be 1
  kVmKeepA = 8,   // a is in registers, left there by the instruction before
  kVmNoStore = 16 // nothing reads the result from its slot
};

struct VmOp {
  uint8_t code;
  uint8_t fill;     // Shr (segment mode): bits shifted in from above are ones; Fill/Load: see codes
  uint8_t flags;    // kVmBar, kVmTrack, kVmTailA
  uint8_t pad;
  int32_t dst;      // Pop: popcount slot index; PopI/IConst/I*: int register
  int32_t a;
  int32_t b;        // Shl / Shr: shift amount (clamped to 64 * n_words); Jz/Jmp: target
};
static_assert(sizeof(VmOp) == 16, "VmOp is 16 bytes");

// Program mode: marks the instructions whose values' tails are not 0 in every
// execution (kVmTrack, kVmTailA), by a fixed point over the slots.
void vm_mark_tails(std::vector<VmOp>& ops, int64_t n_slots);

// Where a value file lives and how many CTAs run a program of `n_slots`
// values of nw words (see vm.cu); `extra` = shared bytes a warp needs beside
// its share of the file.
struct VmPlan {
  int ctas = 0;              // 0: the one-CTA loop kernels (streams too long for a cluster)
  int threads = 0;
  bool smem = false;         // the file fits in the cluster's shared memory
  int64_t dyn_bytes = 0;     // dynamic shared memory per CTA
  int64_t file_words = 0;    // words of the global file (0 when smem)
  int64_t unit = 0;          // a slot's size in the file, in 16-byte units
};
VmPlan vm_plan(int64_t n_slots, int64_t nw, int64_t warp_extra);

// Prepares an instruction list for the cluster engine (plan.ctas > 0):
// * kVmBar: each thread owns its words of every value, so only a shift reads
//   other threads' words: a barrier is needed before a shift whose operand
//   was written since the last barrier, and before a write to a value that a
//   shift has read since.  Instructions that synchronise by themselves (Add,
//   Jz, PopI) count as barriers.  Jump targets start from an unknown state.
// * kVmKeepA, kVmNoStore: operands and results that stay in registers.
// * slot numbers become offsets; operands below 0 are entries of the external
//   table (`n_ext`).
void vm_finish(std::vector<VmOp>& ops, int64_t n_slots, int64_t n_ext, int64_t n_loads, const VmPlan& plan);

struct VmLaunch {
  const VmOp* ops;
  int64_t n_ops;
  int64_t n_loads;           // the first n_loads instructions are kVmLoad (at most kVmWindow)
  const uint64_t* const* ext;   // null: every operand is a slot
  uint64_t* file;            // global slot file (unused when it fits in shared memory)
  int64_t n_slots;
  int64_t nw;
  uint64_t last_mask;
  unsigned long long* pops;
  // The engine zeroes pops[0, n_pops) first and, with `publish` (page-locked
  // host memory), copies them there at the end.
  int64_t n_pops = 0;
  unsigned long long* publish = nullptr;
};

// Program-mode state block, read back after the launch (page-locked host
// memory, written once at the end; device memory for the loop kernels):
// [err u32, pad u32][iregs i64 x n_iregs][tails u8 x n_slots]
struct VmProgLaunch {
  VmLaunch base;             // ops, ext, file, n_slots, nw, last_mask (pops unused)
  uint8_t* state;
  int64_t n_iregs;
};

// Shared bytes per warp of a program's tails and int registers.
inline int64_t vm_prog_warp_bytes(int64_t n_iregs, int64_t n_slots) {
  return 8 * n_iregs + (n_slots + 15) / 16 * 16;
}

inline size_t vm_state_bytes(int64_t n_iregs, int64_t n_slots) {
  return 8 + 8 * static_cast<size_t>(n_iregs) + static_cast<size_t>(n_slots);
}

// Largest stream the automatic policy runs on the VM.
constexpr int64_t kVmMaxWords = 8192;
// Instructions held in shared memory at a time.
constexpr int kVmWindow = 1024;
// Instructions that loading another window for a jump counts as, so that the
// limit on executed instructions stays one on time.
constexpr int kVmStageCost = 32;

// Runs the instruction list on the context's stream as `plan` says (the plan
// of these n_slots and nw).  `file` may be null when the file is in shared
// memory.
void launch_vm(Device& dev, const VmLaunch& L, const VmPlan& plan);
void launch_vm_program(Device& dev, const VmProgLaunch& L, const VmPlan& plan);

}  // namespace bsz
