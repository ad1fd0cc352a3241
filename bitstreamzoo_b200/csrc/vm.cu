// Device-side interpreter for short streams.
//
// At small N the per-op form is launch-bound (a few microseconds per DSL
// operation whatever the stream length; the reference pays the same, plus a
// cudaMalloc per result), and compiling a fused kernel per segment costs far
// more than the segment's work.  The VM runs a whole segment -- possibly
// millions of operations of an unrolled loop nest -- as one launch that walks
// a 16-byte instruction list; program mode (compiled by vmprog.cpp) runs a
// whole program with its if/while control flow in the same way.
//
// Streams of up to 16,384 words run on the cluster engine (k_vm below): one
// CTA, or one thread-block cluster whose CTAs each hold their words of every
// value.  Longer ones (explicit VM mode only) run on the one-CTA loop kernels
// (k_vm_loop, k_vm_program_loop): thread t of T owns words t, t + T, ...,
// the values live in global memory, and every instruction ends with a CTA
// barrier.
//
// A linear scan on the host keeps a segment's value file to its peak live
// count.  POPCOUNT sums all stored words (unmasked, like the per-op kernel).
//
// Every instruction has the exact semantics of the per-op kernel for the
// same node (masking of ~, + and << at the last word; >> filling with the
// operand's tail), so results are bit-identical to the plain form.
#include "vm.h"

#include <algorithm>
#include <mutex>
#include <set>
#include <stdexcept>
#include <string>

namespace bsz {
namespace {

constexpr int64_t kVmSmemLimit = 200 * 1024;

struct VmArgs {
  const VmOp* ops;
  int64_t n_ops;
  const uint64_t* const* ext;
  uint64_t* file;
  int64_t nw;
  uint64_t last_mask;
  unsigned long long* pops;
};

__device__ __forceinline__ VmOp load_op(const VmOp* p) {
  const int4 v = __ldg(reinterpret_cast<const int4*>(p));
  VmOp o;
  o.code = static_cast<uint8_t>(v.x & 0xff);
  o.fill = static_cast<uint8_t>((v.x >> 8) & 0xff);
  o.flags = static_cast<uint8_t>((v.x >> 16) & 0xff);
  o.pad = 0;
  o.dst = v.y;
  o.a = v.z;
  o.b = v.w;
  return o;
}

// The device pointer that a Load or Store carries in two of its fields.
__device__ __forceinline__ uint64_t* op_pointer(int32_t lo, int32_t hi) {
  return reinterpret_cast<uint64_t*>(static_cast<uint64_t>(static_cast<uint32_t>(lo)) |
                                     (static_cast<uint64_t>(static_cast<uint32_t>(hi)) << 32));
}

// ---- per-instruction stream operations of the one-CTA loop kernels -------------
// Thread tid of T owns words tid, tid + T, ...  Callers put a barrier
// between instructions.

__device__ __forceinline__ void vm_not(uint64_t* D, const uint64_t* A, int64_t nw, uint64_t lm, int tid, int T) {
  for (int64_t w = tid; w < nw; w += T) {
    uint64_t r = ~A[w];
    if (w == nw - 1) r &= lm;
    D[w] = r;
  }
}

__device__ __forceinline__ void vm_bitwise(uint8_t code, uint64_t* D, const uint64_t* A, const uint64_t* B,
                                           int64_t nw, uint64_t lm, int tid, int T) {
  for (int64_t w = tid; w < nw; w += T) {
    const uint64_t x = A[w], y = B[w];
    D[w] = code == kVmAnd ? (x & y) : code == kVmOr ? (x | y) : code == kVmXor ? (x ^ y)
           : (x & ~y & (w == nw - 1 ? lm : ~uint64_t(0)));
  }
}

__device__ __forceinline__ void vm_shl(uint64_t* D, const uint64_t* A, int32_t k, int64_t nw, uint64_t lm,
                                       int tid, int T) {
  const int64_t ws = k >> 6;
  const int bs = k & 63;
  for (int64_t w = tid; w < nw; w += T) {
    const int64_t lo = w - ws;
    const uint64_t x = lo >= 0 ? A[lo] : 0;
    const uint64_t y = (bs && lo >= 1) ? A[lo - 1] : 0;
    uint64_t r = bs ? ((x << bs) | (y >> (64 - bs))) : x;
    if (w == nw - 1) r &= lm;
    D[w] = r;
  }
}

__device__ __forceinline__ void vm_shr(uint64_t* D, const uint64_t* A, int32_t k, uint64_t fill, int64_t nw,
                                       int tid, int T) {
  const int64_t ws = k >> 6;
  const int bs = k & 63;
  for (int64_t w = tid; w < nw; w += T) {
    const int64_t lo = w + ws;
    const uint64_t x = lo < nw ? A[lo] : fill;
    const uint64_t y = bs ? (lo + 1 < nw ? A[lo + 1] : fill) : 0;
    D[w] = bs ? ((x >> bs) | (y << (64 - bs))) : x;
  }
}

// Carries per step of T words: two ballots per warp, then the warps'
// (generate, propagate) pairs composed through shared memory.  Each thread
// reads only its own words before writing them, so D may alias A or B.
__device__ __forceinline__ void vm_add(uint64_t* D, const uint64_t* A, const uint64_t* B, int64_t nw,
                                       uint64_t lm, int tid, int T, uint32_t* s_g, uint32_t* s_p) {
  const int lane = tid & 31, warp = tid >> 5, n_warps = T >> 5;
  uint32_t carry = 0;
  for (int64_t base = 0; base < nw; base += T) {
    const int64_t w = base + tid;
    const bool in = w < nw;
    const uint64_t x = in ? A[w] : 0, y = in ? B[w] : 0;
    const uint64_t s = x + y;
    const uint32_t G = __ballot_sync(0xffffffffu, s < x);
    const uint32_t P = __ballot_sync(0xffffffffu, in && s == ~uint64_t(0));
    uint32_t cin, cout;
    if (n_warps == 1) {
      cin = carry;
      cout = static_cast<uint32_t>((static_cast<uint64_t>(G | P) + G + cin) >> 32);
    } else {
      if (lane == 0) {
        s_g[warp] = static_cast<uint32_t>((static_cast<uint64_t>(G | P) + G) >> 32);
        s_p[warp] = P == 0xffffffffu;
      }
      __syncthreads();
      cin = carry;
      for (int v = 0; v < warp; ++v) cin = s_g[v] | (s_p[v] & cin);
      cout = carry;
      for (int v = 0; v < n_warps; ++v) cout = s_g[v] | (s_p[v] & cout);
      __syncthreads();
    }
    const uint64_t z = static_cast<uint64_t>(G | P) + G + cin;
    const uint32_t carries = static_cast<uint32_t>(z) ^ P;
    if (in) {
      uint64_t r = s + ((carries >> lane) & 1u);
      if (w == nw - 1) r &= lm;
      D[w] = r;
    }
    carry = cout;
  }
}

// Popcount of all stored words (unmasked, like the per-op kernel), summed
// over the CTA into *out by one atomic per warp.
__device__ __forceinline__ void vm_popcount(unsigned long long* out, const uint64_t* A, int64_t nw, int tid,
                                            int T) {
  unsigned long long c = 0;
  for (int64_t w = tid; w < nw; w += T) c += __popcll(A[w]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
  if ((tid & 31) == 0 && c) atomicAdd(out, c);
}

__device__ __forceinline__ void vm_barrier(int T) {
  if (T > 32) __syncthreads();
  else __syncwarp();
}

// ---- segment mode ----------------------------------------------------------

__global__ void __launch_bounds__(1024) k_vm_loop(VmArgs args) {
  __shared__ uint32_t s_g[32], s_p[32];
  uint64_t* file = args.file;
  const int T = blockDim.x;
  const int tid = threadIdx.x;
  const int64_t nw = args.nw;
  const uint64_t lm = args.last_mask;
  auto loc = [&](int32_t v) -> uint64_t* {
    return v >= 0 ? file + static_cast<int64_t>(v) * nw : const_cast<uint64_t*>(args.ext[-1 - v]);
  };
  VmOp next = args.n_ops > 0 ? load_op(args.ops) : VmOp{};
  for (int64_t i = 0; i < args.n_ops; ++i) {
    const VmOp op = next;
    if (i + 1 < args.n_ops) next = load_op(args.ops + i + 1);
    const uint64_t* A = loc(op.a);
    switch (op.code) {
      case kVmNot: vm_not(loc(op.dst), A, nw, lm, tid, T); break;
      case kVmAnd: case kVmOr: case kVmXor: case kVmAndNot:
        vm_bitwise(op.code, loc(op.dst), A, loc(op.b), nw, lm, tid, T);
        break;
      case kVmShl: vm_shl(loc(op.dst), A, op.b, nw, lm, tid, T); break;
      case kVmShr: vm_shr(loc(op.dst), A, op.b, op.fill ? ~uint64_t(0) : 0, nw, tid, T); break;
      case kVmAdd: vm_add(loc(op.dst), A, loc(op.b), nw, lm, tid, T, s_g, s_p); break;
      case kVmPop: vm_popcount(args.pops + op.dst, A, nw, tid, T); break;
      default: break;
    }
    vm_barrier(T);
  }
}

// ---- program mode ----------------------------------------------------------
// Control flow runs on the device: a condition is a CTA-wide OR of the
// slot's words (plus its tail), taken by every thread alike.  Thread 0
// updates tails, int registers and op counters; the barrier after every
// instruction publishes them.  Errors stop the program with a code the host
// turns into the reference's message.

struct VmProgArgs {
  VmArgs base;
  uint8_t* state;
  int64_t n_iregs;
};

__global__ void __launch_bounds__(1024) k_vm_program_loop(VmProgArgs P) {
  __shared__ uint32_t s_g[32], s_p[32];
  __shared__ uint32_t s_err;
  __shared__ unsigned long long s_pop;
  const VmArgs& args = P.base;
  uint64_t* file = args.file;
  const int T = blockDim.x;
  const int tid = threadIdx.x;
  const int64_t nw = args.nw;
  const uint64_t lm = args.last_mask;
  uint32_t* g_err = reinterpret_cast<uint32_t*>(P.state);
  long long* iregs = reinterpret_cast<long long*>(P.state + 8);
  uint8_t* tails = P.state + 8 + 8 * P.n_iregs;
  if (tid == 0) {
    s_err = 0;
    s_pop = 0;
  }
  __syncthreads();
  auto slot = [&](int32_t v) -> uint64_t* { return file + static_cast<int64_t>(v) * nw; };
  int64_t pc = 0, executed = 0;
  while (pc < args.n_ops) {
    if (++executed > kVmMaxExecuted) {   // uniform: every thread leaves here
      if (tid == 0) *g_err = kVmErrBudget;
      return;
    }
    const VmOp op = load_op(args.ops + pc);
    ++pc;
    switch (op.code) {
      case kVmNot:
        vm_not(slot(op.dst), slot(op.a), nw, lm, tid, T);
        if (tid == 0) tails[op.dst] = 0;
        break;
      case kVmAnd: case kVmOr: case kVmXor: case kVmAndNot: {
        const uint8_t ta = tails[op.a], tb = tails[op.b];
        vm_bitwise(op.code, slot(op.dst), slot(op.a), slot(op.b), nw, lm, tid, T);
        if (tid == 0)
          tails[op.dst] = op.code == kVmAnd ? (ta & tb) : op.code == kVmOr ? (ta | tb)
                          : op.code == kVmXor ? (ta ^ tb) : 0;
        break;
      }
      case kVmShl:
        vm_shl(slot(op.dst), slot(op.a), op.b, nw, lm, tid, T);
        if (tid == 0) tails[op.dst] = 0;
        break;
      case kVmShr: {
        const uint8_t ta = tails[op.a];
        vm_shr(slot(op.dst), slot(op.a), op.b, ta ? ~uint64_t(0) : 0, nw, tid, T);
        if (tid == 0) tails[op.dst] = ta;
        break;
      }
      case kVmAdd:
        vm_add(slot(op.dst), slot(op.a), slot(op.b), nw, lm, tid, T, s_g, s_p);
        if (tid == 0) tails[op.dst] = 0;
        break;
      case kVmCopy: {
        const uint64_t* A = slot(op.a);
        uint64_t* D = slot(op.dst);
        const uint8_t ta = tails[op.a];
        if (D != A)
          for (int64_t w = tid; w < nw; w += T) D[w] = A[w];
        if (tid == 0) tails[op.dst] = ta;
        break;
      }
      case kVmFill: {
        uint64_t* D = slot(op.dst);
        const uint64_t v = op.fill ? ~uint64_t(0) : 0;
        for (int64_t w = tid; w < nw; w += T) D[w] = (op.fill == 1 && w == nw - 1) ? (v & lm) : v;
        if (tid == 0) tails[op.dst] = op.fill == 2 ? 1 : 0;
        break;
      }
      case kVmLoad: {
        const uint64_t* A = op_pointer(op.a, op.b);
        uint64_t* D = slot(op.dst);
        for (int64_t w = tid; w < nw; w += T) D[w] = A[w];
        if (tid == 0) tails[op.dst] = op.fill;
        break;
      }
      case kVmStore: {
        const uint64_t* A = slot(op.a);
        uint64_t* D = op_pointer(op.dst, op.b);
        for (int64_t w = tid; w < nw; w += T) D[w] = A[w];
        break;
      }
      case kVmJz: {
        const uint64_t* A = slot(op.a);
        int any = 0;
        for (int64_t w = tid; w < nw; w += T) any |= A[w] != 0;
        const int nz = __syncthreads_or(any) || tails[op.a];
        if (!nz) pc = op.b;
        break;
      }
      case kVmJmp:
        pc = op.b;
        break;
      case kVmPopI: {
        if (tails[op.a]) {
          if (tid == 0) s_err = kVmErrNegPop;
          break;
        }
        vm_popcount(&s_pop, slot(op.a), nw, tid, T);
        __syncthreads();
        if (tid == 0) {
          iregs[op.dst] = static_cast<long long>(s_pop);
          s_pop = 0;
        }
        break;
      }
      case kVmIConst:
        if (tid == 0)
          iregs[op.dst] = static_cast<long long>(static_cast<uint64_t>(static_cast<uint32_t>(op.a)) |
                                                 (static_cast<uint64_t>(static_cast<uint32_t>(op.b)) << 32));
        break;
      case kVmIAdd: case kVmISub: case kVmIMul:
        if (tid == 0) {
          // two's-complement wrap, like the int64 host arithmetic
          const unsigned long long x = static_cast<unsigned long long>(iregs[op.a]);
          const unsigned long long y = static_cast<unsigned long long>(iregs[op.b]);
          iregs[op.dst] = static_cast<long long>(op.code == kVmIAdd ? x + y : op.code == kVmISub ? x - y : x * y);
        }
        break;
      case kVmTick:
        if (tid == 0) {
          const long long t = ++iregs[op.dst];
          if (t > 10000) s_err = kVmErrWhile;
        }
        break;
      case kVmInc:
        if (tid == 0) ++iregs[op.dst];
        break;
      case kVmErr:
        if (tid == 0) s_err = static_cast<uint32_t>(op.a);
        break;
      default:
        break;
    }
    __syncthreads();
    if (s_err) break;
  }
  if (tid == 0) *g_err = s_err;
}

// ---- cluster engine ----------------------------------------------------------
// Both modes for streams of up to kMaxCtas x 1024 words.  Words are split
// over the threads of one CTA or of one thread-block cluster, four
// consecutive words to a thread, and every value is a slot of a file that
// each CTA holds its own words of: in its shared memory, or, when the file
// does not fit, in global memory.
//
// What bounds it is the latency of one instruction after another: a few
// hundred kilobytes of data at most, a chain of dependent instructions.  So
//   * instructions are read from shared memory (kVmWindow of them at a time)
//     and the next one is fetched while this one runs; operands come as
//     offsets; the last result stays in registers for the next instruction
//     (kVmKeepA) and is stored only if something else reads it;
//   * a thread's operands are its own words, so &, |, ^, ~, + need no
//     synchronisation on operands; barriers stand only where a shift reads a
//     neighbour's word (kVmBar, placed by vm_finish);
//   * an addition is a 256-bit carry chain per thread, two ballots per warp
//     and one exchange between warps: every warp puts its (generate,
//     propagate) pair into every CTA's table, one barrier, and each warp
//     composes the pairs below it by ballots.  Two tables taken in turn make
//     the one barrier enough;
//   * ints and tails are kept per warp, every warp computing the same ones,
//     so control flow needs a barrier only for a condition's OR and a
//     popcount's sum.
// Inputs are loaded into slots before the first instruction, all in flight
// together.
//
// Measured on a B200 (one instruction, single thread chain; the one-CTA loop
// before it in parentheses): at 3,001 bits x ^ y 133 ns (346), x << 1 274 ns
// (382), x + y 199 ns (742); at 400,009 bits on 16 CTAs 133 (1,458), 594
// (1,922) and 779 ns (10,799).  A 300-op DAG of 400,009 bits: 28 us (244 us)
// between device buffers, 45 us with inputs read from and results written to
// page-locked host memory.
constexpr int kMaxCtas = 16;      // non-portable cluster size
constexpr int kMaxWarps = 8;      // warps per CTA
constexpr int kMaxTotalWarps = kMaxCtas * kMaxWarps;
static_assert(kMaxTotalWarps == 128, "the exchange table is four entries per lane");

struct VmxArgs {
  VmProgArgs prog;         // state, n_iregs: program mode only
  int64_t n_loads;
  int64_t n_slots;
  int64_t n_pops;          // segment mode: popcounts zeroed first ...
  unsigned long long* publish;   // ... and copied here at the end (or null)
  uint32_t unit;           // offset of slot 1 (see Vmx)
  int wpc_log2;            // words per CTA (a power of two) when there are several CTAs
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

extern __shared__ __align__(16) uint64_t s_dyn[];

// SMEM: the file is in shared memory.  SLOTS: every operand is a slot (some
// segments have external operands, below 0).  A slot operand is its offset in
// the CTA's file in units of 16 bytes (vm_finish).
template <bool SMEM, bool SLOTS>
struct Vmx {
  int64_t nw;
  int64_t w0;              // this thread's first word
  uint64_t lm[4];          // its words' masks: bits below the bit length; 0 past the stream
  uint64_t* file;          // this CTA's part of a global file
  const uint64_t* const* ext;
  int wpc_log2;
  int rank, ctas, T, tid, lane, warp, warps;
  uint32_t par;            // exchange table used next
  uint32_t (*ex)[kMaxTotalWarps];

  __device__ __forceinline__ void barrier() const {
    if (ctas > 1) {
      asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    } else if (T > 32) {
      __syncthreads();
    } else {
      __syncwarp();
    }
  }

  // Puts `v` (the same in all lanes) into this warp's entry of every CTA's
  // table and returns the table after a barrier.  A table is written again
  // two exchanges later: its readers have passed the barrier in between.
  __device__ __forceinline__ const uint32_t* exchange(uint32_t v) {
    uint32_t* t = ex[par];
    par ^= 1u;
    uint32_t* e = t + rank * warps + warp;
    if (ctas > 1) {
      if (lane < ctas)
        asm volatile("{ .reg .u32 ra; mapa.shared::cluster.u32 ra, %0, %1; st.shared::cluster.u32 [ra], %2; }" ::"r"(
                         smem_addr(e)),
                     "r"(lane), "r"(v)
                     : "memory");
    } else if (lane == 0) {
      *e = v;
    }
    barrier();
    return t;
  }

  __device__ __forceinline__ ulonglong2* slot(int32_t v) const {
    ulonglong2* f = SMEM ? reinterpret_cast<ulonglong2*>(s_dyn) : reinterpret_cast<ulonglong2*>(file);
    return f + v;
  }

  // A CTA's part of a slot holds the first two words of every thread, then
  // the last two, so that 16-byte accesses of a warp are consecutive.
  __device__ __forceinline__ void load(uint64_t (&x)[4], int32_t v) const {
    if (SLOTS || v >= 0) {
      const ulonglong2* p = slot(v);
      const ulonglong2 a = p[tid], b = p[T + tid];
      x[0] = a.x;
      x[1] = a.y;
      x[2] = b.x;
      x[3] = b.y;
    } else {
      load_ext(x, ext[-1 - v]);
    }
  }
  __device__ __forceinline__ void store(const uint64_t (&x)[4], int32_t v) const {
    if (SLOTS || v >= 0) {
      ulonglong2* p = slot(v);
      p[tid] = make_ulonglong2(x[0], x[1]);
      p[T + tid] = make_ulonglong2(x[2], x[3]);
    } else {
      store_ext(x, const_cast<uint64_t*>(ext[-1 - v]));
    }
  }
  __device__ __forceinline__ void load_ext(uint64_t (&x)[4], const uint64_t* p) const {
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = w0 + j < nw ? p[w0 + j] : 0;
  }
  __device__ __forceinline__ void store_ext(const uint64_t (&x)[4], uint64_t* p) const {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (w0 + j < nw) p[w0 + j] = x[j];
  }
  // Any word in [0, nw) of a value.
  __device__ __forceinline__ uint64_t word(int32_t v, int64_t w) const {
    if (!SLOTS && v < 0) return ext[-1 - v][w];
    int r = 0, l = static_cast<int>(w);
    if (ctas > 1) {
      r = static_cast<int>(w >> wpc_log2);
      l = static_cast<int>(w & ((int64_t(1) << wpc_log2) - 1));
    }
    const int t = l >> 2, j = l & 3;
    const uint64_t* p = reinterpret_cast<const uint64_t*>(slot(v) + ((j >> 1) ? T + t : t)) + (j & 1);
    if (r == rank) return *p;
    if (!SMEM) return p[static_cast<int64_t>(r - rank) * (4 * T)];
    uint64_t x;
    asm volatile("{ .reg .u32 ra; mapa.shared::cluster.u32 ra, %1, %2; ld.shared::cluster.u64 %0, [ra]; }"
                 : "=l"(x)
                 : "r"(smem_addr(p)), "r"(r)
                 : "memory");
    return x;
  }

  // Words past the stream stay zero in every slot; ~, + and << also clear
  // the bits at and above the bit length.
  __device__ __forceinline__ void mask(uint64_t (&x)[4]) const {
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] &= lm[j];
  }

  __device__ __forceinline__ void add(uint64_t (&x)[4], const uint64_t (&y)[4]) {
    uint32_t g;
    asm("add.cc.u64 %0, %0, %5;\n\taddc.cc.u64 %1, %1, %6;\n\taddc.cc.u64 %2, %2, %7;\n\t"
        "addc.cc.u64 %3, %3, %8;\n\taddc.u32 %4, 0, 0;"
        : "+&l"(x[0]), "+&l"(x[1]), "+&l"(x[2]), "+&l"(x[3]), "=r"(g)
        : "l"(y[0]), "l"(y[1]), "l"(y[2]), "l"(y[3]));
    const bool p = (x[0] & x[1] & x[2] & x[3]) == ~uint64_t(0);
    const uint32_t G = __ballot_sync(0xffffffffu, g != 0), P = __ballot_sync(0xffffffffu, p);
    uint32_t cin = 0;
    if (ctas * warps > 1) {
      const uint32_t wg = static_cast<uint32_t>((static_cast<uint64_t>(G | P) + G) >> 32);
      const uint32_t* e = exchange(wg | (P == 0xffffffffu ? 2u : 0u));
      // four warps' pairs per lane, composed; then the carries into the lanes
      const uint4 q = reinterpret_cast<const uint4*>(e)[lane];
      uint32_t cg = q.x & 1u, cp = q.x >> 1;
      cg = (q.y & 1u) | ((q.y >> 1) & cg);
      cp &= q.y >> 1;
      cg = (q.z & 1u) | ((q.z >> 1) & cg);
      cp &= q.z >> 1;
      cg = (q.w & 1u) | ((q.w >> 1) & cg);
      cp &= q.w >> 1;
      const uint32_t GG = __ballot_sync(0xffffffffu, cg != 0), PP = __ballot_sync(0xffffffffu, cp != 0);
      const uint32_t me = rank * warps + warp, grp = me >> 2, r = me & 3;
      cin = ((((GG | PP) + GG) ^ PP) >> grp) & 1u;
      const uint4 m = reinterpret_cast<const uint4*>(e)[grp];
      if (r > 0) cin = (m.x & 1u) | ((m.x >> 1) & cin);
      if (r > 1) cin = (m.y & 1u) | ((m.y >> 1) & cin);
      if (r > 2) cin = (m.z & 1u) | ((m.z >> 1) & cin);
    } else {
      __syncwarp();
    }
    const uint64_t c = (((static_cast<uint32_t>(G | P) + G + cin) ^ P) >> lane) & 1u;
    asm("add.cc.u64 %0, %0, %4;\n\taddc.cc.u64 %1, %1, 0;\n\taddc.cc.u64 %2, %2, 0;\n\taddc.u64 %3, %3, 0;"
        : "+l"(x[0]), "+l"(x[1]), "+l"(x[2]), "+l"(x[3])
        : "l"(c));
    mask(x);
  }

  // r: this thread's words of v
  __device__ __forceinline__ void shl(uint64_t (&r)[4], int32_t v, int32_t k) const {
    const int ws = k >> 6, bs = k & 63;
    uint64_t below;   // the word under this thread's lowest source word
    if (ws == 0) {
      if (SLOTS || v >= 0) {
        // the last word of the thread below, read by every lane (no lane-0
        // branch); the CTA's first thread reads the CTA below's last word
        below = slot(v)[T + max(tid, 1) - 1].y;
        if (tid == 0) below = 0;
        if (ctas > 1 && tid == 0 && rank > 0) below = w0 - 1 < nw ? word(v, w0 - 1) : 0;
      } else {
        below = w0 > 0 && w0 - 1 < nw ? word(v, w0 - 1) : 0;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int64_t w = w0 + j - ws;
        r[j] = w >= 0 && w < nw ? word(v, w) : 0;
      }
      const int64_t w = w0 - 1 - ws;
      below = bs && w >= 0 && w < nw ? word(v, w) : 0;
    }
    if (bs) {
      // eight 32-bit funnel shifts over the halves, taken one half lower when
      // the shift is 32 bits or more
      uint32_t u[10];
      u[0] = static_cast<uint32_t>(below);
      u[1] = static_cast<uint32_t>(below >> 32);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        u[2 + 2 * j] = static_cast<uint32_t>(r[j]);
        u[3 + 2 * j] = static_cast<uint32_t>(r[j] >> 32);
      }
      const bool far = bs >= 32;
#pragma unroll
      for (int i = 9; i > 1; --i) u[i] = far ? u[i - 1] : u[i];
      u[1] = far ? u[0] : u[1];
#pragma unroll
      for (int j = 3; j >= 0; --j) {
        const uint32_t hi = __funnelshift_l(u[2 + 2 * j], u[3 + 2 * j], bs);
        const uint32_t lo = __funnelshift_l(u[1 + 2 * j], u[2 + 2 * j], bs);
        r[j] = static_cast<uint64_t>(lo) | (static_cast<uint64_t>(hi) << 32);
      }
    }
    mask(r);
  }

  __device__ __forceinline__ void shr(uint64_t (&r)[4], int32_t v, int32_t k, uint64_t fill) const {
    const int ws = k >> 6, bs = k & 63;
    uint64_t above;
    if (ws == 0) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (w0 + j >= nw) r[j] = fill;
      above = __shfl_down_sync(0xffffffffu, r[0], 1);
      if (lane == 31) above = w0 + 4 >= nw ? fill : bs ? word(v, w0 + 4) : 0;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int64_t w = w0 + j + ws;
        r[j] = w < nw ? word(v, w) : fill;
      }
      const int64_t w = w0 + 4 + ws;
      above = w < nw ? (bs ? word(v, w) : 0) : fill;
    }
    if (bs) {
#pragma unroll
      for (int j = 0; j < 4; ++j) r[j] = (r[j] >> bs) | ((j < 3 ? r[j + 1] : above) << (64 - bs));
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (w0 + j >= nw) r[j] = 0;
  }

  // Set bits of a value's words, summed over the warp.
  __device__ __forceinline__ uint32_t warp_popcount(const uint64_t (&x)[4]) const {
    return __reduce_add_sync(0xffffffffu, static_cast<uint32_t>(__popcll(x[0]) + __popcll(x[1]) + __popcll(x[2]) +
                                                                __popcll(x[3])));
  }
};

template <bool SMEM, bool SLOTS, bool PROG>
__global__ void __launch_bounds__(kMaxWarps * 32) k_vm(const VmxArgs X) {
  __shared__ __align__(16) uint4 s_ops[kVmWindow + 1];
  __shared__ __align__(16) uint32_t s_ex[2][kMaxTotalWarps];
  const VmArgs& A = X.prog.base;
  Vmx<SMEM, SLOTS> m;
  m.nw = A.nw;
  m.ext = A.ext;
  m.wpc_log2 = X.wpc_log2;
  m.T = blockDim.x;
  m.tid = threadIdx.x;
  m.lane = threadIdx.x & 31;
  m.warp = threadIdx.x >> 5;
  m.warps = blockDim.x >> 5;
  m.rank = blockIdx.x;     // the grid is one cluster
  m.ctas = gridDim.x;
  m.par = 0;
  m.ex = s_ex;
  m.w0 = (static_cast<int64_t>(m.rank) * m.T + m.tid) * 4;
  const int wpc = 4 * m.T;
  m.file = A.file + m.rank * wpc;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    m.lm[j] = m.w0 + j < A.nw - 1 ? ~uint64_t(0) : m.w0 + j == A.nw - 1 ? A.last_mask : 0;
  // program mode: this warp's int registers and tails, after the file
  const int64_t per_warp = 8 * X.prog.n_iregs + (X.n_slots + 15) / 16 * 16;
  long long* iregs = reinterpret_cast<long long*>(reinterpret_cast<char*>(s_dyn + (SMEM ? X.n_slots * wpc : 0)) +
                                                  m.warp * per_warp);
  uint8_t* tails = reinterpret_cast<uint8_t*>(iregs + X.prog.n_iregs);
  for (int i = m.tid; i < 2 * kMaxTotalWarps; i += m.T) (&s_ex[0][0])[i] = 0;
  if (!PROG && m.rank == 0)
    for (int64_t i = m.tid; i < X.n_pops; i += m.T) A.pops[i] = 0;
  if (PROG) {
    for (int64_t i = m.lane; i < X.prog.n_iregs; i += 32) iregs[i] = 0;
    for (int64_t i = m.lane; i < X.n_slots; i += 32) tails[i] = 0;
  }
  // the window of instructions in shared memory: [first, first + cnt)
  int64_t first = 0;
  int cnt = 0;
  auto cta_barrier = [&]() {
    if (m.T > 32) __syncthreads();
    else __syncwarp();
  };
  auto stage = [&](int64_t pc) {
    cta_barrier();
    first = pc;
    cnt = static_cast<int>(A.n_ops - first < kVmWindow ? A.n_ops - first : kVmWindow);
    for (int i = m.tid; i < cnt; i += m.T) s_ops[i] = __ldg(reinterpret_cast<const uint4*>(A.ops + first + i));
    cta_barrier();
  };
  stage(0);
  for (int i = 0; i < X.n_loads; i += 4) {
    uint64_t v[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (i + q < X.n_loads) m.load_ext(v[q], op_pointer(s_ops[i + q].z, s_ops[i + q].w));
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (i + q < X.n_loads) {
        m.store(v[q], s_ops[i + q].y);
        if (PROG) tails[s_ops[i + q].y / X.unit] = (s_ops[i + q].x >> 8) & 0xff;
      }
  }
  m.barrier();   // exchange tables cleared everywhere, inputs loaded
  // A value of the warp's own that its lanes share: all have read what it was
  // computed from before one of them writes it, and see it from then on.
  auto set_shared = [&](auto* p, auto v) {
    __syncwarp();
    if (m.lane == 0) *p = v;
    __syncwarp();
  };
  uint32_t err = kVmOk;
  int64_t executed = 0;    // beyond one pass over the list: jumps back, less what jumps ahead skip
  int i = static_cast<int>(X.n_loads);
  uint64_t x[4] = {0, 0, 0, 0};   // the last instruction's value stays here (kVmKeepA)
  while (true) {
    if (i >= cnt) {   // past this window: the next one
      if (first + i >= A.n_ops) break;
      stage(first + i);
      i = 0;
    }
    uint4 next = s_ops[i];
    int64_t jump = -1;
    while (i < cnt) {
      const uint4 o = next;
      next = s_ops[++i];   // fetched while this one runs (entry cnt is never executed)
      const int dst = static_cast<int>(o.y), a = static_cast<int>(o.z), b = static_cast<int>(o.w);
      const uint32_t code = o.x & 0xff;
      if (o.x & (kVmBar << 16)) m.barrier();
      const bool track = PROG && (o.x & (kVmTrack << 16));
      const bool keep = o.x & (kVmKeepA << 16), keep_out = !(o.x & (kVmNoStore << 16));
      auto tail = [&](int v) -> uint32_t { return tails[v / X.unit]; };
      auto set_tail = [&](int v, uint32_t t) { set_shared(tails + v / X.unit, static_cast<uint8_t>(t)); };
      auto set_int = [&](int r, long long v) { set_shared(iregs + r, v); };
      uint64_t y[4];
      if (code <= kVmAndNot) {   // the commonest first
        if (!keep) m.load(x, a);
        if (code != kVmNot) m.load(y, b);
        if (code == kVmAnd) {
#pragma unroll
          for (int j = 0; j < 4; ++j) x[j] &= y[j];
        } else if (code == kVmOr) {
#pragma unroll
          for (int j = 0; j < 4; ++j) x[j] |= y[j];
        } else if (code == kVmXor) {
#pragma unroll
          for (int j = 0; j < 4; ++j) x[j] ^= y[j];
        } else if (code == kVmAndNot) {
#pragma unroll
          for (int j = 0; j < 4; ++j) x[j] &= ~y[j] & m.lm[j];
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) x[j] = ~x[j] & m.lm[j];
        }
        if (keep_out) m.store(x, dst);
        if (track)
          set_tail(dst, code == kVmAnd ? tail(a) & tail(b) : code == kVmOr ? tail(a) | tail(b)
                        : code == kVmXor ? tail(a) ^ tail(b) : 0);
        continue;
      }
      if (code == kVmAdd) {
        if (!keep) m.load(x, a);
        m.load(y, b);
        m.add(x, y);
        if (keep_out) m.store(x, dst);
        if (track) set_tail(dst, 0);
        continue;
      }
      if (code == kVmShl) {
        if (!keep) m.load(x, a);
        m.shl(x, a, b);
        if (keep_out) m.store(x, dst);
        if (track) set_tail(dst, 0);
        continue;
      }
      switch (code) {
        case kVmShr: {
          const uint32_t t = PROG ? ((o.x & (kVmTailA << 16)) ? tail(a) : 0) : (o.x >> 8) & 0xff;
          if (!keep) m.load(x, a);
          m.shr(x, a, b, t ? ~uint64_t(0) : 0);
          if (keep_out) m.store(x, dst);
          if (track) set_tail(dst, static_cast<uint8_t>(t));
          break;
        }
        case kVmPop: {
          if (!keep) m.load(x, a);
          const uint32_t c = m.warp_popcount(x);
          if (m.lane == 0 && c) atomicAdd(A.pops + dst, static_cast<unsigned long long>(c));
          break;
        }
        case kVmCopy:
          if (!keep) m.load(x, a);
          if (keep_out) m.store(x, dst);
          if (track) set_tail(dst, tail(a));
          break;
        case kVmFill: {
          const uint32_t f = (o.x >> 8) & 0xff;
#pragma unroll
          for (int j = 0; j < 4; ++j) x[j] = f == 0 || m.w0 + j >= m.nw ? 0 : f == 1 ? m.lm[j] : ~uint64_t(0);
          m.store(x, dst);
          if (track) set_tail(dst, f == 2 ? 1 : 0);
          break;
        }
        case kVmLoad:   // inputs past the first kVmWindow
          m.load_ext(x, op_pointer(a, b));
          m.store(x, dst);
          if (track) set_tail(dst, (o.x >> 8) & 0xff);
          break;
        case kVmStore:
          if (!keep) m.load(x, a);
          m.store_ext(x, op_pointer(dst, b));
          break;
        case kVmJz: {
          if (!PROG) break;
          if (!keep) m.load(x, a);
          uint32_t any = __any_sync(0xffffffffu, (x[0] | x[1] | x[2] | x[3]) != 0);
          if (m.ctas * m.warps > 1) {
            const uint4 q = reinterpret_cast<const uint4*>(m.exchange(any))[m.lane];
            any = __any_sync(0xffffffffu, (q.x | q.y | q.z | q.w) != 0);
          } else {
            __syncwarp();
          }
          if (!any && !((o.x & (kVmTailA << 16)) && tail(a))) {
            executed -= b - (first + i);   // skipped
            jump = b;
          }
          break;
        }
        case kVmJmp:   // back to a loop's condition
          if (!PROG) break;
          executed += first + i - b;
          if (executed > kVmMaxExecuted) err = kVmErrBudget;
          jump = b;
          break;
        case kVmPopI: {
          if (!PROG) break;
          if ((o.x & (kVmTailA << 16)) && tail(a)) {
            err = kVmErrNegPop;
            break;
          }
          if (!keep) m.load(x, a);
          uint32_t c = m.warp_popcount(x);
          if (m.ctas * m.warps > 1) {
            const uint4 q = reinterpret_cast<const uint4*>(m.exchange(c))[m.lane];
            c = __reduce_add_sync(0xffffffffu, q.x + q.y + q.z + q.w);
          } else {
            __syncwarp();   // a barrier for the shifts behind it (vm_finish)
          }
          set_int(dst, static_cast<long long>(c));
          break;
        }
        case kVmIConst:
          if (PROG) set_int(dst, static_cast<long long>(reinterpret_cast<uintptr_t>(op_pointer(a, b))));
          break;
        // two's-complement wrap, like the int64 host arithmetic
        case kVmIAdd:
          if (PROG) set_int(dst, static_cast<long long>(static_cast<uint64_t>(iregs[a]) + static_cast<uint64_t>(iregs[b])));
          break;
        case kVmISub:
          if (PROG) set_int(dst, static_cast<long long>(static_cast<uint64_t>(iregs[a]) - static_cast<uint64_t>(iregs[b])));
          break;
        case kVmIMul:
          if (PROG) set_int(dst, static_cast<long long>(static_cast<uint64_t>(iregs[a]) * static_cast<uint64_t>(iregs[b])));
          break;
        case kVmTick: {
          if (!PROG) break;
          const long long t = iregs[dst] + 1;
          set_int(dst, t);
          if (t > 10000) err = kVmErrWhile;
          break;
        }
        case kVmInc:
          if (PROG) set_int(dst, iregs[dst] + 1);
          break;
        case kVmErr:
          if (PROG) err = static_cast<uint32_t>(a);
          break;
        default:
          break;
      }
      if (PROG) {
        if (err) break;
        if (jump >= 0) {
          if (jump < first || jump >= first + cnt) break;
          i = static_cast<int>(jump - first);
          next = s_ops[i];
          jump = -1;
        }
      }
    }
    if (PROG) {
      if (err) break;
      if (jump >= 0) {
        if (jump >= A.n_ops) break;
        stage(jump);
        executed += kVmStageCost;
        i = 0;
      }
    }
  }
  if (PROG && m.rank == 0 && m.warp == 0) {
    __syncwarp();
    uint8_t* st = X.prog.state;
    if (m.lane == 0) *reinterpret_cast<uint32_t*>(st) = err;
    long long* out_iregs = reinterpret_cast<long long*>(st + 8);
    for (int64_t k = m.lane; k < X.prog.n_iregs; k += 32) out_iregs[k] = iregs[k];
    uint8_t* out_tails = st + 8 + 8 * X.prog.n_iregs;
    for (int64_t k = m.lane; k < X.n_slots; k += 32) out_tails[k] = tails[k];
  }
  if (m.ctas > 1 || (!PROG && X.publish)) m.barrier();   // no CTA leaves while another may read its words
  if (!PROG && X.publish && m.rank == 0)
    for (int64_t i = m.tid; i < X.n_pops; i += m.T) X.publish[i] = __ldcg(A.pops + i);
}

int vm_threads(int64_t nw) {
  const int64_t t = ((nw + 31) / 32) * 32;
  return static_cast<int>(std::max<int64_t>(32, std::min<int64_t>(1024, t)));
}

template <bool SMEM, bool SLOTS, bool PROG>
void set_attrs() {
  cudaFuncSetAttribute(k_vm<SMEM, SLOTS, PROG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       static_cast<int>(kVmSmemLimit));
  cudaFuncSetAttribute(k_vm<SMEM, SLOTS, PROG>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}

// Once per device: the engine kernels' shared-memory size and cluster size.
void set_kernel_attrs() {
  static std::mutex mu;
  static std::set<int> done;
  int d = 0;
  cudaGetDevice(&d);
  std::lock_guard<std::mutex> lk(mu);
  if (done.count(d)) return;
  set_attrs<true, true, true>();
  set_attrs<false, true, true>();
  set_attrs<true, true, false>();
  set_attrs<true, false, false>();
  set_attrs<false, false, false>();
  done.insert(d);
}

void check_vm_launch(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw CudaError(std::string(what) + " launch failed: " + cudaGetErrorString(e));
}

void launch_cluster(Device& dev, const VmPlan& plan, bool program, bool slots, VmxArgs x) {
  set_kernel_attrs();
  x.unit = static_cast<uint32_t>(plan.unit);
  x.wpc_log2 = 0;
  while ((int64_t(1) << x.wpc_log2) < 4 * plan.threads) ++x.wpc_log2;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(plan.ctas));
  cfg.blockDim = dim3(static_cast<unsigned>(plan.threads));
  cfg.dynamicSmemBytes = static_cast<size_t>(plan.dyn_bytes);
  cfg.stream = dev.stream();
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = static_cast<unsigned>(plan.ctas);
  at.val.clusterDim.y = 1;
  at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = plan.ctas > 1 ? 1 : 0;
  cudaError_t e;
  if (program) e = plan.smem ? cudaLaunchKernelEx(&cfg, k_vm<true, true, true>, x) : cudaLaunchKernelEx(&cfg, k_vm<false, true, true>, x);
  else if (slots && plan.smem) e = cudaLaunchKernelEx(&cfg, k_vm<true, true, false>, x);
  else e = plan.smem ? cudaLaunchKernelEx(&cfg, k_vm<true, false, false>, x) : cudaLaunchKernelEx(&cfg, k_vm<false, false, false>, x);
  check_vm_launch(e, program ? "vm program" : "vm");
}

}  // namespace

// The fewest CTAs whose shared memory holds the file, at most 8 warps each:
// an exchange or barrier inside one CTA is several times cheaper than one
// across a cluster.  With no such count the file goes to global memory.
VmPlan vm_plan(int64_t n_slots, int64_t nw, int64_t warp_extra) {
  VmPlan p;
  n_slots = std::max<int64_t>(1, n_slots);
  for (int pass = 0; pass < 2; ++pass) {
    for (int ctas = 1; ctas <= kMaxCtas; ctas *= 2) {
      const int64_t need = (nw + 4 * ctas - 1) / (4 * ctas);
      int64_t t = 32;
      if (ctas == 1) t = std::max<int64_t>(32, (need + 31) / 32 * 32);
      else
        while (t < need) t *= 2;   // words per CTA: a power of two
      if (t > kMaxWarps * 32) continue;
      const int64_t file = n_slots * 4 * t * 8, extra = (t / 32) * warp_extra;
      if (extra > kVmSmemLimit || (pass == 0 && file + extra > kVmSmemLimit)) continue;
      p.ctas = ctas;
      p.threads = static_cast<int>(t);
      p.smem = pass == 0;
      p.dyn_bytes = extra + (pass == 0 ? file : 0);
      p.file_words = pass == 0 ? 0 : n_slots * 4 * t * ctas;
      p.unit = 2 * t * (pass == 0 ? 1 : ctas);
      if (p.unit * n_slots > INT32_MAX) break;
      return p;
    }
  }
  p = VmPlan{};
  p.file_words = n_slots * nw;   // the one-CTA loop kernels, file in global memory
  return p;
}

namespace {

bool vm_writes(const VmOp& o) {
  switch (o.code) {
    case kVmNot: case kVmAnd: case kVmOr: case kVmXor: case kVmAndNot: case kVmAdd: case kVmShl: case kVmShr:
    case kVmCopy: case kVmFill: case kVmLoad:
      return true;
    default: return false;
  }
}
bool vm_reads_a(const VmOp& o) {
  return (vm_writes(o) && o.code != kVmFill && o.code != kVmLoad) || o.code == kVmPop || o.code == kVmStore ||
         o.code == kVmJz || o.code == kVmPopI;
}
bool vm_reads_b(const VmOp& o) { return (o.code > kVmNot && o.code <= kVmAndNot) || o.code == kVmAdd; }
bool vm_shifts(const VmOp& o) { return (o.code == kVmShl || o.code == kVmShr) && o.b > 0; }

}  // namespace

void vm_finish(std::vector<VmOp>& ops, int64_t n_slots, int64_t n_ext, int64_t n_loads, const VmPlan& plan) {
  const size_t n = static_cast<size_t>(n_slots + n_ext);
  auto id = [&](int32_t v) { return static_cast<size_t>(v >= 0 ? v : n_slots + (-1 - static_cast<int64_t>(v))); };
  std::vector<uint8_t> target(ops.size() + 1, 0);
  bool straight = true;
  for (const VmOp& o : ops)
    if (o.code == kVmJz || o.code == kVmJmp) {
      target[static_cast<size_t>(o.b)] = 1;
      straight = false;
    }
  // Barriers.
  std::vector<int64_t> written(n, -1), read_across(n, -1);   // epoch of the last one
  int64_t epoch = 0;
  for (size_t i = 0; i < ops.size(); ++i) {
    VmOp& o = ops[i];
    bool bar = target[i] && o.code != kVmJz;   // Jz reads own words only and is a barrier itself
    const bool own_barrier = o.code == kVmAdd || o.code == kVmJz || o.code == kVmPopI;
    if (vm_shifts(o) && written[id(o.a)] == epoch) bar = true;
    if (vm_writes(o) && !own_barrier && read_across[id(o.dst)] == epoch) bar = true;
    if (bar) {
      o.flags |= kVmBar;
      ++epoch;
    }
    if (own_barrier) ++epoch;
    if (vm_shifts(o)) read_across[id(o.a)] = epoch;
    if (vm_writes(o)) written[id(o.dst)] = epoch;
  }
  // The value in registers: an instruction's result, or the operand that it
  // only read.
  bool have = false;
  int32_t held = 0;
  for (size_t i = static_cast<size_t>(n_loads); i < ops.size(); ++i) {
    VmOp& o = ops[i];
    if (target[i]) have = false;
    if (vm_reads_b(o) && o.code != kVmAndNot && have && o.b == held && o.a != held)
      std::swap(o.a, o.b);
    if (vm_reads_a(o) && have && o.a == held) o.flags |= kVmKeepA;
    if (vm_writes(o)) {
      have = true;
      held = o.dst;
    } else if (vm_reads_a(o)) {
      have = true;
      held = o.a;
    }
  }
  // Straight-line code: results that only the next instruction reads, from
  // registers, are not stored.
  if (straight) {
    std::vector<uint8_t> read(n, 0);
    for (size_t i = ops.size(); i-- > 0;) {
      VmOp& o = ops[i];
      if (vm_writes(o)) {
        if (o.dst >= 0 && !read[id(o.dst)] && o.code != kVmLoad) o.flags |= kVmNoStore;
        read[id(o.dst)] = 0;
      }
      if (vm_reads_a(o) && (!(o.flags & kVmKeepA) || vm_shifts(o))) read[id(o.a)] = 1;
      if (vm_reads_b(o)) read[id(o.b)] = 1;
    }
  }
  // Slots as offsets.
  auto offset = [&](int32_t& v) {
    if (v >= 0) v = static_cast<int32_t>(v * plan.unit);
  };
  for (VmOp& o : ops) {
    if (vm_writes(o)) offset(o.dst);
    if (vm_reads_a(o)) offset(o.a);
    if (vm_reads_b(o)) offset(o.b);
  }
}

void vm_mark_tails(std::vector<VmOp>& ops, int64_t n_slots) {
  std::vector<uint8_t> may(static_cast<size_t>(n_slots), 0);
  auto result = [&](const VmOp& o) -> int {
    switch (o.code) {
      case kVmFill: return o.fill == 2;
      case kVmLoad: return o.fill;
      case kVmCopy: case kVmShr: return may[o.a];
      case kVmAnd: return may[o.a] & may[o.b];
      case kVmOr: case kVmXor: return may[o.a] | may[o.b];
      default: return 0;
    }
  };
  for (bool grown = true; grown;) {
    grown = false;
    for (const VmOp& o : ops)
      if (result(o) && !may[o.dst]) {
        may[o.dst] = 1;
        grown = true;
      }
  }
  for (VmOp& o : ops) {
    if (vm_writes(o) && may[o.dst]) o.flags |= kVmTrack;
    if ((o.code == kVmShr || o.code == kVmJz || o.code == kVmPopI) && may[o.a]) o.flags |= kVmTailA;
  }
}

void launch_vm(Device& dev, const VmLaunch& L, const VmPlan& plan) {
  if (L.n_ops <= 0) return;
  VmArgs a{L.ops, L.n_ops, L.ext, L.file, L.nw, L.last_mask, L.pops};
  if (!plan.smem && !L.file && L.n_slots > 0) throw std::invalid_argument("vm: no slot file");
  ProfScope prof(dev, "k_vm");
  if (plan.ctas > 0) {
    launch_cluster(dev, plan, false, L.ext == nullptr, VmxArgs{{a, nullptr, 0}, L.n_loads, L.n_slots, L.n_pops, L.publish, 0, 0});
  } else {
    if (L.n_pops > 0) BSZ_CUDA(cudaMemsetAsync(L.pops, 0, static_cast<size_t>(L.n_pops) * 8, dev.stream()));
    k_vm_loop<<<1, vm_threads(L.nw), 0, dev.stream()>>>(a);
    check_vm_launch(cudaGetLastError(), "vm");
  }
  ++dev.n_launches;
}

void launch_vm_program(Device& dev, const VmProgLaunch& L, const VmPlan& plan) {
  const VmLaunch& B = L.base;
  if (B.n_ops <= 0) return;
  VmProgArgs a{{B.ops, B.n_ops, B.ext, B.file, B.nw, B.last_mask, nullptr}, L.state, L.n_iregs};
  if (!plan.smem && !B.file && B.n_slots > 0) throw std::invalid_argument("vm: no slot file");
  ProfScope prof(dev, "k_vm_program");
  if (plan.ctas > 0) {
    launch_cluster(dev, plan, true, true, VmxArgs{a, B.n_loads, B.n_slots, 0, nullptr, 0, 0});
  } else {
    BSZ_CUDA(cudaMemsetAsync(L.state, 0, vm_state_bytes(L.n_iregs, B.n_slots), dev.stream()));
    k_vm_program_loop<<<1, vm_threads(B.nw), 0, dev.stream()>>>(a);
    check_vm_launch(cudaGetLastError(), "vm program");
  }
  ++dev.n_launches;
}

}  // namespace bsz
