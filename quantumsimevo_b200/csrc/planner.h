// planner.h -- gate-fusion planner: turns the queued gate list of
// Circuit::execute (Circuit.cpp:64-120) into full-state passes, each applied by
// one launch of the tile kernel (tile.cu).
//
// A pass owns a set T of k "tile" qubits.  Every CTA loads the 2^k amplitudes
// that differ only in T (the other, "outer" bits are fixed per CTA), applies a
// run of gates in registers, and writes them back: one HBM read + write per
// pass instead of one per gate.  A non-diagonal gate (H, X, Y, RX, RY, 2x2,
// CNOT target) needs its target in T; diagonal gates (Z, PHASE, RZ, CPHASE,
// MCPHASE) and CNOT controls can sit on any qubit, because each amplitude's
// full index is known inside the kernel.  SWAP costs nothing: it relabels the
// logical->physical qubit map.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

namespace qse {
namespace plan {

// ---- device program records (layout shared with tile.cu) ----
enum KKind : uint8_t {
    K_NOP = 0,
    K_H,           // unscaled Hadamard on register bit p (the pass scale carries 1/sqrt2 per H)
    K_X,           // X on p, controls: register mask f, thread mask tcond, outer mask ocond
    K_Y,           // Y on p, same controls
    K_RX,          // [[c,-is],[-is,c]] on p, (a,b) = (c,s); Options::unit_rot: divided by c, (a,b) = (s/c, 1),
                   // where |c| >= |s|, else by s, (a,b) = (c/s, 0) (the pass scale carries the divisor)
    K_RY,          // [[c,-s],[s,c]] on p, likewise
    K_U,           // generic 2x2 on p, matrix index g, controls as K_X
    K_ACC_THR,     // if thread cond: acc_thr *= group value g
    K_ACC_REG,     // if thread cond: acc[p] *= group value g
    K_PHD,         // if thread cond: amplitudes with (j & f) == f *= group value g
    K_FLUSH_REG,   // amplitudes with bit p *= acc[p]; acc[p] = 1
    K_FLUSH_ALL,   // flush acc[p] for p in f, then all amplitudes *= acc_thr * (a + ib);
                   // q: 0 = the constant is 1, 1 = it has modulus 1, 2 = any
    K_TRANSPOSE,   // exchange through shared memory into layout g
    K_GRAD_X,      // slot g += sum_pairs Im(conj(l0) s1 + conj(l1) s0)         (RX generator)
    K_GRAD_Y,      // slot g += sum_pairs Re(conj(l1) s0) - Re(conj(l0) s1)     (RY generator)
    K_GRAD_Z,      // slot g += sum sign * Im(conj(l) s): sign flips on reg bit p (p<8), thread mask tcond, outer mask ocond
    K_GRAD_P,      // if conds: slot g += sum_{(j&f)==f} Im(conj(l) s)          (phase-type generator, scaled on host)
    K_KIND_COUNT
};

struct alignas(16) KOp {
    uint8_t kind;
    uint8_t p;
    uint8_t q;
    uint8_t f;
    uint16_t tcond;
    uint16_t g;
    uint64_t ocond;
    double a;
    double b;
};
static_assert(sizeof(KOp) == 32, "KOp layout");

// Per-thread-bit entries beyond the layout's thread bits are 0: the interpreter
// always walks kThrBits of them.  wthr/wreg and rthr/rreg are the slot images of
// what a thread writes (the layout before) and reads (this one) in the exchange
// into this layout, so that it does not look them up through two tables.
constexpr uint32_t kThrBits = 10;   // 12 tile qubits, 2 of them in registers
struct alignas(16) LayoutRec {
    uint16_t L[16];        // shared-memory slot image of every tile-local bit (XOR-linear map)
    uint16_t wthr[16];
    uint16_t rthr[16];
    uint16_t wreg[8], rreg[8];
    uint8_t reg[8];        // tile-local bits held in registers (register index bit i <-> reg[i]; rb <= 5)
    uint8_t preg[8];       // their physical qubits
    uint8_t thr[16];       // tile-local bit of thread-index bit t (ascending), t < nthr
    uint8_t pthr[16];      // their physical qubits
    uint8_t nthr;          // number of thread-index bits
    uint8_t pad[15];
};
static_assert(sizeof(LayoutRec) == 192, "LayoutRec layout");

struct TermRec {       // one diagonal term: angle theta if all outer bits of ocond are set
    uint64_t ocond;
    double theta;
};

struct alignas(8) GroupRec {   // terms [first, first+count): value (cos, sin) of their angles' sum, per CTA
    uint32_t first;
    uint32_t count;
};

// An angle-carrying record of a pass and the source gate it came from: a
// K_RX / K_RY op (a, b) = (cos, sin)(theta/2), or a diagonal term's theta.
// Lets a caller rebind angles on the device without planning again.
struct AngleRef {
    uint32_t index;   // into PassProgram::ops or PassProgram::terms
    uint32_t src;     // source-gate index in the planner input
};

struct PassProgram {
    uint32_t k = 0;                 // tile qubits
    uint32_t rb = 4;                // register bits per thread
    bool lane_swaps = false;        // Options::lane_swaps
    uint64_t outer_mask = 0;        // physical qubits not in the tile
    uint8_t tile_phys[16] = {0};    // physical qubit of tile-local bit b (ascending)
    uint32_t layout0 = 0;           // layout at load time (index into layouts)
    std::vector<KOp> ops;
    std::vector<LayoutRec> layouts;
    std::vector<TermRec> terms;
    std::vector<GroupRec> groups;
    std::vector<double> mats;       // 8 doubles per K_U matrix
    std::vector<int32_t> slot_src;  // gradient slot (local) -> gradient occurrence id
    std::vector<AngleRef> op_angles;    // K_RX / K_RY ops
    std::vector<AngleRef> term_angles;  // terms of PHASE / RZ / CPHASE / MCPHASE gates
    std::vector<uint32_t> order;    // source-gate indices absorbed, in execution order
    // debug view, per entry of `order`: physical target, physical control
    // (CNOT / CPHASE) and physical support (diagonal gates); SWAPs come first
    // with zeros (they only relabel)
    std::vector<uint32_t> phys_target;
    std::vector<uint32_t> phys_control;
    std::vector<uint64_t> phys_support;
    uint32_t ngates = 0;            // source gates absorbed
    uint32_t n_nondiag = 0;
    // How the program's numbers follow from the source gates, in emission order,
    // besides op_angles and term_angles (bind_angles walks them): the pending
    // scale of the unscaled Hadamards and rotations and the ops that take it, the RZ gates
    // whose global phase the pass constant carries, and the matrices' gates.
    struct ScaleEvent {
        enum Kind : uint8_t { hadamard, rotation, gradient, flush, last } kind;
        uint32_t op;                // index into ops (rotation: into op_angles; hadamard: none)
    };
    std::vector<ScaleEvent> scale_events;
    std::vector<uint32_t> gphase_src;
    std::vector<uint32_t> mat_src;
    bool deferred = false;          // the pass constant goes to the next pass instead of the last flush
    // SWAPs only, and no constant to apply: the output is the input
    bool idle() const { return n_nondiag == 0 && groups.empty() && slot_src.empty() && (ops.empty() || ops.back().q == 0); }
};

// ---- planner input ----
struct Gate {
    int type = 0;          // qse_gate_type
    uint32_t t = 0;        // target (SWAP: q0)
    uint32_t c = 0;        // control (CNOT, CPHASE; SWAP: q1)
    uint64_t cmask = 0;    // MCPHASE controls (logical)
    double theta = 0.0;    // bound angle
    double m[8] = {0};     // QSE_GATE_2X2
    int32_t grad = -1;     // gradient occurrence id (adjoint reverse sweep), -1 = none
};

// Non-diagonal gates per pass when the passes are compiled into specialised
// kernels: NVRTC's compile time grows faster than linearly with the length of
// the straight-line kernel (a 12-qubit pass of 2400 gates takes over a minute),
// while an extra pass costs one sweep of the state.
constexpr uint32_t kJitMaxGates = 256;

struct Options {
    uint32_t k = 12;             // tile qubits (clamped to n)
    uint32_t rb = 4;             // register bits per thread (at most 5; the interpreter kernel takes 3 or 4)
    uint32_t rb_first = 0;       // the first pass's register bits (0: rb)
    uint32_t max_gates = 0;      // 0 = no cap on non-diagonal gates per pass
    uint32_t max_terms = 1024;   // diagonal terms per pass (shared-memory group table)
    bool grads = false;          // emit K_GRAD_* for gates with grad >= 0
    uint32_t max_slots = 0;      // gradient slots per pass, 0 = no cap
    bool direct_phases = false;  // single-register-bit phase terms without a thread
                                 // condition as K_PHD, not through an accumulator
    bool zz_fuse = false;        // rewrite CNOT(c,t) RZ(th,t) CNOT(c,t) as the diagonal
                                 // RZ(th,c) PHASE(th,t) CPHASE(-2th,c,t) (same three slots;
                                 // bind_angles rewrites the new gates likewise)
    bool lane_swaps = false;     // specialised kernels move physical qubits 0..2 from the registers to the
                                 // lanes by shuffles where a pass reads and writes
    bool low_lanes = false;      // the layouts keep physical qubits 0..2 out of the registers where a pass reads and writes
    bool unit_rot = false;       // rotations divided by their larger entry, one FMA per component instead
                                 // of a multiply and an FMA (kernels that take K_RX / K_RY in that form)
    bool keep_gphase = true;     // false: drop RZ's global phase (expectations and gradients
                                 // do not see it; the pass programs then depend on angles
                                 // only through op_angles / term_angles)
};

// What of a context's settings decides how its states' gates are planned.
struct Settings {
    int jit = 1;                 // qse_ctx_set_jit
    int tile_qubits = 12;        // qse_ctx_set_fusion
    bool exact_tiles = false;
    int max_gates_per_pass = 0;
};

// The options of an n-qubit state's forward passes (compact_input: the first one
// makes its input from a compact state) and of the adjoint sweep's reverse passes.
// qse_plan_compile plans with the same, so what it compiles is what runs.
Options forward_options(const Settings& s, uint32_t n, bool compact_input);
Options adjoint_options(const Settings& s, uint32_t n);
// tile qubits of a state for a setting and rb register bits, at most kmax
uint32_t tile_size(int tile_qubits, uint32_t n, uint32_t rb, uint32_t kmax);

struct Plan {
    std::vector<PassProgram> passes;
    uint32_t perm_final[64];
    uint64_t gates = 0;
};

// The rewrite of Options::zz_fuse on its own: out = gates with every
// CNOT(c,t) RZ(th,t) CNOT(c,t) (no gradient ids) replaced by RZ(th,c)
// PHASE(th,t) CPHASE(-2th,c,t) in the same three slots; false (out untouched)
// when there is none.
bool fuse_zz(const std::vector<Gate>& gates, std::vector<Gate>& out);

// Plans gates (logical qubits) for an n-qubit state whose logical->physical
// map is perm_in.  Throws qse::Error on invalid gates.
Plan build(const std::vector<Gate>& gates, uint32_t n, const uint32_t* perm_in, const Options& opt);

// Everything in a plan but its numbers depends on the gates' types, qubits and
// gradient ids only: this sets the numbers (angles, matrices, constants) of a
// plan built for gates that differ from these in theta and m at most, to what
// build() gives for them, bit for bit.  When memory runs out it throws with every
// number as it was.
void bind_angles(Plan& plan, const std::vector<Gate>& gates, const Options& opt);

// Planner-only debug view used by the CPU tests: for each pass, the tile
// (physical qubits) and the source-gate indices in execution order.
std::string describe(const Plan& p);

}  // namespace plan
}  // namespace qse
