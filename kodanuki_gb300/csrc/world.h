// Device-resident world of the GB300 backend: the cut octree and the kept
// programs of its leaves, in the layout the trace kernel reads.
//
// The octree is a pointer-free array of 32-bit nodes, children of a node
// contiguous (breadth-first per parent).  A node holds the index of its first
// child, or ~leaf for a leaf.  A leaf names a run of kept programs; a program
// is a run of 16-byte GpuSteps whose operands are register slots (a linear
// scan over the straight-line program reuses a slot once its value is dead),
// so the march keeps a program's live values in a few shared-memory slots.
// The same steps keep their SSA operand numbers in a parallel array for the
// single evaluation at a hit that finds the source leaf (sdf/program.cpp:505).
#pragma once

#include <cstdint>

namespace kdn {

// sdf/program.h:20 Opcode values.
enum Op : uint8_t {
	OpConstant, OpArgument, OpPointX, OpPointY, OpPointZ, OpNormalX, OpNormalY, OpNormalZ,
	OpAdd, OpSubtract, OpMultiply, OpDivide, OpNegate, OpSqrt, OpAbs, OpFloor, OpSin, OpCos,
	OpSign, OpAtan2, OpPow, OpMin, OpMax, OpSmin, OpPosSq, OpLess, OpLessEq, OpEqual,
	OpNotEqual, OpAnd, OpOr, OpNot, OpSelect, OpCount
};

// The march form: a program lowered to steps r = post(fma(a, b, c), w).
// +, -, * and negation are one fused multiply-add each (x + y = fma(x, 1,
// y), x - y = fma(y, -1, x), x * y = fma(x, y, 0)); a product that feeds only
// a sum folds into it; sqrt, |x|, max(x, 0)^2, min, max and a smooth minimum
// of constant radius ride on the step that makes their operand where that
// step's result has no other use; double negations cancel.  Operands are
// slots of the thread's column: the first kMarchFirstSlot hold 0, 1, -1, the
// point and the step's immediate.  Every other reference operation is a
// rare step (kMarchRare + opcode) over slots a, b, c.
//
// The runs of steps that signed distances are made of are fused further, into
// steps of two or three units that round at every point the single steps
// round at, so their values are theirs to the bit:
//  - FormPrimitive: up to three slabs of the point, each p - c, |p - c| or
//    -(p - c), then - h and + r; their sum of squares' root, one's positive
//    part, or the one slab itself; a box's inside term; and - e.  A plane, a
//    sphere, and a rounded box with the faces, edges and corners a cut leaves
//    of it are one step each, the same operations for all of them, so a warp
//    whose lanes are at different ones does not split; a coordinate one is
//    joined with is a plane of its own before it;
//  - FormNorm: such a root over slots, where other steps read the slabs too
//    or make them;
//  - FormRepeat: a coordinate taken into the middle cell of a repetition,
//    x - s * floor(x / s + o).
// 98% of the programs the march runs on config 2 and the city are primitives
// alone, joined by the post operations.  A slab that is one single step and is
// read by other forms stays that step.
enum MarchPost : uint8_t { PostNone, PostSqrt, PostAbs, PostPosSq, PostMin, PostMax, PostSminK };
enum MarchForm : uint8_t { FormFma = 0, FormAxis = 8, FormPrimitive = 16, FormNorm = 24, FormRepeat = 32 }; // op = form + post; FormAxis: in the lowering alone
constexpr uint8_t kMarchPostMask = 7, kMarchFormMask = 56;
constexpr uint8_t kMarchRare = 64;
enum AxisSide : uint8_t { SideNone, SideAbs, SideNegative };
// The terms of a root (FormNorm, FormPrimitive): which are in the sum, which
// are squared by their positive part, which are added by a fused multiply-add
enum SumFlag : uint8_t { SumHas0 = 1, SumHas1 = 2, SumHas2 = 4, SumPositive0 = 8, SumPositive1 = 16, SumPositive2 = 32, SumFused1 = 64, SumFused2 = 128 };
// FormNorm's m where it has no inside term
constexpr uint8_t kNoInside = 255;
// FormPrimitive's m: the slab itself; the sum's one term's positive part; an
// inside term, and that it spans a third term; the h and r unit follows; the
// post operation's w is the step before's result; the result is read from its slot
enum PrimitiveFlag : uint8_t { PrimPlain = 1, PrimSingle = 2, PrimInside = 4, PrimThird = 8, PrimSized = 16, PrimPrevious = 32, PrimStored = 64 };
// FormPrimitive's a, b, c: bits 0-1 the axis, bits 2-3 its AxisSide
constexpr uint8_t kTermSideShift = 2;
enum MarchSlot : uint8_t { SlotZero, SlotOne, SlotMinusOne, SlotX, SlotY, SlotZ, SlotImm, kMarchFirstSlot };

struct alignas(16) MarchStep {
	uint8_t op;  // MarchForm + MarchPost, or kMarchRare + reference opcode
	uint8_t dst; // slot of the result
	uint8_t a, b, c;
	uint8_t w;   // the post operation's second operand (min, max, smooth minimum)
	uint8_t m;     // FormNorm: the inside term's slot; FormPrimitive: PrimitiveFlag
	uint8_t flags; // FormNorm, FormPrimitive: SumFlag
	float value;   // the immediate (SlotImm); a smooth minimum's radius; FormRepeat: s
	float quarter; // 0.25 / radius of a smooth minimum; FormRepeat: o
};
static_assert(sizeof(MarchStep) == 16, "MarchStep is 16 bytes");
// A fused step's second unit: FormNorm e; FormPrimitive the terms' c and e,
// and where PrimSized a third, the terms' h and r.
struct alignas(16) MarchParams {
	float v[4];
};
static_assert(sizeof(MarchParams) == sizeof(MarchStep), "a fused step's parameters are one unit");

constexpr uint32_t kNoLeaf     = 0xFFFFFFFFu;
constexpr uint32_t kMaxSlots   = 48;   // register slots a leaf program may use
constexpr uint32_t kMaxSsa     = 1024; // steps a leaf program may hold
constexpr uint32_t kMaxLeafProgs = 64; // kept programs of one leaf
// The most steps a ray is marched (sphere_trace.h:37 sphereSteps): a ray that
// skims a surface for longer meets nothing.
constexpr uint32_t kMarchSteps = 1u << 16;

// A step of a program's full form, read once a hit: register slots a, b,
// c, the reference opcode and constant, and the leaf a step names.
struct alignas(16) GpuStep {
	uint8_t op;
	uint8_t dst;
	uint8_t a, b, c;
	uint8_t imm;
	uint16_t pad1;
	float value;
	uint32_t leaf;
};
static_assert(sizeof(GpuStep) == 16, "GpuStep is 16 bytes");

struct alignas(8) SsaOps {
	uint16_t a, b, c, pad;
};
static_assert(sizeof(SsaOps) == 8, "SsaOps is 8 bytes");

struct alignas(16) GpuProgram {
	uint32_t code;       // first GpuStep of the whole program (read at a hit)
	uint16_t count;      // its steps
	uint16_t result;     // SSA index of the result
	uint8_t slot;        // slot of the result
	uint8_t slots;       // slots used
	uint16_t marchCount; // units of the march form (a fused step takes two or three)
	uint32_t object;     // index into the scene's object programs
	uint32_t march;      // first MarchStep of the march form
	uint16_t marchSlots; // slots the march form uses
	uint16_t marchSteps; // single steps the march form stands for (what the counters count)
	uint32_t pad1[2];
};
static_assert(sizeof(GpuProgram) == 32, "GpuProgram is 32 bytes");

enum Occupancy : uint8_t { Empty = 0, Filled = 1, Surface = 2 };

// A leaf.  An empty one, or one whose one program is a single axis or sphere
// (on config 2, 54% and 34% of the march's steps; on a ray that skims the
// ground, all of them), is marched from the record itself, in registers.
enum LeafShape : uint8_t { ShapeAxis = 0, ShapeSphere = 1, ShapePrograms = 2, ShapeEmpty = 3 }; // bits 0-1
constexpr uint8_t kShapeMask = 3, kShapeAxisShift = 2, kShapeSideShift = 4; // an axis: bits 2-3 which, 4-5 its AxisSide
struct alignas(16) GpuLeaf {
	uint32_t first;     // first GpuProgram
	uint8_t count;      // kept programs
	uint8_t pad0;
	uint8_t shape;      // LeafShape
	uint8_t pad1;
	// the first program's march form, read with the leaf
	uint32_t march;
	uint16_t marchCount;
	uint16_t marchSteps;
	float params[4]; // of an axis c, h, r, e; of a sphere its centre and radius
};
static_assert(sizeof(GpuLeaf) == 32, "GpuLeaf is 32 bytes");

// Locating a point.  The tree's walls down to its finest level (kMostFine at
// most) are tabled per axis: the descent's own midpoints, 0.5 * (lo + hi)
// level by level in FP32, so a point's place among them, whose bits are the
// descent's choices, is the place the descent from the root would give it.
// The place is estimated by one multiply-add, a quarter of a place low, and
// set right by the one wall above it; the build checks that the estimate is
// never off by more (fineLevelOf) and tables fewer levels where it would be.
// The octree cut across at kGridLevel gives what is there by one load, and
// below it bricks of 4 x 4 x 4 give two levels by one load each (most steps of
// a march end in an empty cell, whose size is all it needs to know: three
// dependent loads for a cell of level 11, where child by child and its leaf's
// record were six).  Leaves below the finest tabled level go on by midpoints.
//
// A grid or brick entry: a leaf (kEntryLeaf; kEntryEmpty where it is empty;
// its level in four bits, its index in 26); else above the finest tabled level
// a brick, and there the first child of an octree node.
constexpr uint32_t kEntryLeaf = 1u << 31, kEntryEmpty = 1u << 30, kEntryLevelShift = 26, kEntryIndex = (1u << 26) - 1u;
constexpr uint32_t kBrick = 64; // entries a brick, x fastest
constexpr uint32_t kGridLevel = 7, kMostFine = 12;
constexpr uint64_t kMostCells = uint64_t(kEntryIndex) + 1u; // cells a tree may have: an entry names any leaf

// Everything the trace kernel reads, as device pointers.
struct DeviceWorld {
	const int32_t* nodes;
	const GpuLeaf* leaves;
	const GpuProgram* programs;
	const GpuStep* steps;
	const MarchStep* march;
	const SsaOps* ssa;
	const uint32_t* leaf_material;
	const uint32_t* grid;   // the entries of the (2^gridLevel)^3 cells, x fastest
	const uint32_t* bricks;
	const float* walls;   // per axis 2^fineLevel + 1 walls
	uint32_t gridLevel, fineLevel;
	float scale[3], bias[3]; // a point's place: p * scale + bias, rounded down
	float lower[3];
	float size[3];
	uint32_t leaf_count;
	uint32_t material_count;
	uint32_t marchSlots; // the most slots a march-form program uses: the trace kernel's shared memory a ray
};

} // namespace kdn
