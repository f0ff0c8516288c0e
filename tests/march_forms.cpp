// The forms a program's march steps take (test_march_forms.py): the steps of
// stdin, five numbers each (opcode, a, b, c, value), flattened whole; one line
// a march step: its form, its post operation and whether it is rare.
#include "octree.h"

#include <cstdio>

int main() {
	auto p = std::make_shared<kdn::Prog>();
	unsigned op, a, b, c;
	double value;
	while (std::scanf("%u %u %u %u %lf", &op, &a, &b, &c, &value) == 5) {
		kdn_step s {};
		s.opcode = uint8_t(op);
		s.a      = a;
		s.b      = b;
		s.c      = c;
		s.value  = value;
		p->steps.push_back(s);
	}
	p->result = uint32_t(p->steps.size() - 1);
	kdn::Octree tree;
	tree.cells.resize(1);
	tree.cells[0].occupancy = kdn::Surface;
	tree.cells[0].programs.push_back(p);
	kdn::FlatWorld flat;
	const std::string error = kdn::flattenOctree(tree, flat);
	if (!error.empty()) return std::fprintf(stderr, "%s\n", error.c_str()), 1;
	const kdn::GpuProgram& g = flat.programs[0];
	for (uint32_t i = 0; i < g.marchCount;) {
		const kdn::MarchStep& s = flat.march[g.march + i];
		const bool rare         = s.op >= kdn::kMarchRare;
		const uint32_t form     = rare ? 0u : s.op & kdn::kMarchFormMask;
		std::printf("%u %u %d\n", form, rare ? 0u : s.op & kdn::kMarchPostMask, int(rare));
		i += rare || form == kdn::FormFma || form == kdn::FormRepeat ? 1 : form == kdn::FormPrimitive && (s.m & kdn::PrimSized) ? 3 : 2;
	}
	return 0;
}
