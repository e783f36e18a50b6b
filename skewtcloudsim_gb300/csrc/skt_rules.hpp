// Rules of the launches that need no GPU, in a form that host code compiles alone.
#pragma once

namespace skt {

// The reductions of the one-launch PCG are told apart by a tag that counts on from launch to launch, kept by
// block 0: the one it stores after its last reduction, the next launch's first being one more. Where a wait
// ran out, block 0 gave up at `tag`, and a block that saw the late partial after all went on and sent its
// partial of the next reduction, but not one beyond, which would take block 0's. That tag is passed over, so
// that no partial of an abandoned launch is taken for one of the next.
constexpr unsigned tag_after(unsigned tag, bool stuck) { return stuck ? tag + 1 : tag; }

}  // namespace skt
