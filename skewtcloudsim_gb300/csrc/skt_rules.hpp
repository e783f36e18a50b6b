// Rules of the launches that need no GPU, in a form that host code compiles alone.
#pragma once

namespace skt {

// The reductions of the one-launch PCG are told apart by a tag that counts on from launch to launch, kept by
// block 0: the one it stores after its last reduction, the next launch's first being one more. Where a wait
// ran out, block 0 gave up at `tag`, and a block that saw the late partial after all went on and sent its
// partial of the next reduction, but not one beyond, which would take block 0's. That tag is passed over, so
// that no partial of an abandoned launch is taken for one of the next.
constexpr unsigned tag_after(unsigned tag, bool stuck) { return stuck ? tag + 1 : tag; }

// blocks of `per` cells for a grid of n (any n >= 1 that an int holds)
constexpr int blocks_for(int n, int per) { return (n - 1) / per + 1; }

// The faces on the far sides, those of x = X-1, y = Y-1 and z = Z-1: up to 1.5 * 2^31 of them on a grid below
// 2^31 cells with two rows and one plane
constexpr unsigned far_faces(int X, int Y, int Z) { return unsigned(X) * unsigned(Y) + unsigned(X) * unsigned(Z) + unsigned(Y) * unsigned(Z); }

}  // namespace skt
