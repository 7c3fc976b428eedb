"""What handles share is shared by device and CUDA context (csrc/per_context.hpp):
a context that has changed, as after a cudaDeviceReset, makes it empty."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cassert>
#include "per_context.hpp"
struct Share {
    int device;
    uint64_t context;
    int kept = 0;
    Share(int d, uint64_t c) : device(d), context(c) {}
};
int main() {
    mcg::PerContext<Share> known;
    auto a = known.get(0, 1);
    a->kept = 5;
    assert(known.get(0, 1) == a);           // another handle of the same context
    auto other = known.get(1, 7);           // another device
    assert(other != a && other->kept == 0 && other->device == 1 && other->context == 7);
    auto b = known.get(0, 2);               // device 0 was reset with a handle open
    assert(b != a && b->kept == 0 && b->context == 2);
    assert(known.get(0, 2) == b && a->kept == 5);
    a.reset();                              // the old handle goes late
    assert(known.get(0, 2) == b && known.get(1, 7) == other);
    b->kept = 3;
    b.reset();                              // the last handle: what it shared goes with it
    assert(known.get(0, 2)->kept == 0);
    return 0;
}
"""


def test_shared_objects_follow_the_context(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "multicomponent_color_gradient_b200", "csrc"),
                    str(src), "-o", str(exe), "-pthread"], check=True)
    subprocess.run([str(exe)], check=True)
