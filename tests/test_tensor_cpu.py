"""CPU: core::Tensor's companion planes, which a layer attaches to what it wrote and the next layer reads in its place, do not outlive the value."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "turbotransformers_b200")

PROGRAM = """
#include <cstdio>
#include <utility>
#include "core.h"
using namespace turbo_transformers::core;
static int bad = 0;
#define EXPECT(x) if (!(x)) { std::printf("%d: %s\\n", __LINE__, #x); ++bad; }
static void attach(Tensor& t) {
  TensorExtras& e = t.NewExtras();
  e.lo.Reshape<float>({4}, kDLCPU, 0);
  e.hi.Reshape<float>({4}, kDLCPU, 0);
}
int main() {
  Tensor t(nullptr);
  t.Reshape<float>({4}, kDLCPU, 0);
  attach(t);
  const Tensor& seen = t;
  EXPECT(seen.raw() && seen.data<float>() && t.lo() && t.hi());  // reading keeps them
  Tensor moved(std::move(t));
  EXPECT(moved.lo() && moved.hi());
  moved.mutableData<float>()[0] = 1.f;  // a caller's own kernel would write here
  EXPECT(!moved.lo() && !moved.hi());
  attach(moved);
  EXPECT(moved.raw_mut() && !moved.lo() && !moved.hi());
  attach(moved);
  moved.Reshape<float>({4}, kDLCPU, 0);
  EXPECT(!moved.lo() && !moved.hi());
  return bad;
}
"""


def test_companions_go_with_the_value_they_belong_to(built, tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "include"), "-I", os.path.join(PKG, "csrc", "host"), str(src),
                    os.path.join(PKG, "csrc", "host", "core.cpp"), "-L", PKG, "-l:libttb.so", "-Wl,-rpath," + PKG, "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
