/* Where a call may work in the caller's memory itself: the rules on plain values, no device needed. */
#include <cstdio>

#include "../../axomae_b200/csrc/caller_memory.cuh"

static int failed = 0;
static void check(bool ok, const char *what) {
  if (!ok) std::printf("failed: %s\n", what), failed = 1;
}

static cudaPointerAttributes at(cudaMemoryType type, int device) {
  cudaPointerAttributes a{};
  a.type = type;
  a.device = device;
  return a;
}

static std::vector<char> direct(std::vector<nb::Span> films) { return nb::direct_films(films); }
using Want = std::vector<char>;

int main() {
  check(nb::on_device(at(cudaMemoryTypeDevice, 1), 1), "the GPU's own memory");
  check(!nb::on_device(at(cudaMemoryTypeDevice, 0), 1), "another GPU's memory");
  check(!nb::on_device(at(cudaMemoryTypeHost, 1), 1), "pinned host memory");
  check(!nb::on_device(at(cudaMemoryTypeManaged, 1), 1), "managed memory");
  check(!nb::on_device(at(cudaMemoryTypeUnregistered, -2), 0), "pageable host memory");
  check(!nb::on_device(cudaPointerAttributes{}, 0), "a pointer without attributes");

  check(nb::overlap({4096, 64, true}, {4096, 64, true}) && nb::overlap({4096, 64, true}, {4159, 64, true}) &&
            nb::overlap({4159, 64, true}, {4096, 64, true}) && nb::overlap({4096, 64, true}, {4100, 4, true}),
        "spans that overlap");
  check(!nb::overlap({4096, 64, true}, {4160, 64, true}) && !nb::overlap({4160, 64, true}, {4096, 64, true}),
        "spans end to end");

  check(direct({}) == Want{}, "no films");
  check(direct({{4096, 64, true}}) == Want{1}, "one film");
  check(direct({{0, 64, false}, {0, 64, false}}) == (Want{0, 0}), "no device films");
  check(direct({{4096, 64, false}, {8192, 64, true}}) == (Want{0, 1}), "a film elsewhere");
  check(direct({{4100, 64, true}, {4104, 64, true}}) == (Want{0, 0}), "not on 16 bytes");
  check(direct({{4160, 64, true}, {4096, 64, true}}) == (Want{1, 1}), "films end to end");
  check(direct({{4144, 64, true}, {4096, 64, true}, {8192, 16, true}}) == (Want{0, 0, 1}), "films that overlap");
  check(direct({{4096, 64, true}, {8192, 16, true}, {4096, 16, true}}) == (Want{0, 1, 0}), "one buffer for two");
  check(direct({{4096, 4096, true}, {4112, 16, true}, {4160, 16, true}, {8192, 16, true}}) == (Want{0, 0, 0, 1}),
        "a film over two others");
  check(direct({{4096, 64, false}, {4112, 16, true}}) == (Want{0, 0}), "over a film elsewhere");
  check(direct({{0, 64, false}, {16, 64, true}}) == (Want{0, 1}), "no film and a low address");
  return failed;
}
