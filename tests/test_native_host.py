"""Host rules of the engine that no entry point shows, through small C++
programs against its headers."""
import pytest

import native_driver


@pytest.mark.parametrize("kept", [True, False])
@pytest.mark.parametrize("call", ["hfx::DevBuf<int> d; d.upload(%s, nullptr);",
                                  "hfx::TeamPlanDev d; d.upload(%s, 1, nullptr);"], ids=["buffer", "plan"])
def test_upload_refuses_a_temporary(tmp_path, call, kept):
    """An upload's copy may read its host data after the call: data that dies
    with the statement does not compile, data that is kept does."""
    T = "std::vector<int>" if "DevBuf" in call else "hfx::TeamPlanHost"
    body = T + " v; " + call % "v" if kept else call % (T + "{}")
    r = native_driver.compile_driver('#include "hfx_engine.hpp"\nvoid f() { %s }\nint main() {}\n' % body,
                                     tmp_path / "prog", link=False)
    assert (r.returncode == 0) == kept, r.stderr
    assert kept or "deleted" in r.stderr


def test_shared_memory_limit_is_raised_once_per_device_and_kernel(tmp_path):
    """A second device needs its own limit; a failed attempt is repeated."""
    out = native_driver.run_driver(r"""
#include <cstdio>
#include "hfx_smem.hpp"
int main()
{
    hfx::OncePerDevice once;
    int a, b, calls = 0;
    auto ok = [&] { ++calls; return cudaSuccess; };
    auto bad = [&] { ++calls; return cudaErrorInvalidValue; };
    std::printf("%d ", once.run(0, &a, bad) != cudaSuccess);
    for (int dev : {0, 0, 1, 1, 0})
        for (const void* k : {(const void*)&a, (const void*)&b}) once.run(dev, k, ok);
    std::printf("%d\n", calls);
}
""", tmp_path / "prog")
    assert out.split() == ["1", "5"]


def test_every_launch_of_a_build_is_placed_once(tmp_path):
    """Side by side below the threshold, FP64 and FP32 on lanes of their own;
    from there on the FP32 class kernels by decreasing work before a join, then
    the launches that use shared memory; one kind alone on every lane."""
    out = native_driver.run_driver(r"""
#include <cstdio>
#include "hfx_engine.hpp"
struct Sink final : hfx::OpSink {
    void zero(int, void*, size_t) override {}
    void kernel(int, const hfx::KernelSpec&, void**) override {}
    void fork() override { std::printf("fork "); }
    void join() override { std::printf("join "); }
};
int main()
{
    for (double flops : {1e9, hfx::kClassesFirstFlops})
        for (int team : {0, 13})
            for (int fp32 = 0; fp32 < 3; ++fp32) {    // none, class kernels, class and warp kernels
                std::vector<hfx::LaunchGroup> g;
                for (int k = 0; k < 6 * (fp32 > 0); ++k) {
                    hfx::LaunchGroup x{};
                    x.kind = fp32 == 2 && k % 3 == 2;
                    x.n = k == 4 ? 0 : 1;
                    x.flops = x.kind ? 1e15 : flops * (k + 1) / 2.0;
                    g.push_back(x);
                }
                Sink sk;
                hfx::place_launches(sk, team, g, 12, [&](int lane, bool fp64, size_t i) {
                    std::printf("%s%zu@%d ", fp64 ? "t" : g[i].kind ? "w" : "c", i, lane);
                });
                std::printf("\n");
            }
}
""", tmp_path / "prog")
    team = ["t%d@%%d" % i for i in range(13)]
    apart = [t % (i % 12) for i, t in enumerate(team)]
    beside = [t % (i % 8) for i, t in enumerate(team)]
    small, large = out.splitlines()[:6], out.splitlines()[6:]
    cls = ["c5@0", "c3@1", "c2@2", "c1@3", "c0@4"]
    mix = ["c3@0", "c1@1", "c0@2"]
    assert [x.split() for x in small] == [
        [], cls, mix + ["w2@3", "w5@4"],
        apart, beside + ["c0@11", "c1@10", "c2@9", "c3@8", "c5@11"],
        beside + ["c0@11", "c1@10", "w2@11", "c3@9", "w5@11"]]
    assert [x.split() for x in large] == [
        [], cls, mix + ["join", "fork", "w2@3", "w5@4"],
        apart, cls + ["join", "fork"] + apart, mix + ["join", "fork"] + apart + ["w2@3", "w5@4"]]
