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
