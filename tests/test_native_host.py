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
