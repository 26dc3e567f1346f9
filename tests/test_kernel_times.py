"""The breakdown by kernel knows every launching function (host side only)."""
import inspect

from llm_steadyinfer_b200.csrc import ops
from llm_steadyinfer_b200.engine.kernel_times import KINDS


def test_every_launching_function_has_a_name_in_the_breakdown():
    """A function that is not listed would be missing from the shares, and the others would look larger."""
    launching = {n for n, f in inspect.getmembers(ops, inspect.isfunction)
                 if f.__module__ == ops.__name__ and not n.startswith("_") and "_stream()" in inspect.getsource(f)}
    assert len(launching) > 40
    assert launching - set(KINDS) - {n for n in launching if n.startswith("selftest")} == set()
    assert all(hasattr(ops, n) for n in KINDS)
