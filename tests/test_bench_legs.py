"""bench.py's legs beside the headline: a failed one leaves its error and the
next runs; one that lost the CUDA context ends the rest, which are not called."""
import importlib
import sys


def test_legs():
    argv, sys.argv = sys.argv, ["bench.py"]
    try:
        bench = importlib.import_module("bench")
    finally:
        sys.argv = argv
    state = {"usable": True, "called": []}

    def leg(name, error=None, loses=False):
        def fn():
            state["called"].append(name)
            if loses:
                state["usable"] = False
            if error:
                raise RuntimeError(error)
            return {"ran": name}
        return fn

    legs = bench.Legs({"a", "b", "c", "d"}, lambda: state["usable"])
    assert legs.run("other", leg("other")) is None
    assert legs.run("a", leg("a")) == {"ran": "a"}
    assert legs.run("b", leg("b", error="refused")) == {"error": "RuntimeError: refused"}
    assert legs.lost is None
    assert legs.run("c", leg("c", error="illegal address", loses=True)) == {"error": "RuntimeError: illegal address"}
    assert legs.lost == "c"
    assert "not run" in legs.run("d", leg("d"))["error"]
    assert state["called"] == ["a", "b", "c"]
