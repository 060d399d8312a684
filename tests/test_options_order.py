"""Options are accepted by position too: a new one goes behind those that were there."""
import dataclasses

from mcpdlp import PdlpOptions


def test_starting_point_keeps_its_place():
    names = [f.name for f in dataclasses.fields(PdlpOptions)]
    at = names.index("warm_start_guard")
    assert names[at:at + 3] == ["warm_start_guard", "initial_primal", "initial_dual"]
