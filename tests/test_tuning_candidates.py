"""The autotuner times every launch configuration once: its candidates differ in what
the launch depends on (the scheduler selects nothing)."""


def test_candidates_are_different_launches(gc):
    launches = [c[1:] for c in gc.AUTOTUNE_CANDIDATES]
    assert len(set(launches)) == len(launches)
    assert {c[0] for c in gc.AUTOTUNE_CANDIDATES} <= {0, 1}
