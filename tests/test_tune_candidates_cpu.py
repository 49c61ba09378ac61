"""CPU test of the launch autotuner's default candidates: no two are the same
launch (at m = 1 more than 3 CTAs per SM are taken as 3)."""


def test_default_candidates_are_distinct_launches():
    from ncs_b200 import tune
    launches = [(min(c["ctas_per_sm"], 3) if c["m"] == 1 else c["ctas_per_sm"], c["m"])
                for c in tune.DEFAULT_CANDIDATES]
    assert len(set(launches)) == len(launches) == 8
