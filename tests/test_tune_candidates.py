"""The candidates of the autotuner are different launches (CPU): the last field, contacts on a second stream, has an
effect with a positive block size only."""
from woodem_gb300 import tune


def test_candidates_differ():
    seen = [(b, c, g, s if b > 0 else None) for b, c, g, s in tune.DEFAULT_CANDIDATES]
    assert len(set(seen)) == len(seen)
    assert seen[0] == (-256, 32, False, None)  # the default shape comes first
