"""The autotuner against the table it maintains (CPU only)."""
from xted import autotune as A


def test_table_rows_are_among_the_candidates():
    """Running the tuner can keep what is there: every row of the compiled table
    is one it measures, and no candidate differs from
    another only in the column without effect."""
    rows = {r[1:] for r in A.read_header()}
    full = [(rr, nw, hw) for rr in A.RUN_ROWS for nw in A.NARROW for hw in A.HALF]
    assert rows <= set(full)
    assert len({c[:2] for c in full}) == len(full)
