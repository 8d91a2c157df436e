"""The autotuner's choice: a shape is written to the table only where it beats the
built-in one at every side that was timed."""
from cat_cpu_b200 import autotune

BUILT_IN = (2, 0)


def test_built_in_is_kept_unless_beaten():
    assert autotune.choose({4096: {BUILT_IN: 1.0, (2, 64): 1.5}}, BUILT_IN) is None
    assert autotune.choose({4096: {BUILT_IN: 1.0, (2, 64): 0.99}}, BUILT_IN) is None  # within the margin
    assert autotune.choose({4096: {BUILT_IN: 1.0, (2, 64): 0.9, (3, 32): 0.8}}, BUILT_IN) == (3, 32)


def test_a_class_is_not_set_from_one_of_its_sides():
    """64 rows a band are best at 4096 and three times too slow at 1024."""
    times = {1024: {BUILT_IN: 4.0, (2, 64): 12.9, (2, 16): 4.0}, 4096: {BUILT_IN: 13.0, (2, 64): 11.0, (2, 16): 14.0}}
    assert autotune.choose(times, BUILT_IN) is None
    times[1024][(2, 16)], times[4096][(2, 16)] = 3.5, 12.5
    assert autotune.choose(times, BUILT_IN) == (2, 16)


def test_table_in_use_names_no_single_grid_shape():
    """The built-in choices follow the sides; nothing in the table holds them back."""
    import os
    path = os.path.join(os.path.dirname(autotune.__file__), "tuning", "ltl_tuning.txt")
    lines = [x for x in open(path) if x.strip() and not x.startswith("#")]
    assert all(x.startswith("variant=batch ") for x in lines), lines
