"""A batch's options are filled by column: each curve's as a single search's
are, field by field, whatever integers, texts and intervals they hold."""

import pytest

INTEGERS = [0, 1, -1, True, 2 ** 31 - 1, 2 ** 31, 2 ** 32, 2 ** 33 + 7, 2 ** 63, 2 ** 64 + 3, -2 ** 63, 7.9, "12"]


def fields(options):
    values = {}
    for name, _ in type(options)._fields_:
        value = getattr(options, name)
        if name == "coefficients":
            value = [value[i] for i in range(options.coefficient_count)]
        elif name == "intervals":
            value = [(value[i].lower, value[i].upper) for i in range(options.interval_count)]
        values[name] = value
    return values


@pytest.mark.parametrize("name", ["bound", "first", "last", "include_infinity", "square"])
def test_columns_hold_what_fields_hold(rpg, name):
    curves = [{"coefficients": [["1", "0", "1"], "1 -2 3", [4, -5, 6, 7], []][i % 4], "bound": 10, "first": 1, "last": 5,
               "intervals": [(), [("0", "1.5")], [(None, "2"), (-1, None)]][i % 3], name: value}
              for i, value in enumerate(INTEGERS)]
    filled, _keep = rpg._batch_options(curves)
    for i, c in enumerate(curves):
        single = rpg.SearchOptions()
        _buffers = rpg._fill_options(single, rpg.coefficients_of(c["coefficients"]), c["bound"], c["first"], c["last"],
                                     c["intervals"], c.get("include_infinity", True), square=c.get("square", False))
        assert fields(filled[i]) == fields(single), c
