"""Reading weights ahead of the stream is asked for, not taken: the default of every entry point of the few-row product."""
import inspect


def test_early_is_off_by_default(pkg, ext, capi):
    assert "early: bool = False" in ext.linear.__doc__
    assert capi.LinearArgs().early == 0
    for f in (capi.linear, pkg.mixers.few_rows, pkg.mixers.linear, pkg.mixers.product32):
        assert inspect.signature(f).parameters["early"].default is False
