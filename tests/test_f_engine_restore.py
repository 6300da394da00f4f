"""What set_f_engine (and the C getter) returns brings back the engine that was
set, the default 'auto' among them."""
import pytest

from pyscf_wb97mv_fast_gb300 import _native, cosx


@pytest.fixture
def engine_kept():
    code = _native.lib().wb_ozaki_get_f_engine()
    yield
    assert _native.lib().wb_ozaki_set_f_engine(code) == _native.WB_OK


@pytest.mark.parametrize('first', sorted(cosx.F_ENGINES))
@pytest.mark.parametrize('second', sorted(cosx.F_ENGINES))
def test_set_and_restore(engine_kept, first, second):
    get = _native.lib().wb_ozaki_get_f_engine
    cosx.set_f_engine(first)
    assert get() == cosx.F_ENGINES[first]
    assert cosx.get_f_engine() in cosx.F_ENGINES
    prev = cosx.set_f_engine(second)
    assert get() == cosx.F_ENGINES[second]
    cosx.set_f_engine(prev)
    assert get() == cosx.F_ENGINES[first]


def test_default_is_auto():
    import subprocess
    import sys
    code = ('from pyscf_wb97mv_fast_gb300 import _native; '
            'raise SystemExit(_native.lib().wb_ozaki_get_f_engine())')
    assert subprocess.run([sys.executable, '-c', code]).returncode == cosx.F_ENGINES['auto']
