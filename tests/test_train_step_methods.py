"""WarmMLP.train_step with a method of its own that a subclass, an instance or a patched class has replaced: the step
is then made of those methods, as it was before it became one library call.  CPU: the library is a recorder."""
import pytest

from arpeggio_b200 import _lib, warm

PARTS = ['forward', 'backward', 'adam', 'pack', 'view']


class Recorder:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*a):
            self.calls.append(name)
            return 0
        return call


class Flat:
    """Stands for a flat parameter tensor."""
    def __getitem__(self, _):
        return self

    def __getattr__(self, name):
        return lambda *a, **k: self


def bare(cls):
    m = cls.__new__(cls)
    for name in 'w wb w2p grad m v H1 H2 Z dZ3 dZ2 dZ1 loss correct status'.split():
        setattr(m, name, Flat())
    m.part = type('Part', (Flat,), {'numel': lambda self: 80})()
    m.reserve = lambda rows, train=False: None
    m.offs, o = {}, 0
    for name, shp in m.LAYOUT:
        m.offs[name] = (o, shp)
    m.C, m.n, m.steps = 3, 10, 0
    return m


@pytest.fixture
def library(monkeypatch):
    r = Recorder()
    monkeypatch.setattr(_lib, 'lib', lambda: r)
    monkeypatch.setattr(_lib, 'ptr', lambda t: None)
    monkeypatch.setattr(_lib, 'stream_ptr', lambda s=None: None)
    return r


def wrapped(name, seen):
    f = getattr(warm.WarmMLP, name)

    def method(self, *a, **k):
        seen.append(name)
        return f(self, *a, **k)
    return method


def test_unchanged_class_takes_the_one_call(library):
    m = bare(warm.WarmMLP)
    m.train_step(Flat(), Flat(), 32)
    assert library.calls == ['arp_mlp_train_step'] and m.steps == 1


@pytest.mark.parametrize('how', ['subclass', 'instance', 'class'])
@pytest.mark.parametrize('name', PARTS)
def test_replaced_methods_take_part(library, monkeypatch, name, how):
    seen = []
    method = wrapped(name, seen)
    if how == 'subclass':
        m = bare(type('Sub', (warm.WarmMLP,), {name: method}))
    elif how == 'class':
        monkeypatch.setattr(warm.WarmMLP, name, method)
        m = bare(warm.WarmMLP)
    else:
        m = bare(warm.WarmMLP)
        setattr(m, name, method.__get__(m))
    m.train_step(Flat(), Flat(), 32)
    assert seen and 'arp_mlp_train_step' not in library.calls and m.steps == 1
