"""Mechanisms beyond the built-in ones, made from the 9-species one, and a second library that holds
them (the product's sources, other generated units)."""
import concurrent.futures as cf
import contextlib
import copy
import os
import shutil
import subprocess

from pelelm_gb300 import _build, _lib, workloads
from pelelm_gb300.mech import codegen
from pelelm_gb300.mech.model import Arrhenius, Reaction


def trio():
    """Coefficients of 3 on either side (net 2 and 3), a third-body reaction that is not the last, an
    elementary last one, N2 as a listed collider, H2O2 in the total alone."""
    m = workloads.load_mechanism("lidryer_syn")
    m.name = "trio_syn"
    keep = [r for r in m.reactions if "H2O2" not in r.reactants and "H2O2" not in r.products]
    third = [r for r in keep if r.kind == "three_body"]
    third[0].efficiencies["N2"] = 0.4
    # barriers a little above the heats of reaction: moderate rates either way
    threes = [Reaction("elementary", {"HO2": 1, "H2O": 1}, {"OH": 3}, True, Arrhenius(1e15, 0.0, 42e3)),
              Reaction("elementary", {"OH": 3}, {"H2": 1, "HO2": 1, "O": 1}, True, Arrhenius(1e15, 0.0, 90e3)),
              Reaction("elementary", {"O2": 1, "O": 1}, {"O": 3}, True, Arrhenius(1e13, 0.0, 120e3))]
    m.reactions = third + threes + [r for r in keep if r.kind != "three_body"]
    assert m.reactions[-1].kind == "elementary"
    return m


def jump():
    """H2, H and N2, whose enthalpies fall by 20 K R at the common Tmid."""
    m = workloads.load_mechanism("lidryer_syn")
    m.name = "jump_syn"
    m.species = [s for s in m.species if s.name in ("H2", "H", "N2")]
    for s in m.species:
        s.high[5] -= 20.0
    m.reactions = [Reaction("three_body", {"H": 2}, {"H2": 1}, True, Arrhenius(1e18, -1.0, 0.0))]
    return m


def reduced(base, name, ns):
    """`base` with ns species (CH4, its products and air among them), the least connected ones left out,
    and the reactions of those alone."""
    m = workloads.load_mechanism(base)
    m.name = name
    held = {"CH4", "O2", "N2", "H", "O", "OH", "CO2", "H2O"}
    keep = [s.name for s in m.species]
    while len(keep) > ns:
        uses = {s: sum(s in r.reactants or s in r.products for r in m.reactions) for s in keep if s not in held}
        keep.remove(min(uses, key=uses.get))
        m.reactions = [r for r in m.reactions if all(s in keep for s in [*r.reactants, *r.products])]
    m.species = [s for s in m.species if s.name in keep]
    for r in m.reactions:
        r.efficiencies = {s: e for s, e in r.efficiencies.items() if s in keep}
    return m


def reduced_cells(cs, base, m):
    """The states of `base` on the species of `m`."""
    cols = [base.index(s.name) for s in m.species]
    cs = copy.deepcopy(cs)
    cs.rY, cs.rYsrc = cs.rY[:, cols].copy(), cs.rYsrc[:, cols].copy()
    rho = cs.rY.sum(1)
    cs.rE = rho * workloads.mixture_h(m, cs.T, cs.rY / rho[:, None])
    return cs


def build(outdir, mechs):
    """Library of `mechs` alone in outdir; returns its path. Units that hold no mechanism are the
    product's objects."""
    csrc = os.path.join(outdir, "pelelm_gb300", "csrc")
    gen = os.path.join(csrc, "gen")
    shutil.copytree(_build.CSRC, csrc)
    shutil.copytree(os.path.join(_build.ROOT, "include"), os.path.join(outdir, "include"))
    names = [m.name for m in mechs]
    with mechanisms(outdir, mechs):
        codegen.main(gen, names=names)
        codegen.write_tables(gen, names=names)
        units = codegen.write_units(gen, names)

    def compile_unit(src):
        obj = os.path.join(outdir, os.path.splitext(os.path.basename(src))[0] + ".o")
        subprocess.run([_build.nvcc(), *_build.NVFLAGS, *_build.ARCH, "-c", src, "-o", obj], check=True)
        return obj

    with cf.ThreadPoolExecutor() as ex:
        objs = list(ex.map(compile_unit, units + [os.path.join(csrc, "reactor.cu")]))
    objs += [os.path.join(_build.BUILD, os.path.splitext(u)[0] + ".o") for u in _build.UNITS if u != "reactor.cu"]
    so = os.path.join(outdir, "libextra.so")
    subprocess.run([_build.nvcc(), *_build.ARCH, "-shared", "-o", so, *objs], check=True)
    return so


@contextlib.contextmanager
def mechanisms(outdir, mechs):
    """load_mechanism and mech_path know `mechs`."""
    by_name = {m.name: m for m in mechs}
    load, path = workloads.load_mechanism, workloads.mech_path
    for m in mechs:
        m.to_flat(os.path.join(outdir, m.name + ".mech"))
    workloads.load_mechanism = lambda n: copy.deepcopy(by_name[n]) if n in by_name else load(n)
    workloads.mech_path = lambda n, ext="mech": os.path.join(outdir, f"{n}.{ext}") if n in by_name else path(n, ext)
    try:
        yield
    finally:
        workloads.load_mechanism, workloads.mech_path = load, path


@contextlib.contextmanager
def library(so):
    """Calls go to the library `so`."""
    saved = _lib.LIB, _lib._lib
    _lib.LIB, _lib._lib = so, None
    try:
        yield
    finally:
        _lib.LIB, _lib._lib = saved
