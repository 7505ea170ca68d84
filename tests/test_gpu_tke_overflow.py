"""The tke step where the scan of a column's pivots overflows at the top level while
everything that the fast divisions see stays in their range (GPU): b' is infinite
there and the solution finite.  Such columns need diffusivities and mixing lengths of
both signs that cancel; these four came out of a random search.  Bit for bit against
the CPU oracle."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W = importlib.import_module("futhark-benchmarks_b200.workloads")
tke_mod = importlib.import_module("futhark-benchmarks_b200.tke")

# dzw, kappaM, tketau, mxl by level
COLUMNS = [
    ([0.0016465565422549844, 0.0003099308523815125, 74.90926361083984, 0.022549405694007874],
     [0.0, 4814810.5, -4814815.0, 2.8654589427318784e+16],
     [1.4551915228366852e-11, 0.00390625, 4194304.0, 281474976710656.0],
     [-4.996551783431613e-12, -2.8162049515306764e-12, -3.7477390982254555e-12, -4.620923435560975e-12]),
    ([1.0280942888130085e-06, 60.36153030395508, 982.1019897460938, 159.22804260253906],
     [0.0, -12537562.0, 25075118.0, -2.8751074579133235e+18],
     [4096.0, 1.3877787807814457e-17, 268435456.0, 68719476736.0],
     [3.674125673841511e-12, -3.95514021533927e-09, 3.9176023536313664e-12, 5.081285218977438e-12]),
    ([0.0009723299881443381, 745.97705078125, 178053.65625, 12431.044921875],
     [0.0, -698.9840698242188, 698.9840698242188, -1.9442352591532533e+22],
     [1.4551915228366852e-11, 1.3877787807814457e-17, 274877906944.0, 281474976710656.0],
     [3.716867525566103e-12, -4.139525699997648e-08, 3.3610109053533455e-12, 3.754454646481831e-12]),
    ([2.183982132919482e-06, 847.9747314453125, 0.4152442216873169, 0.0031239136587828398],
     [0.0, 358343456.0, -384885056.0, 1693255020314624.0],
     [1048576.0, 1.3877787807814457e-17, 268435456.0, 17592186044416.0],
     [-4.375897214026203e-12, -2.461616910309772e-09, -2.8125449018368e-12, -2.708350470975729e-12]),
]


@pytest.mark.parametrize("column", range(len(COLUMNS)))
def test_overflow_at_the_top_level(oracle, column):
    ins = list(W.tke_inputs(6, 6, 4, seed=1))
    dzw, kappaM, tketau, mxl = COLUMNS[column]
    put = {"dzw": dzw, "kappaM": kappaM, "tketau": tketau, "mxl": mxl, "dzt": 0.5, "kbot": 1}
    put.update({n: 0.0 for n in ("utau", "vtau", "wtau", "forc", "dtketau", "dtketaum1", "forc_tke_surface")})
    put.update({n: 1.0 for n in ("dxt", "dxu", "dyt", "dyu", "cost", "cosu", "maskU", "maskV", "maskW")})
    for name, v in put.items():
        k = tke_mod.INPUT_NAMES.index(name)
        ins[k] = np.ascontiguousarray(np.broadcast_to(np.asarray(v, ins[k].dtype), ins[k].shape))
    with np.errstate(all="ignore"):
        want = oracle.tke(*ins)
    assert np.all(np.isfinite(want[1]))
    with tke_mod.TkeContext() as tctx:
        for g, w in zip(tctx.main(*ins), want):
            assert np.array_equal(g.view(np.int32), w.view(np.int32))
