"""The step's launch counter (last_step_counters) counts every kernel of the Linearized solve: the refined solve, one
kernel or, from 448 lines, three or four around the cluster, and the elimination behind it; beyond 768 lines the
elimination alone. Counted against the same step with the SimpleIterative solver, whose solve is one kernel."""
import pytest

from stormbird_gb300 import Simulation
from stormbird_gb300 import setups as S

from .test_linearized_refined import row, step

pytestmark = pytest.mark.gpu
NO_VISCOUS = {"Linearized": {"disable_viscous_corrections": True}}


@pytest.mark.parametrize("panels,solver,solve", [(32, None, 2), (447, None, 2), (448, None, 5), (448, NO_VISCOUS, 4), (768, None, 5),
                                                 (769, None, 1)])
def test_linearized(gpu_lib, panels, solver, solve):
    count = {}
    for name, s in (("linearized", solver), ("iterative", S.simple_iterative(3, 0.05, 0.0, 0.0))):
        sim = Simulation(row(1, panels, solver=s))
        step(sim, [5.0, 8.0, 0.0])
        count[name] = sim.last_step_counters()["kernel_launches"]
    assert count["linearized"] - count["iterative"] == solve - 1
