"""sw_get_kernel_config reports a cut-over only where one is used: the time model
decides in place of the built-in table's, a caller's table keeps its own."""
import pytest

from swhybrid_b200 import autotune, capi, synth

pytestmark = pytest.mark.gpu


def test_cutover_of_the_built_in_table_and_of_a_callers():
    table = autotune.load_table(autotune.DEFAULT_TABLE)
    hi, cfg = next((row[0], row[1]) for row in table if row[1][4] > 0)
    db = synth.small_db(5, 300)
    with capi.Context(0) as c:
        c.load_db(db.residues, db.offsets)
        assert c.kernel_config(hi) == (*cfg[:4], 0)
        c.search(synth.query(3, 150))
        c.set_tuning(table)
        assert c.kernel_config(hi) == tuple(cfg)
        c.set_kernel_config((16, 32, 8, 16, 777))
        assert c.kernel_config(hi) == (16, 32, 8, 16, 777)
