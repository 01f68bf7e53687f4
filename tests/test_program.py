"""Which recorded calls zc_end_record joins, and other decisions made on the host."""
from helpers import run_cpp


def test_what_is_worth_being_joined():
    run_cpp("test_program_worth")


def test_how_moe_layers_are_laid_out():
    run_cpp("test_moe_layout")


def test_tile_widths_are_chosen_for_the_device():
    run_cpp("test_tile_width")
