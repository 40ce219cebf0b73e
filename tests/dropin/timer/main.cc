// Fields that follow the simulation time alone: n integrates it (an explicit block on old_1), m adds
// it to the new n (a second explicit block), on 2-D Q1 elements.
#include "custom_pde.h"

#include <prismspf/core/parse_cmd_options.h>
#include <prismspf/core/problem.h>

using namespace prismspf;

int
main(int argc, char *argv[])
{
  prismspf::MPIInitFinalize mpi_init(argc, argv);
  ParseCMDOptions           cli_options(argc, argv);

  constexpr unsigned int dim    = 2;
  constexpr unsigned int degree = 1;

  std::vector<FieldAttributes> fields = {FieldAttributes("n", Scalar), FieldAttributes("m", Scalar)};
  std::vector<SolveBlock> blocks;
  blocks.push_back(SolveBlock(1, Explicit, Primary, {0}, make_dependency_set(fields, {"old_1(n)"})));
  blocks.push_back(SolveBlock(2, Explicit, Secondary, {1}, make_dependency_set(fields, {"n"})));

  UserInputParameters<dim>       user_inputs(cli_options.get_parameters_filename());
  PhaseFieldTools<dim>           pf_tools;
  CustomPDE<dim, degree, double> pde(user_inputs, pf_tools);
  Problem<dim, degree, double>   problem(fields, blocks, user_inputs, pf_tools, pde);
  problem.solve();
  return 0;
}
