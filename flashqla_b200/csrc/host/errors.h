// Errors raised towards Python with the exception types of the Python-level checks they replace.
#pragma once
#include <stdexcept>
#include <string>

namespace fqla_host {

struct PyError : std::runtime_error {
  enum Kind { Assertion, Type, Value, NotImplemented, Fqla };
  Kind kind;
  PyError(Kind k, const std::string& what) : std::runtime_error(what), kind(k) {}
};

}  // namespace fqla_host
