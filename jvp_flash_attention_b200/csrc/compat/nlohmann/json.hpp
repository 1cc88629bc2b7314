// Stands in for the JSON library that ATen/functorch/Interpreter.h includes for its serialisation members and that torch
// does not ship with its headers.  Nothing here is ever called: the members only have to be declarable.
#pragma once
#include <string>

namespace nlohmann {
struct json {
  json() = default;
  template <typename T>
  json(const T&) {}
  std::string dump() const { return {}; }
  static json parse(const std::string&) { return {}; }
  template <typename T>
  T get() const;
};
}  // namespace nlohmann
